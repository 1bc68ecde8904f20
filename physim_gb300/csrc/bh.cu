// bh.cu -- Barnes-Hut gravity on the GPU: the astro2 (octree) and astro
// (quadtree) elements, astro/src/transformers.rs:31-69,122-160, over the
// reference's tree semantics (astro/src/octree.rs, astro/src/quadtree.rs).
//
// Pipeline, all on the device (no host round trip, so it can be captured):
//   1. extent    X = max_i max(|x_i|,|y_i|,|z_i|) in f64 (transformers.rs:126-131);
//                the root cell is centred at the origin with half-width X.
//   2. keys      per axis the cell index q at the finest level D, with the
//                reference's octant rule (p > centre goes high, ties low,
//                octree.rs:160-165), interleaved x-lowest into a Morton key:
//                octree 21 levels x 3 bits = 63 bits, quadtree 31 x 2 = 62.
//                Bodies within a rounding margin of a cell boundary re-derive
//                q by replaying the reference's f64 centre arithmetic.
//   3. sort      stable radix sort of (key, body) pairs, 9-bit digits.
//                Up to 1.2M bodies steps 1-3 are one launch (tree_sort_kernel).
//   4. tree      not path-compressed (as the reference's pointer tree): a
//                cell with more than leaf_size bodies that are not all at
//                one key splits into its non-empty children; breadth-first
//                layout (levels contiguous, children contiguous in key
//                order), built flat for all levels at once from the
//                key-prefix boundaries (section 4).  Geometric centres are
//                computed exactly as the reference does (child = parent +-
//                extent/2, octree.rs:167-215).
//   5. cells     geometry, mass, centre of mass (double-float sums) and optionally
//                second moments (f32) of every cell, all cells at once from
//                sums over groups of consecutive sorted bodies.
//   6. traversal one warp per 32 consecutive sorted bodies, DFS with a shared
//                stack, the reference's opening rule extent/|x - centre| < theta
//                (octree.rs:137-144).  EXACT: every body keeps its own
//                interaction list (the reference's); WARP: a cell is accepted
//                only if all 32 bodies accept it, and the common list is
//                batched through shared memory.  Pair law in FP32 with one
//                MUFU.RSQ per pair and compensated per-body sums.
#include <stdio.h>
#include <string.h>

#include <cuda/atomic>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "engine.h"
#include "plugin_state.h"

namespace pg {

namespace {

constexpr int kRadixBits = 9;
constexpr int kRadixBuckets = 1 << kRadixBits;
// 8,192 keys per tile: few tiles keep the look-back chains of a pass short
// (all tiles of a 1M-key sort are resident at once, so a pass's time is set
// by how far an inclusive prefix must travel from tile 0)
constexpr int kSortThreads = 512;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kSortWarps = kSortThreads / 32;
constexpr size_t kSortSmem = (size_t)kSortTile * (sizeof(uint64_t) + sizeof(uint32_t));  // staged tile

constexpr int kMaxLevels = 31;


// flags[0]: node capacity exceeded (tree truncated; results stay exact)
// flags[1]: traversal stack overflow (results of the affected warp invalid)
// flags[2]: a radix-sort look-back wait gave up (sort order invalid)
constexpr int kFlagNodes = 0;
constexpr int kFlagStack = 1;
constexpr int kFlagSort = 2;

// Radix sort of the 63-bit (62-bit) keys: 7 passes of 9-bit digits (512
// digits: one look-back thread each in a 512-thread tile).
constexpr int kSortPasses = 7;
// Look-back spin limit per digit (each spin is one L2 load, ~0.5 us worst
// case), far above any wait of a running predecessor tile; the default of
// physim_gpu_set_wait_limit.
constexpr int kLookbackSpins = 1 << 20;
// Predecessor tiles a look-back reads per round trip.
constexpr int kLookbackWindow = 8;

struct LevelInfo {
    int32_t begin[kMaxLevels + 2];  // first node of each level
    int32_t count[kMaxLevels + 2];  // nodes of each level
    int32_t total;                  // nodes in the tree
    int32_t max_level;              // deepest level built (below D only if capacity ran out)
};

__host__ __device__ inline int tree_levels(int nchild) { return nchild == 8 ? 21 : 31; }
__host__ __device__ inline int level_bits(int nchild) { return nchild == 8 ? 3 : 2; }

// ---------------------------------------------------------------------------
// 1. extent
// ---------------------------------------------------------------------------
// |coordinate| maxima on the f64 bit patterns: non-negative doubles order like
// their bit patterns, so integer maxima replace f64 ones (GB300 issues f64
// instructions at a small fraction of its integer rate).  NaN coordinates are
// skipped, as f64::max skips a NaN operand.
__device__ __forceinline__ unsigned long long abs_bits(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return b > 0x7ff0000000000000ull ? 0ull : b;
}

__global__ void extent_kernel(const double *__restrict__ x, const double *__restrict__ y,
                              const double *__restrict__ z, int n,
                              unsigned long long *__restrict__ out_bits)
{
    unsigned long long m = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        m = max(m, abs_bits(x[i]));
        m = max(m, abs_bits(y[i]));
        m = max(m, abs_bits(z[i]));
    }
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ unsigned long long wm[32];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? wm[threadIdx.x] : 0ull;
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) atomicMax(out_bits, m);
    }
}

// ---------------------------------------------------------------------------
// 2. keys
// ---------------------------------------------------------------------------
// Cell index of coordinate p at the finest level D: the reference descends
// from centre 0 / half-width X deciding `p > centre` at every level.
// u = (p + X) * 2^(D-1) / X is the position in finest-cell units; unless u is
// within 2^-mbits of a cell boundary, the cell is floor(u), read off u's bits
// with integer instructions (two f64 operations per axis).  Close to a
// boundary, or for u < 1, the reference's centre arithmetic is replayed in
// f64.  The margin: u carries three roundings (< 2^(D-51)), the reference's
// centres at most D of 2^-53 X each (< 2^(D-49) of a cell), together under
// 2^(D-48); mbits = 46 - D leaves a factor of four.  A replay is a chain of D
// dependent f64 steps (3 us for the one body that needs it, and its whole sort
// waits), so a margin as wide as 2^(D-40) was felt at 100,000 bodies, where it
// caught about one body per step.
__host__ __device__ inline int key_margin_bits(int D) { return 46 - D; }

// axis_cell_fast reads the cell off u, or sets `replay` where that may not be
// the reference's cell.
__device__ __forceinline__ uint32_t axis_cell_fast(double p, double X, double scale, int D,
                                                   int mbits, bool &replay)
{
    const uint32_t lim = (1u << D) - 1u;
    const double u = __dmul_rn(__dadd_rn(p, X), scale);
    const unsigned long long bits = (unsigned long long)__double_as_longlong(u);
    const int ex = (int)((bits >> 52) & 0x7ff) - 1023;
    if (ex == 1024) return 0;  // NaN (or infinite) coordinate
    const unsigned long long mant = (bits & 0xfffffffffffffull) | (1ull << 52);
    const int fb = 52 - ex;  // fraction bits of u
    // (shift counts outside 0..63 are only formed where `replay` discards the result)
    const unsigned long long ip = mant >> (fb & 63);
    const unsigned long long top = (mant >> ((fb - mbits) & 63)) & ((1ull << mbits) - 1ull);
    const bool inside = ex >= 0 && ex <= 52 - mbits && top != 0ull && top != (1ull << mbits) - 1ull;
    replay = replay || !inside;
    return ip > lim ? lim : (uint32_t)ip;
}

__device__ __noinline__ uint32_t axis_cell_replay(double p, double X, int D)
{
    // The body that sets the extent sits on a boundary in every state: every
    // centre lies strictly between -X and X (D <= 31 halvings of a normal X
    // round to at most X (1 - 2^-D)), so p = X is above and p = -X below all.
    const unsigned long long xb = (unsigned long long)__double_as_longlong(X);
    if (abs_bits(p) == xb && (xb >> 52) > 64) return p > 0.0 ? (1u << D) - 1u : 0u;
    double c = 0.0, ext = X;
    uint32_t q = 0;
    for (int d = 0; d < D; ++d) {
        const bool hi = p > c;
        const double h = __dmul_rn(ext, 0.5);  // ext / 2, exact
        c = hi ? __dadd_rn(c, h) : __dsub_rn(c, h);
        ext = h;
        q = (q << 1) | (hi ? 1u : 0u);
    }
    return q;
}

__device__ __forceinline__ uint64_t spread3(uint32_t v)
{
    uint64_t x = v & 0x1fffffu;
    x = (x | x << 32) & 0x1f00000000ffffull;
    x = (x | x << 16) & 0x1f0000ff0000ffull;
    x = (x | x << 8) & 0x100f00f00f00f00full;
    x = (x | x << 4) & 0x10c30c30c30c30c3ull;
    x = (x | x << 2) & 0x1249249249249249ull;
    return x;
}

__device__ __forceinline__ uint64_t spread2(uint32_t v)
{
    uint64_t x = v & 0x7fffffffu;
    x = (x | x << 16) & 0x0000ffff0000ffffull;
    x = (x | x << 8) & 0x00ff00ff00ff00ffull;
    x = (x | x << 4) & 0x0f0f0f0f0f0f0f0full;
    x = (x | x << 2) & 0x3333333333333333ull;
    x = (x | x << 1) & 0x5555555555555555ull;
    return x;
}

// Morton key of a body (X > 0; scale = 2^(D-1) / X).
__device__ __forceinline__ uint64_t body_key(double x, double y, double z, double X, double scale,
                                             int nchild)
{
    const int D = tree_levels(nchild), mbits = key_margin_bits(D);
    bool rx = false, ry = false, rz = false;
    uint32_t qx = axis_cell_fast(x, X, scale, D, mbits, rx);
    uint32_t qy = axis_cell_fast(y, X, scale, D, mbits, ry);
    uint32_t qz = nchild == 8 ? axis_cell_fast(z, X, scale, D, mbits, rz) : 0u;
    if (rx || ry || rz) {
        if (rx) qx = axis_cell_replay(x, X, D);
        if (ry) qy = axis_cell_replay(y, X, D);
        if (rz) qz = axis_cell_replay(z, X, D);
    }
    if (nchild != 8) return spread2(qx) | (spread2(qy) << 1);
    return spread3(qx) | (spread3(qy) << 1) | (spread3(qz) << 2);
}

// Keys, plus the histograms of all 7 radix digits of all keys (block-local in
// shared memory, then one global atomic per non-empty bucket), for the
// one-sweep sort.  ghist [7][512] must be zero on entry.  Block 0 also resets
// the sort's tile counters and grid barrier and advances its epoch (see
// radix_pass_kernel).
__global__ void __launch_bounds__(256)
keys_kernel(const double *__restrict__ x, const double *__restrict__ y,
            const double *__restrict__ z, int n, int nchild,
            const unsigned long long *__restrict__ extent_bits, uint64_t *__restrict__ keys,
            uint32_t *__restrict__ vals, uint32_t *__restrict__ ghist,
            uint32_t *__restrict__ tile_ctr, uint32_t *__restrict__ epoch,
            uint32_t *__restrict__ sort_bar)
{
    __shared__ double s_scale;
    __shared__ uint32_t h[kSortPasses][kRadixBuckets];
    const double X = __longlong_as_double((long long)*extent_bits);
    const int D = tree_levels(nchild);
    for (int k = threadIdx.x; k < kSortPasses * kRadixBuckets; k += blockDim.x) (&h[0][0])[k] = 0;
    if (threadIdx.x == 0) s_scale = X > 0.0 ? __ddiv_rn(ldexp(1.0, D - 1), X) : 0.0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        for (int p = 0; p < kSortPasses; ++p) tile_ctr[p] = 0;
        *sort_bar = 0;
        *epoch += 1u;
    }
    __syncthreads();
    const double scale = s_scale;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint64_t key = X > 0.0 ? body_key(x[i], y[i], z[i], X, scale, nchild) : 0ull;
        keys[i] = key;
        vals[i] = (uint32_t)i;
#pragma unroll
        for (int p = 0; p < kSortPasses; ++p)
            atomicAdd(&h[p][(uint32_t)(key >> (kRadixBits * p)) & (kRadixBuckets - 1)], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kSortPasses * kRadixBuckets; k += blockDim.x) {
        const uint32_t c = (&h[0][0])[k];
        if (c) atomicAdd(&ghist[k], c);
    }
}

// ---------------------------------------------------------------------------
// 3. radix sort (stable, LSD, 9-bit digits)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t lanemask_lt()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Block-wide exclusive scan of one value per thread (blockDim.x <= 1024).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *warp_sums,
                                                         uint32_t &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < nw ? warp_sums[lane] : 0;
        uint32_t wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < nw) warp_sums[lane] = wi - w;
        if (lane == 31) warp_sums[32] = wi;
    }
    __syncthreads();
    const uint32_t r = warp_sums[warp] + incl - v;
    total = warp_sums[32];
    __syncthreads();
    return r;
}

// One tile of one pass of the radix sort (the body shared by the per-pass
// kernel and the single-launch sort): ranks the tile's keys by digit,
// publishes and looks back, and scatters through shared memory.  digit_base
// is this thread's digit's first place in the output (the scan of the
// pass's global histogram); h must be zero on entry.  The key and value
// pointers carry no __restrict__: in the single-launch sort a pass reads what
// other blocks of the same launch wrote, which the read-only cache path may
// not serve.
__device__ __forceinline__ void sort_tile(
    const uint64_t *keys_in, const uint32_t *vals_in, uint64_t *keys_out, uint32_t *vals_out,
    int n, int pass, int tile,
    uint32_t digit_base, unsigned long long *__restrict__ status,
    const uint32_t *__restrict__ epoch_ptr, uint32_t *__restrict__ flags, int spin_limit,
    int stall_tile, uint32_t (*h)[kRadixBuckets], uint32_t *digit_off, uint32_t *local_start,
    uint32_t *ws)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int shift = kRadixBits * pass;
    const int base = tile * kSortTile + warp * (kSortItems * 32);
    uint64_t kk[kSortItems];
    uint32_t vv[kSortItems];
    uint32_t rank[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int idx = base + r * 32 + lane;
        const bool valid = idx < n;
        kk[r] = valid ? keys_in[idx] : 0;
        vv[r] = valid ? (vals_in ? vals_in[idx] : (uint32_t)idx) : 0;
    }
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int idx = base + r * 32 + lane;
        const bool valid = idx < n;
        // lanes with this lane's digit: one vote per digit bit (MATCH.ANY is
        // several times slower here)
        const uint32_t d = valid ? (uint32_t)(kk[r] >> shift) & (kRadixBuckets - 1) : 0u;
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int b = 0; b < kRadixBits; ++b) {
            const uint32_t bit = (d >> b) & 1u;
            const uint32_t vote = __ballot_sync(0xffffffffu, bit);
            peers &= bit ? vote : ~vote;
        }
        const uint32_t before = __popc(peers & lanemask_lt());
        uint32_t cur = 0;
        if (valid) cur = h[warp][d];
        __syncwarp();
        if (valid && before == 0) h[warp][d] = cur + __popc(peers);
        __syncwarp();
        rank[r] = cur + before;
    }
    __syncthreads();
    // this tile's count of digit d, and the warps' exclusive offsets within it
    // (threads 0..255, one digit each)
    const int d = threadIdx.x;
    if (d < kRadixBuckets) {
        uint32_t count = 0;
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = h[w][d];
            h[w][d] = count;
            count += c;
        }
        {
            uint32_t total;
            local_start[d] = block_exclusive_scan(count, ws, total);
        }
        // tag base of this sort and pass: the passes share the status array
        const unsigned long long ep =
            ((unsigned long long)(*epoch_ptr & 0x03ffffffu) * kSortPasses + (unsigned)pass) * 4ull;
        volatile unsigned long long *st = status;
        uint32_t excl = 0;
        if (tile == 0) {
            st[d] = ((ep + 2ull) << 32) | count;
        } else {
            st[(size_t)tile * kRadixBuckets + d] = ((ep + 1ull) << 32) | count;
            // walk back kLookbackWindow tiles per round trip: the window's words
            // are loaded together, then summed up to the first inclusive prefix
            int t = tile - 1;
            int spins = 0;
            const bool stall = tile == stall_tile;
            for (;;) {
                unsigned long long w[kLookbackWindow];
#pragma unroll
                for (int j = 0; j < kLookbackWindow; ++j)
                    w[j] = t - j >= 0 && !stall ? st[(size_t)(t - j) * kRadixBuckets + d] : 0ull;
                int used = 0;
                bool done = false;
#pragma unroll
                for (int j = 0; j < kLookbackWindow; ++j) {
                    if (done || used != j) continue;
                    const unsigned long long tag = w[j] >> 32;
                    if (tag == ep + 2ull) {
                        excl += (uint32_t)w[j];
                        done = true;
                    } else if (tag == ep + 1ull) {
                        excl += (uint32_t)w[j];
                        ++used;  // t - j > 0 here: tile 0 publishes its inclusive prefix at once
                    }
                }
                if (done) break;
                t -= used;
                if (used == 0 && ++spins > spin_limit) {
                    atomicOr(&flags[kFlagSort], 1u);
                    break;
                }
            }
            st[(size_t)tile * kRadixBuckets + d] = ((ep + 2ull) << 32) | (excl + count);
        }
        digit_off[d] = digit_base + excl;
    }
    __syncthreads();
    // the tile in digit order in shared memory, then each digit's run written
    // to its place in one contiguous stretch (scattered 8-byte stores cost
    // a third of the pass)
    extern __shared__ uint64_t skeys[];  // kSortTile keys, then kSortTile values
    uint32_t *svals = reinterpret_cast<uint32_t *>(skeys + kSortTile);
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const int idx = base + r * 32 + lane;
        if (idx >= n) continue;
        const uint32_t dg = (uint32_t)(kk[r] >> shift) & (kRadixBuckets - 1);
        const uint32_t lp = local_start[dg] + h[warp][dg] + rank[r];
        skeys[lp] = kk[r];
        svals[lp] = vv[r];
    }
    __syncthreads();
    const int cnt = min(kSortTile, n - tile * kSortTile);
    for (int j = threadIdx.x; j < cnt; j += kSortThreads) {
        const uint64_t key = skeys[j];
        const uint32_t dg = (uint32_t)(key >> shift) & (kRadixBuckets - 1);
        const uint32_t pos = digit_off[dg] + (uint32_t)j - local_start[dg];
        keys_out[pos] = key;
        vals_out[pos] = svals[j];
    }
}

// One stable counting pass of the one-sweep LSD radix sort (single-pass
// chained scan with decoupled look-back, after Merrill & Garland 2016 and
// Adinets & Merrill 2022).  Tiles of kSortTile keys are claimed in launch
// order from an atomic counter, so every tile a block looks back at is held
// by a block that is already running.  Each block ranks its keys by digit
// (warp by warp, stable, lanes of equal digit found by one ballot per digit
// bit), publishes its per-digit counts, then walks back over the preceding
// tiles' published words until it meets an inclusive prefix, publishes its
// own inclusive prefix, and scatters: the tile is first put in digit order
// in shared memory, so each digit's keys leave in one contiguous run.  A status word is
// (epoch * 4 + flag) << 32 | count, flag 1 = tile count, 2 = inclusive
// prefix, and epoch counts (sort, pass) pairs; words of earlier passes and
// sorts carry older epochs and read as not ready, so the status array needs
// no clearing.  A wait that exceeds
// the wait limit (kLookbackSpins unless physim_gpu_set_wait_limit set one)
// sets flags[kFlagSort] and gives up: the tile still scatters, at positions no
// higher than the right ones (its prefix is a partial sum), so every write
// stays in bounds; every later kernel of the build and the traversal see the
// flag and return at once, so nothing reads the invalid order or an unbuilt
// tree, and the host reports PHYSIM_ERR_TIMEOUT.  stall_tile >= 0
// (physim_gpu_test_stall_sort) makes that tile's look-back see no
// predecessor word, so the limit is reached for sure.
__global__ void __launch_bounds__(kSortThreads)
radix_pass_kernel(const uint64_t *__restrict__ keys_in, const uint32_t *__restrict__ vals_in,
                  uint64_t *__restrict__ keys_out, uint32_t *__restrict__ vals_out, int n,
                  int pass, const uint32_t *__restrict__ ghist, uint32_t *__restrict__ tile_ctr,
                  unsigned long long *__restrict__ status, const uint32_t *__restrict__ epoch_ptr,
                  uint32_t *__restrict__ flags, int spin_limit, int stall_tile)
{
    static_assert(kSortThreads >= kRadixBuckets, "one thread per digit");
    __shared__ uint32_t h[kSortWarps][kRadixBuckets];
    __shared__ uint32_t digit_off[kRadixBuckets];
    __shared__ uint32_t local_start[kRadixBuckets];  // the digit's first key in the staged tile
    __shared__ uint32_t ws[33];
    __shared__ int s_tile, s_stop;
    // an earlier wait failed: the whole block leaves (one read, shared, since
    // another block of this launch may raise the flag meanwhile)
    if (threadIdx.x == 0) {
        s_stop = *(volatile const uint32_t *)&flags[kFlagSort] != 0u;
        s_tile = (int)atomicAdd(&tile_ctr[pass], 1u);
    }
    __syncthreads();
    if (s_stop) return;
    for (int k = threadIdx.x; k < kSortWarps * kRadixBuckets; k += kSortThreads)
        (&h[0][0])[k] = 0;
    uint32_t digit_base;
    {
        uint32_t total;
        const uint32_t c = threadIdx.x < kRadixBuckets ? ghist[pass * kRadixBuckets + threadIdx.x]
                                                       : 0u;
        digit_base = block_exclusive_scan(c, ws, total);
    }
    sort_tile(keys_in, vals_in, keys_out, vals_out, n, pass, s_tile, digit_base, status,
              epoch_ptr, flags, spin_limit, stall_tile, h, digit_off, local_start, ws);
}

// All seven passes in one cooperative launch (every block resident, up to
// one per SM): each block takes tiles blockIdx.x, blockIdx.x + gridDim.x, ...
// of every pass, and a grid barrier separates the passes (a pass reads keys
// that every tile of the previous one wrote).  Every tile a look-back waits on
// is lower-numbered, so it is held by a resident block that reaches it after
// lower tiles only: the waits end.  The barrier is a counter each block adds
// to once per pass (reset by keys_kernel); its wait gives up after the wait
// limit, or at once when the sort's error flag is up, raising the flag, so no
// block waits for one that has left.  Against one launch per pass this saves
// six launch gaps and the tail of each pass.
__device__ __forceinline__ bool sort_grid_barrier(uint32_t *bar, uint32_t target,
                                                  uint32_t *flags, int spin_limit, int *s_ok)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        int spins = 0;
        while (*(volatile uint32_t *)bar < target) {
            if (*(volatile uint32_t *)&flags[kFlagSort] != 0u) break;
            if (++spins > spin_limit) {
                atomicOr(&flags[kFlagSort], 1u);
                break;
            }
        }
        __threadfence();
        *s_ok = *(volatile uint32_t *)&flags[kFlagSort] == 0u;
    }
    __syncthreads();
    return *s_ok != 0;
}

__global__ void __launch_bounds__(kSortThreads, 1)
radix_sort_kernel(uint64_t *k0, uint32_t *v0, uint64_t *k1, uint32_t *v1, int n,
                  const uint32_t *__restrict__ ghist, unsigned long long *__restrict__ status,
                  const uint32_t *__restrict__ epoch_ptr, uint32_t *__restrict__ flags,
                  int spin_limit, int stall_tile, uint32_t *bar)
{
    static_assert(kSortThreads == kRadixBuckets, "one thread per digit");
    __shared__ uint32_t h[kSortWarps][kRadixBuckets];
    __shared__ uint32_t digit_off[kRadixBuckets];
    __shared__ uint32_t local_start[kRadixBuckets];
    __shared__ uint32_t ws[33];
    __shared__ int s_ok;
    if (threadIdx.x == 0) s_ok = *(volatile const uint32_t *)&flags[kFlagSort] == 0u;
    __syncthreads();
    if (!s_ok) return;
    const int tiles = (n + kSortTile - 1) / kSortTile;
    for (int pass = 0; pass < kSortPasses; ++pass) {
        const uint64_t *keys_in = (pass & 1) ? k1 : k0;
        const uint32_t *vals_in = pass == 0 ? nullptr : ((pass & 1) ? v1 : v0);
        uint64_t *keys_out = (pass & 1) ? k0 : k1;
        uint32_t *vals_out = (pass & 1) ? v0 : v1;
        uint32_t digit_base;
        {
            uint32_t total;
            digit_base = block_exclusive_scan(ghist[pass * kRadixBuckets + threadIdx.x], ws, total);
        }
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            for (int k = threadIdx.x; k < kSortWarps * kRadixBuckets; k += kSortThreads)
                (&h[0][0])[k] = 0;
            __syncthreads();
            sort_tile(keys_in, vals_in, keys_out, vals_out, n, pass, tile, digit_base, status,
                      epoch_ptr, flags, spin_limit, stall_tile, h, digit_off, local_start, ws);
            __syncthreads();  // the staged tile, h and the offsets serve the next tile
        }
        if (pass + 1 < kSortPasses &&
            !sort_grid_barrier(bar, (uint32_t)(pass + 1) * gridDim.x, flags, spin_limit, &s_ok))
            return;
    }
}

// ---------------------------------------------------------------------------
// Extent, keys and sort in one launch, for states whose sort tiles are all
// resident (one block per tile, at most one per SM: up to 1.2M bodies).
// ---------------------------------------------------------------------------
// The sort's cost is latency: a pass moves 24 B a key through L2, but each is
// a chain of load, rank, exchange of the tiles' digit counts, scatter.  So:
//   * tiles of kSortThreads x ITEMS keys, ITEMS the smallest that keeps every
//     tile resident: a small state's passes are spread over more SMs;
//   * the tiles exchange counts through one grid barrier (a tile adds its
//     counts to its group of kSortGroup tiles, then sums the groups and the
//     group's tiles before it: at most 10 + 15 loads in flight together)
//     instead of a look-back's dependent reads;
//   * the passes cover only the top kSortTopPasses digits (36 bits), then
//     every key finds its place among the few that share those bits (a run)
//     by comparing whole keys in shared memory.  If some run has more than
//     kFixRun keys that are not all equal, every block learns it at the last
//     barrier and all seven passes run over the order reached so far, which
//     holds equal keys in body order: the result is the same stable order.  That
//     is a state with a dense core or one body far away (1,000 core radii in these
//     figures); a step, theta 0.7, leaf 16, of a Plummer sphere / the same with such
//     a body, and with the look-back sort (us): 20,011 bodies 78 / 108, 141 / 129;
//     100,003 99 / 134, 163 / 151; 300,007 139 / 182, 212 / 201; 1,000,003 314 /
//     366, 353 / 336;
//   * the extent and the keys are computed in the same launch (the keys go
//     from registers into the first pass), and the digits' places come from
//     the counts exchanged anyway, so no histogram pass is needed.
// Measured against extent, keys and the look-back sort of all seven digits in
// three launches (us, whole state): 8,195 bodies 96 -> 30, 100,003 bodies
// 110 -> 37, 1,048,580 bodies 160 -> 92, of which the f64 pipe takes 17 for
// the keys (2 f64 operations an axis) and each pass 15.  Beyond the resident
// sizes the look-back sort, whose blocks take several tiles, stays.
constexpr int kSortTopPasses = 4;
constexpr int kSortGroup = 16;   // tiles per count group
constexpr int kFixRun = 64;      // keys either side that share the top digits
constexpr uint32_t kBarPoison = 0x40000000u;  // the barrier's "a wait gave up" bit

struct TreeSortArgs {
    const double *x, *y, *z;
    int n, nchild;
    unsigned long long *extent_bits;  // out
    unsigned long long *blockmax;     // one per block
    uint64_t *k0, *k1;                // the sorted keys end in k1
    uint32_t *v0, *v1;
    uint32_t *tile_cnt;  // [tiles][512]
    uint32_t *grp;       // [2][groups][512]
    uint32_t *bar;       // [0] barrier count, [1] blocks that left, [2] a run was too long
    unsigned long long *stats;  // the traversal's two counts, cleared
    uint32_t *flags;
    int spin_limit, stall_tile;
};

// Grid barrier of the resident kernels: the count must reach `want`.  A wait
// that exceeds the limit raises the sort's error flag and sets the poison bit,
// which ends every other wait.  False: some wait gave up.
__device__ __forceinline__ bool grid_barrier(uint32_t *count, uint32_t *flags, int spin_limit,
                                             uint32_t want, int *s_ok)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        cuda::atomic_ref<uint32_t, cuda::thread_scope_device> bar(*count);
        bar.fetch_add(1u, cuda::memory_order_release);
        int spins = 0;
        uint32_t v;
        while ((v = bar.load(cuda::memory_order_acquire)) < want) {
            if (++spins > spin_limit) {
                atomicOr(&flags[kFlagSort], 1u);
                v = bar.fetch_or(kBarPoison, cuda::memory_order_relaxed) | kBarPoison;
                break;
            }
        }
        *s_ok = v < kBarPoison;
    }
    __syncthreads();
    return *s_ok != 0;
}

__device__ __forceinline__ bool tree_sort_barrier(const TreeSortArgs &a, uint32_t target,
                                                  int *s_ok)
{
    // the test hook's tile waits for a count that nothing reaches
    return grid_barrier(a.bar, a.flags, a.spin_limit,
                        (int)blockIdx.x == a.stall_tile ? kBarPoison : target, s_ok);
}

// The extent (bits of the largest |coordinate|) in wm[0] of every block, from
// each thread's maximum m, and to extent_bits; one barrier.
template <int kWarps>
__device__ __forceinline__ bool grid_extent(const TreeSortArgs &a, unsigned long long m,
                                            unsigned long long *wm, uint32_t &target, int *s_ok)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto block_max = [&]() {  // m of thread 0
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) wm[warp] = m;
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 1; w < kWarps; ++w) m = max(m, wm[w]);
    };
    block_max();
    if (threadIdx.x == 0) a.blockmax[blockIdx.x] = m;
    target += gridDim.x;
    if (!tree_sort_barrier(a, target, s_ok)) return false;
    m = 0;
    for (int t = threadIdx.x; t < (int)gridDim.x; t += kWarps * 32)
        m = max(m, __ldcg(&a.blockmax[t]));
    block_max();
    if (threadIdx.x == 0) {
        wm[0] = m;
        if (blockIdx.x == 0) *a.extent_bits = m;
    }
    __syncthreads();
    return true;
}

// 2^(D - 1) / X, one thread's division.
__device__ __forceinline__ double key_scale(double X, int nchild, double *s_scale)
{
    if (threadIdx.x == 0)
        *s_scale = X > 0.0 ? __ddiv_rn(ldexp(1.0, tree_levels(nchild) - 1), X) : 0.0;
    __syncthreads();
    return *s_scale;
}

// The last block to leave resets the barrier for the next build.
__device__ __forceinline__ void leave_grid(uint32_t *bar)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&bar[1], 1u) == gridDim.x - 1) {
            bar[0] = 0u;
            bar[1] = 0u;
        }
    }
}

template <int ITEMS>
struct TreeSortShared {
    uint32_t h[kSortWarps][kRadixBuckets];
    uint32_t digit_off[kRadixBuckets];
    uint32_t local_start[kRadixBuckets];
    unsigned long long wm[kSortWarps];
    uint32_t ws[33];
    int ok;
};

// One pass over digit `pass`: this block's tile (keys in kk / vv) goes to its
// place in keys_out / vals_out.  Ends with the grid barrier after the writes.
template <int ITEMS>
__device__ __forceinline__ bool tree_sort_pass(const TreeSortArgs &a, int pass, int seq,
                                               uint32_t &target, const uint64_t (&kk)[ITEMS],
                                               const uint32_t (&vv)[ITEMS], uint64_t *keys_out,
                                               uint32_t *vals_out, TreeSortShared<ITEMS> &sh,
                                               uint64_t *skeys)
{
    constexpr int kTile = kSortThreads * ITEMS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int shift = kRadixBits * pass;
    const int tile = blockIdx.x, tiles = gridDim.x;
    const int groups = (tiles + kSortGroup - 1) / kSortGroup;
    const int base = tile * kTile + warp * (ITEMS * 32);
    uint32_t *svals = reinterpret_cast<uint32_t *>(skeys + kTile);
    uint32_t *grp = a.grp + (size_t)(seq & 1) * groups * kRadixBuckets;
    // the other half of the group counts is free (read before the last
    // barrier): cleared for the next pass
    {
        uint32_t *nxt = a.grp + (size_t)((seq & 1) ^ 1) * groups * kRadixBuckets;
        for (int k = tile * kSortThreads + threadIdx.x; k < groups * kRadixBuckets;
             k += tiles * kSortThreads)
            nxt[k] = 0u;
    }
    for (int k = threadIdx.x; k < kSortWarps * kRadixBuckets; k += kSortThreads)
        (&sh.h[0][0])[k] = 0;
    __syncthreads();
    uint32_t rank[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const bool valid = base + r * 32 + lane < a.n;
        const uint32_t d = valid ? (uint32_t)(kk[r] >> shift) & (kRadixBuckets - 1) : 0u;
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int b = 0; b < kRadixBits; ++b) {
            const uint32_t bit = (d >> b) & 1u;
            const uint32_t vote = __ballot_sync(0xffffffffu, bit);
            peers &= bit ? vote : ~vote;
        }
        const uint32_t before = __popc(peers & lanemask_lt());
        uint32_t cur = 0;
        if (valid) cur = sh.h[warp][d];
        __syncwarp();
        if (valid && before == 0) sh.h[warp][d] = cur + __popc(peers);
        __syncwarp();
        rank[r] = cur + before;
    }
    __syncthreads();
    const int d = threadIdx.x;  // one digit per thread
    uint32_t count = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = sh.h[w][d];
        sh.h[w][d] = count;
        count += c;
    }
    a.tile_cnt[(size_t)tile * kRadixBuckets + d] = count;
    if (count) atomicAdd(&grp[(size_t)(tile / kSortGroup) * kRadixBuckets + d], count);
    {
        uint32_t total;
        sh.local_start[d] = block_exclusive_scan(count, sh.ws, total);
    }
    __syncthreads();
    // the tile in digit order in shared memory
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        if (base + r * 32 + lane >= a.n) continue;
        const uint32_t dg = (uint32_t)(kk[r] >> shift) & (kRadixBuckets - 1);
        const uint32_t lp = sh.local_start[dg] + sh.h[warp][dg] + rank[r];
        skeys[lp] = kk[r];
        svals[lp] = vv[r];
    }
    target += tiles;
    if (!tree_sort_barrier(a, target, &sh.ok)) return false;
    // this digit's keys in lower tiles, and in the whole state
    uint32_t before = 0, all = 0;
    for (int g = 0; g < groups; ++g) {
        const uint32_t c = __ldcg(&grp[(size_t)g * kRadixBuckets + d]);
        all += c;
        if (g < tile / kSortGroup) before += c;
    }
#pragma unroll 4
    for (int t = tile / kSortGroup * kSortGroup; t < tile; ++t)
        before += __ldcg(&a.tile_cnt[(size_t)t * kRadixBuckets + d]);
    {
        uint32_t total;
        sh.digit_off[d] = block_exclusive_scan(all, sh.ws, total) + before - sh.local_start[d];
    }
    __syncthreads();
    const int cnt = min(kTile, a.n - tile * kTile);
    for (int j = threadIdx.x; j < cnt; j += kSortThreads) {
        const uint64_t key = skeys[j];
        const uint32_t dg = (uint32_t)(key >> shift) & (kRadixBuckets - 1);
        const uint32_t pos = sh.digit_off[dg] + (uint32_t)j;
        keys_out[pos] = key;
        vals_out[pos] = svals[j];
    }
    target += tiles;
    return tree_sort_barrier(a, target, &sh.ok);
}

template <int ITEMS>
__device__ __forceinline__ void tree_sort_body(const TreeSortArgs &a, TreeSortShared<ITEMS> &sh,
                                               uint64_t *skeys)
{
    constexpr int kTile = kSortThreads * ITEMS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x, tiles = gridDim.x;
    const int base = tile * kTile + warp * (ITEMS * 32);
    uint32_t target = 0;
    // positions in batches whose loads are in flight together (a batch is a
    // thread's whole share up to 4 keys: then the keys need no second read)
    constexpr int kBatch = ITEMS < 4 ? ITEMS : 4;
    double px[kBatch], py[kBatch], pz[kBatch];
    auto load_positions = [&](int r0) {
#pragma unroll
        for (int r = 0; r < kBatch; ++r) {
            const int i = base + (r0 + r) * 32 + lane;
            const bool valid = r0 + r < ITEMS && i < a.n;
            px[r] = valid ? a.x[i] : 0.0;
            py[r] = valid ? a.y[i] : 0.0;
            pz[r] = valid ? a.z[i] : 0.0;
        }
    };
    // extent: the tiles' maxima, and the first pass's group counts cleared
    {
        const int groups = (tiles + kSortGroup - 1) / kSortGroup;
        for (int k = tile * kSortThreads + threadIdx.x; k < groups * kRadixBuckets;
             k += tiles * kSortThreads)
            a.grp[k] = 0u;
        if (tile == 0 && threadIdx.x == 0) a.bar[2] = 0u;
        if (tile == 0 && threadIdx.x < 2) a.stats[threadIdx.x] = 0ull;
        unsigned long long m = 0;
#pragma unroll 1
        for (int r0 = 0; r0 < ITEMS; r0 += kBatch) {
            load_positions(r0);
#pragma unroll
            for (int r = 0; r < kBatch; ++r)
                m = max(max(m, abs_bits(px[r])), max(abs_bits(py[r]), abs_bits(pz[r])));
        }
        if (!grid_extent<kSortWarps>(a, m, sh.wm, target, &sh.ok)) return;
    }
    const double X = __longlong_as_double((long long)sh.wm[0]);
    uint64_t kk[ITEMS];
    uint32_t vv[ITEMS];
    {
        __shared__ double s_scale;
        const double scale = key_scale(X, a.nchild, &s_scale);
        // through shared memory: the loop stays rolled (unrolled over all keys
        // its code outgrows the instruction cache) and the keys in registers
#pragma unroll 1
        for (int r0 = 0; r0 < ITEMS; r0 += kBatch) {
            if (ITEMS > kBatch) load_positions(r0);
#pragma unroll
            for (int r = 0; r < kBatch; ++r) {
                if (r0 + r >= ITEMS) break;
                const int i = base + (r0 + r) * 32 + lane;
                skeys[i - tile * kTile] =
                    i < a.n && X > 0.0 ? body_key(px[r], py[r], pz[r], X, scale, a.nchild) : 0ull;
            }
        }
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const int i = base + r * 32 + lane;  // written by this thread
            kk[r] = skeys[i - tile * kTile];
            vv[r] = (uint32_t)i;
        }
    }
    int seq = 0;
    uint64_t *kin = a.k0, *kout = a.k1;
    uint32_t *vin = a.v0, *vout = a.v1;
    auto load = [&]() {
#pragma unroll
        for (int r = 0; r < ITEMS; ++r) {
            const int i = base + r * 32 + lane;
            kk[r] = i < a.n ? __ldcg(&kin[i]) : 0ull;
            vv[r] = i < a.n ? __ldcg(&vin[i]) : 0u;
        }
    };
    auto swap = [&]() {
        uint64_t *tk = kin;
        kin = kout;
        kout = tk;
        uint32_t *tv = vin;
        vin = vout;
        vout = tv;
    };
    static_assert(kSortTopPasses % 2 == 0 && kSortPasses % 2 == 1, "the order ends in k1, v1");
#pragma unroll 1
    for (int pass = kSortPasses - kSortTopPasses; pass < kSortPasses; ++pass) {
        if (seq > 0) load();
        if (!tree_sort_pass<ITEMS>(a, pass, seq, target, kk, vv, kout, vout, sh, skeys)) return;
        ++seq;
        swap();
    }
    // kin (k0) is in order of the top digits; each key's place among those
    // that share them, into k1
    {
        const int shift = kRadixBits * (kSortPasses - kSortTopPasses);
        const int t0 = tile * kTile;
#pragma unroll 4  // loads in flight together
        for (int t = threadIdx.x; t < kTile + 2 * kFixRun; t += kSortThreads) {
            const int i = t0 - kFixRun + t;
            skeys[t] = i >= 0 && i < a.n ? __ldcg(&kin[i]) : ~0ull;  // no key has bit 63
        }
        uint32_t *sv = reinterpret_cast<uint32_t *>(skeys + kTile + 2 * kFixRun);
#pragma unroll 4
        for (int t = threadIdx.x; t < kTile; t += kSortThreads)
            sv[t] = t0 + t < a.n ? __ldcg(&vin[t0 + t]) : 0u;
        __syncthreads();
        // a key and the kFixRun-th after it differ and share the top digits: the run is
        // too long for sure, and no place in it need be looked for
        bool too_long = false;
        for (int t = threadIdx.x; t < kTile && t0 + t < a.n; t += kSortThreads) {
            const uint64_t k = skeys[kFixRun + t], o = skeys[2 * kFixRun + t];
            too_long |= k != o && !((k ^ o) >> shift);
        }
        const bool place = !__syncthreads_or(too_long);
#pragma unroll 1
        for (int t = threadIdx.x; place && t < kTile && t0 + t < a.n; t += kSortThreads) {
            const uint64_t *p = skeys + kFixRun + t;
            const uint64_t k = p[0];
            int left = 0, right = 0, rank = 0;
            bool differ = false;
            while (left < kFixRun) {
                const uint64_t o = p[-(left + 1)];
                if ((o ^ k) >> shift) break;
                ++left;
                rank += o <= k;
                differ |= o != k;
            }
            while (right < kFixRun) {
                const uint64_t o = p[right + 1];
                if ((o ^ k) >> shift) break;
                ++right;
                rank += o < k;
                differ |= o != k;
            }
            too_long |= differ && (left == kFixRun || right == kFixRun);
            const int at = t0 + t;
            const int to = at - left + rank;  // within the run: always in [0, n)
            kout[to] = k;
            vout[to] = sv[t];
        }
        if (__syncthreads_or(too_long) && threadIdx.x == 0) atomicOr(&a.bar[2], 1u);
    }
    target += tiles;
    if (!tree_sort_barrier(a, target, &sh.ok)) return;
    if (__ldcg(&a.bar[2]) == 0u) return;
#pragma unroll 1
    for (int pass = 0; pass < kSortPasses; ++pass) {
        load();
        if (!tree_sort_pass<ITEMS>(a, pass, seq, target, kk, vv, kout, vout, sh, skeys)) return;
        ++seq;
        swap();
    }
}

template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads, 1) tree_sort_kernel(TreeSortArgs a)
{
    static_assert(kSortThreads == kRadixBuckets, "one thread per digit");
    __shared__ TreeSortShared<ITEMS> sh;
    extern __shared__ uint64_t skeys_dyn[];
    tree_sort_body<ITEMS>(a, sh, skeys_dyn);
    leave_grid(a.bar);
}

// The same for few bodies, by ranks instead of digits: each block sorts a tile of
// kRankTile keys (a bitonic network), then every key's place is its place in its
// own tile plus the keys below it in each other tile, by binary search over all
// the tiles' keys in shared memory.  Keys compare whole and equal ones keep the
// order of their tiles and places, so any state takes the same time, with two
// barriers where the digit passes take ten.  A key's searches and the keys each
// block reads grow with n.  Step times by digits / by ranks (us), theta 1.0, leaf
// 16, Plummer and cube: 255 bodies 50 / 42 and 53 / 41, 2,003 67 / 51 and 67 / 51,
// 8,195 74 / 62 and 73 / 58, 16,384 74 / 70 and 74 / 67, 20,011 76 / 77 and 73 /
// 73, 24,576 77 / 81 and 77 / 79.
constexpr int kRankTile = 256;
constexpr int kRankMax = 18432;

__device__ __forceinline__ void rank_sort_body(const TreeSortArgs &a, uint64_t *all)
{
    __shared__ unsigned long long wm[kRankTile / 32];
    __shared__ double s_scale;
    __shared__ int s_ok;
    const int t = threadIdx.x, tile = blockIdx.x, tiles = gridDim.x;
    const int i = tile * kRankTile + t;
    if (tile == 0 && t < 2) a.stats[t] = 0ull;
    uint32_t target = 0;
    double x = 0.0, y = 0.0, z = 0.0;
    if (i < a.n) {
        x = a.x[i];
        y = a.y[i];
        z = a.z[i];
    }
    if (!grid_extent<kRankTile / 32>(a, max(abs_bits(x), max(abs_bits(y), abs_bits(z))), wm, target,
                                     &s_ok))
        return;
    const double X = __longlong_as_double((long long)wm[0]);
    const double scale = key_scale(X, a.nchild, &s_scale);
    // (no key has bit 63: the places after the last body sort to the end)
    uint64_t k = i >= a.n ? ~0ull : X > 0.0 ? body_key(x, y, z, X, scale, a.nchild) : 0ull;
    uint32_t v = t;
    // the tile, by (key, place)
    {
        uint32_t *sv = reinterpret_cast<uint32_t *>(all + 2 * kRankTile);
        int buf = 0;
#pragma unroll 1
        for (int size = 2; size <= kRankTile; size <<= 1) {
#pragma unroll 1
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                uint64_t pk;
                uint32_t pv;
                if (stride >= 32) {
                    all[buf + t] = k;
                    sv[buf + t] = v;
                    __syncthreads();
                    pk = all[buf + (t ^ stride)];
                    pv = sv[buf + (t ^ stride)];
                    buf ^= kRankTile;  // (read again only after the next barrier)
                } else {
                    pk = __shfl_xor_sync(0xffffffffu, k, stride);
                    pv = __shfl_xor_sync(0xffffffffu, v, stride);
                }
                const bool less = k < pk || (k == pk && v < pv);
                if (less != (((t & stride) == 0) == ((t & size) == 0))) {
                    k = pk;
                    v = pv;
                }
            }
        }
    }
    if (i < a.n) a.k0[i] = k;
    target += tiles;
    if (!tree_sort_barrier(a, target, &s_ok)) return;
    // all keys, 16 bytes at a time; no key is below the places after the last
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(all);
    for (int p = t; p < a.n / 2; p += kRankTile)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * p),
                     "l"(a.k0 + 2 * p)
                     : "memory");
    for (int p = (a.n & ~1) + t; p < tiles * kRankTile; p += kRankTile)
        all[p] = p < a.n ? __ldcg(&a.k0[p]) : ~0ull;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (i >= a.n) return;
    int to = t;
#pragma unroll 4
    for (int o = 0; o < tiles; ++o) {
        if (o == tile) continue;
        const uint64_t *q = all + o * kRankTile;
        const uint64_t below = k + (o < tile);  // equal keys of earlier tiles come first
        int at = 0;
#pragma unroll
        for (int step = kRankTile / 2; step > 0; step >>= 1)
            at += q[at + step - 1] < below ? step : 0;
        to += at + (q[at] < below);
    }
    a.k1[to] = k;
    a.v1[to] = (uint32_t)(tile * kRankTile) + v;
}

__global__ void __launch_bounds__(kRankTile, 1) rank_sort_kernel(TreeSortArgs a)
{
    extern __shared__ __align__(16) uint64_t rank_keys[];  // (16-byte asynchronous copies)
    rank_sort_body(a, rank_keys);
    leave_grid(a.bar);
}

// ---------------------------------------------------------------------------
// node arrays
// ---------------------------------------------------------------------------
struct NodeArrays {
    int32_t *begin, *count, *child;
    uint8_t *nchild, *level;
    float4 *geo;     // cx, cy, cz, extent (f32)
    float4 *geo_lo;  // the centre's f64 value less its f32 one (exact traversal only)
    float4 *com;   // x, y, z, mass (f32)
    int4 *meta;    // (id | nchild << 28, first child, first body, body count)
    int32_t *parent;   // parent node, -1 for the root
    float4 *quad_a;    // second moments about the centre of mass: Sxx, Syy, Szz, trace
    float4 *quad_b;    // Sxy, Sxz, Syz, 0
    int cap;
};

// ---------------------------------------------------------------------------
// double-float helpers
// ---------------------------------------------------------------------------
// (ah, al) + (bh, bl) as a normalised double-float pair.
__device__ __forceinline__ void df_add(float &ah, float &al, float bh, float bl)
{
    float s, e;
    two_sum(ah, bh, s, e);
    e += al + bl;
    ah = s + e;
    al = e - (ah - s);
}

// f32 rounding of (sh + sl) / (mh + ml): an f32 quotient corrected once with
// its exact residual (TwoProduct by FMA).
__device__ __forceinline__ float df_div(float sh, float sl, float mh, float ml)
{
    const float q = sh / mh;
    const float p = q * mh;
    const float pe = fmaf(q, mh, -p);
    const float r = fmaf(-q, ml, ((sh - p) - pe) + sl);
    return q + r / mh;
}

__device__ __forceinline__ float4 df_com(const float4 h, const float4 l, float4 geo)
{
    if (h.x == 0.f && l.x == 0.f) return make_float4(geo.x, geo.y, geo.z, 0.f);
    return make_float4(df_div(h.y, l.y, h.x, l.x), df_div(h.z, l.z, h.x, l.x),
                       df_div(h.w, l.w, h.x, l.x), h.x + l.x);
}

// m * p added exactly-rounded into the double-float (hi, lo)
__device__ __forceinline__ void df_add_prod(float &hi, float &lo, float m, float p)
{
    const float pr = m * p;
    const float pe = fmaf(m, p, -pr);
    df_add(hi, lo, pr, pe);
}

// ---------------------------------------------------------------------------
// 4. tree build (flat: a few launches for all levels)
// ---------------------------------------------------------------------------
// The tree is the reference's non-path-compressed one over the sorted keys: a
// node at level l is a maximal run of bodies sharing the first l digits of
// their keys, and it exists iff l = 0 or the run one level up (its parent)
// splits, i.e. holds more than leaf_size bodies whose keys are not all equal,
// at a level below D.  Node numbering is breadth first: levels one after the
// other, each in key order, so a node's children are contiguous and in
// octant order, as a level-by-level serial build lays them out.
//
// With L(i) the number of leading digits keys[i-1] and keys[i] share, a run
// at level l starts at body i iff i = 0 or L(i) < l, and everything about
// the runs starting at i follows from L near i:
//   * the run at level l starting at i has more than `leaf` bodies iff
//     L(i+1..i+leaf) are all >= l (those bodies exist);
//   * it is not uniform iff the first body after i with a different key,
//     u(i), has L(u(i)) >= l;
//   * so it splits iff l <= c(i) = min(m(i), L(u(i)), D - 1), m(i) the
//     minimum of L over the next leaf boundaries;
//   * a run at level l > L(i) + 1 starting at i exists iff its parent (the
//     run at l - 1 starting at i) splits, i.e. l <= c(i) + 1;
//   * the run at level L(i) + 1 exists iff the run at level L(i) containing
//     i - 1 and i (not uniform: those keys differ) has more than leaf
//     bodies, which a scan of L over leaf boundaries either side decides.
// Each body's existing runs form a bit mask over levels; a node's index is
// the start of its level plus the count of set bits of that level before its
// body (block counts, one scan over blocks, warp ballots within a block).
// The deepest run a body starts is a leaf; its end (the next boundary below
// its level) is read off the same shared tile of L.

constexpr int kTreeBlock = 1024;   // bodies per block of the mask and node kernels
constexpr int kTreeHalo = 72;      // boundaries read either side (> the largest leaf + 1)
constexpr int kMaxLeaf = 64;
constexpr uint8_t kLongLeaf = 255;  // leaf count marker: longer than the shared tile reaches

__device__ __forceinline__ bool sort_failed(const uint32_t *flags)
{
    return *(volatile const uint32_t *)&flags[kFlagSort] != 0u;
}

// Sums over groups of consecutive sorted bodies, from which cell_kernel reads
// any cell's moments without waiting for its children: level k holds groups of
// kSegBase 2^k bodies, complete groups only, level after level.  A group keeps
// its mass and mass-weighted position sums (M, Mx, My, Mz) as double-float
// pairs (hi + lo) and, for quadrupole builds, its f32 centre of mass and second
// moments about it.  Sums are additions of sub-sums only (no differences of
// prefixes), so a cell is as exact beside a heavy neighbour as alone.
constexpr int kSegBase = 4;
constexpr int kSegLevels = 30;
constexpr int kSegBlock = 1024;                   // bodies whose groups one block sums
constexpr int kSegBlockLevel = 8;                 // kSegBase << 8 = kSegBlock

struct Segments {
    float4 *hi, *lo;
    float4 *com, *qa, *qb;  // quadrupole builds
    int n;                  // bodies
    int off[kSegLevels];    // first group of each level
    __host__ __device__ int groups(int level) const { return n / kSegBase >> level; }
};

struct GroupSum {
    float4 h, l;
};

__device__ __forceinline__ void df_add4(GroupSum &a, const GroupSum &b)
{
    df_add(a.h.x, a.l.x, b.h.x, b.l.x);
    df_add(a.h.y, a.l.y, b.h.y, b.l.y);
    df_add(a.h.z, a.l.z, b.h.z, b.l.z);
    df_add(a.h.w, a.l.w, b.h.w, b.l.w);
}

__device__ __forceinline__ void df_add_body(GroupSum &a, float4 p)
{
    df_add(a.h.x, a.l.x, p.w, 0.f);
    df_add_prod(a.h.y, a.l.y, p.w, p.x);
    df_add_prod(a.h.z, a.l.z, p.w, p.y);
    df_add_prod(a.h.w, a.l.w, p.w, p.z);
}

__device__ __forceinline__ GroupSum group_zero()
{
    GroupSum g;
    g.h = g.l = make_float4(0.f, 0.f, 0.f, 0.f);
    return g;
}

// Second moments: xx, yy, zz, xy, xz, yz.
struct Quad6 {
    float v[6];
};

// q += m d d^T + s (s about its own centre, d from the new centre to it)
__device__ __forceinline__ void quad_shift_add(Quad6 &q, const Quad6 &s, float m, float dx,
                                               float dy, float dz)
{
    q.v[0] += fmaf(m * dx, dx, s.v[0]);
    q.v[1] += fmaf(m * dy, dy, s.v[1]);
    q.v[2] += fmaf(m * dz, dz, s.v[2]);
    q.v[3] += fmaf(m * dx, dy, s.v[3]);
    q.v[4] += fmaf(m * dx, dz, s.v[4]);
    q.v[5] += fmaf(m * dy, dz, s.v[5]);
}

__device__ __forceinline__ void quad_body_add(Quad6 &q, float4 p, float4 com)
{
    const float dx = p.x - com.x, dy = p.y - com.y, dz = p.z - com.z;
    q.v[0] = fmaf(p.w * dx, dx, q.v[0]);
    q.v[1] = fmaf(p.w * dy, dy, q.v[1]);
    q.v[2] = fmaf(p.w * dz, dz, q.v[2]);
    q.v[3] = fmaf(p.w * dx, dy, q.v[3]);
    q.v[4] = fmaf(p.w * dx, dz, q.v[4]);
    q.v[5] = fmaf(p.w * dy, dz, q.v[5]);
}

__device__ __forceinline__ Quad6 quad_load(const Segments &sg, int at)
{
    const float4 a = sg.qa[at], b = sg.qb[at];
    return {{a.x, a.y, a.z, b.x, b.y, b.z}};
}

__device__ __forceinline__ void group_store(const Segments &sg, int at, const GroupSum &g)
{
    sg.hi[at] = g.h;
    sg.lo[at] = g.l;
}

__device__ __forceinline__ void group_store_quad(const Segments &sg, int at, float4 com,
                                                 const Quad6 &q)
{
    sg.com[at] = com;
    sg.qa[at] = make_float4(q.v[0], q.v[1], q.v[2], q.v[0] + q.v[1] + q.v[2]);
    sg.qb[at] = make_float4(q.v[3], q.v[4], q.v[5], 0.f);
}

// A group and its quadrupole from its two halves.
template <bool kQuad>
__device__ __forceinline__ void group_join(GroupSum &g, float4 &com, Quad6 &q, const GroupSum &o,
                                           float4 ocom, const Quad6 &oq)
{
    df_add4(g, o);
    if (kQuad) {
        const float4 c = df_com(g.h, g.l, com);
        Quad6 t = {{0.f, 0.f, 0.f, 0.f, 0.f, 0.f}};
        quad_shift_add(t, q, com.w, com.x - c.x, com.y - c.y, com.z - c.z);
        quad_shift_add(t, oq, ocom.w, ocom.x - c.x, ocom.y - c.y, ocom.z - c.z);
        com = c;
        q = t;
    }
}

__device__ __forceinline__ float4 shfl_down4(float4 v, int o)
{
    return make_float4(__shfl_down_sync(0xffffffffu, v.x, o), __shfl_down_sync(0xffffffffu, v.y, o),
                       __shfl_down_sync(0xffffffffu, v.z, o),
                       __shfl_down_sync(0xffffffffu, v.w, o));
}

__device__ __forceinline__ float4 shfl_xor4(float4 v, int o)
{
    return make_float4(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o),
                       __shfl_xor_sync(0xffffffffu, v.z, o), __shfl_xor_sync(0xffffffffu, v.w, o));
}

// Sums of the next levels over the block's threads (thread t holds group
// first + t of `level`, complete where first + t < groups(level)), by shuffles
// within a warp and then over the warps' sums in shared memory; each complete
// group is stored.
// kThreads threads take part, the block's first; fewer than the whole block
// (kShare) meet at a named barrier.
template <int kThreads, bool kShare>
__device__ __forceinline__ void share_sync()
{
    if (kShare)
        asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
    else
        __syncthreads();
}

template <bool kQuad, int kThreads, bool kShare>
__device__ __forceinline__ void block_groups(const Segments &sg, int level, int first,
                                             GroupSum g, float4 com, Quad6 q,
                                             GroupSum *warp_sum, float4 *warp_com,
                                             Quad6 *warp_quad)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto fold = [&](int at, int lanes) {  // `at`: this thread's group of `level`
        for (int o = 1; o < lanes; o <<= 1) {
            GroupSum p;
            p.h = shfl_down4(g.h, o);
            p.l = shfl_down4(g.l, o);
            float4 pc = com;
            Quad6 pq = q;
            if (kQuad) {
                pc = shfl_down4(com, o);
#pragma unroll
                for (int c = 0; c < 6; ++c) pq.v[c] = __shfl_down_sync(0xffffffffu, q.v[c], o);
            }
            ++level;
            at >>= 1;
            if (lane < lanes && (lane & (2 * o - 1)) == 0) {
                group_join<kQuad>(g, com, q, p, pc, pq);
                if (level < kSegLevels && at < sg.groups(level)) {
                    group_store(sg, sg.off[level] + at, g);
                    if (kQuad) group_store_quad(sg, sg.off[level] + at, com, q);
                }
            }
        }
    };
    fold(first + (int)threadIdx.x, 32);
    if (lane == 0) {
        warp_sum[warp] = g;
        if (kQuad) {
            warp_com[warp] = com;
            warp_quad[warp] = q;
        }
    }
    share_sync<kThreads, kShare>();
    constexpr int warps = kThreads / 32;
    if (warp == 0) {
        const int w = lane < warps ? lane : 0;
        g = warp_sum[w];
        if (kQuad) {
            com = warp_com[w];
            q = warp_quad[w];
        }
        fold((first >> 5) + lane, warps);
    }
}

// L(k) for k >= 1: the number of leading digits that a and b (keys k - 1 and k)
// share, D for equal keys.
__device__ __forceinline__ int shared_digits(uint64_t a, uint64_t b, int nchild)
{
    const int D = tree_levels(nchild), B = level_bits(nchild);
    const uint64_t x = a ^ b;
    // keys use the low B * D bits: 64 - B * D leading bits are always 0
    return x == 0 ? D : (__clzll((long long)x) - (64 - B * D)) / B;
}

struct GatherArgs {
    const uint64_t *keys;
    const uint32_t *order;
    int n, nchild;
    const float4 *body4;
    const double *bx, *by, *bz;
    float4 *sbody, *sbody_lo;
    uint8_t *lcp;  // null: not kept
    Segments sg;
};

template <int kThreads>
struct GatherShared {
    GroupSum sum[kThreads / 32];
    float4 com[kThreads / 32];
    Quad6 quad[kThreads / 32];
};

// The sorted f32 bodies (with kExact what f32 dropped of their f64 positions),
// the L of lcp, and the group sums of kThreads * kSegBase bodies from group
// `first` on, by the block's first kThreads threads.  Four bodies a thread: the
// keys and the order come as 16-byte words and a thread's bodies are its first
// group.
template <bool kQuad, bool kExact, int kThreads, bool kShare>
__device__ __forceinline__ void gather_groups(const GatherArgs &a, int first,
                                              GatherShared<kThreads> &sh)
{
    static_assert(kSegBase == 4, "a thread's bodies are one 16-byte word of the order");
    const int g0 = first + (int)threadIdx.x;  // this thread's group
    const int k0 = g0 * kSegBase;
    const int cnt = max(0, min(kSegBase, a.n - k0));
    uint64_t key[kSegBase] = {0, 0, 0, 0};
    uint32_t ord[kSegBase] = {0, 0, 0, 0};
    if (cnt == kSegBase) {
        const uint4 o = *reinterpret_cast<const uint4 *>(a.order + k0);
        ord[0] = o.x;
        ord[1] = o.y;
        ord[2] = o.z;
        ord[3] = o.w;
        if (a.lcp) {
            const ulonglong2 u = *reinterpret_cast<const ulonglong2 *>(a.keys + k0);
            const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(a.keys + k0 + 2);
            key[0] = u.x;
            key[1] = u.y;
            key[2] = v.x;
            key[3] = v.y;
        }
    } else {
#pragma unroll
        for (int u = 0; u < kSegBase; ++u)
            if (u < cnt) {
                ord[u] = a.order[k0 + u];
                if (a.lcp) key[u] = a.keys[k0 + u];
            }
    }
    uint64_t prev = a.lcp && k0 > 0 && cnt > 0 ? a.keys[k0 - 1] : 0ull;
    float4 p[kSegBase];
#pragma unroll
    for (int u = 0; u < kSegBase; ++u)
        p[u] = u < cnt ? a.body4[ord[u]] : make_float4(0.f, 0.f, 0.f, 0.f);
    GroupSum g = group_zero();
#pragma unroll
    for (int u = 0; u < kSegBase; ++u) {
        if (u >= cnt) continue;
        if (a.lcp) {
            const int L = shared_digits(prev, key[u], a.nchild);
            prev = key[u];
            a.lcp[k0 + u] = (uint8_t)(k0 + u == 0 ? 0 : L);
        }
        a.sbody[k0 + u] = p[u];
        if (kExact) {
            const uint32_t i = ord[u];
            a.sbody_lo[k0 + u] = make_float4((float)(a.bx[i] - (double)p[u].x),
                                             (float)(a.by[i] - (double)p[u].y),
                                             (float)(a.bz[i] - (double)p[u].z), 0.f);
        }
        df_add_body(g, p[u]);
    }
    float4 com = p[0];
    Quad6 q = {{0.f, 0.f, 0.f, 0.f, 0.f, 0.f}};
    if (kQuad) {
        com = df_com(g.h, g.l, p[0]);
#pragma unroll
        for (int u = 0; u < kSegBase; ++u)
            if (u < cnt) quad_body_add(q, p[u], com);
    }
    if (g0 < a.sg.groups(0)) {
        group_store(a.sg, a.sg.off[0] + g0, g);
        if (kQuad) group_store_quad(a.sg, a.sg.off[0] + g0, com, q);
    }
    block_groups<kQuad, kThreads, kShare>(a.sg, 0, first, g, com, q, sh.sum, sh.com, sh.quad);
}

template <bool kQuad, bool kExact>
__global__ void __launch_bounds__(kSegBlock / kSegBase)
boundary_kernel(GatherArgs a, const uint32_t *__restrict__ flags)
{
    pdl_wait();
    if (sort_failed(flags)) return;
    constexpr int kThreads = kSegBlock / kSegBase;
    __shared__ GatherShared<kThreads> sh;
    gather_groups<kQuad, kExact, kThreads, false>(a, blockIdx.x * kThreads, sh);
}

// The group sums above level `from`, by one block of kThreads threads
// (log2(kThreads) levels per round).
template <bool kQuad, int kThreads>
__device__ __forceinline__ void top_groups(const Segments &sg, int from)
{
    constexpr int kLevels = kThreads == 1024 ? 10 : 9;
    static_assert(kThreads == 1 << kLevels, "512 or 1,024 threads");
    __shared__ GatherShared<kThreads> sh;
    for (int level = from; level < kSegLevels && sg.groups(level) > 1; level += kLevels) {
        const int m = sg.groups(level);
        for (int first = 0; first < m; first += kThreads) {
            const int at = first + (int)threadIdx.x;
            GroupSum g = group_zero();
            float4 com = make_float4(0.f, 0.f, 0.f, 0.f);
            Quad6 q = {{0.f, 0.f, 0.f, 0.f, 0.f, 0.f}};
            if (at < m) {
                g.h = __ldcg(&sg.hi[sg.off[level] + at]);
                g.l = __ldcg(&sg.lo[sg.off[level] + at]);
                if (kQuad) {
                    com = __ldcg(&sg.com[sg.off[level] + at]);
                    const float4 a = __ldcg(&sg.qa[sg.off[level] + at]);
                    const float4 b = __ldcg(&sg.qb[sg.off[level] + at]);
                    q = {{a.x, a.y, a.z, b.x, b.y, b.z}};
                }
            }
            block_groups<kQuad, kThreads, false>(sg, level, first, g, com, q, sh.sum, sh.com,
                                                 sh.quad);
            __syncthreads();  // the warps' sums serve the next chunk, the groups the next round
        }
    }
}

// First index j in [lo, n) with keys[j] != keys[i] (keys sorted), or n.
__device__ __forceinline__ int next_key_change(const uint64_t *__restrict__ keys, int i, int lo,
                                               int n)
{
    const uint64_t ki = keys[i];
    int hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (keys[mid] == ki)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Level masks of the bodies (bit l: a node at level l starts at this body),
// per-block counts of every level (blk_cnt[l * nblk + block]) and the body
// count of the leaf starting at each body (the deepest run it starts; 0: no
// node starts here, kLongLeaf: longer than the shared tile reaches).  The questions about L near a body (the minimum
// over the next `leaf` boundaries; how many consecutive boundaries either side,
// or after the body, are at or below a level) are answered from tables of
// window minima over 1, 2, 4, ..., 64 boundaries of the block's tile: the
// minimum over any window of up to 64 from two overlapping entries, a run
// length by binary lifting (the longest run is the sum of the powers of two
// whose windows, taken largest first, stay at or below the level), so every
// body takes the same few steps instead of a loop of data-dependent length.
constexpr int kMinTables = 7;  // windows of 2^0 .. 2^6 boundaries
static_assert(kMaxLeaf <= (1 << (kMinTables - 1)) && kMaxLeaf + 1 < kTreeHalo,
              "leaf windows fit the tables and the halo");

template <int kBlock>
struct MaskShared {
    // m[p][t]: minimum of L over boundaries t .. t + 2^p - 1 of the tile
    // (clipped at the tile's end; every query below stays inside it)
    int8_t m[kMinTables][kBlock + 2 * kTreeHalo];
    uint32_t cnt[32];
};

// One tile of kBlock bodies, one thread each: its body's mask m and leaf count
// lc, and the tile's counts to blk_cnt; shared(j) gives L(j).
template <int kBlock, typename Shared>
__device__ __forceinline__ void level_masks(const uint64_t *__restrict__ keys, Shared shared,
                                            int tile, int n, int nchild, int leaf,
                                            uint32_t *__restrict__ blk_cnt, int nblk,
                                            MaskShared<kBlock> &sh, uint32_t &m, uint8_t &lc)
{
    constexpr int kTile = kBlock + 2 * kTreeHalo;
    const int D = tree_levels(nchild);
    const int base = tile * kBlock;
    // boundaries base - halo .. base + block + halo; -1 marks "no boundary
    // beyond here" (index 0 starts every run, indices >= n end them)
    for (int t = threadIdx.x; t < kTile; t += blockDim.x) {
        const int j = base - kTreeHalo + t;
        sh.m[0][t] = (j >= 1 && j < n) ? (int8_t)shared(j) : (int8_t)-1;
    }
    if (threadIdx.x < 32) sh.cnt[threadIdx.x] = 0u;
    __syncthreads();
    for (int q = 1; q < kMinTables; ++q) {
        const int h = 1 << (q - 1);
        for (int t = threadIdx.x; t < kTile; t += blockDim.x) {
            const int a = sh.m[q - 1][t];
            sh.m[q][t] = (int8_t)(t + h < kTile ? min(a, (int)sh.m[q - 1][t + h]) : a);
        }
        __syncthreads();
    }
    const int8_t *sL = sh.m[0];
    const int i = base + threadIdx.x;
    m = 0u;
    lc = 0;
    if (i < n) {
        const int s = threadIdx.x + kTreeHalo;  // i's slot in the tile
        const int Li = i == 0 ? -1 : sL[s];
        // m(i): min of L over the next leaf boundaries, -1 if fewer remain
        int mi = -1;
        if (i + leaf <= n - 1) {
            const int q = 31 - __clz(leaf);
            mi = min((int)sh.m[q][s + 1], (int)sh.m[q][s + leaf + 1 - (1 << q)]);
        }
        // u(i): the next body with another key; L(u(i)), -1 if none
        int Lu = -1;
        {
            int j = i + 1, t = s + 1;
            while (j < n && t < kTile && sL[t] == D) {
                ++j;
                ++t;
            }
            if (j < n && t >= kTile) j = next_key_change(keys, i, j, n);
            if (j < n) Lu = shared(j);
        }
        const int c = min(min(mi, Lu), D - 1);
        if (i == 0) {
            m = 1u;  // the root
            for (int l = 1; l <= c + 1; ++l) m |= 1u << l;
        } else if (Li < D) {
            // the run at level Li containing i - 1 and i: more than leaf bodies?
            // (lft, rgt: consecutive boundaries at or below Li before and
            // after i, up to leaf each)
            int lft = 0, rgt = 0;
#pragma unroll
            for (int q = kMinTables - 1; q >= 0; --q) {
                const int k = 1 << q;
                if (lft + k <= leaf && sh.m[q][s - lft - k] >= Li) lft += k;
                if (rgt + k <= leaf && sh.m[q][s + rgt + 1] >= Li) rgt += k;
            }
            if (lft + rgt + 2 > leaf) {
                m |= 1u << (Li + 1);
                for (int l = Li + 2; l <= c + 1; ++l) m |= 1u << l;
            }
        }
        // the leaf starting here (the deepest run; unless the capacity stops
        // the tree above it) runs to the next boundary below its level
        if (m != 0u) {
            const int lf = 31 - __clz(m);
            const int room = kTile - 1 - s;  // boundaries after i in the tile
            int run = 0;
            while (run + 64 <= room && sh.m[6][s + 1 + run] >= lf) run += 64;
#pragma unroll
            for (int q = kMinTables - 2; q >= 0; --q) {
                const int k = 1 << q;
                if (run + k <= room && sh.m[q][s + 1 + run] >= lf) run += k;
            }
            const int e = i + 1 + run, t = s + 1 + run;
            lc = (e < n && t >= kTile) || e - i >= (int)kLongLeaf ? kLongLeaf
                                                                      : (uint8_t)(e - i);
        }
    }
    // per-level counts: only the levels some lane of the warp starts
    uint32_t present = __reduce_or_sync(0xffffffffu, m);
    while (present) {
        const int l = __ffs(present) - 1;
        present &= present - 1u;
        const uint32_t b = __ballot_sync(0xffffffffu, (m >> l) & 1u);
        if ((threadIdx.x & 31) == 0) atomicAdd(&sh.cnt[l], (uint32_t)__popc(b));
    }
    __syncthreads();
    if (threadIdx.x < 32) blk_cnt[(size_t)threadIdx.x * nblk + tile] = sh.cnt[threadIdx.x];
}

__global__ void __launch_bounds__(kTreeBlock)
mask_kernel(const uint64_t *__restrict__ keys, const uint8_t *__restrict__ lcp, int n,
            int nchild, int leaf, uint32_t *__restrict__ mask, uint32_t *__restrict__ blk_cnt,
            int nblk, uint8_t *__restrict__ leafcnt, const uint32_t *__restrict__ flags)
{
    pdl_wait();
    if (sort_failed(flags)) return;
    __shared__ MaskShared<kTreeBlock> sh;
    uint32_t m;
    uint8_t lc;
    level_masks<kTreeBlock>(
        keys, [&](int j) { return (int)lcp[j]; }, blockIdx.x, n, nchild, leaf, blk_cnt, nblk, sh,
        m, lc);
    const int i = blockIdx.x * kTreeBlock + threadIdx.x;
    if (i < n) {
        mask[i] = m;
        leafcnt[i] = lc;
    }
}

// The levels' first nodes and counts from their totals, by one warp.  If the
// nodes do not fit the node arrays, the tree stops at the deepest level that
// fits (its nodes become leaves: results stay exact, slower) and
// flags[kFlagNodes] is raised.
__device__ __forceinline__ void level_starts(const uint32_t *total_of, int D, int cap,
                                             LevelInfo &lv, uint32_t *flags)
{
    static_assert(kMaxLevels <= 32, "a level per lane");
    const int q = threadIdx.x & 31;
    const long long c = q <= D ? (long long)total_of[q] : 0;
    long long end = c;  // of level q's nodes
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, end, o);
        if (q >= o) end += t;
    }
    const uint32_t over = __ballot_sync(0xffffffffu, end > cap);
    const int max_level = over ? min(D, __ffs(over) - 2) : D;
    const int total = max_level < 0 ? 0 : (int)__shfl_sync(0xffffffffu, end, max_level & 31);
    for (int l = q; l < kMaxLevels + 2; l += 32) {
        const bool built = l == q && l <= max_level;
        lv.begin[l] = built ? (int32_t)(end - c) : total;
        lv.count[l] = built ? (int32_t)c : 0;
    }
    if (q == 0) {
        lv.total = total;
        lv.max_level = max_level;
        if (over) atomicOr(&flags[kFlagNodes], 1u);
    }
}

// Block 0: per level, the exclusive scan of the block counts (blk_off,
// same layout as blk_cnt) and the level's first node; block 1: the group sums
// of over kSegBlock bodies.  Warp l scans row l, 32 blocks per step.
__global__ void __launch_bounds__(1024)
level_scan_kernel(const uint32_t *__restrict__ blk_cnt, int nblk, int nchild,
                  uint32_t *__restrict__ blk_off, LevelInfo *lv, int cap,
                  uint32_t *__restrict__ flags, Segments sg, int quad)
{
    pdl_wait();
    if (sort_failed(flags)) return;
    if (blockIdx.x == 1) {
        if (quad)
            top_groups<true, 1024>(sg, kSegBlockLevel);
        else
            top_groups<false, 1024>(sg, kSegBlockLevel);
        return;
    }
    __shared__ uint32_t total_of[32];
    const int D = tree_levels(nchild);
    const int l = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t *row = blk_cnt + (size_t)l * nblk;
    uint32_t *orow = blk_off + (size_t)l * nblk;
    uint32_t carry = 0;
    constexpr int kAhead = 4;  // row chunks loaded before they are scanned
    for (int c0 = 0; c0 < nblk; c0 += 32 * kAhead) {
        uint32_t v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int b = c0 + u * 32 + lane;
            v[u] = b < nblk ? row[b] : 0u;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            uint32_t incl = v[u];
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const int b = c0 + u * 32 + lane;
            if (b < nblk) orow[b] = carry + incl - v[u];
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    if (lane == 0) total_of[l] = carry;
    __syncthreads();
    if (threadIdx.x < 32) level_starts(total_of, D, cap, *lv, flags);
}

// Node records: per body, one node per set bit of its mask.  Leaves get
// their body count here; an internal node's count, its child count and its
// traversal metadata, and every node's geometry and moments, are cell_kernel's.
template <int kBlock>
struct NodeShared {
    uint32_t bal[kBlock / 32][32];  // per warp and level: lanes with that bit
    uint32_t off[kBlock / 32][32];  // ... and the level's nodes before the warp
};

// One tile of kBlock bodies, one thread each, with its body's mask m and leaf
// count lc; before(l): the nodes of level l in the tiles before it.
template <int kBlock, typename Before>
__device__ __forceinline__ void node_records(const uint64_t *__restrict__ keys, uint32_t m,
                                             uint8_t lc, Before before, int tile, int n,
                                             int nchild, const NodeArrays &nd,
                                             const LevelInfo &lv, NodeShared<kBlock> &sh)
{
    const int D = tree_levels(nchild), B = level_bits(nchild);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = tile * kBlock + threadIdx.x;
    for (int l = 0; l < 32; ++l) {
        const uint32_t b = __ballot_sync(0xffffffffu, (m >> l) & 1u);
        if (lane == 0) {
            sh.bal[warp][l] = b;
            sh.off[warp][l] = (uint32_t)__popc(b);
        }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t run = before(threadIdx.x);
        for (int w = 0; w < kBlock / 32; ++w) {
            const uint32_t v = sh.off[w][threadIdx.x];
            sh.off[w][threadIdx.x] = run;
            run += v;
        }
    }
    __syncthreads();
    if (m == 0u) return;
    const int max_level = lv.max_level;
    const uint32_t lt = (1u << lane) - 1u, le = lt | (1u << lane);
    const int top = min(31 - __clz(m), max_level);
    for (int l = __ffs(m) - 1; l <= top; ++l) {
        if (!((m >> l) & 1u)) continue;
        const int x = lv.begin[l] + (int)sh.off[warp][l] + __popc(sh.bal[warp][l] & lt);
        int parent = -1;
        if (l > 0) {
            // the last node of level l - 1 starting at or before body i
            parent = lv.begin[l - 1] + (int)sh.off[warp][l - 1] + __popc(sh.bal[warp][l - 1] & le) - 1;
        }
        const bool splits = l + 1 <= max_level && ((m >> (l + 1)) & 1u);
        const int first_child =
            splits ? lv.begin[l + 1] + (int)sh.off[warp][l + 1] + __popc(sh.bal[warp][l + 1] & lt) : -1;
        nd.begin[x] = i;
        nd.level[x] = (uint8_t)l;
        nd.parent[x] = parent;
        nd.child[x] = first_child;
        if (!splits) {
            // a leaf: its bodies run to the next boundary below level l
            int cnt = lc;
            if (cnt == kLongLeaf || l != 31 - __clz(m)) {
                // a long run (equal keys, or a node the capacity kept from
                // splitting): the end of its level-l key prefix
                const int shift = B * (D - l);
                const uint64_t p = keys[i] >> shift;
                int lo = i + 1, hi = n;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if ((keys[mid] >> shift) == p)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                cnt = lo - i;
            }
            nd.count[x] = cnt;
            nd.nchild[x] = 0;
            nd.meta[x] = make_int4(x, -1, i, cnt);
        }
    }
}

__global__ void __launch_bounds__(kTreeBlock)
node_kernel(const uint64_t *__restrict__ keys, const uint8_t *__restrict__ leafcnt,
            const uint32_t *__restrict__ mask, const uint32_t *__restrict__ blk_off, int nblk,
            int n, int nchild, NodeArrays nd, const LevelInfo *__restrict__ lv,
            const uint32_t *__restrict__ flags)
{
    pdl_wait();
    if (sort_failed(flags)) return;
    __shared__ NodeShared<kTreeBlock> sh;
    __shared__ LevelInfo s_lv;
    if (threadIdx.x < kMaxLevels + 2) s_lv.begin[threadIdx.x] = lv->begin[threadIdx.x];
    if (threadIdx.x == 0) s_lv.max_level = lv->max_level;
    // (node_records synchronises before it reads the levels)
    const int i = blockIdx.x * kTreeBlock + threadIdx.x;
    node_records<kTreeBlock>(
        keys, i < n ? mask[i] : 0u, i < n ? leafcnt[i] : (uint8_t)0,
        [&](int l) { return blk_off[(size_t)l * nblk + blockIdx.x]; }, blockIdx.x, n, nchild, nd,
        s_lv, sh);
}

__device__ __forceinline__ uint32_t compact3(uint64_t x)
{
    x &= 0x1249249249249249ull;
    x = (x ^ (x >> 2)) & 0x10c30c30c30c30c3ull;
    x = (x ^ (x >> 4)) & 0x100f00f00f00f00full;
    x = (x ^ (x >> 8)) & 0x1f0000ff0000ffull;
    x = (x ^ (x >> 16)) & 0x1f00000000ffffull;
    x = (x ^ (x >> 32)) & 0x1fffffull;
    return (uint32_t)x;
}

__device__ __forceinline__ uint32_t compact2(uint64_t x)
{
    x &= 0x5555555555555555ull;
    x = (x | (x >> 1)) & 0x3333333333333333ull;
    x = (x | (x >> 2)) & 0x0f0f0f0f0f0f0f0full;
    x = (x | (x >> 4)) & 0x00ff00ff00ff00ffull;
    x = (x | (x >> 8)) & 0x0000ffff0000ffffull;
    x = (x | (x >> 16)) & 0x00000000ffffffffull;
    return (uint32_t)x;
}

// ---------------------------------------------------------------------------
// 5. cells: geometry, counts, mass, centre of mass and (optionally) second
//    moments of every node, one thread per node, all nodes at once
// ---------------------------------------------------------------------------
// Nothing is passed up the tree: a node's bodies are the range [begin, end) of
// the sorted order, and its sums are those of the O(log count) complete groups
// (Segments) that tile the range, with up to three bodies at either end.  The
// end of an internal node is its next sibling's begin, or its parent's end if it
// is the last child.  A bottom-up pass (each parent finished by its last child
// to arrive) took 37 us at 8,195 bodies, 45 at 1,048,580 (leaf 16) and 124 at
// 250,007 with one body per leaf: three dependent round trips to L2 per level of
// the tree, whatever the size, after a centre pass of 6, 12 and 70 (the f64
// chain of every centre).  This takes 9, 23 and 24 for both, and the group
// sums add 1, 3 and 5 to the boundary pass.
//
// Each product m x is taken exactly (TwoProduct by FMA) and summed as
// double-float (hi + lo f32) pairs -- FP32 arithmetic only, as GB300 issues f64
// instructions at a small fraction of its f32 rate.  The f32 centre of mass
// c = S / M is the double-float quotient rounded once.  A leaf whose bodies all
// sit at one position keeps that exact position, so a body there cancels
// against it as the reference's equal-centre skip does; a massless cell sits at
// its geometric centre.  Second moments (kQuad) are f32, combined with the
// parallel-axis rule S = sum [S_g + M_g (c_g - c)(c_g - c)^T] over the groups.
//
// Geometry: X (2q + 1 - 2^l) / 2^l from the cell index q, one f64 product per
// axis rounded to f32 (geo), and for the exact traversal (kExact) what that
// rounding dropped (geo_lo), within 2^-48 X of the reference's f64 centre; the
// traversal replays the reference's own centre arithmetic (cell_centre) only
// for the openings those bounds leave open.

// The reference's f64 centre and half-width of the level-l cell with key `key`
// (child = parent +- half-width / 2 per level, octree.rs:167-215,
// quadtree.rs:167-194).
__device__ __forceinline__ void cell_centre(uint64_t key, int l, int nchild, double X, double &cx,
                                            double &cy, double &cz, double &ext)
{
    const int D = tree_levels(nchild), B = level_bits(nchild);
    const uint32_t dmask = (uint32_t)nchild - 1u;
    cx = cy = cz = 0.0;
    ext = X;
    for (int j = 1; j <= l; ++j) {
        const uint32_t q = (uint32_t)(key >> (B * (D - j))) & dmask;
        const double h = __dmul_rn(ext, 0.5);  // ext / 2, exact
        cx = (q & 1) ? __dadd_rn(cx, h) : __dsub_rn(cx, h);
        cy = (q & 2) ? __dadd_rn(cy, h) : __dsub_rn(cy, h);
        if (nchild == 8) cz = (q & 4) ? __dadd_rn(cz, h) : __dsub_rn(cz, h);
        ext = h;
    }
}

// The centres of a tree snapshot: planes cx, cy, cz, half-width of m entries.
__global__ void snapshot_centre_kernel(const uint64_t *__restrict__ keys, NodeArrays nd, int m,
                                       int nchild,
                                       const unsigned long long *__restrict__ extent_bits,
                                       double *__restrict__ out)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= m) return;
    double c[4];
    cell_centre(keys[nd.begin[x]], nd.level[x], nchild,
                __longlong_as_double((long long)*extent_bits), c[0], c[1], c[2], c[3]);
    for (int p = 0; p < 4; ++p) out[(size_t)p * m + x] = c[p];
}

// The bodies [b, e) as pieces: at most three bodies before and three after the
// complete groups, and per level k of the groups the one at its lower end if
// that is odd and the one at its upper end if that is odd, where groups remain
// (lo(k) < hi(k)).
struct RangePieces {
    int b, lo, hi, head, bodies;  // `bodies` loose ones, `head` of them before
    __device__ __forceinline__ RangePieces(int begin, int end)
    {
        b = begin;
        lo = (begin + kSegBase - 1) / kSegBase;
        hi = end / kSegBase;
        if (lo < hi) {
            head = lo * kSegBase - begin;
            bodies = head + end - hi * kSegBase;
        } else {
            head = bodies = end - begin;
        }
    }
    __device__ __forceinline__ int body(int t) const
    {
        return t < head ? b + t : hi * kSegBase + t - head;
    }
    __device__ __forceinline__ int lo_at(int k) const { return (lo + (1 << k) - 1) >> k; }
    __device__ __forceinline__ int hi_at(int k) const { return hi >> k; }
};

// One lane per node, or eight: they share out the loose bodies and the groups'
// levels, so that all of a node's reads are in flight together, and add their
// sums by shuffles; the first three take an axis each for the geometry (f64) and
// the quotients.  cell_lanes picks.
template <bool kQuad, bool kExact, int kLanes>
__device__ __forceinline__ void cell_nodes(const uint64_t *__restrict__ keys,
                                           const float4 *sbody, const NodeArrays &nd, int total,
                                           int nchild, const Segments &sg,
                                           const unsigned long long *__restrict__ extent_bits)
{
    const int D = tree_levels(nchild), B = level_bits(nchild);
    const double X = __longlong_as_double((long long)*extent_bits);
    constexpr int kBatch = kLanes == 1 ? 3 : 1;  // loose bodies read at a time
    const int l = threadIdx.x & (kLanes - 1);  // lane of the node
    const unsigned full = 0xffffffffu;
    const int shift = (int)(threadIdx.x & 31) & ~(kLanes - 1);
    const int per_grid = gridDim.x * (blockDim.x / kLanes);
    const int first = (blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
    // (whole warps take part in the shuffles: the last turn repeats the last node)
    for (int x0 = first - (threadIdx.x & 31) / kLanes; x0 < total; x0 += per_grid) {
        const bool live = x0 + shift / kLanes < total;
        const int x = live ? x0 + shift / kLanes : total - 1;
        const int level = nd.level[x], b = nd.begin[x], fc = nd.child[x];
        const uint64_t key = keys[b];
        int e;
        if (fc < 0) {
            e = b + nd.count[x];
        } else {
            // siblings are consecutive: the next sibling's begin, or the parent's end
            int s = x, par = nd.parent[x];
            for (;;) {
                if (par < 0) {
                    e = sg.n;
                    break;
                }
                if (s + 1 < total && nd.parent[s + 1] == par) {
                    e = nd.begin[s + 1];
                    break;
                }
                s = par;
                par = nd.parent[s];
            }
        }
        // children: the nodes from fc on whose parent this is
        int nc = 0;
#pragma unroll
        for (int k = 0; k < 8; k += kLanes) {
            const bool mine = fc >= 0 && k + l < nchild && fc + k + l < total &&
                              nd.parent[fc + k + l] == x;
            if constexpr (kLanes == 1)
                nc += mine;
            else
                nc += __popc((__ballot_sync(full, mine) >> shift) & ((1u << kLanes) - 1u));
        }
        // moments
        const RangePieces pc(b, e);
        GroupSum g = group_zero();
        for (int t = l; t < pc.bodies; t += kLanes * kBatch) {
            float4 p[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) p[u] = sbody[pc.body(min(t + u, pc.bodies - 1))];
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                if (t + u < pc.bodies) df_add_body(g, p[u]);
        }
        for (int k = l; pc.lo_at(k) < pc.hi_at(k); k += kLanes) {
            const int lo = pc.lo_at(k), hi = pc.hi_at(k);
            GroupSum p = group_zero(), r = p;
            if (lo & 1) {
                p.h = sg.hi[sg.off[k] + lo];
                p.l = sg.lo[sg.off[k] + lo];
            }
            if (hi & 1) {
                r.h = sg.hi[sg.off[k] + hi - 1];
                r.l = sg.lo[sg.off[k] + hi - 1];
            }
            if (lo & 1) df_add4(g, p);
            if (hi & 1) df_add4(g, r);
        }
        __syncwarp();
#pragma unroll
        for (int o = 1; o < kLanes; o <<= 1) {
            GroupSum p;
            p.h = shfl_xor4(g.h, o);
            p.l = shfl_xor4(g.l, o);
            df_add4(g, p);
        }
        // geometry
        const uint64_t pre = level == 0 ? 0ull : key >> (B * (D - level));
        const double h = X * pow2d(-level);  // the half-width, exact
        const long long span = 1ll << level;
        auto axis = [&](int c) {
            const uint32_t q = nchild == 8 ? compact3(pre >> c) : compact2(pre >> c);
            return c == 2 && nchild != 8 ? 0.0 : h * (double)(2ll * q + 1 - span);
        };
        float4 geo, low = make_float4(0.f, 0.f, 0.f, 0.f);
        geo.w = (float)h;
        if constexpr (kLanes == 1) {
            const double dx = axis(0), dy = axis(1), dz = axis(2);
            geo.x = (float)dx;
            geo.y = (float)dy;
            geo.z = (float)dz;
            if (kExact)
                low = make_float4((float)(dx - (double)geo.x), (float)(dy - (double)geo.y),
                                  (float)(dz - (double)geo.z), 0.f);
        } else {  // an axis per lane
            const double d = axis(l < 3 ? l : 0);
            const float df = (float)d;
            geo.x = __shfl_sync(full, df, shift);
            geo.y = __shfl_sync(full, df, shift + 1);
            geo.z = __shfl_sync(full, df, shift + 2);
            if (kExact) {
                const float dl = (float)(d - (double)df);
                low = make_float4(__shfl_sync(full, dl, shift), __shfl_sync(full, dl, shift + 1),
                                  __shfl_sync(full, dl, shift + 2), 0.f);
            }
        }
        bool same = fc < 0;  // a leaf's bodies all at one position
        const float4 p0 = sbody[b];
        for (int j = b + 1; same && j < e; ++j) {
            const float4 p = sbody[j];
            same = p.x == p0.x && p.y == p0.y && p.z == p0.z;
        }
        __syncwarp();
        float4 com;
        if constexpr (kLanes == 1) {
            com = df_com(g.h, g.l, geo);
        } else {  // df_com, a quotient per lane
            const float qh = l == 1 ? g.h.z : l == 2 ? g.h.w : g.h.y;
            const float ql = l == 1 ? g.l.z : l == 2 ? g.l.w : g.l.y;
            const float quot = df_div(qh, ql, g.h.x, g.l.x);
            com = make_float4(__shfl_sync(full, quot, shift), __shfl_sync(full, quot, shift + 1),
                              __shfl_sync(full, quot, shift + 2), g.h.x + g.l.x);
            if (g.h.x == 0.f && g.l.x == 0.f) com = make_float4(geo.x, geo.y, geo.z, 0.f);
        }
        if (same) com = make_float4(p0.x, p0.y, p0.z, g.h.x + g.l.x);
        if (live && l == 0) {
            if (fc >= 0) {
                nd.count[x] = e - b;
                nd.nchild[x] = (uint8_t)nc;
                nd.meta[x] = make_int4(x | (nc << 28), fc, b, e - b);
            }
            nd.geo[x] = geo;
            if (kExact) nd.geo_lo[x] = low;
            nd.com[x] = com;
        }
        if (kQuad) {
            Quad6 q = {{0.f, 0.f, 0.f, 0.f, 0.f, 0.f}};
            if (!same) {
                for (int t = l; t < pc.bodies; t += kLanes)
                    quad_body_add(q, sbody[pc.body(t)], com);
                for (int k = l; pc.lo_at(k) < pc.hi_at(k); k += kLanes) {
                    const int lo = pc.lo_at(k), hi = pc.hi_at(k);
                    if (lo & 1) {
                        const float4 c = sg.com[sg.off[k] + lo];
                        quad_shift_add(q, quad_load(sg, sg.off[k] + lo), c.w, c.x - com.x,
                                       c.y - com.y, c.z - com.z);
                    }
                    if (hi & 1) {
                        const float4 c = sg.com[sg.off[k] + hi - 1];
                        quad_shift_add(q, quad_load(sg, sg.off[k] + hi - 1), c.w, c.x - com.x,
                                       c.y - com.y, c.z - com.z);
                    }
                }
            }
            __syncwarp();
#pragma unroll
            for (int o = 1; o < kLanes; o <<= 1)
#pragma unroll
                for (int c = 0; c < 6; ++c) q.v[c] += __shfl_xor_sync(full, q.v[c], o);
            if (live && l == 0) {
                nd.quad_a[x] = make_float4(q.v[0], q.v[1], q.v[2], q.v[0] + q.v[1] + q.v[2]);
                nd.quad_b[x] = make_float4(q.v[3], q.v[4], q.v[5], 0.f);
            }
        }
    }
}

template <bool kQuad, bool kExact, int kLanes>
__global__ void __launch_bounds__(256)
cell_kernel(const uint64_t *__restrict__ keys, const float4 *__restrict__ sbody, NodeArrays nd,
            const LevelInfo *__restrict__ lv, int nchild, Segments sg,
            const unsigned long long *__restrict__ extent_bits,
            const uint32_t *__restrict__ flags)
{
    pdl_wait();
    if (sort_failed(flags)) return;
    cell_nodes<kQuad, kExact, kLanes>(keys, sbody, nd, lv->total, nchild, sg, extent_bits);
}

// ---------------------------------------------------------------------------
// The tree of few bodies in one launch
// ---------------------------------------------------------------------------
// The five kernels above take 6 + 7 + 5 + 7 + 9 us for 8,195 bodies and hardly
// less for 300: their beginnings and ends and the round trips to L2 in each.
// Where an SM's block of kBuildBlock threads has no more than one tile of bodies,
// this takes the same stages in 23 us, with a grid barrier (1.2 us) between
// them: sorted bodies,
// group sums and level masks; node records (each block adds up the level counts
// of the tiles before its own, so there is no scan kernel, and the last block
// makes the top group sums); cells.  Masks and leaf counts stay in registers.
// What other blocks of the launch wrote is never read through the read-only
// cache.
constexpr int kBuildBlock = 512;

struct BuildArgs {
    GatherArgs gather;
    int leaf;
    uint32_t *blk_cnt;
    NodeArrays nd;
    LevelInfo *lv;
    const unsigned long long *extent_bits;
    uint32_t *bar;  // [0] barrier count, [1] blocks that left
    uint32_t *flags;
    int spin_limit, stall_tile;
    bool early;  // SMs are free for the next kernel's blocks
};

template <bool kQuad, bool kExact, int kLanes>
__global__ void __launch_bounds__(kBuildBlock, 1) tree_build_kernel(BuildArgs a)
{
    constexpr int kGather = kBuildBlock / kSegBase;  // threads of the gather
    constexpr int kGatherLevel = 7;                  // its last level of group sums
    static_assert(kSegBase << kGatherLevel == kBuildBlock, "a group of all the tile's bodies");
    __shared__ union {
        struct {
            GatherShared<kGather> gather;
            MaskShared<kBuildBlock> mask;
        } first;
        NodeShared<kBuildBlock> node;
    } sh;
    __shared__ uint32_t total_of[32], before_of[32];
    __shared__ LevelInfo lv;
    __shared__ int s_ok;
    if (threadIdx.x == 0) s_ok = !sort_failed(a.flags);
    __syncthreads();
    const int n = a.gather.n, nchild = a.gather.nchild;
    const uint64_t *keys = a.gather.keys;
    const int tiles = (n + kBuildBlock - 1) / kBuildBlock;  // at most gridDim.x
    const int tile = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t m = 0u;
    uint8_t lc = 0;
    bool ok = s_ok != 0;  // (else an earlier kernel gave up: there is no order to read)
    if (ok) {
        if (tile < tiles) {
            if (threadIdx.x < kGather)
                gather_groups<kQuad, kExact, kGather, true>(a.gather, tile * kGather,
                                                            sh.first.gather);
            level_masks<kBuildBlock>(
                keys, [&](int j) { return shared_digits(keys[j - 1], keys[j], nchild); }, tile, n,
                nchild, a.leaf, a.blk_cnt, tiles, sh.first.mask, m, lc);
        }
        // the test hook's block waits for a count that nothing reaches
        ok = grid_barrier(a.bar, a.flags, a.spin_limit,
                          (int)blockIdx.x == a.stall_tile ? kBarPoison : gridDim.x, &s_ok);
    }
    if (ok) {
        // the levels' totals and starts, the same in every block, and the nodes
        // of the tiles before this block's
        for (int l = warp; l < 32; l += kBuildBlock / 32) {
            uint32_t sum = 0, before = 0;
            for (int t = lane; t < tiles; t += 32) {
                const uint32_t v = __ldcg(&a.blk_cnt[(size_t)l * tiles + t]);
                sum += v;
                before += t < tile ? v : 0u;
            }
            sum = __reduce_add_sync(0xffffffffu, sum);
            before = __reduce_add_sync(0xffffffffu, before);
            if (lane == 0) {
                total_of[l] = sum;
                before_of[l] = before;
            }
        }
        __syncthreads();
        if (threadIdx.x < 32) level_starts(total_of, tree_levels(nchild), a.nd.cap, lv, a.flags);
        __syncthreads();
        if (blockIdx.x == 0 && threadIdx.x < sizeof lv / sizeof(int32_t))
            reinterpret_cast<int32_t *>(a.lv)[threadIdx.x] =
                reinterpret_cast<const int32_t *>(&lv)[threadIdx.x];
        if (tile < tiles)
            node_records<kBuildBlock>(
                keys, m, lc, [&](int l) { return before_of[l]; }, tile, n, nchild, a.nd, lv,
                sh.node);
        if (blockIdx.x == gridDim.x - 1)
            top_groups<kQuad, kBuildBlock>(a.gather.sg, kGatherLevel);
        ok = grid_barrier(a.bar, a.flags, a.spin_limit, 2u * gridDim.x, &s_ok);
    }
    // the traversal's blocks may come in beside the cells; with the counts it adds to
    // cleared by the sort instead of a memset between the two, and the integrator as
    // dependent launch after it, a step of 8,195 bodies takes 67.3 us instead of 74.1
    // (not where this grid holds every SM, 50,021 bodies with one per leaf 80.1
    // instead of 77.9 us)
    if (a.early) pdl_trigger();
    if (ok)
        cell_nodes<kQuad, kExact, kLanes>(keys, a.gather.sbody, a.nd, lv.total, nchild,
                                          a.gather.sg, a.extent_bits);
    leave_grid(a.bar);
}

// ---------------------------------------------------------------------------
// 6. traversal
// ---------------------------------------------------------------------------
struct TravArgs {
    NodeArrays nd;
    const float4 *sbody;
    const float4 *sbody_lo;      // f64 positions less their f32 values (exact traversal)
    const uint64_t *keys;
    int nchild;
    const double *bx, *by, *bz;  // the f64 state, unsorted (body order[k] is sorted body k)
    const uint32_t *order;
    const LevelInfo *lv;
    int n;
    float theta, e;
    double theta64;
    float extent;  // root half-width X (set on the device before the traversal)
    uint32_t *flags;
    double *partial;
    const unsigned long long *extent_bits;
    unsigned long long *stats;  // [0] node visits, [1] pair interactions (lanes)
    // accuracy options (not reference behaviour): quadrupole correction of
    // accepted cells, and a centre-of-mass guard that also requires
    // b_max < com_theta * |x - c| (b_max = sqrt(3) extent + |c - centre|
    // bounds the distance of the cell's bodies from c); 0 disables it.
    int quad;
    float com_theta;
    // pair-law scale (PairScale in engine.h), set on the device from the root
    // half-width X and the total mass M (the largest cell): bodies and cells
    // enter pair_acc / quad_acc at p 2^-sk with mass m 2^-skm, second moments
    // as S 2^-(2sk + skm), the easing as e 2^-2sk (es), and the sums leave
    // multiplied by 2^(skm - 2sk); opening tests use unscaled positions
    int sk, skm;
    float sc, msc, es;
};

__device__ __forceinline__ float load_extent(const TravArgs &a)
{
    return (float)__longlong_as_double((long long)*a.extent_bits);
}

__device__ __forceinline__ void set_pair_scale(TravArgs &a)
{
    a.sk = pair_scale_exp(a.extent, a.e);
    a.skm = mass_scale_exp(a.n > 0 ? a.nd.com[0].w : 0.f);  // root: the total mass
    a.sc = pow2f(-a.sk);
    a.msc = pow2f(-a.skm);
    a.es = a.e * pow2f(-2 * a.sk);
}

// (x, y, z, m) scaled by sc and msc
__device__ __forceinline__ float4 scaled(float4 p, float sc, float msc)
{
    return make_float4(p.x * sc, p.y * sc, p.z * sc, p.w * msc);
}

// second moments scaled by f = sc^2 msc
__device__ __forceinline__ float4 scaled2(float4 q, float f)
{
    return make_float4(q.x * f, q.y * f, q.z * f, q.w * f);
}

// The reference's opening rule `extent / r < theta` (octree.rs:137-144) in
// FP32, re-evaluated in f64 with the reference's arithmetic near the edge.
// ql / gl: what f32 dropped of the body's position and the cell's centre.
__device__ __forceinline__ bool accept_cell(const TravArgs &a, int node, float4 geo, float4 gl,
                                            float4 q, float4 ql, int k)
{
    const float dx = (q.x - geo.x) + (ql.x - gl.x);
    const float dy = (q.y - geo.y) + (ql.y - gl.y);
    const float dz = (q.z - geo.z) + (ql.z - gl.z);
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float inv = rsqrt_approx(r2);
    const float ratio = geo.w * inv;
    // Bound on the relative error of `ratio` against the reference's f64
    // value.  Each difference is the f64 one to a relative 3 * 2^-24 (the f32
    // difference rounds once, the sum with the dropped parts once) and to an
    // absolute 2^-45 X (the dropped parts round at 2^-24 of themselves, the
    // centre is within 2^-48 X of the reference's); the squares, rsqrt.approx
    // and the f32 extent add 4e-7.  Decisions inside twice that band are redone
    // in f64 with the reference's operations.  (From f32 positions alone the
    // band is 6.4e-7 X / r wide: at a cell of level 15 two percent of theta, so
    // most warps had a lane that took the f64 branch.)
    const float band = fabsf(a.theta) * (1e-13f * a.extent * inv + 1.5e-6f) + 1e-30f;
    if (fabsf(ratio - a.theta) > band && ratio == ratio && r2 > 1e-30f)
        return ratio < a.theta;
    const uint32_t i = a.order[k];
    double cx, cy, cz, ext;
    cell_centre(a.keys[a.nd.begin[node]], a.nd.level[node], a.nchild,
                __longlong_as_double((long long)*a.extent_bits), cx, cy, cz, ext);
    const double d0 = a.bx[i] - cx;
    const double d1 = a.by[i] - cy;
    const double d2 = a.bz[i] - cz;
    const double r64 = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
    return ext / r64 < a.theta64;
}

__device__ __forceinline__ void pair_acc(float qx, float qy, float qz, float4 b, float e,
                                         float &ax, float &ay, float &az)
{
    const float dx = b.x - qx, dy = b.y - qy, dz = b.z - qz;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    const float w = r2 + e;
    const float q = fmaf(r2, w * w, kPairGuard);
    const float s = b.w * rsqrt_approx(q);
    ax = fmaf(dx, s, ax);
    ay = fmaf(dy, s, ay);
    az = fmaf(dz, s, az);
}

// Quadrupole correction of a cell with centre of mass c and second moments S
// (about c) for the reference's law a = sum m d / (|d| (|d|^2 + e)):
// expanding d g(|d|), g(r) = 1/(r (r^2 + e)), to second order about c gives
//   a_2 = h S D + (h tr S + h' / r  D.S.D) D / 2,  D = c - x,
// h = g'(r)/r = -A / (r u^2), h'/r = (-6 + A (1/r^2 + 2 A / (u r))) / (r u^2),
// u = r (r^2 + e), A = 3 r^2 + e (e = 0 gives the Newtonian -3/r^5, 15/r^7).
__device__ __forceinline__ void quad_acc(float qx, float qy, float qz, float4 c, float4 qa,
                                         float4 qb, float e, float &ax, float &ay, float &az)
{
    const float dx = c.x - qx, dy = c.y - qy, dz = c.z - qz;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    if (!(r2 > 1e-30f)) return;
    const float ir = rsqrt_approx(r2);
    const float iu = ir * __fdividef(1.f, r2 + e);
    const float A = fmaf(3.f, r2, e);
    const float base = ir * iu * iu;
    const float h = -A * base;
    const float hp = base * fmaf(A, fmaf(2.f * A, iu * ir, ir * ir), -6.f);
    const float sdx = fmaf(qa.x, dx, fmaf(qb.x, dy, qb.y * dz));
    const float sdy = fmaf(qb.x, dx, fmaf(qa.y, dy, qb.z * dz));
    const float sdz = fmaf(qb.y, dx, fmaf(qb.z, dy, qa.z * dz));
    const float dsd = fmaf(dx, sdx, fmaf(dy, sdy, dz * sdz));
    const float k = 0.5f * fmaf(h, qa.w, hp * dsd);
    ax = fmaf(h, sdx, fmaf(k, dx, ax));
    ay = fmaf(h, sdy, fmaf(k, dy, ay));
    az = fmaf(h, sdz, fmaf(k, dz, az));
}

// Monopole + quadrupole terms of two accepted cells for one body (nq =
// -position), the cells' (x, y, z, m) and second moments given as float2
// planes, through packed FP32 instructions.  Per lane the monopole and the
// quadrupole share one reciprocal square root: 1/sqrt(r^2 (r^2 + e)^2) = 1/u
// and 1/r = (r^2 + e)/u; the quadrupole term is that of quad_acc.
__device__ __forceinline__ void cell_quad_acc2(float2 nqx, float2 nqy, float2 nqz, float2 cx,
                                               float2 cy, float2 cz, float2 cm, float2 qax,
                                               float2 qay, float2 qaz, float2 qaw, float2 qbx,
                                               float2 qby, float2 qbz, float2 e2, float2 &ax,
                                               float2 &ay, float2 &az)
{
    const float2 dx = add2(cx, nqx), dy = add2(cy, nqy), dz = add2(cz, nqz);
    float2 r2 = mul2(dz, dz);
    r2 = fma2(dy, dy, r2);
    r2 = fma2(dx, dx, r2);
    const float2 w = add2(r2, e2);
    const float2 arg = fma2(r2, mul2(w, w), make_float2(kPairGuard, kPairGuard));
    const float2 iu = make_float2(rsqrt_approx(arg.x), rsqrt_approx(arg.y));
    const float2 s = mul2(cm, iu);
    float2 ir = mul2(iu, w);
    ir.x = r2.x > 1e-30f ? ir.x : 0.f;  // no quadrupole term at r = 0
    ir.y = r2.y > 1e-30f ? ir.y : 0.f;
    const float2 A = fma2(make_float2(3.f, 3.f), r2, e2);
    const float2 base = mul2(mul2(ir, iu), iu);
    const float2 h = mul2(make_float2(-A.x, -A.y), base);
    const float2 hp =
        mul2(base, fma2(A, fma2(mul2(make_float2(2.f, 2.f), A), mul2(iu, ir), mul2(ir, ir)),
                        make_float2(-6.f, -6.f)));
    const float2 sdx = fma2(qax, dx, fma2(qbx, dy, mul2(qby, dz)));
    const float2 sdy = fma2(qbx, dx, fma2(qay, dy, mul2(qbz, dz)));
    const float2 sdz = fma2(qby, dx, fma2(qbz, dy, mul2(qaz, dz)));
    const float2 dsd = fma2(dx, sdx, fma2(dy, sdy, mul2(dz, sdz)));
    const float2 k = fma2(make_float2(0.5f, 0.5f), fma2(h, qaw, mul2(hp, dsd)), s);
    ax = fma2(h, sdx, fma2(k, dx, ax));
    ay = fma2(h, sdy, fma2(k, dy, ay));
    az = fma2(h, sdz, fma2(k, dz, az));
}

// The centre-of-mass guard for one body: b_max < com_theta |x - c|.
__device__ __forceinline__ bool com_guard(const TravArgs &a, float4 geo, float4 c, float qx,
                                          float qy, float qz)
{
    if (a.com_theta <= 0.f) return true;
    const float ox = c.x - geo.x, oy = c.y - geo.y, oz = c.z - geo.z;
    const float bmax = fmaf(1.7320509f, geo.w, sqrtf(fmaf(ox, ox, fmaf(oy, oy, oz * oz))));
    const float dx = c.x - qx, dy = c.y - qy, dz = c.z - qz;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    return bmax * bmax < a.com_theta * a.com_theta * r2;
}

// Two interactions of one body (nq = -position, both lanes) with sources
// (x, y, z, m) given as float2 planes, through packed FP32 instructions; the
// arithmetic of each lane is that of pair_acc.
__device__ __forceinline__ void pair_acc2(float2 nqx, float2 nqy, float2 nqz, float2 x, float2 y,
                                          float2 z, float2 m, float2 e2, float2 &ax, float2 &ay,
                                          float2 &az)
{
    const float2 dx = add2(x, nqx), dy = add2(y, nqy), dz = add2(z, nqz);
    float2 r2 = mul2(dz, dz);
    r2 = fma2(dy, dy, r2);
    r2 = fma2(dx, dx, r2);
    const float2 w = add2(r2, e2);
    const float2 q = fma2(r2, mul2(w, w), make_float2(kPairGuard, kPairGuard));
    const float2 s = mul2(m, make_float2(rsqrt_approx(q.x), rsqrt_approx(q.y)));
    ax = fma2(dx, s, ax);
    ay = fma2(dy, s, ay);
    az = fma2(dz, s, az);
}

__device__ __forceinline__ void fold(float &hi, float &lo, float &t)
{
    float s, err;
    two_sum(hi, t, s, err);
    hi = s;
    lo += err;
    t = 0.f;
}

// An opened cell: its children and the bodies that opened it.
struct StackEntry {
    int32_t first, count;
    uint32_t mask;
};

// A warp walks its 32 bodies' own lists together: a stack of opened cells, each
// with the mask of the bodies that opened it.  A turn takes up to 32 / nchild
// opened cells and reads all their children at once, one lane each (geometry,
// centre of mass, record), then tests child after child for the bodies of its
// parent's mask.  Nothing is read inside that: an opened leaf of one body is its
// own centre of mass, and the record of an opened cell goes on the stack.  (One
// cell per turn, with its record, its leaves' bodies and its centres read when
// they were needed, was three or four L2 round trips per cell: 71 us at 50,021
// bodies, theta 0.5.)
// As in the warp traversal a team of S warps walks for one group, sharing the
// stack: each warp takes its share of a turn's cells and keeps its opened ones
// aside until the team puts them on the stack, in warp order.
template <int S>
__global__ void __launch_bounds__(S * 32, S > 1 ? 24 / S : 24)
traverse_exact_kernel(TravArgs a_in)
{
    constexpr int kCap = S == 1 ? 320 : 192 * S;
    __shared__ StackEntry stack[kCap];
    __shared__ StackEntry aside[S > 1 ? S : 1][S > 1 ? 32 : 1];
    __shared__ int aside_count[S];
    __shared__ float4 child_geo[S][32];  // the children being tested
    __shared__ float4 child_lo[S][32];
    __shared__ float4 child_com[S][32];
    __shared__ int4 child_meta[S][32];
    pdl_wait();
    // a failed sort left no tree to walk (the node arrays may hold anything)
    if (sort_failed(a_in.flags)) return;
    TravArgs a = a_in;
    a.extent = load_extent(a_in);
    set_pair_scale(a);
    const float sc2 = a.sc * a.sc * a.msc;
    unsigned long long visits = 0, pairs = 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k0 = blockIdx.x * 32;
    const int k = k0 + lane;
    const bool valid = k < a.n;
    const uint32_t active = __ballot_sync(0xffffffffu, valid);
    const float4 q = valid ? a.sbody[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 ql = valid ? a.sbody_lo[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 qs = scaled(q, a.sc, a.msc);
    float ax = 0.f, ay = 0.f, az = 0.f, hx = 0.f, hy = 0.f, hz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
    int sp = 0;
    int put = 0;  // S > 1: cells kept aside this turn
    int since_fold = 0;
    bool overflow = false;
    // Tests cell `node` (geometry `geo`, record `meta`) for the lanes of
    // `mask`, each with the reference's own opening rule for its body:
    // accepted lanes take the cell's monopole (and quadrupole); the lanes that
    // open a leaf take its bodies here; an internal cell opened by any lane
    // goes on the stack with those lanes, to have its children tested.
    auto visit = [&](int node, uint32_t mask, float4 geo, float4 gl, float4 com, int4 meta) {
        const bool in = (mask >> lane) & 1u;
        bool acc = false;
        if (in) {
            acc = accept_cell(a, node, geo, gl, q, ql, k);
            if (acc && a.com_theta > 0.f) acc = com_guard(a, geo, com, q.x, q.y, q.z);
        }
        const uint32_t open = mask & ~__ballot_sync(0xffffffffu, acc);
        ++visits;
        if (acc) {
            const float4 cm = scaled(com, a.sc, a.msc);
            pair_acc(qs.x, qs.y, qs.z, cm, a.es, ax, ay, az);
            if (a.quad)
                quad_acc(qs.x, qs.y, qs.z, cm, scaled2(a.nd.quad_a[node], sc2),
                         scaled2(a.nd.quad_b[node], sc2), a.es, ax, ay, az);
            ++pairs;
        }
        ++since_fold;
        if (!open) return;
        if (meta.y < 0) {
            const int b = meta.z, c = meta.w;
            const bool mine = (open >> lane) & 1u;
            if (c == 1) {  // the leaf's body is its centre of mass
                if (mine) pair_acc(qs.x, qs.y, qs.z, scaled(com, a.sc, a.msc), a.es, ax, ay, az);
            } else {
                for (int j = b; j < b + c; ++j) {
                    const float4 bj = scaled(a.sbody[j], a.sc, a.msc);
                    if (mine) pair_acc(qs.x, qs.y, qs.z, bj, a.es, ax, ay, az);
                }
            }
            if (mine) pairs += c;
            since_fold += c;
        } else if (S > 1) {  // at most 32 per turn
            if (lane == 0)
                aside[warp][put] = {meta.y, (int32_t)((uint32_t)meta.x >> 28), open};
            ++put;
        } else if (sp < kCap) {
            if (lane == 0) stack[sp] = {meta.y, (int32_t)((uint32_t)meta.x >> 28), open};
            ++sp;
        } else {
            overflow = true;
        }
        if (since_fold >= 64) {
            fold(hx, lx, ax);
            fold(hy, ly, ay);
            fold(hz, lz, az);
            since_fold = 0;
        }
    };
    // the cells kept aside go on the stack, in warp order
    auto settle = [&]() {
        if (S == 1) return;
        if (lane == 0) aside_count[warp] = put;
        __syncthreads();  // also: every warp has taken its cells
        int at = sp, total = 0;
#pragma unroll
        for (int w = 0; w < S; ++w) {
            const int c = aside_count[w];
            if (w < warp) at += c;
            total += c;
        }
        if (sp + total > kCap)
            overflow = true;
        else if (lane < put)
            stack[at + lane] = aside[warp][lane];
        sp += total;
        put = 0;
        __syncthreads();
    };
    if (warp == 0)
        visit(0, active, a.nd.geo[0], a.nd.geo_lo[0], a.nd.com[0], a.nd.meta[0]);
    settle();
    const int slots = a.nchild;  // lanes per taken cell
    const int per_warp = 32 / slots;
    const int slot = lane / slots, which = lane - slot * slots;
    while (sp > 0 && !overflow) {
        // (one cell a turn where the stack is deep: each level then adds at most 7)
        const int m = sp > kCap - S * 32 - 7 * kMaxLevels ? 1 : min(S * per_warp, sp);
        __syncwarp();
        StackEntry mine = {0, 0, 0u};
        // dealt to the warps in turn
        const int take = slot * S + warp;
        if (slot < per_warp && take < m) mine = stack[sp - 1 - take];
        sp -= m;
        if (which < mine.count) {
            const int x = mine.first + which;
            child_geo[warp][lane] = a.nd.geo[x];
            child_lo[warp][lane] = a.nd.geo_lo[x];
            child_com[warp][lane] = a.nd.com[x];
            child_meta[warp][lane] = a.nd.meta[x];
        }
        __syncwarp();  // also: every lane has read the stack
#pragma unroll 1
        for (uint32_t todo = __ballot_sync(0xffffffffu, which < mine.count); todo;
             todo &= todo - 1u) {
            const int l = __ffs(todo) - 1;
            visit(__shfl_sync(0xffffffffu, mine.first + which, l),
                  __shfl_sync(0xffffffffu, mine.mask, l), child_geo[warp][l], child_lo[warp][l],
                  child_com[warp][l], child_meta[warp][l]);
        }
        settle();
    }
    if (overflow && lane == 0) atomicOr(&a.flags[kFlagStack], 1u);
    fold(hx, lx, ax);
    fold(hy, ly, ay);
    fold(hz, lz, az);
    for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    if (lane == 0) {
        atomicAdd(&a.stats[0], visits);
        atomicAdd(&a.stats[1], pairs);
    }
    if (S > 1) {
        // the warps' sums, added in warp order (child_geo is free)
        __syncthreads();
        float *part = reinterpret_cast<float *>(&child_geo[0][0]);  // [S][3][32], then lows
        float *low = reinterpret_cast<float *>(&child_com[0][0]);
        part[(warp * 3 + 0) * 32 + lane] = hx;
        part[(warp * 3 + 1) * 32 + lane] = hy;
        part[(warp * 3 + 2) * 32 + lane] = hz;
        low[(warp * 3 + 0) * 32 + lane] = lx;
        low[(warp * 3 + 1) * 32 + lane] = ly;
        low[(warp * 3 + 2) * 32 + lane] = lz;
        __syncthreads();
        if (warp > 0) return;
        for (int w = 1; w < S; ++w) {
            const int o = w * 3 * 32 + lane;
            float sum, err;
            two_sum(hx, part[o], sum, err);
            hx = sum;
            lx += err + low[o];
            two_sum(hy, part[o + 32], sum, err);
            hy = sum;
            ly += err + low[o + 32];
            two_sum(hz, part[o + 64], sum, err);
            hz = sum;
            lz += err + low[o + 64];
        }
    }
    if (valid) {
        const uint32_t i = a.order[k];
        const double unsc = pow2d(a.skm - 2 * a.sk);
        a.partial[i] = ((double)hx + (double)lx) * unsc;
        a.partial[a.n + i] = ((double)hy + (double)ly) * unsc;
        a.partial[2 * (size_t)a.n + i] = ((double)hz + (double)lz) * unsc;
    }
}

// Warp traversal: the 32 bodies of a group (consecutive in Morton order) walk
// the tree together, and the lanes work on different cells.  Each round takes
// pending cells from the top of a shared stack, one per lane, and tests each
// against the group's bounding box: a cell is accepted when
//     extent * (1 + 2e-6) < theta * (r_min - 6e-7 X),
// r_min = distance from the cell centre to the box.  Every body of the group
// is at least r_min (less f32 rounding of positions and centres, <= 2.1e-7 X)
// from the centre, so an accepted cell passes every body's own f64 reference
// test extent / r < theta; cells that some body would open are opened.
// Accepted cells and the bodies of opened leaves are queued (>= 0 body,
// < 0 cell) and gathered 32 at a time into shared memory, where all lanes
// evaluate them against their own body.
//
// A group is walked by a team of S warps: S x 32 lanes share the stack, the
// queue and the rounds, and the queued tiles of 32 are dealt to the warps in
// turn (so the sums do not depend on timing).  One warp per group is the least
// work, but its walk is a chain of 15 to 60 rounds of L2 latency, 50 us at
// 8,195 bodies and 540 at 100,003 with quadrupoles, with 2 to 20 warps an SM to
// hide it; bh_team picks S.  A block is one team, so a warp's slot is free again
// when its own walk ends (four groups to a block kept 22.8 of 28 warps running,
// one 24.2).
//
// At 1,048,580 bodies and theta 0.5 the kernel is bound by instruction issue
// (72%; FMA pipe 56%), half of it the walk's bookkeeping: 13 rounds and 334 cells
// per group, 532 interactions per body.  397M -> 343M warp instructions and 472
// -> 405 us came from testing squared distances, the sample bodies, the unrolled
// pushes and four packed pairs in flight.
constexpr int kTeamTake(int S) { return S == 1 ? 16 : 8; }  // bodies a lane queues at a time
template <int S>
struct TeamSize {
    static constexpr int kLanes = 32 * S;                      // a block is a team
    static constexpr int kStackCap = S == 1 ? 1024 : 512 * S;  // pending cells
    // above this, pop one cell at a time (each level then adds at most 7)
    static constexpr int kWide = kStackCap - 8 * kLanes - 8 * 22;
    static constexpr int kFlush = S == 1 ? 256 : 128 * S;      // queued before evaluating
    static constexpr int kQueue = S == 1 ? 640 : kFlush + kLanes * kTeamTake(S);
    static_assert(kWide > 0, "a full round fits");
};
constexpr int kSamples = 4;  // bodies a rejected cell is tried against before all of them

__device__ __forceinline__ int warp_exclusive_scan(int v, int lane, int &total)
{
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += t;
    }
    total = __shfl_sync(0xffffffffu, x, 31);
    return x - v;
}

// kQuad: quadrupole corrections of accepted cells (the quadrupole tiles are
// only sized in that instantiation, so the monopole kernel keeps its
// registers and occupancy).
// kGuard: the centre-of-mass guard may be on.  Its cells' centres are then read
// with the cells, so neither the samples nor the per-body test below goes back to
// memory (a broadcast load per asked cell was most of the quadrupole walk: 260
// cells per group at 100,003 bodies).
template <bool kQuad, bool kGuard, int S>
__global__ void __launch_bounds__(S * 32, S > 1 ? (kGuard ? 6 : 7) : (kGuard ? 24 : 28))
traverse_warp_kernel(TravArgs a_in)
{
    using T = TeamSize<S>;
    __shared__ int32_t stack[T::kStackCap];
    __shared__ int32_t queue[T::kQueue];
    __shared__ float4 tile[S][32];
    __shared__ float4 tqa[kQuad ? S : 1][32];
    __shared__ float4 tqb[kQuad ? S : 1][32];
    __shared__ float4 sample_xy[kSamples / 2];  // negated (x, x', y, y')
    __shared__ float2 sample_z[kSamples / 2];
    __shared__ int warp_total[2][S];
    pdl_wait();
    // a failed sort left no tree to walk (the node arrays may hold anything)
    if (sort_failed(a_in.flags)) return;
    TravArgs a = a_in;
    a.extent = load_extent(a_in);
    set_pair_scale(a);
    const float sc = a.sc, msc = a.msc, sc2 = a.sc * a.sc * a.msc;
    const int tw = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tl = threadIdx.x;  // lane within the team
    const int k0 = blockIdx.x * 32;
    auto team_sync = [&]() {
        if (S == 1)
            __syncwarp();
        else
            __syncthreads();
    };
    int scans = 0;
    // exclusive scan over the team's lanes (S > 1: also a barrier of the team)
    auto team_scan = [&](int v, int &total) {
        int x = warp_exclusive_scan(v, lane, total);
        if (S > 1) {
            int *wt = warp_total[scans++ & 1];
            if (lane == 0) wt[tw] = total;
            __syncthreads();
            total = 0;
#pragma unroll
            for (int w = 0; w < S; ++w) {
                const int t = wt[w];
                if (w < tw) x += t;
                total += t;
            }
        }
        return x;
    };
    const int k = k0 + lane;
    const bool valid = k < a.n;
    const int nvalid = __popc(__ballot_sync(0xffffffffu, valid));
    const float4 q = valid ? a.sbody[k] : a.sbody[k0];
    float lo_x = q.x, hi_x = q.x, lo_y = q.y, hi_y = q.y, lo_z = q.z, hi_z = q.z;
    for (int o = 16; o > 0; o >>= 1) {
        lo_x = fminf(lo_x, __shfl_xor_sync(0xffffffffu, lo_x, o));
        hi_x = fmaxf(hi_x, __shfl_xor_sync(0xffffffffu, hi_x, o));
        lo_y = fminf(lo_y, __shfl_xor_sync(0xffffffffu, lo_y, o));
        hi_y = fmaxf(hi_y, __shfl_xor_sync(0xffffffffu, hi_y, o));
        lo_z = fminf(lo_z, __shfl_xor_sync(0xffffffffu, lo_z, o));
        hi_z = fmaxf(hi_z, __shfl_xor_sync(0xffffffffu, hi_z, o));
    }
    // largest coordinate magnitude in the box: bounds the f32 rounding of the
    // group's positions
    const float bmax = fmaxf(fmaxf(fmaxf(fabsf(lo_x), fabsf(hi_x)), fmaxf(fabsf(lo_y), fabsf(hi_y))),
                             fmaxf(fabsf(lo_z), fabsf(hi_z)));
    const float pmax = fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fabsf(q.z));
    const float theta = a.theta;
    const float need = (1.f + 2.5e-6f) / theta;
    const float ct2 = a.com_theta * a.com_theta;
    if (tw == 0) {
        // four bodies spread over the group
#pragma unroll
        for (int u = 0; u < kSamples; ++u)
            if (lane == u * 31 / (kSamples - 1)) {
                float *xy = reinterpret_cast<float *>(&sample_xy[u >> 1]) + (u & 1);
                xy[0] = -q.x;
                xy[2] = -q.y;
                reinterpret_cast<float *>(&sample_z[u >> 1])[u & 1] = -q.z;
            }
    }
    float ax = 0.f, ay = 0.f, az = 0.f, hx = 0.f, hy = 0.f, hz = 0.f, lx = 0.f, ly = 0.f, lz = 0.f;
    unsigned long long visits = 0, pairs = 0;
    int nq = 0;
    int sp = 1;
    // The root is opened by every body when theta sqrt(3) < 1: no body is
    // further than sqrt(3) X from its centre.
    {
        const int4 root = a.nd.meta[0];
        if (root.y >= 0 && theta > 0.f && theta * 1.7320515f < 1.f) {
            sp = (int)((uint32_t)root.x >> 28);
            visits = 1;
            if (tl < sp) stack[tl] = root.y + tl;
        } else if (tl == 0) {
            stack[0] = 0;
        }
    }
    team_sync();
    // Bodies are queued from the front of the queue, accepted cells from the
    // back, so each is evaluated by its own loop: plain pairs for bodies,
    // pair + quadrupole (kQuad) for cells.
    int nc = 0;  // queued cells
    const float2 nqx = make_float2(-q.x * sc, -q.x * sc), nqy = make_float2(-q.y * sc, -q.y * sc);
    const float2 nqz = make_float2(-q.z * sc, -q.z * sc), e2 = make_float2(a.es, a.es);
    // Evaluates this warp's tiles of `count` queued interactions whose (x, y, z,
    // m) load(t) gives: entries 2k and 2k + 1 are staged interleaved as (x, x',
    // y, y')(z, z', m, m'), so two 128-bit loads give the float2 operands of two
    // interactions, which go through packed FADD2/FMUL2/FFMA2 (a tile is padded
    // to a multiple of eight with massless entries, which add exactly zero, so
    // four pairs are in flight at a time); the next tile is loaded while the
    // current one is evaluated.
    auto eval_packed = [&](int count, auto load) {
        float4 nb = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tw * 32 + lane < count) nb = load(tw * 32 + lane);
        for (int j0 = tw * 32; j0 < count; j0 += T::kLanes) {
            const int m = min(32, count - j0);
            __syncwarp();
            const float4 bj = nb;
            nb = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j0 + T::kLanes + lane < count) nb = load(j0 + T::kLanes + lane);
            float *pl = reinterpret_cast<float *>(&tile[tw][lane & ~1]) + (lane & 1);
            pl[0] = bj.x * sc;
            pl[2] = bj.y * sc;
            pl[4] = bj.z * sc;
            pl[6] = bj.w * msc;
            __syncwarp();
            float2 sx = make_float2(0.f, 0.f), sy = sx, sz = sx;
            for (int jj = 0; jj < m; jj += 8) {
#pragma unroll
                for (int u = 0; u < 8; u += 2) {
                    const float4 A = tile[tw][jj + u], B = tile[tw][jj + u + 1];
                    pair_acc2(nqx, nqy, nqz, make_float2(A.x, A.y), make_float2(A.z, A.w),
                              make_float2(B.x, B.y), make_float2(B.z, B.w), e2, sx, sy, sz);
                }
            }
            ax += sx.x + sx.y;
            ay += sy.x + sy.y;
            az += sz.x + sz.y;
        }
    };
    auto flush = [&]() {
        team_sync();  // every lane's queue entries
        // leaf bodies, then accepted cells (monopoles packed like bodies;
        // with quadrupoles one cell per lane step)
        eval_packed(nq, [&](int t) { return a.sbody[queue[t]]; });
        if (!kQuad) {
            eval_packed(nc, [&](int t) { return a.nd.com[-queue[T::kQueue - 1 - t] - 1]; });
        } else {
            // cells with quadrupoles, two per packed instruction: centre of
            // mass and both moment vectors staged interleaved like bodies
            for (int j0 = tw * 32; j0 < nc; j0 += T::kLanes) {
                const int m = min(32, nc - j0);
                __syncwarp();
                float4 c4 = make_float4(0.f, 0.f, 0.f, 0.f), qa = c4, qb = c4;
                if (lane < m) {
                    const int c = -queue[T::kQueue - 1 - (j0 + lane)] - 1;
                    c4 = scaled(a.nd.com[c], sc, msc);
                    qa = scaled2(a.nd.quad_a[c], sc2);
                    qb = scaled2(a.nd.quad_b[c], sc2);
                }
                const int slot = lane & ~1, half = lane & 1;
                float *pc = reinterpret_cast<float *>(&tile[tw][slot]) + half;
                float *pa = reinterpret_cast<float *>(&tqa[tw][slot]) + half;
                float *pb = reinterpret_cast<float *>(&tqb[tw][slot]) + half;
                pc[0] = c4.x; pc[2] = c4.y; pc[4] = c4.z; pc[6] = c4.w;
                pa[0] = qa.x; pa[2] = qa.y; pa[4] = qa.z; pa[6] = qa.w;
                pb[0] = qb.x; pb[2] = qb.y; pb[4] = qb.z; pb[6] = qb.w;
                __syncwarp();
                float2 sx = make_float2(0.f, 0.f), sy = sx, sz = sx;
                for (int jj = 0; jj < (m + 1) >> 1; ++jj) {
                    const float4 C0 = tile[tw][2 * jj], C1 = tile[tw][2 * jj + 1];
                    const float4 A0 = tqa[tw][2 * jj], A1 = tqa[tw][2 * jj + 1];
                    const float4 B0 = tqb[tw][2 * jj], B1 = tqb[tw][2 * jj + 1];
                    cell_quad_acc2(nqx, nqy, nqz, make_float2(C0.x, C0.y), make_float2(C0.z, C0.w),
                                   make_float2(C1.x, C1.y), make_float2(C1.z, C1.w),
                                   make_float2(A0.x, A0.y), make_float2(A0.z, A0.w),
                                   make_float2(A1.x, A1.y), make_float2(A1.z, A1.w),
                                   make_float2(B0.x, B0.y), make_float2(B0.z, B0.w),
                                   make_float2(B1.x, B1.y), e2, sx, sy, sz);
                }
                ax += sx.x + sx.y;
                ay += sy.x + sy.y;
                az += sz.x + sz.y;
            }
        }
        pairs += nq + nc;
        fold(hx, lx, ax);
        fold(hy, ly, ay);
        fold(hz, lz, az);
        nq = 0;
        nc = 0;
        team_sync();  // the queue is free again
    };
    bool overflow = false;
    while (sp > 0) {
        const int m = sp > T::kWide ? 1 : min(T::kLanes, sp);
        int cell = 0;
        if (tl < m) cell = stack[sp - m + tl];
        if (S == 1) __syncwarp();  // (S > 1: the scan below is a barrier)
        sp -= m;
        visits += m;
        int qref = 0, qcnt = 0, nchild = 0, first_child = 0;
        float4 geo = make_float4(0.f, 0.f, 0.f, 0.f);
        float cx = 0.f, cy = 0.f, cz = 0.f, bm2 = 0.f;  // kGuard: centre of mass, b_max^2
        bool acc = false, maybe = false;
        if (tl < m) {
            geo = a.nd.geo[cell];
            const int4 meta = a.nd.meta[cell];
            if (kGuard && ct2 > 0.f) {
                const float4 cm = a.nd.com[cell];
                cx = cm.x;
                cy = cm.y;
                cz = cm.z;
                const float ox = cx - geo.x, oy = cy - geo.y, oz = cz - geo.z;
                const float bm =
                    fmaf(1.7320509f, geo.w, sqrtf(fmaf(ox, ox, fmaf(oy, oy, oz * oz))));
                bm2 = bm * bm;
            }
            const float cmax = fmaxf(fmaxf(fabsf(geo.x), fabsf(geo.y)), fabsf(geo.z));
            const float dx = fmaxf(fmaxf(lo_x - geo.x, geo.x - hi_x), 0.f);
            const float dy = fmaxf(fmaxf(lo_y - geo.y, geo.y - hi_y), 0.f);
            const float dz = fmaxf(fmaxf(lo_z - geo.z, geo.z - hi_z), 0.f);
            // f32 rounding of positions and centre moves r by at most
            // 1.1e-7 (|p| + |c|) + 3.5e-7 r against the reference's f64 value:
            // rmin = r - (2e-7 (bmax + cmax) + 5e-7 r) must exceed extent (1 + 2e-6) /
            // theta.  Squared, for a root less; what is as near as the rounding of
            // the squares (1e-6, one cell in a million) is decided by rmin itself.
            const float t = fmaf(geo.w, need, 2.000001e-7f * (bmax + cmax));
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz)), t2 = t * t;
            acc = theta > 0.f && r2 > t2;
            if (fabsf(r2 - t2) <= 1e-6f * t2) {
                const float r = sqrtf(r2);
                const float rmin = r - (2e-7f * (bmax + cmax) + 5e-7f * r);
                acc = theta > 0.f && rmin > 0.f && geo.w * (1.f + 2e-6f) < theta * rmin;
            }
            if (kGuard && acc && ct2 > 0.f) {
                // centre-of-mass guard against the whole box (distance from c
                // to the box is a lower bound of every body's |x - c|)
                const float ex = fmaxf(fmaxf(lo_x - cx, cx - hi_x), 0.f);
                const float ey = fmaxf(fmaxf(lo_y - cy, cy - hi_y), 0.f);
                const float ez = fmaxf(fmaxf(lo_z - cz, cz - hi_z), 0.f);
                acc = bm2 < ct2 * fmaf(ex, ex, fmaf(ey, ey, ez * ez));
            }
            if (acc) {
                qref = -cell - 1;
                qcnt = 1;
            } else if (meta.y < 0) {
                qref = meta.z;  // first body of the leaf
                qcnt = meta.w;
            } else {
                nchild = (int)((uint32_t)meta.x >> 28);
                first_child = meta.y;
                maybe = theta > 0.f;
            }
        }
        // Internal cells the box test rejects: accept them if every body of
        // the group passes its own test (with the same rounding margin).  Most
        // fail for some of four sample bodies, by more than the margin (r theta
        // <= extent, f32 rounding under 2e-6), and are opened without asking
        // the rest: of 60 such cells per group at theta 0.5, 1M bodies, 42 are
        // opened, each asked of every body by four shuffles and a vote.
        if (__any_sync(0xffffffffu, maybe)) {
            const float t2 = theta * theta, w2 = geo.w * geo.w;
#pragma unroll
            for (int u = 0; u < kSamples / 2; ++u) {
                const float4 xy = sample_xy[u];
                const float2 dx = add2(make_float2(xy.x, xy.y), make_float2(geo.x, geo.x));
                const float2 dy = add2(make_float2(xy.z, xy.w), make_float2(geo.y, geo.y));
                const float2 dz = add2(sample_z[u], make_float2(geo.z, geo.z));
                const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
                maybe = maybe && !(t2 * r2.x <= w2) && !(t2 * r2.y <= w2);
                if (kGuard && ct2 > 0.f) {
                    const float2 ex = add2(make_float2(xy.x, xy.y), make_float2(cx, cx));
                    const float2 ey = add2(make_float2(xy.z, xy.w), make_float2(cy, cy));
                    const float2 ez = add2(sample_z[u], make_float2(cz, cz));
                    const float2 c2 = fma2(ex, ex, fma2(ey, ey, mul2(ez, ez)));
                    maybe = maybe && bm2 < ct2 * c2.x && bm2 < ct2 * c2.y;
                }
            }
        }
        uint32_t pend = __ballot_sync(0xffffffffu, maybe);
        while (pend) {
            const int src = __ffs(pend) - 1;
            pend &= pend - 1;
            const float gx = __shfl_sync(0xffffffffu, geo.x, src);
            const float gy = __shfl_sync(0xffffffffu, geo.y, src);
            const float gz = __shfl_sync(0xffffffffu, geo.z, src);
            const float gw = __shfl_sync(0xffffffffu, geo.w, src);
            const float ddx = q.x - gx, ddy = q.y - gy, ddz = q.z - gz;
            const float r2 = fmaf(ddx, ddx, fmaf(ddy, ddy, ddz * ddz));
            const float r = r2 * rsqrt_approx(r2);
            const float cm = fmaxf(fmaxf(fabsf(gx), fabsf(gy)), fabsf(gz));
            const float rl = r - (2e-7f * (pmax + cm) + 5e-7f * r);
            bool ok = !valid || (rl > 0.f && gw * (1.f + 2e-6f) < theta * rl);
            if (kGuard && ct2 > 0.f) {
                // com_guard for this body
                const float ex = __shfl_sync(0xffffffffu, cx, src) - q.x;
                const float ey = __shfl_sync(0xffffffffu, cy, src) - q.y;
                const float ez = __shfl_sync(0xffffffffu, cz, src) - q.z;
                const float b2 = __shfl_sync(0xffffffffu, bm2, src);
                ok = ok && (!valid || b2 < ct2 * fmaf(ex, ex, fmaf(ey, ey, ez * ez)));
            }
            if (__all_sync(0xffffffffu, ok) && lane == src) {
                qref = -cell - 1;
                qcnt = 1;
                nchild = 0;
            }
        }
        // push the children of opened cells, queue the accepted ones (back)
        const bool is_cell = qref < 0;
        int total;
        const int off = team_scan(nchild | (is_cell ? 1 << 16 : 0), total);
        const int kids = total & 0xffff, cells = total >> 16;
        if (sp + kids > T::kStackCap) {
            overflow = true;
            break;
        }
#pragma unroll
        for (int c = 0; c < 8; ++c)
            if (c < nchild) stack[sp + (off & 0xffff) + c] = first_child + c;
        sp += kids;
        if (nq + nc + cells > T::kQueue) flush();
        if (is_cell) {
            queue[T::kQueue - 1 - (nc + (off >> 16))] = qref;
            qcnt = 0;
        }
        nc += cells;
        // queue leaf bodies (front), a bounded number per lane and turn
        for (bool more = S > 1 || __any_sync(0xffffffffu, qcnt > 0); more;) {
            const int take = min(qcnt, kTeamTake(S));
            int btotal;
            const int boff = team_scan(take | (qcnt > take ? 1 << 16 : 0), btotal) & 0xffff;
            more = btotal >> 16;
            btotal &= 0xffff;
            if (nq + nc + btotal > T::kQueue) flush();
            for (int j = 0; j < take; j += 4) {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (j + u < take) queue[nq + boff + j + u] = qref + j + u;
            }
            qref += take;
            qcnt -= take;
            nq += btotal;
        }
        team_sync();  // the pushed cells
        if (nq + nc >= T::kFlush) flush();
    }
    flush();
    if (tl == 0) {
        if (overflow) atomicOr(&a.flags[kFlagStack], 1u);
        atomicAdd(&a.stats[0], visits);
        atomicAdd(&a.stats[1], pairs * (unsigned long long)nvalid);
    }
    if (S > 1) {
        // the warps' sums, added in warp order (the stack is free: flush was a barrier)
        float *part = reinterpret_cast<float *>(stack);
        const float v[6] = {hx, hy, hz, lx, ly, lz};
#pragma unroll
        for (int c = 0; c < 6; ++c) part[(tw * 6 + c) * 32 + lane] = v[c];
        __syncthreads();
        if (tw > 0) return;
        for (int w = 1; w < S; ++w) {
            const float *o = part + w * 6 * 32 + lane;
            float s, err;
            two_sum(hx, o[0], s, err);
            hx = s;
            lx += err + o[3 * 32];
            two_sum(hy, o[32], s, err);
            hy = s;
            ly += err + o[4 * 32];
            two_sum(hz, o[2 * 32], s, err);
            hz = s;
            lz += err + o[5 * 32];
        }
    }
    if (valid) {
        const uint32_t i = a.order[k];
        const double unsc = pow2d(a.skm - 2 * a.sk);
        a.partial[i] = ((double)hx + (double)lx) * unsc;
        a.partial[a.n + i] = ((double)hy + (double)ly) * unsc;
        a.partial[2 * (size_t)a.n + i] = ((double)hz + (double)lz) * unsc;
    }
}

inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

}  // namespace

// ---------------------------------------------------------------------------
// workspace + host driver
// ---------------------------------------------------------------------------
namespace {
// per device: the sort's kernel attributes are set, and how many blocks of the
// single-launch sort an SM holds (0 = one launch per pass)
std::atomic<bool> g_sort_ready[64];
std::atomic<int> g_sort_coop_per_sm[64];

constexpr int kTreeSortItems[] = {1, 2, 4, 6, 8, 10, 12, 14, 16};

const void *tree_sort_fn(int items)
{
    switch (items) {
    case 1: return (const void *)tree_sort_kernel<1>;
    case 2: return (const void *)tree_sort_kernel<2>;
    case 4: return (const void *)tree_sort_kernel<4>;
    case 6: return (const void *)tree_sort_kernel<6>;
    case 8: return (const void *)tree_sort_kernel<8>;
    case 10: return (const void *)tree_sort_kernel<10>;
    case 12: return (const void *)tree_sort_kernel<12>;
    case 14: return (const void *)tree_sort_kernel<14>;
    default: return (const void *)tree_sort_kernel<16>;
    }
}

size_t tree_sort_smem(int items)
{
    // the staged tile; its runs are placed with kFixRun keys either side
    return (size_t)kSortThreads * items * (sizeof(uint64_t) + sizeof(uint32_t)) +
           2 * kFixRun * sizeof(uint64_t);
}

size_t rank_sort_smem(int n)
{
    // all keys; the tile's two buffers of keys and places before them
    const size_t keys = (size_t)cdiv(n, kRankTile) * kRankTile * sizeof(uint64_t);
    return std::max(keys, (size_t)2 * kRankTile * (sizeof(uint64_t) + sizeof(uint32_t)));
}

int tree_sort_attributes()
{
    PG_CUDA(cudaFuncSetAttribute((const void *)rank_sort_kernel,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)rank_sort_smem(kRankMax)));
    for (int items : kTreeSortItems)
        PG_CUDA(cudaFuncSetAttribute(tree_sort_fn(items),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)tree_sort_smem(items)));
    return PHYSIM_OK;
}

// Keys per thread of the resident sort of n bodies: the fewest that give
// every tile a block of its own on `blocks` resident blocks (0: none does).
int resident_items(size_t n, int blocks)
{
    for (int items : kTreeSortItems)
        if (((n + (size_t)kSortThreads * items - 1) / ((size_t)kSortThreads * items)) <=
            (size_t)blocks)
            return items;
    return 0;
}

// Tiles that the resident sort of up to n bodies can need.
int resident_tiles(size_t n, int blocks)
{
    return (int)std::min<size_t>((n + kSortThreads - 1) / kSortThreads, (size_t)blocks);
}
}  // namespace

struct BhWorkspace {
    int device = 0;
    cudaStream_t stream = nullptr;  // allocations and frees are ordered on it
    size_t cap_n = 0;
    uint64_t *keys[2] = {nullptr, nullptr};
    uint32_t *vals[2] = {nullptr, nullptr};
    // sort_meta: digit histograms of the passes, then the passes' tile
    // counters, the epoch and the single-launch sort's grid barrier;
    // sort_status: look-back words, tiles x digits
    uint32_t *sort_meta = nullptr;
    unsigned long long *sort_status = nullptr;
    // the resident sort: tiles' digit counts, their groups' counts (two
    // halves), blocks' extents, and barrier words
    uint32_t *tile_cnt = nullptr, *tile_grp = nullptr, *tree_bar = nullptr;
    unsigned long long *blockmax = nullptr;
    float4 *sbody = nullptr;
    uint8_t *lcp = nullptr;        // L(k): leading digits keys[k-1] and keys[k] share
    uint32_t *mask = nullptr;      // level mask of each sorted body
    uint8_t *leafcnt = nullptr;    // bodies of the leaf starting at each sorted body
    uint32_t *blk_cnt = nullptr;   // per level and tree block: nodes starting in it
    uint32_t *blk_off = nullptr;   // ... and the level's nodes before the block
    float4 *sbody_lo = nullptr;    // what f32 dropped of the sorted positions
    Segments sg = {};              // group sums (n and off are set per build)
    NodeArrays nd = {};
    LevelInfo *lv = nullptr;
    unsigned long long *extent_bits = nullptr;
    unsigned long long *stats = nullptr;  // node visits, pair interactions of the last traversal
    uint32_t *flags = nullptr;
    int launches = 0;
    // which key/val buffer holds the sorted result
    int sorted = 0;
    int leaf_min = 1;  // smallest leaf size the node capacity was sized for
    int nchild = 8;     // of the last build
    bool exact = false;
    // optional events around the traversal kernel (recorded into graphs too)
    bool profiling = false;
    cudaEvent_t trav_ev[2] = {nullptr, nullptr};
};

static void ws_release(BhWorkspace *ws)
{
    void *p[] = {ws->keys[0],     ws->keys[1],    ws->vals[0],    ws->vals[1],
                 ws->sort_meta,   ws->sort_status, ws->sbody,     ws->lcp,
                 ws->mask,        ws->leafcnt,    ws->blk_cnt,    ws->blk_off,
                 ws->sbody_lo,    ws->sg.hi,      ws->sg.lo,      ws->nd.begin,
                 ws->nd.count,    ws->nd.child,   ws->nd.nchild,  ws->nd.level,
                 ws->nd.geo_lo,   ws->nd.geo,     ws->nd.com,     ws->lv,
                 ws->extent_bits, ws->flags,      ws->nd.meta,    ws->stats,
                 ws->nd.parent,   ws->nd.quad_a,  ws->nd.quad_b,  ws->sg.com,
                 ws->sg.qa,       ws->sg.qb,
                 ws->tile_cnt,    ws->tile_grp,   ws->tree_bar,   ws->blockmax};
    for (void *q : p) dev_free(q, ws->stream);
}

template <typename T>
static int wsalloc(T *&p, size_t count, cudaStream_t st)
{
    return dev_alloc(p, count, st);
}

int bh_reserve(BhWorkspace *&ws, size_t n, int device, const BhParams &p, cudaStream_t stream)
{
    const int leaf = p.leaf_size < 1 ? 1 : p.leaf_size;
    const bool quad = p.multipole == kMultipoleQuadrupole;
    const bool exact = p.traversal != PHYSIM_TRAVERSAL_WARP;
    if (ws && n <= ws->cap_n && leaf >= ws->leaf_min && (ws->nd.quad_a || !quad) &&
        (ws->nd.geo_lo || !exact))
        return PHYSIM_OK;
    if (ws) {
        ws_release(ws);
        delete ws;
        ws = nullptr;
    }
    // the radix sort stages its tile in 96 KB of dynamic shared memory; set
    // once per device, here (never inside a stream capture), with the number
    // of single-launch sort blocks an SM holds (0: no cooperative launch)
    if (device >= 0 && device < 64 && !g_sort_ready[device].load()) {
        PG_CUDA(cudaFuncSetAttribute(radix_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kSortSmem));
        PG_CUDA(cudaFuncSetAttribute(radix_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kSortSmem));
        int coop = 0, per_sm = 0;
        PG_TRY(tree_sort_attributes());
        PG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
        if (coop)
            PG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, radix_sort_kernel,
                                                                  kSortThreads, kSortSmem));
        g_sort_coop_per_sm[device].store(per_sm);
        g_sort_ready[device].store(true);
    }
    BhWorkspace *w = new (std::nothrow) BhWorkspace();
    PG_CHECK(w, PHYSIM_ERR_MEMORY, "out of host memory");
    w->device = device;
    w->stream = stream;
    const size_t cap = n < 64 ? 64 : n;
    w->cap_n = cap;
    const int tiles = cdiv((long long)cap, kSortTile);
    const int resident_blocks = device_sm_count(device);
    const size_t tree_blocks = (size_t)cdiv((long long)cap, kTreeBlock);
    // Node capacity: leaves hold about leaf/4 bodies on average, so 8N/leaf
    // (at most 4N) nodes hold every non-degenerate distribution; deeper
    // chains only leave levels unsplit (exact, slower) and raise a flag.
    const size_t ncap = std::min<size_t>(4 * cap, 8 * cap / (size_t)leaf) + 4096 + 64 * kMaxLevels;
    w->leaf_min = leaf;
    int rc = PHYSIM_OK;
#define PG_WA(ptr, cnt)                                                                     \
    if (rc == PHYSIM_OK) rc = wsalloc(ptr, cnt, stream)
    PG_WA(w->keys[0], cap);
    PG_WA(w->keys[1], cap);
    PG_WA(w->vals[0], cap);
    PG_WA(w->vals[1], cap);
    PG_WA(w->sort_meta, (size_t)kSortPasses * kRadixBuckets + kSortPasses + 2);
    PG_WA(w->sort_status, (size_t)kRadixBuckets * tiles);
    const size_t rtiles = (size_t)resident_tiles(cap, resident_blocks);
    PG_WA(w->tile_cnt, rtiles * kRadixBuckets);
    PG_WA(w->tile_grp, 2 * ((rtiles + kSortGroup - 1) / kSortGroup) * kRadixBuckets);
    PG_WA(w->blockmax, 2 * rtiles);  // (a rank tile is half a sort tile)
    PG_WA(w->tree_bar, 8);
    PG_WA(w->sbody, cap);
    PG_WA(w->lcp, cap);
    PG_WA(w->mask, cap);
    PG_WA(w->leafcnt, cap);
    // (tree_build_kernel counts tiles of kBuildBlock, mask_kernel of kTreeBlock)
    static_assert(kBuildBlock <= kTreeBlock, "the finer tiles");
    PG_WA(w->blk_cnt, (size_t)32 * cdiv((long long)cap, kBuildBlock));
    PG_WA(w->blk_off, 32 * tree_blocks);
    if (exact) PG_WA(w->sbody_lo, cap);
    const size_t groups = cap / 2 + kSegLevels;  // all levels of cap / 4, cap / 8, ...
    PG_WA(w->sg.hi, groups);
    PG_WA(w->sg.lo, groups);
    if (quad) {
        PG_WA(w->sg.com, groups);
        PG_WA(w->sg.qa, groups);
        PG_WA(w->sg.qb, groups);
        PG_WA(w->nd.quad_a, ncap);
        PG_WA(w->nd.quad_b, ncap);
    }
    PG_WA(w->nd.begin, ncap);
    PG_WA(w->nd.count, ncap);
    PG_WA(w->nd.child, ncap);
    PG_WA(w->nd.nchild, ncap);
    PG_WA(w->nd.level, ncap);
    if (exact) PG_WA(w->nd.geo_lo, ncap);
    PG_WA(w->nd.geo, ncap);
    PG_WA(w->nd.com, ncap);
    PG_WA(w->nd.meta, ncap);
    PG_WA(w->nd.parent, ncap);
    PG_WA(w->stats, 4);
    PG_WA(w->lv, 1);
    PG_WA(w->extent_bits, 1);
    PG_WA(w->flags, 4);
#undef PG_WA
    w->nd.cap = (int)ncap;
    if (rc == PHYSIM_OK &&
        (cudaMemsetAsync(w->flags, 0, 4 * sizeof(uint32_t), stream) != cudaSuccess ||
         cudaMemsetAsync(w->lv, 0, sizeof(LevelInfo), stream) != cudaSuccess ||
         cudaMemsetAsync(w->tree_bar, 0, 8 * sizeof(uint32_t), stream) != cudaSuccess ||
         cudaMemsetAsync(w->sort_meta, 0,
                         ((size_t)kSortPasses * kRadixBuckets + kSortPasses + 2) * sizeof(uint32_t),
                         stream) != cudaSuccess ||
         cudaMemsetAsync(w->sort_status, 0,
                         (size_t)kRadixBuckets * tiles * sizeof(unsigned long long),
                         stream) != cudaSuccess))
        rc = PHYSIM_ERR_CUDA;
    if (rc != PHYSIM_OK) {
        ws_release(w);
        delete w;
        return rc;
    }
    ws = w;
    return PHYSIM_OK;
}

void bh_free(BhWorkspace *ws)
{
    if (!ws) return;
    for (cudaEvent_t e : ws->trav_ev)
        if (e) cudaEventDestroy(e);
    ws_release(ws);
    delete ws;
}

int bh_set_profiling(BhWorkspace *ws, bool enable)
{
    PG_CHECK(ws, PHYSIM_ERR_ARGUMENT, "null workspace");
    if (enable && !ws->trav_ev[0])
        for (cudaEvent_t &e : ws->trav_ev) PG_CUDA(cudaEventCreate(&e));
    ws->profiling = enable;
    return PHYSIM_OK;
}

int bh_traversal_ms(BhWorkspace *ws, double *ms)
{
    PG_CHECK(ws && ms && ws->profiling, PHYSIM_ERR_ARGUMENT, "profiling is off");
    PG_CUDA(cudaEventSynchronize(ws->trav_ev[1]));
    float t = 0.f;
    PG_CUDA(cudaEventElapsedTime(&t, ws->trav_ev[0], ws->trav_ev[1]));
    *ms = t;
    return PHYSIM_OK;
}

int bh_launches(const BhWorkspace *ws) { return ws ? ws->launches : 0; }

const uint32_t *bh_flags(const BhWorkspace *ws) { return ws->flags; }

bool bh_failed(const uint32_t f[4]) { return f[kFlagStack] != 0 || f[kFlagSort] != 0; }

int bh_check(BhWorkspace *ws, cudaStream_t st)
{
    if (!ws) return PHYSIM_OK;
    uint32_t f[4];
    PG_CUDA(cudaMemcpyAsync(f, ws->flags, sizeof f, cudaMemcpyDeviceToHost, st));
    PG_CUDA(cudaStreamSynchronize(st));
    if (!bh_failed(f)) return PHYSIM_OK;
    PG_CUDA(cudaMemsetAsync(ws->flags + kFlagStack, 0, 2 * sizeof(uint32_t), st));
    PG_CUDA(cudaStreamSynchronize(st));
    if (f[kFlagSort]) {
        set_error("Barnes-Hut build: a bounded wait (radix sort look-back or pass barrier, "
                  "or tree level) gave up; "
                  "results are invalid");
        return PHYSIM_ERR_TIMEOUT;
    }
    set_error("Barnes-Hut traversal stack overflow; results are invalid");
    return PHYSIM_ERR_TREE;
}

int bh_stats(BhWorkspace *ws, cudaStream_t st, uint64_t out[2])
{
    PG_CHECK(ws && out, PHYSIM_ERR_ARGUMENT, "null argument");
    unsigned long long h[2] = {0, 0};
    PG_CUDA(cudaMemcpyAsync(h, ws->stats, sizeof h, cudaMemcpyDeviceToHost, st));
    PG_CUDA(cudaStreamSynchronize(st));
    out[0] = h[0];
    out[1] = h[1];
    return PHYSIM_OK;
}

namespace {
std::atomic<uint32_t> g_wait_limit{0};  // 0: kLookbackSpins
std::atomic<int32_t> g_stall_tile{-1}, g_stall_build{-1};
std::atomic<int> g_sort_single{1};
}  // namespace

int wait_limit()
{
    const uint32_t v = g_wait_limit.load();
    return v == 0u ? kLookbackSpins : (int)std::min<uint32_t>(v, (uint32_t)INT32_MAX);
}

static bool rank_sort(int n, int sms) { return n <= std::min(kRankMax, sms * kRankTile); }

// Extent, keys and sort of a state whose tiles are all resident.
static int launch_tree_sort(BhWorkspace *ws, const DeviceBodies &b, const BhParams &p, int n,
                            int items, cudaStream_t st)
{
    TreeSortArgs a;
    a.x = b.x;
    a.y = b.y;
    a.z = b.z;
    a.n = n;
    a.nchild = p.nchild;
    a.extent_bits = ws->extent_bits;
    a.blockmax = ws->blockmax;
    a.k0 = ws->keys[0];
    a.k1 = ws->keys[1];
    a.v0 = ws->vals[0];
    a.v1 = ws->vals[1];
    a.tile_cnt = ws->tile_cnt;
    a.grp = ws->tile_grp;
    a.bar = ws->tree_bar;
    a.stats = ws->stats;
    a.flags = ws->flags;
    a.spin_limit = wait_limit();
    a.stall_tile = (int)g_stall_tile.load();
    void *args[] = {&a};
    if (rank_sort(n, device_sm_count(ws->device))) {
        PG_CUDA(cudaLaunchCooperativeKernel((const void *)rank_sort_kernel,
                                            dim3((unsigned)cdiv(n, kRankTile)), dim3(kRankTile),
                                            args, rank_sort_smem(n), st));
        return PHYSIM_OK;
    }
    PG_CUDA(cudaLaunchCooperativeKernel(tree_sort_fn(items),
                                        dim3((unsigned)cdiv(n, kSortThreads * items)),
                                        dim3(kSortThreads), args, tree_sort_smem(items), st));
    return PHYSIM_OK;
}

// The same as separate launches: extent, keys with the digits' histograms, and
// the one-sweep radix sort of all seven digits, in one cooperative launch
// where the device allows it (blocks then sort several tiles), else one launch
// per pass.
static int launch_split_sort(BhWorkspace *ws, const DeviceBodies &b, const BhParams &p, int n,
                             int per_sm, int sms, cudaStream_t st, int *cur_out, int *launches)
{
    PG_CUDA(cudaMemsetAsync(ws->extent_bits, 0, sizeof(unsigned long long), st));
    PG_CUDA(cudaMemsetAsync(ws->stats, 0, 2 * sizeof(unsigned long long), st));
    extent_kernel<<<sms * 2, 256, 0, st>>>(b.x, b.y, b.z, n, ws->extent_bits);
    uint32_t *ghist = ws->sort_meta;
    uint32_t *tile_ctr = ws->sort_meta + kSortPasses * kRadixBuckets;
    uint32_t *epoch = tile_ctr + kSortPasses;
    uint32_t *sort_bar = epoch + 1;
    PG_CUDA(cudaMemsetAsync(ghist, 0, kSortPasses * kRadixBuckets * sizeof(uint32_t), st));
    keys_kernel<<<std::min(cdiv(n, 256), sms * 8), 256, 0, st>>>(
        b.x, b.y, b.z, n, p.nchild, ws->extent_bits, ws->keys[0], ws->vals[0], ghist, tile_ctr,
        epoch, sort_bar);
    *launches += 2;
    // one-sweep radix sort over 9-bit digits: all passes in one cooperative
    // launch where the device allows it, else one launch per pass
    const int tiles = cdiv(n, kSortTile);
    int cur = 0;
    if (g_sort_single.load() && per_sm > 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)std::min(tiles, per_sm * sms));
        cfg.blockDim = dim3(kSortThreads);
        cfg.dynamicSmemBytes = kSortSmem;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        PG_CUDA(cudaLaunchKernelEx(&cfg, radix_sort_kernel, ws->keys[0], ws->vals[0], ws->keys[1],
                                   ws->vals[1], n, (const uint32_t *)ghist, ws->sort_status,
                                   (const uint32_t *)epoch, ws->flags, wait_limit(),
                                   (int)g_stall_tile.load(), sort_bar));
        cur = kSortPasses & 1;
        *launches += 1;
    } else {
        for (int pass = 0; pass < kSortPasses; ++pass) {
            radix_pass_kernel<<<tiles, kSortThreads, kSortSmem, st>>>(
                ws->keys[cur], pass == 0 ? nullptr : ws->vals[cur], ws->keys[cur ^ 1],
                ws->vals[cur ^ 1], n, pass, ghist, tile_ctr, ws->sort_status, epoch, ws->flags,
                wait_limit(), g_stall_tile.load());
            cur ^= 1;
            *launches += 1;
        }
    }
    *cur_out = cur;
    return PHYSIM_OK;
}

template <int kLanes>
static int launch_cells_lanes(const uint64_t *keys, BhWorkspace *ws, const BhParams &p,
                              const Segments &sg, bool quad, bool exact, int blocks,
                              cudaStream_t st)
{
    auto cells = quad ? (exact ? cell_kernel<true, true, kLanes> : cell_kernel<true, false, kLanes>)
                      : (exact ? cell_kernel<false, true, kLanes>
                               : cell_kernel<false, false, kLanes>);
    return launch_pdl(cells, blocks, 256, st, keys, (const float4 *)ws->sbody, ws->nd,
                      (const LevelInfo *)ws->lv, p.nchild, sg,
                      (const unsigned long long *)ws->extent_bits, (const uint32_t *)ws->flags);
}

// Lanes per node of the cells: eight while the nodes (about 1.5 per body with
// one body per leaf, an eighth per body with 16) leave the SMs idle.  One lane
// vs eight (us): leaf 16, 2,003 bodies 12.0 / 7.9, 100,003 15.1 / 9.4, 200,003
// 15.9 / 13.8, 400,009 17.2 / 23.4; with quadrupoles 100,003 25.0 / 11.4, 400,009
// 28.7 / 29.4; leaf 1, 2,003 bodies 12.3 / 8.5, 20,011 13.5 / 12.9, 50,021 15.1 /
// 19.0.
static int cell_lanes(int n, const BhParams &p)
{
    const double leaf = std::max(1.0, 0.625 * p.leaf_size);
    const bool quad = p.multipole == kMultipoleQuadrupole;
    return n <= (quad ? 30000.0 : 20000.0) * leaf ? 8 : 1;
}

// Whether the tree is built in one launch: a tile per SM.  Step times, separate
// launches vs one (us): theta 1.0, leaf 16, 303 bodies 54.3 / 52.6, 8,195 77.6 /
// 73.9, 50,021 83.5 / 79.5, and with several tiles per block 100,003 97.0 /
// 100.5, 300,007 139.6 / 149.0; leaf 1, 8,195 80.4 / 75.9, 250,007 150.5 / 175.8;
// quadrupoles, 8,195 104.5 / 98.8, 100,003 242.4 / 246.0.
static bool resident_build(int n, int per_sm, int sms)
{
    return g_sort_single.load() && per_sm > 0 && n <= sms * kBuildBlock;
}

template <int kLanes>
static const void *tree_build_fn(bool quad, bool exact)
{
    auto f = quad ? (exact ? tree_build_kernel<true, true, kLanes>
                           : tree_build_kernel<true, false, kLanes>)
                  : (exact ? tree_build_kernel<false, true, kLanes>
                           : tree_build_kernel<false, false, kLanes>);
    return (const void *)f;
}

static int launch_build(BhWorkspace *ws, const GatherArgs &ga, const BhParams &p, bool quad,
                        bool exact, int sms, cudaStream_t st)
{
    BuildArgs a;
    a.gather = ga;
    a.gather.lcp = nullptr;
    a.leaf = p.leaf_size;
    a.blk_cnt = ws->blk_cnt;
    a.nd = ws->nd;
    a.lv = ws->lv;
    a.extent_bits = ws->extent_bits;
    a.bar = ws->tree_bar + 4;
    a.flags = ws->flags;
    a.spin_limit = wait_limit();
    a.stall_tile = (int)g_stall_build.load();
    // blocks for the tiles, one for the top group sums, and more if the cells
    // are more than those blocks' threads
    const int lanes = cell_lanes(ga.n, p);
    const int nodes = (int)(1.6 * ga.n / std::max(1.0, 0.625 * p.leaf_size)) + 1;
    const int blocks = std::min(
        sms, std::max(cdiv(ga.n, kBuildBlock) + 1, cdiv(nodes * lanes, kBuildBlock)));
    a.early = blocks < sms;
    void *args[] = {&a};
    PG_CUDA(cudaLaunchCooperativeKernel(
        lanes == 8 ? tree_build_fn<8>(quad, exact) : tree_build_fn<1>(quad, exact),
        dim3((unsigned)blocks), dim3(kBuildBlock), args, 0, st));
    return PHYSIM_OK;
}

static int bh_build(BhWorkspace *ws, const DeviceBodies &b, const BhParams &p, cudaStream_t st)
{
    const int n = (int)b.n;
    int launches = 0;
    const int sms = device_sm_count(ws->device);
    const int per_sm = ws->device >= 0 && ws->device < 64 ? g_sort_coop_per_sm[ws->device].load() : 0;
    const int items = per_sm > 0 ? resident_items((size_t)n, sms) : 0;
    int cur = 0;
    if (g_sort_single.load() && items > 0) {
        PG_TRY(launch_tree_sort(ws, b, p, n, items, st));
        cur = 1;
        launches += 1;
    } else {
        PG_TRY(launch_split_sort(ws, b, p, n, per_sm, sms, st, &cur, &launches));
    }
    ws->sorted = cur;
    // the tree: boundaries, sorted bodies and group sums; level masks; one scan
    // (and the top group sums); node records; cells
    const uint64_t *keys = ws->keys[cur];
    const bool quad = p.multipole == kMultipoleQuadrupole;
    const bool exact = p.traversal == PHYSIM_TRAVERSAL_EXACT;
    Segments &sg = ws->sg;
    sg.n = n;
    for (int k = 0, at = 0; k < kSegLevels; ++k) {
        sg.off[k] = at;
        at += sg.groups(k);
    }
    PG_CHECK(p.leaf_size >= 1 && p.leaf_size <= kMaxLeaf, PHYSIM_ERR_ARGUMENT,
             "leaf size %d outside 1..%d", p.leaf_size, kMaxLeaf);
    GatherArgs ga;
    ga.keys = keys;
    ga.order = ws->vals[cur];
    ga.n = n;
    ga.nchild = p.nchild;
    ga.body4 = (const float4 *)b.body4;
    ga.bx = b.x;
    ga.by = b.y;
    ga.bz = b.z;
    ga.sbody = ws->sbody;
    ga.sbody_lo = ws->sbody_lo;
    ga.lcp = ws->lcp;
    ga.sg = sg;
    ws->nchild = p.nchild;
    ws->exact = exact;
    if (resident_build(n, per_sm, sms)) {
        PG_TRY(launch_build(ws, ga, p, quad, exact, sms, st));
        ws->launches = launches + 1;
        return PHYSIM_OK;
    }
    auto boundary = quad ? (exact ? boundary_kernel<true, true> : boundary_kernel<true, false>)
                         : (exact ? boundary_kernel<false, true> : boundary_kernel<false, false>);
    PG_TRY(launch_pdl(boundary, cdiv(n, kSegBlock), kSegBlock / kSegBase, st, ga,
                      (const uint32_t *)ws->flags));
    const int tree_blocks = cdiv(n, kTreeBlock);
    PG_TRY(launch_pdl(mask_kernel, tree_blocks, kTreeBlock, st, keys, (const uint8_t *)ws->lcp, n,
                      p.nchild, p.leaf_size, ws->mask, ws->blk_cnt, tree_blocks, ws->leafcnt,
                      (const uint32_t *)ws->flags));
    PG_TRY(launch_pdl(level_scan_kernel, 2, 1024, st, (const uint32_t *)ws->blk_cnt, tree_blocks,
                      p.nchild, ws->blk_off, ws->lv, ws->nd.cap, ws->flags, sg, quad ? 1 : 0));
    PG_TRY(launch_pdl(node_kernel, tree_blocks, kTreeBlock, st, keys, (const uint8_t *)ws->leafcnt,
                      (const uint32_t *)ws->mask, (const uint32_t *)ws->blk_off, tree_blocks, n,
                      p.nchild, ws->nd, (const LevelInfo *)ws->lv, (const uint32_t *)ws->flags));
    PG_TRY(cell_lanes(n, p) == 8
               ? launch_cells_lanes<8>(keys, ws, p, sg, quad, exact, sms * 8, st)
               : launch_cells_lanes<1>(keys, ws, p, sg, quad, exact, sms * 8, st));
    launches += 5;
    PG_CUDA(cudaGetLastError());
    ws->launches = launches;
    return PHYSIM_OK;
}

// Warps per group of 32 bodies of the warp traversal.  A team of four shortens
// each walk's chain of rounds but spends about 1.6 times the instructions, so it
// pays while a walk is long (theta below 0.8, or the accuracy options) and the
// groups are too few to hide it.  Step times, one warp vs four (us): theta 0.5,
// Plummer, 8,195 bodies 116 vs 99, 20,011 127 vs 109, 50,021 141 vs 150; theta
// 1.0, 20,011 bodies 87 vs 90; quadrupoles and com_theta 0.6, 20,011 bodies 291
// vs 197, 100,003 673 vs 639, 300,007 1,538 vs 1,754.  (Teams of two and eight
// were never the best by more than 1%.)
static int bh_team(int n, const BhParams &p, int sms)
{
    const bool options = p.multipole == kMultipoleQuadrupole || p.com_theta > 0.0;
    const long long groups_per_sm = cdiv(n, 32) / sms;
    if (options) return groups_per_sm < 24 ? 4 : 1;
    return p.theta < 0.8 && groups_per_sm < 8 ? 4 : 1;
}

// Warps per group of the exact traversal, by the same trade.  Step times with
// one / four / eight warps (us), leaf 1, Plummer: theta 0.3, 1,003 bodies 282 /
// 145 / 119, 20,011 605 / 277 / 273, 250,007 2,015 / 2,009; theta 0.5, 1,003
// bodies 190 / 114 / 103, 10,007 - / 148 / 127, 20,011 291 / 164 / 177, 50,021
// 335 / 257 / 277, 100,003 406 / 413; quadtree, theta 0.5, 50,021 bodies 160 /
// 153, 100,003 183 / 203; theta 1.0, 20,011 bodies 88 / 91 / 93.
static int exact_team(int n, const BhParams &p, int sms)
{
    const double groups_per_sm = n / 32.0 / sms;
    if (p.theta >= 0.8 || groups_per_sm > 16.0) return 1;
    return groups_per_sm > 2.5 ? 4 : 8;
}

template <bool kQuad, bool kGuard>
static int launch_traverse_warp(const TravArgs &a, int team, cudaStream_t st)
{
    const int groups = cdiv(a.n, 32);
    if (team == 4)
        return launch_pdl(traverse_warp_kernel<kQuad, kGuard, 4>, groups, 128, st, a);
    return launch_pdl(traverse_warp_kernel<kQuad, kGuard, 1>, groups, 32, st, a);
}

int bh_accelerations(BhWorkspace *ws, const DeviceBodies &b, const BhParams &p, double *partial,
                     cudaStream_t st)
{
    PG_CHECK(ws && b.x, PHYSIM_ERR_ARGUMENT, "Barnes-Hut needs the f64 body state");
    PG_CHECK(p.nchild == 8 || p.nchild == 4, PHYSIM_ERR_ARGUMENT, "nchild must be 8 or 4");
    PG_CHECK(b.n <= ws->cap_n, PHYSIM_ERR_ARGUMENT, "workspace too small");
    const int n = (int)b.n;
    if (n == 0) return PHYSIM_OK;
    PG_TRY(bh_build(ws, b, p, st));
    TravArgs a;
    a.nd = ws->nd;
    a.sbody = ws->sbody;
    a.sbody_lo = ws->sbody_lo;
    a.keys = ws->keys[ws->sorted];
    a.nchild = p.nchild;
    a.bx = b.x;
    a.by = b.y;
    a.bz = b.z;
    a.order = ws->vals[ws->sorted];
    a.lv = ws->lv;
    a.n = n;
    a.theta = (float)p.theta;
    a.theta64 = p.theta;
    a.e = (float)p.e;
    a.flags = ws->flags;
    a.partial = partial;
    a.extent = 0.f;  // read on the device from extent_bits
    a.extent_bits = ws->extent_bits;
    a.stats = ws->stats;
    a.quad = p.multipole == kMultipoleQuadrupole ? 1 : 0;
    a.com_theta = (float)p.com_theta;
    a.sk = a.skm = 0;  // set on the device (extent, total mass)
    a.sc = a.msc = 1.f;
    a.es = a.e;
    // external records, so they also time the kernel when replayed from a graph
    if (ws->profiling)
        PG_CUDA(cudaEventRecordWithFlags(ws->trav_ev[0], st, cudaEventRecordExternal));
    if (p.traversal == PHYSIM_TRAVERSAL_WARP) {
        const int team = bh_team(n, p, device_sm_count(ws->device));
        if (a.quad)
            PG_TRY((launch_traverse_warp<true, true>(a, team, st)));
        else if (a.com_theta > 0.f)
            PG_TRY((launch_traverse_warp<false, true>(a, team, st)));
        else
            PG_TRY((launch_traverse_warp<false, false>(a, team, st)));
    } else
    {
        const int team = exact_team(n, p, device_sm_count(ws->device)), groups = cdiv(n, 32);
        if (team == 8)
            PG_TRY(launch_pdl(traverse_exact_kernel<8>, groups, 256, st, a));
        else if (team == 4)
            PG_TRY(launch_pdl(traverse_exact_kernel<4>, groups, 128, st, a));
        else
            PG_TRY(launch_pdl(traverse_exact_kernel<1>, groups, 32, st, a));
    }
    PG_CUDA(cudaGetLastError());
    if (ws->profiling)
        PG_CUDA(cudaEventRecordWithFlags(ws->trav_ev[1], st, cudaEventRecordExternal));
    ws->launches += 1;
    return PHYSIM_OK;
}

// Copies the tree of the last build to host arrays (tests / diagnostics).
int bh_snapshot(BhWorkspace *ws, size_t n, cudaStream_t st, PhysimTreeSnapshot *out)
{
    PG_CHECK(ws && out, PHYSIM_ERR_ARGUMENT, "null argument");
    LevelInfo lv;
    uint32_t flags[4];
    unsigned long long xb = 0;
    PG_CUDA(cudaMemcpyAsync(&lv, ws->lv, sizeof lv, cudaMemcpyDeviceToHost, st));
    PG_CUDA(cudaMemcpyAsync(flags, ws->flags, sizeof flags, cudaMemcpyDeviceToHost, st));
    PG_CUDA(cudaMemcpyAsync(&xb, ws->extent_bits, sizeof xb, cudaMemcpyDeviceToHost, st));
    PG_CUDA(cudaStreamSynchronize(st));
    double X;
    memcpy(&X, &xb, sizeof X);
    out->extent = X;
    out->n_bodies = n;
    out->n_nodes = (size_t)lv.total;
    out->flags = flags[kFlagNodes] | (flags[kFlagStack] << 1) | (flags[kFlagSort] << 2);
    const size_t nn = out->n_nodes < out->cap_nodes ? out->n_nodes : out->cap_nodes;
    auto cp = [&](void *dst, const void *src, size_t bytes) -> int {
        if (dst && bytes) PG_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
        return PHYSIM_OK;
    };
    PG_TRY(cp(out->keys, ws->keys[ws->sorted], n * sizeof(uint64_t)));
    PG_TRY(cp(out->order, ws->vals[ws->sorted], n * sizeof(uint32_t)));
    PG_TRY(cp(out->node_begin, ws->nd.begin, nn * sizeof(int32_t)));
    PG_TRY(cp(out->node_count, ws->nd.count, nn * sizeof(int32_t)));
    PG_TRY(cp(out->node_child, ws->nd.child, nn * sizeof(int32_t)));
    PG_TRY(cp(out->node_nchild, ws->nd.nchild, nn));
    PG_TRY(cp(out->node_level, ws->nd.level, nn));
    if (out->node_centre && ws->exact && nn) {
        double *c64 = nullptr;
        PG_TRY(dev_alloc(c64, 4 * nn, st));
        snapshot_centre_kernel<<<cdiv((long long)nn, 256), 256, 0, st>>>(
            ws->keys[ws->sorted], ws->nd, (int)nn, ws->nchild, ws->extent_bits, c64);
        const int rc = cp(out->node_centre, c64, 4 * nn * sizeof(double));
        dev_free(c64, st);
        PG_TRY(rc);
    }
    PG_TRY(cp(out->node_com, ws->nd.com, nn * sizeof(float4)));
    if (out->node_quad && ws->nd.quad_a) {
        PG_TRY(cp(out->node_quad, ws->nd.quad_a, nn * sizeof(float4)));
        PG_TRY(cp(out->node_quad + 4 * nn, ws->nd.quad_b, nn * sizeof(float4)));
    }
    PG_CUDA(cudaStreamSynchronize(st));
    return PHYSIM_OK;
}

}  // namespace pg

extern "C" int physim_gpu_set_wait_limit(uint32_t polls)
{
    pg::g_wait_limit.store(polls);
    return PHYSIM_OK;
}

extern "C" int physim_gpu_set_sort_single_launch(int32_t on)
{
    pg::g_sort_single.store(on ? 1 : 0);
    return PHYSIM_OK;
}

extern "C" int physim_gpu_test_stall_sort(int32_t tile)
{
    pg::g_stall_tile.store(tile < 0 ? -1 : tile);
    return PHYSIM_OK;
}

extern "C" int physim_gpu_test_stall_build(int32_t block)
{
    pg::g_stall_build.store(block < 0 ? -1 : block);
    return PHYSIM_OK;
}
