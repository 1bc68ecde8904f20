// direct_sym.cu -- simple_astro pair forces with every unordered pair
// evaluated once (astro/src/transformers.rs:219-244, force law
// astro/src/lib.rs:84-113).
//
// The reference's force is antisymmetric: F_ji = -F_ij.  With
//     s_ij = 1 / sqrt(r^2 (r^2 + e)^2),   d = x_j - x_i,
// body i gains  m_j s_ij d  and body j gains  -m_i s_ij d  from one
// evaluation of d, r^2 and the reciprocal square root.  Per unordered pair
// that is 17 FP32 FMA-pipe operations (3 differences, 3 for r^2, 3 for the
// argument, m_j s and the 3-term update of a_i, -m_i s and the 3-term
// update of a_j) and one MUFU.RSQ, against 2 x 13 operations and 2 MUFU when
// each ordered pair is evaluated on its own.  The FMA pipe bounds the pair
// kernels, so this is up to 1.53x the interactions per second.
//
// Schedule.  Bodies form tiles of 1,024 (the body padding unit).  A block
// holds the 1,024 bodies of one tile I in registers (2 warps, 16 per thread,
// as 8 packed FFMA2 pairs); a warp takes the bodies of a tile J 32 at a
// time, one per lane, and rotates them through its lanes with shuffles:
// after 32 steps every lane's bodies have met all 32, and each travelling
// body's accumulated reaction is back at its home lane (sym_pair_core).  The
// diagonal tile pair (I, I) evaluates all ordered pairs of the tile and
// updates a_i only.
//
// Two schedules share that core.  With few tiles (one [3][n] f32 slot per
// tile fits in kSymPairsSlotBytes) every tile pair (I, J), I <= J, is one
// block, or one cluster of up to eight that share out tile J (pair_parts;
// sym_tile_pair in direct_sym_tile.cuh): tile J's contribution to tile
// I goes to slot J, tile I's to tile J to slot I, and a reduce adds each
// body's T slots.  That keeps every SM busy at any size and is the faster of
// the two, but its slots grow as 12 T n bytes (12.9 GB at 1,048,580 bodies),
// so once they would exceed kSymPairsSlotBytes (4 GiB, about 600,000 bodies)
// the group schedule below takes over.
//
// Group schedule.  A block of four teams (of two warps) holds an SM.  It takes
// the I tiles g*8 .. g*8+7 and a run of kSymRun (16) J tiles r*16 .. r*16+15,
// the pairs with I <= J: for each J tile first I tiles 0..3 of the group, one
// per team, then 4..7.  A tile's a_i accumulates over the whole run and is
// written once, to slot r of its tile's i-side slots: after each J tile a thread
// folds its register sums into its bodies' compensated (TwoSum) sums in shared
// memory (high part f32, low part bf16: the low part only carries rounding
// errors), so every tile's contribution is compensated as when each tile pair
// had a slot of its own.  A team's two warps add their reactions to tile J into
// the team's buffer; the block adds the buffers (I tiles in order,
// TwoSum-compensated) and writes the sums of all eight once, to slot g of tile
// J's j-side slots.  Per unit of up to 8 x 16 tile pairs that is 8 + 16 slot
// writes of 12 KB instead of 2 per tile pair.  All of it stays on one SM: the
// same units as clusters of eight blocks of two warps, adding through
// distributed shared memory, took 293 ms for the 1,048,580-body force pass where
// this takes 257 (tile pairs with a slot each: 248); a cluster waits for the
// slowest of its blocks at every J tile, and an SM that is left over in its
// group of SMs holds none.
// The units on the diagonal are half as long and come last, where the SMs run
// out of units.
// Group schedule output.  Tile K has Rn - floor(K / 16) i-side slots (the runs r whose last
// J tile is >= K) and floor(K / 8) + 1 j-side slots (the groups g with
// 8 g <= K), each [3][1024] f32, packed tile after tile (offsets in closed
// form, sym_iside_base / sym_jside_base): 1.2 GB at 1,048,580 bodies,
// against 12.9 GB for one slot per tile pair.  A second kernel sums each
// body's slots with compensated (TwoSum) arithmetic in a fixed order (i-side
// by run, then j-side by group) into the f64 partial-sum layout the
// integrators read (one split).  The result is deterministic, and the slot
// sums act as the per-tile compensation of the one-pair kernels.
#include <math.h>

#include <cuda_bf16.h>

#include <atomic>

#include "common.cuh"
#include "direct_sym_tile.cuh"
#include "engine.h"

namespace pg {

namespace {

// The tile-pair schedule while its slot buffer (12 B per body per tile) fits
// in 4 GiB (up to about 600,000 bodies) or the physim_gpu_set_symmetric_pairs_limit.
constexpr size_t kSymPairsSlotBytes = size_t(4) << 30;
std::atomic<uint64_t> g_pairs_limit{0};

// States below this many bodies, which the one-pair kernels would take otherwise,
// are summed as exactly as those do (FINE, sym_pair_core), in slots of two f32, the
// sum and what its rounding dropped.  RMS error against f64 at e = 0.01 (1e-8 of the
// acceleration), one-pair kernels / chains of a tile and one f32 per slot / FINE:
// Plummer 8,192 bodies 3.3 / 4.2 / 2.8, 16,387 4.8 / 4.9 / 4.0, 20,479 3.0 / 3.5 /
// 2.9, cube with four heavy stars 8,192 5.7 / 8.7 / 5.7, 20,479 5.7 / 7.8 / 5.7.
// FINE costs 2 to 6% of a step (16,387 bodies 89 -> 92 us, one-pair 154) and, where
// masses differ, some 10% (97 -> 107).  From 20,480 on, plain chains as ever.
constexpr int kSymFine = 20480;

constexpr int kSymTeams = 4;    // I tiles in registers at a time, two warps each
constexpr int kSymGroup = 8;    // I tiles per unit
constexpr int kSymRun = 16;     // J tiles per run

// Slots of tile K (see the file comment), in units of one [3][1024] slot.
__host__ __device__ inline long long sym_iside_count(int K, int runs)
{
    return runs - K / kSymRun;
}

__host__ __device__ inline long long sym_iside_base(int K, int runs)
{
    const long long q = K / kSymRun, rem = K - q * kSymRun;
    return (long long)K * runs - (kSymRun * q * (q - 1) / 2 + q * rem);
}

__host__ __device__ inline long long sym_jside_base(int K)
{
    const long long q = K / kSymGroup, rem = K - q * kSymGroup;
    return (long long)K + kSymGroup * q * (q - 1) / 2 + q * rem;
}

constexpr int kSlot = 3 * kSymTile;  // floats per slot

// Units: I group g (tiles 8g .. 8g+7) with the J runs r >= floor(8g / 16).
__host__ __device__ inline long long sym_units(int T)
{
    const int groups = (T + kSymGroup - 1) / kSymGroup;
    const int runs = (T + kSymRun - 1) / kSymRun;
    long long c = 0;
    for (int g = 0; g < groups; ++g) c += runs - (g * kSymGroup) / kSymRun;
    return c;
}

// Unit u: those past the diagonal, group by group, then the groups' first runs.
__device__ __forceinline__ void sym_unit(int u, int T, int &g, int &r)
{
    const int groups = (T + kSymGroup - 1) / kSymGroup;
    const int runs = (T + kSymRun - 1) / kSymRun;
    for (g = 0; g < groups; ++g) {
        const int first = (g * kSymGroup) / kSymRun, c = runs - first - 1;
        if (u < c) {
            r = first + 1 + u;
            return;
        }
        u -= c;
    }
    g = u;
    r = (g * kSymGroup) / kSymRun;
}

// Dynamic shared memory of the pair kernel: the teams' reaction buffers
// ([4][1024][3] f32), the reactions' sums over the I tiles so far (high and low
// part), then the compensated i-side sums of the run ([8] x hi[3][1024] f32,
// lo[3][1024] bf16): 216 KB, one block per SM.
constexpr int kSymBlock = kSymTeams * kSymThreads;
constexpr size_t kSymSmem = ((kSymTeams + 2) * sizeof(float) +
                             kSymGroup * (sizeof(float) + sizeof(__nv_bfloat16))) * kSlot;

// 256 threads of up to 255 registers (about 245 used).
__global__ void __launch_bounds__(kSymBlock, 1)
direct_sym_kernel(const float4 *__restrict__ body, const float *__restrict__ mass256, int n, int T,
                  float e, ScaleRef scale, float *__restrict__ Pi, float *__restrict__ Pj)
{
    extern __shared__ float4 smem4[];
    float *jacc = reinterpret_cast<float *>(smem4);  // [team][1024][3]
    float *jhi = jacc + kSymTeams * kSlot, *jlo = jhi + kSlot;
    float *ihi = jlo + kSlot;  // [I tile of the group][3][1024]
    __nv_bfloat16 *ilo = reinterpret_cast<__nv_bfloat16 *>(ihi + kSymGroup * kSlot);
    const int team = threadIdx.x / kSymThreads;
    const int ib = threadIdx.x & (kSymThreads - 1);  // this thread's first body of its tile
    int g, r;
    sym_unit((int)blockIdx.x, T, g, r);
    const int J0 = r * kSymRun, nJ = min(J0 + kSymRun, T) - J0;
    const int sk = pair_scale_exp(__uint_as_float(*scale.ext), e);
    const int skm = mass_scale_exp(__uint_as_float(*scale.mass));
    const float sc = pow2f(-sk), msc = pow2f(-skm);
    const float es = e * pow2f(-2 * sk);
    const float2 e2 = make_float2(es, es);
    for (int x = threadIdx.x; x < kSymTeams * kSlot; x += kSymBlock) jacc[x] = 0.f;
    for (int x = threadIdx.x; x < kSymGroup * kSlot; x += kSymBlock) {
        ihi[x] = 0.f;
        ilo[x] = __float2bfloat16_rn(0.f);
    }
    __syncthreads();
    for (int t = 0; t < nJ; ++t) {
        const int J = J0 + t;
        if (g * kSymGroup > J) continue;  // no I tile of the group reaches tile J
#pragma unroll 1
        for (int half = 0; half < kSymGroup / kSymTeams; ++half) {
            const int slot = half * kSymTeams + team;
            const int I = g * kSymGroup + slot;
            if (I < T && I <= J) {
                float2 nx[kSymQ], ny[kSymQ], nz[kSymQ], nm[kSymQ];
                float2 ax[kSymQ], ay[kSymQ], az[kSymQ];
                sym_load_i(body, I, sc, msc, nx, ny, nz, nm);
#pragma unroll
                for (int q = 0; q < kSymQ; ++q) ax[q] = ay[q] = az[q] = make_float2(0.f, 0.f);
                float mi = 0.f, mj = 0.f;
                bool uni = common_mass(mass256, I * 4, I * 4 + 4, mi);
                uni = common_mass(mass256, J * 4, J * 4 + 4, mj) && uni;
                float (*jw)[3] = reinterpret_cast<float (*)[3]>(jacc + team * kSlot);
                if (I < J)
                    sym_pair<false, true, false>(uni, mi * msc, mj * msc, body, J, 0, kSymGroups, sc,
                                          msc, e2, nx, ny, nz, nm, ax, ay, az, jw);
                else
                    sym_pair<true, false, false>(uni, mi * msc, mj * msc, body, J, 0, kSymGroups, sc,
                                          msc, e2, nx, ny, nz, nm, ax, ay, az, jw);
                // this tile's partial sums into the compensated run sums
                float *hi = ihi + slot * kSlot;
                __nv_bfloat16 *lo = ilo + slot * kSlot;
#pragma unroll
                for (int q = 0; q < kSymQ; ++q) {
                    const float v[2][3] = {{ax[q].x, ay[q].x, az[q].x},
                                           {ax[q].y, ay[q].y, az[q].y}};
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const int at = c * kSymTile + ib + (2 * q + h) * kSymThreads;
                            float sum, err;
                            two_sum(hi[at], v[h][c], sum, err);
                            hi[at] = sum;
                            lo[at] = __float2bfloat16_rn(__bfloat162float(lo[at]) + err);
                        }
                }
            }
            __syncthreads();
            // tile J's reactions, I tiles in order; the buffers are zero again
            float *dst = Pj + (sym_jside_base(J) + g) * kSlot;
            for (int x = threadIdx.x; x < kSlot; x += kSymBlock) {  // x = 3 jj + c
                float hi = half == 0 ? 0.f : jhi[x], lo = half == 0 ? 0.f : jlo[x];
#pragma unroll
                for (int w = 0; w < kSymTeams; ++w) {
                    float sum, err;
                    two_sum(hi, jacc[w * kSlot + x], sum, err);
                    hi = sum;
                    lo += err;
                    jacc[w * kSlot + x] = 0.f;
                }
                if (half == 0) {
                    jhi[x] = hi;
                    jlo[x] = lo;
                } else {
                    const int jj = x / 3, c = x - 3 * jj;
                    if (J * kSymTile + jj < n) dst[c * kSymTile + jj] = hi + lo;
                }
            }
            __syncthreads();
        }
    }
    // the I tiles' sums over the run: i-side slot r
    for (int k = 0; k < kSymGroup; ++k) {
        const int I = g * kSymGroup + k;
        if (I >= T || J0 + nJ - 1 < I) break;
        float *dst = Pi + (sym_iside_base(I, (T + kSymRun - 1) / kSymRun) + (r - I / kSymRun)) * kSlot;
        for (int x = threadIdx.x; x < kSlot; x += kSymBlock)
            if (I * kSymTile + x % kSymTile < n)
                dst[x] = ihi[k * kSlot + x] + __bfloat162float(ilo[k * kSlot + x]);
    }
}

// The factor that takes the scaled sums back: 2^(km - 2k).
__device__ __forceinline__ double unscale(ScaleRef scale, float e)
{
    return pow2d(mass_scale_exp(__uint_as_float(*scale.mass)) -
                 2 * pair_scale_exp(__uint_as_float(*scale.ext), e));
}

// out[c*n + k] = the sum of body k's slots (i-side by run, then j-side by
// group), TwoSum-compensated f32, rounded once to f64 and unscaled
// (x 2^(km - 2k)).
__global__ void sym_reduce_kernel(const float *__restrict__ Pi, const float *__restrict__ Pj,
                                  int n, int T, ScaleRef scale, float e,
                                  double *__restrict__ out)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 3ll * n) return;
    const int c = (int)(idx / n), k = (int)(idx - (long long)c * n);
    const int K = k / kSymTile, local = k - K * kSymTile;
    const int runs = (T + kSymRun - 1) / kSymRun;
    float hi = 0.f, lo = 0.f;
    const float *p = Pi + sym_iside_base(K, runs) * kSlot + c * kSymTile + local;
    const int ni = (int)sym_iside_count(K, runs);
    for (int t = 0; t < ni; ++t) {
        const float v = __ldcs(p + (size_t)t * kSlot);
        float s, err;
        two_sum(hi, v, s, err);
        hi = s;
        lo += err;
    }
    p = Pj + sym_jside_base(K) * kSlot + c * kSymTile + local;
    const int nj = K / kSymGroup + 1;
    for (int t = 0; t < nj; ++t) {
        const float v = __ldcs(p + (size_t)t * kSlot);
        float s, err;
        two_sum(hi, v, s, err);
        hi = s;
        lo += err;
    }
    out[idx] = ((double)hi + (double)lo) * unscale(scale, e);
}

// The tile-pair schedule: `parts` consecutive blocks (a thread-block cluster)
// take tile pair (I, J) (unit_tiles).
template <bool FINE>
__global__ void __launch_bounds__(kSymThreads, 4)
direct_sym_pairs_kernel(const float4 *__restrict__ body, const float *__restrict__ mass256, int n,
                        float e, ScaleRef scale, float *__restrict__ P, int parts)
{
    __shared__ float smem[kSymWarps * kSymTile * 3];
    int I, J;
    const int u = (int)blockIdx.x / parts, rank = (int)blockIdx.x - u * parts;
    unit_tiles(u, I, J);
    const int sk = pair_scale_exp(__uint_as_float(*scale.ext), e);
    const int skm = mass_scale_exp(__uint_as_float(*scale.mass));
    if (I == J)
        sym_tile_pair<true, FINE, false>(body, mass256, n, I, J, e, sk, skm, P, FINE, smem, rank, parts);
    else
        sym_tile_pair<false, FINE, false>(body, mass256, n, I, J, e, sk, skm, P, FINE, smem, rank, parts);
}

// out[idx] = the sum of entry idx of the T slots P[t][3][n], in slot order,
// TwoSum-compensated, rounded once to f64 and unscaled (x 2^(km - 2k)); FINE: the
// slots are float2 (sym_tile_pair).
template <bool FINE>
__global__ void sym_pairs_reduce_kernel(const float *__restrict__ P, long long n3, int T,
                                        ScaleRef scale, float e, double *__restrict__ out)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n3) return;
    float hi = 0.f, lo = 0.f;
#pragma unroll 8
    for (int t = 0; t < T; ++t) {
        const size_t at = (size_t)t * n3 + idx;
        float2 v = make_float2(0.f, 0.f);
        if (FINE)
            v = __ldcs(reinterpret_cast<const float2 *>(P) + at);
        else
            v.x = __ldcs(P + at);
        float s, err;
        two_sum(hi, v.x, s, err);
        hi = s;
        lo += FINE ? err + v.y : err;
    }
    out[idx] = ((double)hi + (double)lo) * unscale(scale, e);
}

}  // namespace

DirectPlan make_symmetric_plan(int n)
{
    // 216 KB of dynamic shared memory per block, and the largest carveout.  Set here, when a plan is made (never inside a stream capture), per device.
    static std::atomic<bool> attrs_set[64];
    int device = 0;
    if (cudaGetDevice(&device) == cudaSuccess && device >= 0 && device < 64 &&
        !attrs_set[device].load()) {
        if (cudaFuncSetAttribute(direct_sym_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kSymSmem) == cudaSuccess)
            attrs_set[device].store(true);
        else
            (void)cudaGetLastError();  // the launch then reports the error
        if (cudaFuncSetAttribute(direct_sym_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess)
            (void)cudaGetLastError();  // a hint only: the kernel runs without it
        for (auto *pairs : {direct_sym_pairs_kernel<false>, direct_sym_pairs_kernel<true>})
            if (cudaFuncSetAttribute(pairs, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess)
                (void)cudaGetLastError();
    }
    DirectPlan p;
    p.symmetric = true;
    p.block = kSymThreads;
    p.ipt = kSymIpt;
    p.n = n;
    p.compensated = true;
    p.splits = 1;
    p.tiles = (int)(pad_bodies((size_t)n) / kSymTile);
    p.n_itiles = p.tiles;
    p.n_jtiles = p.tiles;
    p.chunk_tiles = p.tiles;
    const uint64_t limit = g_pairs_limit.load();
    p.grouped = (size_t)p.tiles * 12 * (size_t)(n > 0 ? n : 1) >
                 (limit ? (size_t)limit : kSymPairsSlotBytes);
    return p;
}

// f32 floats of the symmetric plan's i-side and j-side slots
static size_t sym_slot_floats(int T, size_t *jside_at)
{
    const int runs = (T + kSymRun - 1) / kSymRun;
    const size_t ni = (size_t)sym_iside_base(T, runs) * kSlot;
    const size_t nj = (size_t)sym_jside_base(T) * kSlot;
    if (jside_at) *jside_at = ni;
    return ni + nj;
}

size_t direct_partial_doubles(const DirectPlan &p)
{
    const size_t n3 = 3 * (size_t)(p.n > 0 ? p.n : 1);
    if (!p.symmetric) return (size_t)p.splits * n3;
    // f64 sums, then the f32 slots carved after them
    if (!p.grouped) return n3 + ((p.n < kSymFine ? 2 : 1) * (size_t)p.tiles * n3 + 1) / 2;
    return n3 + (sym_slot_floats(p.tiles, nullptr) + 1) / 2;
}

// Blocks per tile pair.  A block's two warps go to two of an SM's four
// schedulers, so an SM's time is that of its blocks rounded up to an even
// number, each 1 / parts of a tile pair; while more blocks than are resident at
// once (four per SM) follow one another, the last ones run beside idle slots,
// about one block's time more; up to two per SM leave a scheduler one warp, 3%;
// and each doubling of the parts costs some 3% (the cluster's exchange).  A model:
// over 21 sizes its choice was 0.5% slower than the best on the average, 2% at most
// where it changes every thousand bodies (35,000 to 61,500).  Steps
// at 1 / 2 / 4 / 8 parts (us): 12,600 bodies 164 / 96 / 92 / 70, 16,387 164 / 96 /
// 92 / 99, 22,000 166 / 170 / 160 / 150, 24,000 164 / 169 / 180 / 175, 30,011 310 /
// 254 / 258 / 256, 50,000 703 / 667 / 650 / 663, 65,537 1,032 / 1,051 / 1,086 /
// 1,103.
static int pair_parts(int n, int sms)
{
    const double tiles = (double)n / kSymTile;
    if (tiles > 60.0) return 1;
    const double pairs = tiles * (tiles + 1.0) / 2.0;
    int best = 1;
    double best_time = 1e300;
    for (int parts = 1, step = 0; parts <= 8; parts *= 2, ++step) {
        const double blocks = pairs * parts;
        double time = 2.0 * ceil(blocks / sms / 2.0);
        if (blocks > 4.0 * sms) time += 1.0;
        if (blocks <= 2.0 * sms) time *= 1.03;
        time *= (1.0 + 0.03 * step) / parts;
        if (time < best_time) {
            best_time = time;
            best = parts;
        }
    }
    return best;
}

int launch_direct_symmetric(const DirectPlan &plan, const float4 *body4, const float *mass256,
                            float e, ScaleRef scale, double *partial, cudaStream_t stream,
                            cudaEvent_t pairs_done)
{
    if (plan.n <= 0) return PHYSIM_OK;
    if (!plan.grouped) {
        const long long T = plan.tiles;
        const long long units = T * (T + 1) / 2;
        PG_CHECK(units < (1ll << 31), PHYSIM_ERR_ARGUMENT, "too many bodies for one pass: %d",
                 plan.n);
        const long long n3 = 3ll * plan.n;
        float *P = (float *)(partial + n3);
        int device = 0;
        PG_CUDA(cudaGetDevice(&device));
        const int parts = pair_parts(plan.n, device_sm_count(device));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(units * parts));
        cfg.blockDim = dim3(kSymThreads);
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)parts;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = parts > 1 ? 1 : 0;
        PG_CUDA(cudaLaunchKernelEx(
            &cfg, plan.n < kSymFine ? direct_sym_pairs_kernel<true> : direct_sym_pairs_kernel<false>,
            body4, mass256, plan.n, e, scale, P, parts));
        if (pairs_done) PG_TRY(record_event(pairs_done, stream));
        auto reduce = plan.n < kSymFine ? sym_pairs_reduce_kernel<true>
                                        : sym_pairs_reduce_kernel<false>;
        reduce<<<(unsigned)((n3 + 255) / 256), 256, 0, stream>>>(P, n3, (int)T, scale, e, partial);
        PG_CUDA(cudaGetLastError());
        return PHYSIM_OK;
    }
    const int T = plan.tiles;
    const long long blocks = sym_units(T);
    PG_CHECK(blocks < (1ll << 31), PHYSIM_ERR_ARGUMENT, "too many bodies for one pass: %d",
             plan.n);
    const long long n3 = 3ll * plan.n;
    size_t jside_at = 0;
    sym_slot_floats(T, &jside_at);
    float *Pi = (float *)(partial + n3);
    float *Pj = Pi + jside_at;
    direct_sym_kernel<<<(unsigned)blocks, kSymBlock, kSymSmem, stream>>>(
        body4, mass256, plan.n, T, e, scale, Pi, Pj);
    PG_CUDA(cudaGetLastError());
    if (pairs_done) PG_TRY(record_event(pairs_done, stream));
    sym_reduce_kernel<<<(unsigned)((n3 + 255) / 256), 256, 0, stream>>>(Pi, Pj, plan.n, T,
                                                                         scale, e, partial);
    PG_CUDA(cudaGetLastError());
    return PHYSIM_OK;
}

}  // namespace pg

extern "C" int physim_gpu_set_symmetric_pairs_limit(uint64_t bytes)
{
    pg::g_pairs_limit.store(bytes);
    return PHYSIM_OK;
}
