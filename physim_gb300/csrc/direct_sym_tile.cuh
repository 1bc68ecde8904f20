// direct_sym_tile.cuh -- one tile pair of the symmetric direct sum (each
// unordered pair evaluated once, both bodies updated), shared by the
// per-simulation kernel (direct_sym.cu) and the batched ensemble kernel
// (ensemble.cu) so both evaluate bit-identical arithmetic.  The schedule and
// the slot-buffer layout are described in direct_sym.cu.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "engine.h"

namespace pg {

constexpr int kSymWarps = 2;
constexpr int kSymThreads = kSymWarps * 32;
constexpr int kSymIpt = 16;                         // bodies of tile I per thread
constexpr int kSymTile = kSymThreads * kSymIpt;     // 1,024
constexpr int kSymGroups = kSymTile / 32;           // groups of 32 bodies of tile J
static_assert(kSymTile == kBodyPad, "tiles are whole units of the body padding");

// Tile pair of block u: J-major order, u = J (J + 1) / 2 + I, 0 <= I <= J.
__device__ __forceinline__ void unit_tiles(long long u, int &I, int &J)
{
    long long j = (long long)((sqrt(8.0 * (double)u + 1.0) - 1.0) * 0.5);
    while (j > 0 && j * (j + 1) / 2 > u) --j;
    while ((j + 1) * (j + 2) / 2 <= u) ++j;
    J = (int)j;
    I = (int)(u - j * (j + 1) / 2);
}

// Tile I's bodies in registers: positions (negated) scaled by sc, masses
// (negated) by msc (PairScale in engine.h).  Thread layout: bodies
// I*1024 + p*64 + t, p = 2q (x half) and 2q+1 (y half), t = 0..63 within the
// two warps that hold the tile.
constexpr int kSymQ = kSymIpt / 2;

__device__ __forceinline__ void sym_load_i(const float4 *__restrict__ body, int I, float sc,
                                           float msc, float2 (&nx)[kSymQ], float2 (&ny)[kSymQ],
                                           float2 (&nz)[kSymQ], float2 (&nm)[kSymQ])
{
    const int ib = I * kSymTile + (threadIdx.x & (kSymThreads - 1));
#pragma unroll
    for (int q = 0; q < kSymQ; ++q) {
        const float4 b0 = body[ib + (2 * q) * kSymThreads];
        const float4 b1 = body[ib + (2 * q + 1) * kSymThreads];
        nx[q] = make_float2(-b0.x * sc, -b1.x * sc);
        ny[q] = make_float2(-b0.y * sc, -b1.y * sc);
        nz[q] = make_float2(-b0.z * sc, -b1.z * sc);
        nm[q] = make_float2(-b0.w * msc, -b1.w * msc);
    }
}

// *p += v on a shared-memory float, atomically (PTX red.shared.add.f32).
__device__ __forceinline__ void red_shared_add(float *p, float v)
{
    asm volatile("red.shared.add.f32 [%0], %1;"
                 :
                 : "r"((unsigned)__cvta_generic_to_shared(p)), "f"(v)
                 : "memory");
}

// The mass that all bodies of 256-body blocks [b0, b1) have (DeviceBodies::
// mass256); false where there is none.
__device__ __forceinline__ bool common_mass(const float *__restrict__ mass256, int b0, int b1,
                                            float &m)
{
    m = mass256[b0];
    bool same = m == m;
    for (int b = b0 + 1; b < b1; ++b) same = same && mass256[b] == m;
    return same;
}

// a += g with what the addition drops in g (TwoSum).
__device__ __forceinline__ void fold2(float2 &a, float2 &g)
{
    const float2 minus = make_float2(-1.f, -1.f);
    const float2 s = add2(a, g);
    const float2 gp = fma2(a, minus, s), ap = fma2(gp, minus, s);
    g = add2(fma2(ap, minus, a), fma2(gp, minus, g));
    a = s;
}

// Tile I (in registers) against groups [g0, g1) of 32 bodies of tile J: a_i +=
// the pairs' terms (scaled, see sym_load_i); unless DIAG, tile J's reactions go
// to shared memory, jw[j][c] for body j from group g0 on: stored (this warp's own slice), or with ADD added to
// a slice that starts at zero and that both warps of the block add to (two
// terms added onto zero round the same in either order, so the sum does not
// depend on which warp comes first).  With DIAG (I == J) every ordered pair
// of the tile is evaluated for a_i only (a body meets itself with d = 0,
// which contributes 0 through the r^2 guard).
// With UNI the bodies of either tile all have one mass: the pairs' terms are
// summed without masses (15 FMA-pipe operations and 9 shuffles per 16 pairs
// instead of 17 and 10), the reactions leave multiplied by nmi (minus tile I's
// scaled mass), and the caller multiplies a_i by tile J's.  One rounding per sum
// takes the place of one per term.
// With FINE the sums are as exact as the one-pair kernels' (direct_tile.cuh: chains
// of 128 terms, folded by TwoSum): a_i takes each group's 32 terms as one sum, and
// a travelling body's reaction each step's eight, so that no chain is longer than
// 32 (1,024 and 256 otherwise).  A group in which one body outweighs the others by
// far is folded every four terms, by TwoSum: after such a body's term each plain add
// rounds at its size.
template <bool DIAG, bool ADD, bool UNI, bool FINE>
__device__ __forceinline__ void sym_pair_core(const float4 *__restrict__ body, int J, int g0,
                                              int g1, float sc, float msc, float nmi, float2 e2,
                                              const float2 (&nx)[kSymQ],
                                              const float2 (&ny)[kSymQ],
                                              const float2 (&nz)[kSymQ],
                                              const float2 (&nm)[kSymQ], float2 (&ax)[kSymQ],
                                              float2 (&ay)[kSymQ], float2 (&az)[kSymQ],
                                              float (*jw)[3])
{
    const int lane = threadIdx.x & 31;
    const float2 g2 = make_float2(kPairGuard, kPairGuard);
    const unsigned full = 0xffffffffu;
    const int src = (lane + 1) & 31;
    // steps per turn of the loop, by what the registers' rotation costs in moves:
    // ADD (131,072 bodies by groups) 1 / 2 / 4 / 8 / 16: - / 9.90 / 9.59 / 9.35 / 9.37
    // ms; else (524,288 bodies by tile pairs) 1 / 2 / 4: 62.4 / 64.0 / 64.3 ms, with
    // masses of their own 69.2 / 70.0 / -
    constexpr int kUnroll = ADD ? 8 : 1;

    float2 gx[FINE ? kSymQ : 1], gy[FINE ? kSymQ : 1], gz[FINE ? kSymQ : 1];
    if (FINE) {
#pragma unroll
        for (int q = 0; q < kSymQ; ++q) gx[q] = gy[q] = gz[q] = make_float2(0.f, 0.f);
    }
    float4 next = body[J * kSymTile + g0 * 32 + lane];
    for (int g = g0; g < g1; ++g) {
        const float4 bj = next;
        // the next group's body is loaded while this group is evaluated
        if (g + 1 < g1) next = body[J * kSymTile + (g + 1) * 32 + lane];
        float xj = bj.x * sc, yj = bj.y * sc, zj = bj.z * sc, mj = bj.w * msc;
        float2 jx = make_float2(0.f, 0.f), jy = jx, jz = jx;
        int run = 32;  // FINE: steps between two folds
        if (FINE && !UNI) {
            float sum = fabsf(mj);
            const float most =
                __uint_as_float(__reduce_max_sync(full, __float_as_uint(sum)));
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(full, sum, o);
            if (most > 0.125f * sum) run = 4;  // four times the mean
        }
        auto step = [&]() {
            const float2 xj2 = make_float2(xj, xj);
            const float2 yj2 = make_float2(yj, yj);
            const float2 zj2 = make_float2(zj, zj);
            const float2 mj2 = make_float2(mj, mj);
            // the next body's coordinates do not depend on this step
            xj = __shfl_sync(full, xj, src);
            yj = __shfl_sync(full, yj, src);
            zj = __shfl_sync(full, zj, src);
            if (!UNI) mj = __shfl_sync(full, mj, src);
            float2 rx, ry, rz;  // FINE: this step's reaction
#pragma unroll
            for (int q = 0; q < kSymQ; ++q) {
                const float2 dx = add2(xj2, nx[q]);
                const float2 dy = add2(yj2, ny[q]);
                const float2 dz = add2(zj2, nz[q]);
                float2 r2 = mul2(dz, dz);
                r2 = fma2(dy, dy, r2);
                r2 = fma2(dx, dx, r2);
                const float2 w = add2(r2, e2);
                const float2 ww = mul2(w, w);
                const float2 qv = fma2(r2, ww, g2);
                const float2 inv = make_float2(rsqrt_approx(qv.x), rsqrt_approx(qv.y));
                const float2 fi = UNI ? inv : mul2(mj2, inv);
                if (FINE) {
                    gx[q] = fma2(dx, fi, gx[q]);
                    gy[q] = fma2(dy, fi, gy[q]);
                    gz[q] = fma2(dz, fi, gz[q]);
                } else {
                    ax[q] = fma2(dx, fi, ax[q]);
                    ay[q] = fma2(dy, fi, ay[q]);
                    az[q] = fma2(dz, fi, az[q]);
                }
                if (!DIAG) {
                    const float2 fj = UNI ? inv : mul2(nm[q], inv);
                    if (FINE) {
                        rx = q == 0 ? mul2(dx, fj) : fma2(dx, fj, rx);
                        ry = q == 0 ? mul2(dy, fj) : fma2(dy, fj, ry);
                        rz = q == 0 ? mul2(dz, fj) : fma2(dz, fj, rz);
                    } else {
                        jx = fma2(dx, fj, jx);
                        jy = fma2(dy, fj, jy);
                        jz = fma2(dz, fj, jz);
                    }
                }
            }
            if (!DIAG && FINE) {
                jx = add2(jx, rx);
                jy = add2(jy, ry);
                jz = add2(jz, rz);
            }
            if (!DIAG) {
                jx.x = __shfl_sync(full, jx.x, src);
                jx.y = __shfl_sync(full, jx.y, src);
                jy.x = __shfl_sync(full, jy.x, src);
                jy.y = __shfl_sync(full, jy.y, src);
                jz.x = __shfl_sync(full, jz.x, src);
                jz.y = __shfl_sync(full, jz.y, src);
            }
        };
        if (FINE && !UNI) {
#pragma unroll 1
            for (int k = 0; k < 32; k += run) {
#pragma unroll 1
                for (int u = 0; u < run; ++u) step();
                if (run == 32) break;
#pragma unroll
                for (int q = 0; q < kSymQ; ++q) {
                    fold2(ax[q], gx[q]);
                    fold2(ay[q], gy[q]);
                    fold2(az[q], gz[q]);
                }
            }
        } else {
#pragma unroll kUnroll
            for (int k = 0; k < 32; ++k) step();
        }
        if (FINE) {
#pragma unroll
            for (int q = 0; q < kSymQ; ++q) {
                ax[q] = add2(ax[q], gx[q]);
                ay[q] = add2(ay[q], gy[q]);
                az[q] = add2(az[q], gz[q]);
                gx[q] = gy[q] = gz[q] = make_float2(0.f, 0.f);
            }
        }
        if (!DIAG) {
            // after 32 rotations lane `lane` holds body g*32 + lane's reaction again
            float *dst = jw[(g - g0) * 32 + lane];
            const float f = UNI ? nmi : 1.f;
            const float rx = (jx.x + jx.y) * f, ry = (jy.x + jy.y) * f, rz = (jz.x + jz.y) * f;
            if (ADD) {
                red_shared_add(dst + 0, rx);
                red_shared_add(dst + 1, ry);
                red_shared_add(dst + 2, rz);
            } else {
                dst[0] = rx;
                dst[1] = ry;
                dst[2] = rz;
            }
        }
    }
}

// sym_pair_core with the variant that the tiles' masses allow.  uni: tile I's
// scaled mass mi and the groups' mj are common.  a_i must enter as zero.
template <bool DIAG, bool ADD, bool FINE>
__device__ __forceinline__ void sym_pair(bool uni, float mi, float mj,
                                         const float4 *__restrict__ body, int J, int g0, int g1,
                                         float sc, float msc, float2 e2,
                                         const float2 (&nx)[kSymQ], const float2 (&ny)[kSymQ],
                                         const float2 (&nz)[kSymQ], const float2 (&nm)[kSymQ],
                                         float2 (&ax)[kSymQ], float2 (&ay)[kSymQ],
                                         float2 (&az)[kSymQ], float (*jw)[3])
{
    if (uni) {
        sym_pair_core<DIAG, ADD, true, FINE>(body, J, g0, g1, sc, msc, -mi, e2, nx, ny, nz, nm, ax, ay,
                                       az, jw);
        const float2 m2 = make_float2(mj, mj);
#pragma unroll
        for (int q = 0; q < kSymQ; ++q) {
            ax[q] = mul2(ax[q], m2);
            ay[q] = mul2(ay[q], m2);
            az[q] = mul2(az[q], m2);
        }
    } else {
        sym_pair_core<DIAG, ADD, false, FINE>(body, J, g0, g1, sc, msc, 0.f, e2, nx, ny, nz, nm, ax, ay,
                                        az, jw);
    }
}

// Part `rank` of `parts` of one tile pair (I, J): tile I against that share of
// tile J's groups.  Tile J's contribution to tile I's bodies goes to slot J,
// tile I's to tile J's bodies to slot I, of P[T][3][n] (f32, left scaled:
// positions entering as p 2^-sk, masses as m 2^-skm; the reduction multiplies by
// 2^(skm - 2sk) in f64).  With parts > 1 the blocks of one thread-block cluster
// take the parts: their sums for tile I are added through distributed shared
// memory, ranks in order with TwoSum, each block adding and writing its share
// of the bodies, so there is one slot per tile pair whatever the parts.
// EIGHTHS: the sums for tile I are those of eight parts whether eight blocks take one
// each or one block takes all (parts 8 or 1), which adds them up in shared memory the
// same way, so the result does not depend on the parts.
// pairs: the slots are float2, the sum and what its rounding to f32 dropped.
// smem: 6 x 1,024 floats; EIGHTHS with one part 12 x 1,024.
template <bool DIAG, bool FINE, bool EIGHTHS>
__device__ __forceinline__ void sym_tile_pair(const float4 *__restrict__ body,
                                              const float *__restrict__ mass256, int n, int I,
                                              int J, float e, int sk, int skm,
                                              float *__restrict__ P, bool pairs, float *smem,
                                              int rank = 0, int parts = 1)
{
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const size_t n3 = 3 * (size_t)n;
    const int ib = warp * 32 + lane;
    const float sc = pow2f(-sk), msc = pow2f(-skm);
    const float es = e * pow2f(-2 * sk);
    const float2 e2 = make_float2(es, es);
    // the groups of tile J that hold bodies, shared out over the parts
    const int groups = min(kSymGroups, (n - J * kSymTile + 31) / 32);
    const int shares = EIGHTHS ? 8 : parts;
    const int s0 = rank * shares / parts, s1 = (rank + 1) * shares / parts;
    const int g0 = s0 * groups / shares, g1 = s1 * groups / shares;
    const int rows = (g1 - g0) * 32;  // <= 512 with two parts or more
    float (*jacc)[3] = reinterpret_cast<float (*)[3]>(smem);  // [kSymWarps][rows][3]
    float2 nx[kSymQ], ny[kSymQ], nz[kSymQ], nm[kSymQ], ax[kSymQ], ay[kSymQ], az[kSymQ];
    sym_load_i(body, I, sc, msc, nx, ny, nz, nm);
    float mi = 0.f;
    const bool uni_i = common_mass(mass256, I * 4, I * 4 + 4, mi);
    auto share = [&](int a, int b) {
#pragma unroll
        for (int q = 0; q < kSymQ; ++q) ax[q] = ay[q] = az[q] = make_float2(0.f, 0.f);
        if (a == b) return;
        float mj = 0.f;
        const bool uni = common_mass(mass256, J * 4 + a / 8, J * 4 + (b + 7) / 8, mj) && uni_i;
        sym_pair<DIAG, false, FINE>(uni, mi * msc, mj * msc, body, J, a, b, sc, msc, e2, nx, ny,
                                    nz, nm, ax, ay, az, jacc + warp * rows + (a - g0) * 32);
    };
    float *ihi = smem + 2 * 3 * kSymTile, *ilo = ihi + 3 * kSymTile;  // [3][1,024]
    if (EIGHTHS && parts == 1) {
#pragma unroll 1
        for (int k = 0; k < 8; ++k) {
            share(k * groups / 8, (k + 1) * groups / 8);
#pragma unroll
            for (int q = 0; q < kSymQ; ++q) {
                const float v[2][3] = {{ax[q].x, ay[q].x, az[q].x}, {ax[q].y, ay[q].y, az[q].y}};
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const int at = c * kSymTile + ib + (2 * q + h) * kSymThreads;
                        float sum, err;
                        two_sum(k == 0 ? 0.f : ihi[at], v[h][c], sum, err);
                        ihi[at] = sum;
                        ilo[at] = k == 0 ? err : ilo[at] + err;
                    }
            }
        }
    } else {
        share(g0, g1);
    }
    auto put = [&](int slot, int c, int k, float hi, float lo) {
        const size_t at = (size_t)slot * n3 + (size_t)c * n + k;
        if (pairs)
            reinterpret_cast<float2 *>(P)[at] = make_float2(hi, lo);
        else
            P[at] = hi + lo;
    };
    // tile J's contribution to tile I's bodies: slot J
    if (EIGHTHS && parts == 1) {
        for (int p = 0; p < kSymIpt; ++p) {  // (this thread's own sums)
            const int b = ib + p * kSymThreads, i = I * kSymTile + b;
            if (i >= n) break;
#pragma unroll
            for (int c = 0; c < 3; ++c)
                put(J, c, i, ihi[c * kSymTile + b], ilo[c * kSymTile + b]);
        }
        if (!DIAG) __syncthreads();
    } else if (parts == 1) {
#pragma unroll
        for (int q = 0; q < kSymQ; ++q) {
            const int i0 = I * kSymTile + ib + (2 * q) * kSymThreads;
            const int i1 = i0 + kSymThreads;
            if (i0 < n) {
                put(J, 0, i0, ax[q].x, 0.f);
                put(J, 1, i0, ay[q].x, 0.f);
                put(J, 2, i0, az[q].x, 0.f);
            }
            if (i1 < n) {
                put(J, 0, i1, ax[q].y, 0.f);
                put(J, 1, i1, ay[q].y, 0.f);
                put(J, 2, i1, az[q].y, 0.f);
            }
        }
        if (!DIAG) __syncthreads();
    } else {
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        float *mine = smem + 3 * kSymTile;  // [3][1,024], past the reactions
#pragma unroll
        for (int q = 0; q < kSymQ; ++q) {
            const int b0 = ib + (2 * q) * kSymThreads, b1 = b0 + kSymThreads;
            mine[b0] = ax[q].x;
            mine[kSymTile + b0] = ay[q].x;
            mine[2 * kSymTile + b0] = az[q].x;
            mine[b1] = ax[q].y;
            mine[kSymTile + b1] = ay[q].y;
            mine[2 * kSymTile + b1] = az[q].y;
        }
        cluster.sync();
        const int own = kSymTile / parts, first = rank * own;
        for (int t = threadIdx.x; t < 3 * own; t += kSymThreads) {
            const int c = t / own, b = first + t - c * own;
            const int i = I * kSymTile + b;
            if (i >= n) continue;
            float v[8];
#pragma unroll
            for (int r = 0; r < 8; ++r)
                v[r] = r < parts ? cluster.map_shared_rank(mine, r)[c * kSymTile + b] : 0.f;
            float hi = 0.f, lo = 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                if (r >= parts) break;
                float s, err;
                two_sum(hi, v[r], s, err);
                hi = s;
                lo += err;
            }
            put(J, c, i, hi, lo);
        }
    }
    if (!DIAG) {
        // tile I's contribution to tile J's bodies: slot I, warps added in order
        static_assert(kSymWarps == 2, "one sum");
        for (int j = threadIdx.x; j < rows; j += kSymThreads) {
            const int k = J * kSymTile + g0 * 32 + j;
            if (k >= n) break;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                float s, err;
                two_sum(jacc[j][c], jacc[rows + j][c], s, err);
                put(I, c, k, s, pairs ? err : 0.f);
            }
        }
    }
    // every block's shared memory stays until the others have read it
    if (parts > 1) cooperative_groups::this_cluster().sync();
}

}  // namespace pg
