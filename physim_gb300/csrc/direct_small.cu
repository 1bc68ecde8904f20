// direct_small.cu -- simple_astro for small states (astro/src/transformers.rs:
// 219-244, force law astro/src/lib.rs:84-113) in blocks that own their bodies:
// one force pass, or a run of whole verlet steps, in one launch.
//
// The tiled pair kernels (direct.cu) split the j range over blocks, so each
// step is a pair kernel, partial sums through memory and an integrator kernel,
// and at a few thousand bodies most of it is launch latency and the ends of the
// kernels: 25 us per step at 4,098 bodies, 16 at 1,002, where the pair
// arithmetic is 5.4 and 0.3.  Here a block owns n / grid bodies (27 of 4,098)
// outright: its threads hold the state's bodies j in registers, two to a packed
// FP32 lane, and loop over the owned bodies i, so the sums for a body never
// leave the block.
//
//   * j bodies in units of 64 (one packed pair per lane), units dealt to the
//     8 warps in turn, up to kMaxPacks units per warp in registers at a time;
//   * per four bodies i: the pair loop (13 FMA-pipe operations and one MUFU per
//     pair, as direct_tile), then for each two of them six sums over the lanes by
//     a transposing butterfly (8 shuffles instead of 30), one partial per warp in
//     shared memory; the eight warps' partials are added with TwoSum in warp
//     order.  The chains of plain FP32 adds are at most 16 long: nine units, the
//     two halves of a lane, five steps over the lanes, and above 4,608 bodies the
//     second pass (128 and 256 in the tiled kernels).  RMS error against f64 at
//     e = 0.01, against the tiled kernels' plan of the same size: Plummer 0.2 (300
//     bodies) to 0.95 of it, a cube with heavy stars 0.4 to 0.7 in any order of the
//     bodies but the stars last, where the tiled chains end, and then 0.3 to 1.1;
//   * whole steps: the owned bodies' f64 state stays in registers, one thread
//     per coordinate, which applies verlet as integrate.cu does (same
//     operations, same order); the f32 positions go to the other of two body
//     arrays, and one grid barrier per step (1.2 us, every block resident by a
//     cooperative launch) lets the next step read them.
// Step times against the best tiled plan (us): 300 bodies 14.4 -> 3.7, 1,002 16.5
// -> 4.1, 4,098 24.7 -> 11.7, 7,400 49 -> 31.6, and each pair once / here: 7,401
// 32 / 32, with masses that differ 39 / 32, 8,192 33 / 38 and 39 / 38, 9,001 58 /
// 47 and 60 / 47, 10,240 52 / 57 and 61 / 58, 12,001 70 / 74 and 73 / 74.  The line
// is at 7,400: above it the other plan's error is no larger in any order of the
// bodies (kSymFine in direct_sym.cu), for up to 20% of a step between 8,200 and
// 9,800 bodies.  Bound by the FMA pipe (60% busy) from about 6,000 bodies, below by
// the barrier and one pass of latency.  Eight warps of 255 registers, four bodies i
// at a time: sixteen of 128, two at a time, left the pipe waiting on each chain
// (4,098 bodies 14.1).  A wait at the barrier that exceeds the wait limit raises an
// error flag and ends the launch in every block; the next synchronising call
// reports PHYSIM_ERR_TIMEOUT, and the state is invalid until the next upload (the
// blocks may have given up at different steps).
#include <cuda/atomic>

#include <algorithm>

#include "common.cuh"
#include "engine.h"
#include "verlet_axis.cuh"

namespace pg {

namespace {

constexpr int kSmallThreads = 256;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kMaxPacks = 8;     // units every warp holds at a time (some one more)
constexpr int kMaxOwned = 84;    // bodies per block at most (a thread per coordinate; 49
                                 // of 7,400 on 152 SMs)
constexpr int kTurn = 4;         // owned bodies per turn of the pair loop
constexpr int kUnit = 64;        // bodies of a unit
constexpr int kSmallOwned = 16;  // bodies per block until every SM has one
constexpr uint32_t kPoison = 0x40000000u;

struct SmallShared {
    float4 ixy[kMaxOwned];  // owned bodies, negated and scaled: (x, x, y, y)
    float2 iz[kMaxOwned];   // (z, z)
    float part[kSmallWarps][kMaxOwned * 3];
    uint32_t top[kSmallWarps];
    int ok;
};

// Six sums over the warp's lanes: afterwards lane 4 g (g < 6) holds the sum of
// v[g].  Each step halves the values a lane holds while it halves the lanes.
__device__ __forceinline__ float reduce6(float (&v)[6], int lane)
{
    const unsigned full = 0xffffffffu;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    // lanes 0..15 keep v[0..3], lanes 16..31 keep v[4], v[5]
    const float s0 = b4 ? v[0] : v[4], s1 = b4 ? v[1] : v[5];
    float a = (b4 ? v[4] : v[0]) + __shfl_xor_sync(full, s0, 16);
    float b = (b4 ? v[5] : v[1]) + __shfl_xor_sync(full, s1, 16);
    // v[2], v[3] of the upper lanes join the lower lanes'
    const float c = v[2] + __shfl_xor_sync(full, v[2], 16);
    const float d = v[3] + __shfl_xor_sync(full, v[3], 16);
    // lanes with bit 3 clear keep (a, b), set keep (c, d); of the upper lanes
    // those with bit 3 set hold nothing that is used
    const float t0 = b3 ? a : c, t1 = b3 ? b : d;
    a = (b3 ? c : a) + __shfl_xor_sync(full, t0, 8);
    b = (b3 ? d : b) + __shfl_xor_sync(full, t1, 8);
    const float u = b2 ? a : b;
    a = (b2 ? b : a) + __shfl_xor_sync(full, u, 4);
    a += __shfl_xor_sync(full, a, 2);
    a += __shfl_xor_sync(full, a, 1);
    return a;
}

// The owned bodies against P units per warp from unit u0 on (u0 + warp, + 8, ...)
// and, with `extra`, one more; `first`: sh.part is written, else added to.  The
// P units are straight-line code, so their chains overlap (with a branch per
// unit this loop ran at half the FMA pipe).
template <int P>
__device__ __forceinline__ void owned_units(const float4 *body, int u0, bool extra, bool first,
                                            int m, float sc, float msc, float2 e2,
                                            SmallShared &sh)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float2 g2 = make_float2(kPairGuard, kPairGuard);
    float2 jx[P + 1], jy[P + 1], jz[P + 1], jm[P + 1];
    auto load = [&](int p) {
        const int b = (u0 + warp + p * kSmallWarps) * kUnit + lane;
        const float4 q0 = __ldcg(&body[b]), q1 = __ldcg(&body[b + 32]);
        jx[p] = make_float2(q0.x * sc, q1.x * sc);
        jy[p] = make_float2(q0.y * sc, q1.y * sc);
        jz[p] = make_float2(q0.z * sc, q1.z * sc);
        jm[p] = make_float2(q0.w * msc, q1.w * msc);
    };
#pragma unroll
    for (int p = 0; p < P; ++p) load(p);
    if (extra) load(P);
    if (first) __syncthreads();  // the owned bodies are in shared memory
    if (P == 0 && !extra) return;
#pragma unroll 1
    for (int i = 0; i < m; i += kTurn) {
        float4 xy[kTurn];
        float2 z[kTurn], ax[kTurn], ay[kTurn], az[kTurn];
#pragma unroll
        for (int h = 0; h < kTurn; ++h) {
            const int k = min(i + h, m - 1);
            xy[h] = sh.ixy[k];
            z[h] = sh.iz[k];
            ax[h] = ay[h] = az[h] = make_float2(0.f, 0.f);
        }
        auto unit = [&](int p) {
#pragma unroll
            for (int h = 0; h < kTurn; ++h) {
                const float2 dx = add2(jx[p], make_float2(xy[h].x, xy[h].y));
                const float2 dy = add2(jy[p], make_float2(xy[h].z, xy[h].w));
                const float2 dz = add2(jz[p], z[h]);
                float2 r2 = mul2(dz, dz);
                r2 = fma2(dy, dy, r2);
                r2 = fma2(dx, dx, r2);
                const float2 w = add2(r2, e2);
                const float2 q = fma2(r2, mul2(w, w), g2);
                const float2 f = mul2(jm[p], make_float2(rsqrt_approx(q.x), rsqrt_approx(q.y)));
                ax[h] = fma2(dx, f, ax[h]);
                ay[h] = fma2(dy, f, ay[h]);
                az[h] = fma2(dz, f, az[h]);
            }
        };
#pragma unroll
        for (int p = 0; p < P; ++p) unit(p);
        if (extra) unit(P);
        float s[kTurn / 2];
#pragma unroll
        for (int h = 0; h < kTurn; h += 2) {
            float v[6] = {ax[h].x + ax[h].y,         ay[h].x + ay[h].y,
                          az[h].x + az[h].y,         ax[h + 1].x + ax[h + 1].y,
                          ay[h + 1].x + ay[h + 1].y, az[h + 1].x + az[h + 1].y};
            s[h / 2] = reduce6(v, lane);
        }
        // lane 4 g holds v[g], g = 3 h + c (lanes 16, 20: v[4], v[5])
        const int g = lane >> 2;
        if ((lane & 3) == 0 && g < 6) {
#pragma unroll
            for (int h = 0; h < kTurn; h += 2) {
                const int at = (i + h) * 3 + g;
                float *dst = &sh.part[warp][at];
                if (at < 3 * m) *dst = first ? s[h / 2] : *dst + s[h / 2];
            }
        }
    }
}

// Partial sums of the owned bodies [0, m) (in sh.ixy / sh.iz) over all n bodies
// of `body`, per warp, into sh.part; ends with a block barrier.
__device__ __forceinline__ void owned_forces(const float4 *body, int n, int m, float sc, float msc,
                                             float es, SmallShared &sh)
{
    const int units = (n + kUnit - 1) / kUnit;
    const float2 e2 = make_float2(es, es);
    // the arrays are padded with massless bodies to whole tiles, so the last
    // unit can be read whole
    for (int u0 = 0; u0 < units;) {
        int here = units - u0;
        if (here >= kSmallWarps * (kMaxPacks + 1)) here = kSmallWarps * kMaxPacks;
        const bool extra = (int)(threadIdx.x >> 5) < here % kSmallWarps, first = u0 == 0;
        switch (here / kSmallWarps) {
        case 0: owned_units<0>(body, u0, extra, first, m, sc, msc, e2, sh); break;
        case 1: owned_units<1>(body, u0, extra, first, m, sc, msc, e2, sh); break;
        case 2: owned_units<2>(body, u0, extra, first, m, sc, msc, e2, sh); break;
        case 3: owned_units<3>(body, u0, extra, first, m, sc, msc, e2, sh); break;
        case 4: owned_units<4>(body, u0, extra, first, m, sc, msc, e2, sh); break;
        case 5: owned_units<5>(body, u0, extra, first, m, sc, msc, e2, sh); break;
        case 6: owned_units<6>(body, u0, extra, first, m, sc, msc, e2, sh); break;
        case 7: owned_units<7>(body, u0, extra, first, m, sc, msc, e2, sh); break;
        default: owned_units<8>(body, u0, extra, first, m, sc, msc, e2, sh); break;
        }
        u0 += here;
    }
    __syncthreads();
}

// The sum of coordinate c of owned body i over the warps' partials.
__device__ __forceinline__ double owned_sum(const SmallShared &sh, int t, int warps)
{
    float hi = 0.f, lo = 0.f;
#pragma unroll
    for (int w = 0; w < kSmallWarps; ++w) {
        if (w >= warps) break;
        float s, err;
        two_sum(hi, sh.part[w][t], s, err);
        hi = s;
        lo += err;
    }
    return (double)hi + (double)lo;
}

// Warps that hold at least one unit (the others' partials are not written).
__device__ __forceinline__ int working_warps(int n) { return min(kSmallWarps, (n + kUnit - 1) / kUnit); }

__device__ __forceinline__ void put_owned(SmallShared &sh, int t, float4 p, float sc)
{
    const float x = -p.x * sc, y = -p.y * sc, z = -p.z * sc;
    sh.ixy[t] = make_float4(x, x, y, y);
    sh.iz[t] = make_float2(z, z);
}

// One force pass: out[c * n + i], f64 and unscaled.
__global__ void __launch_bounds__(kSmallThreads, 1)
small_forces_kernel(const float4 *__restrict__ body, int n, float e, ScaleRef scale, int early,
                    double *__restrict__ out)
{
    pdl_wait(early != 0);
    __shared__ SmallShared sh;
    const int i0 = (int)((long long)blockIdx.x * n / gridDim.x);
    const int m = (int)((long long)(blockIdx.x + 1) * n / gridDim.x) - i0;
    const int sk = pair_scale_exp(__uint_as_float(*scale.ext), e);
    const int skm = mass_scale_exp(__uint_as_float(*scale.mass));
    const float sc = pow2f(-sk), msc = pow2f(-skm), es = e * pow2f(-2 * sk);
    if ((int)threadIdx.x < m) put_owned(sh, threadIdx.x, body[i0 + threadIdx.x], sc);
    owned_forces(body, n, m, sc, msc, es, sh);
    const int t = threadIdx.x;
    if (t < 3 * m) {
        const int i = t / 3, c = t - 3 * i;
        out[(size_t)c * n + i0 + i] =
            owned_sum(sh, t, working_warps(n)) * pow2d(skm - 2 * sk);
    }
}

struct SmallSteps {
    float4 *body[2];  // the current state and the other array
    const double *mass;
    const uint8_t *fixed;
    double *x[3], *v[3], *p[3];
    int n, steps, initial;
    float e;
    Divisor dt;
    uint32_t *ext;         // the state's largest |coordinate|: in and out
    const uint32_t *mass_max;
    uint32_t *ring;        // three maxima in turn
    uint32_t *bar;         // [0] barrier count, [1] blocks that left
    uint32_t *flag;        // raised when a wait gave up
    int spin_limit;
};

__device__ __forceinline__ bool steps_barrier(const SmallSteps &a, uint32_t target, int *s_ok)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        cuda::atomic_ref<uint32_t, cuda::thread_scope_device> bar(*a.bar);
        bar.fetch_add(1u, cuda::memory_order_release);
        int spins = 0;
        uint32_t v;
        while ((v = bar.load(cuda::memory_order_acquire)) < target) {
            if (++spins > a.spin_limit) {
                atomicOr(a.flag, 1u);
                v = bar.fetch_or(kPoison, cuda::memory_order_relaxed) | kPoison;
                break;
            }
        }
        *s_ok = v < kPoison;
    }
    __syncthreads();
    return *s_ok != 0;
}

__global__ void __launch_bounds__(kSmallThreads, 1) small_steps_kernel(SmallSteps a)
{
    __shared__ SmallShared sh;
    const int n = a.n;
    const int i0 = (int)((long long)blockIdx.x * n / gridDim.x);
    const int m = (int)((long long)(blockIdx.x + 1) * n / gridDim.x) - i0;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const bool live = t < 3 * m;
    const int oi = live ? t / 3 : 0, c = live ? t - 3 * oi : 0, i = i0 + oi;
    const int skm = mass_scale_exp(__uint_as_float(*a.mass_max));
    const float msc = pow2f(-skm);
    const int warps = working_warps(n);
    // the owned bodies: f64 state one thread per coordinate, f32 copy of both
    double x = 0.0, v = 0.0, p = 0.0;
    bool fixed = false, massless = false;
    if (live) {
        x = a.x[c][i];
        v = a.v[c][i];
        p = a.p[c][i];
        fixed = a.fixed[i] != 0;
        massless = a.mass[i] == 0.0;
    }
    uint32_t ext = *a.ext;
    if (t < m) a.body[1][i0 + t] = a.body[0][i0 + t];  // (its mass, and for a stray reader)
    if (blockIdx.x == 0) {
        // the other array's padding is the state's: massless bodies at the origin
        const int pad = (n + kBodyPad - 1) / kBodyPad * kBodyPad;
        for (int k = n + t; k < pad; k += kSmallThreads)
            a.body[1][k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < 3) a.ring[t] = 0u;
    }
    uint32_t target = gridDim.x;
    bool ok = steps_barrier(a, target, &sh.ok);  // the ring is clear
    const double dt2 = __dmul_rn(a.dt.value, a.dt.value);
    int cur = 0;
    for (int s = 0; ok && s < a.steps; ++s) {
        const int sk = pair_scale_exp(__uint_as_float(ext), a.e);
        const float sc = pow2f(-sk), es = a.e * pow2f(-2 * sk);
        if (t < m) put_owned(sh, t, __ldcg(&a.body[cur][i0 + t]), sc);
        owned_forces(a.body[cur], n, m, sc, msc, es, sh);
        uint32_t top = 0;
        if (live) {
            double acc = 0.0;
            if (!fixed) {
                acc += owned_sum(sh, t, warps) * pow2d(skm - 2 * sk);
                if (massless) acc = __longlong_as_double(0x7ff8000000000000LL);
            }
            verlet_axis(x, v, p, acc, a.dt, dt2, a.initial && s == 0);
            const float f = (float)x;
            reinterpret_cast<float *>(&a.body[cur ^ 1][i])[c] = f;
            top = __float_as_uint(f) & 0x7fffffffu;
            if (top >= 0x7f800000u) top = 0;  // NaN and infinities skipped
        }
        top = __reduce_max_sync(0xffffffffu, top);
        if (lane == 0) sh.top[warp] = top;
        __syncthreads();
        if (t == 0) {
            for (int w = 1; w < kSmallWarps; ++w) top = max(top, sh.top[w]);
            if (top) atomicMax(&a.ring[(s + 1) % 3], top);
            // read by every block before the last barrier
            if (blockIdx.x == 0) a.ring[(s + 2) % 3] = 0u;
        }
        target += gridDim.x;
        ok = steps_barrier(a, target, &sh.ok);
        ext = __ldcg(&a.ring[(s + 1) % 3]);
        cur ^= 1;
    }
    if (ok) {
        if (live) {
            a.x[c][i] = x;
            a.v[c][i] = v;
            a.p[c][i] = p;
        }
        if (cur == 1 && t < m) a.body[0][i0 + t] = __ldcg(&a.body[1][i0 + t]);
        if (blockIdx.x == 0 && t == 0) *a.ext = ext;
    }
    // the last block to leave resets the barrier for the next launch
    __syncthreads();
    if (t == 0) {
        __threadfence();
        if (atomicAdd(&a.bar[1], 1u) == gridDim.x - 1) {
            a.bar[0] = 0u;
            a.bar[1] = 0u;
        }
    }
}

// Blocks: sixteen bodies each until every SM has one, then n / SMs.  (Fewer per
// block would shorten the smallest steps by 0.4 us, but a block takes a whole
// SM's registers, and several such simulations side by side would queue.)
int small_grid(int n, int sms)
{
    return std::max(1, std::min(sms, (n + kSmallOwned - 1) / kSmallOwned));
}

}  // namespace

int direct_small_limit(int device)
{
    return std::min(kDirectSmallMax, kMaxOwned * device_sm_count(device));
}

int launch_direct_small(const float4 *body4, int n, float e, ScaleRef scale, double *partial,
                        cudaStream_t stream)
{
    int device = 0;
    PG_CUDA(cudaGetDevice(&device));
    // Where this kernel fills every SM's registers, the next one must not be let in
    // early: it finds no room, and a force pass and integrator of 3,000 bodies take
    // 17.6 us instead of 10.4.
    const int sms = device_sm_count(device), grid = small_grid(n, sms);
    return launch_pdl(small_forces_kernel, grid, kSmallThreads, stream, body4, n, e, scale,
                      grid < sms ? 1 : 0, partial);
}

int reserve_small(SmallWork &w, const DeviceBodies &b, int device, cudaStream_t stream)
{
    int coop = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop) {
        (void)cudaGetLastError();
        return PHYSIM_OK;  // no whole steps: force passes and integrator launches
    }
    PG_TRY(dev_alloc(w.words, 8, stream));
    PG_CUDA(cudaMemsetAsync(w.words, 0, 8 * sizeof(uint32_t), stream));
    return dev_alloc(w.body4, b.cap, stream);
}

int small_steps_per_launch(int n)
{
    // about 5 ms of steps: 4 us each and 2.6e12 pairs/s
    const double us = 4.0 + (double)n * n / 2.6e6;
    return (int)std::min(1000.0, std::max(1.0, 5000.0 / us));
}

int launch_small_steps(DeviceBodies &b, SmallWork &w, float e, double dt, int steps, bool initial,
                       cudaStream_t stream)
{
    int device = 0;
    PG_CUDA(cudaGetDevice(&device));
    PG_CHECK(w.words && w.body4, PHYSIM_ERR_ARGUMENT, "no workspace for whole steps");
    // a caller's graph keeps the addresses of the maxima (PairScale)
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    PG_CUDA(cudaStreamIsCapturing(stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) b.halves_fixed = w.captured = true;
    SmallSteps a;
    a.body[0] = b.body4;
    a.body[1] = w.body4;
    a.mass = b.m;
    a.fixed = b.fixed;
    double *x[3] = {b.x, b.y, b.z}, *v[3] = {b.vx, b.vy, b.vz}, *p[3] = {b.px, b.py, b.pz};
    for (int c = 0; c < 3; ++c) {
        a.x[c] = x[c];
        a.v[c] = v[c];
        a.p[c] = p[c];
    }
    a.n = (int)b.n;
    a.steps = steps;
    a.initial = initial ? 1 : 0;
    a.e = e;
    a.dt = make_divisor(dt);
    a.ext = &b.scale->ext[b.ext_half];
    a.mass_max = &b.scale->mass[b.mass_half];
    a.ring = w.words;
    a.bar = w.words + 4;
    a.flag = w.words + 6;
    a.spin_limit = wait_limit();
    void *args[] = {&a};
    PG_CUDA(cudaLaunchCooperativeKernel((const void *)small_steps_kernel,
                                        dim3((unsigned)small_grid(a.n, device_sm_count(device))),
                                        dim3(kSmallThreads), args, 0, stream));
    w.unchecked = true;
    return PHYSIM_OK;
}

int check_small_steps(SmallWork &w, cudaStream_t stream)
{
    if (!w.unchecked && !w.captured) return PHYSIM_OK;
    w.unchecked = false;
    uint32_t f = 0;
    PG_CUDA(cudaMemcpyAsync(&f, w.words + 6, sizeof f, cudaMemcpyDeviceToHost, stream));
    PG_CUDA(cudaStreamSynchronize(stream));
    if (f == 0) return PHYSIM_OK;
    PG_CUDA(cudaMemsetAsync(w.words + 6, 0, sizeof f, stream));
    set_error("direct sum: the wait between two steps gave up; results are invalid");
    return PHYSIM_ERR_TIMEOUT;
}

void free_small(SmallWork &w, cudaStream_t stream)
{
    dev_free(w.words, stream);
    dev_free(w.body4, stream);
    w = SmallWork();
}

}  // namespace pg
