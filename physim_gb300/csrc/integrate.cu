// integrate.cu -- body staging and the integrators on the device: verlet
// (integrators/src/verlet.rs:24-107), euler (integrators/src/euler.rs:17-49)
// and rk4 (integrators/src/rk4.rs:24-178).
//
// The integrator runs in f64 with the reference's operation order, written
// with explicit round-to-nearest intrinsics so the compiler cannot contract
// a*b+c into an FMA (Rust does not either).  Given the same accelerations,
// new positions and velocities are therefore bit-identical to the reference.
// The same kernel combines the pair kernel's partial sums, so one launch
// does combine + kick + drift + refresh of the f32 body copy.
#include <string.h>

#include <atomic>

#include "common.cuh"
#include "engine.h"
#include "host_pages.h"
#include "verlet_axis.cuh"

namespace pg {

namespace {

constexpr int kThreads = 256;

inline int blocks_for(size_t n) { return (int)((n + kThreads - 1) / kThreads); }

// Copies `bytes` (a multiple of 8) between global memory -- HBM, or the
// caller's host array reached through the host's page tables -- and shared
// memory with every thread of the block, as consecutive 16-byte words when
// both ends are 16-byte aligned, else 8-byte words.  An array of structs read
// one struct per thread touches a 32-byte sector per 8-byte field; this moves
// whole runs instead, which is what a link to host memory needs.
__device__ __forceinline__ void block_copy(void *dst, const void *src, int bytes)
{
    if (((((uintptr_t)dst | (uintptr_t)src) & 15) == 0) && (bytes & 15) == 0) {
        const int4 *s = (const int4 *)src;
        int4 *d = (int4 *)dst;
        for (int w = threadIdx.x; w < bytes / 16; w += blockDim.x) d[w] = s[w];
    } else {
        const long long *s = (const long long *)src;
        long long *d = (long long *)dst;
        for (int w = threadIdx.x; w < bytes / 8; w += blockDim.x) d[w] = s[w];
    }
}

// |v| as f32 bits, 0 for NaN and infinities (bit patterns order like the
// non-negative values).
__device__ __forceinline__ uint32_t finite_abs_bits(float v)
{
    const uint32_t b = __float_as_uint(v) & 0x7fffffffu;
    return b < 0x7f800000u ? b : 0u;
}

__device__ __forceinline__ uint32_t max_abs_bits(float4 b)
{
    return max(finite_abs_bits(b.x), max(finite_abs_bits(b.y), finite_abs_bits(b.z)));
}

// The half of a maximum (PairScale) that this kernel fills, and the one it
// clears; null: the state keeps none.
struct Track {
    uint32_t *fill = nullptr, *clear = nullptr;
};

// Adds the block's largest `m` to the tracked maximum (every thread of the
// block takes part).
__device__ __forceinline__ void track_max(const Track &t, uint32_t m)
{
    if (!t.fill) return;
    __shared__ uint32_t wm[kThreads / 32];
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = max(m, wm[w]);
        if (m) atomicMax(t.fill, m);
        if (blockIdx.x == 0) *t.clear = 0u;
    }
    __syncthreads();  // wm may serve another maximum
}

__global__ void unpack_kernel(const Entity *__restrict__ in, int n, int n_pad, float4 *body4,
                              uint8_t *fixed, double *x, double *y, double *z, double *vx,
                              double *vy, double *vz, double *m, double *radius, uint64_t *id,
                              Track ext, Track mass, float *mass256)
{
    pdl_trigger();
    static_assert(kThreads == 256, "a block fills one entry of mass256");
    __shared__ __align__(16) Entity s_in[kThreads];
    const int base = blockIdx.x * kThreads;
    const int count = min(kThreads, n - base);  // <= 0 for blocks of the padded tail
    if (count > 0) block_copy(s_in, in + base, count * (int)sizeof(Entity));
    __syncthreads();
    const int i = base + threadIdx.x;  // n_pad is a multiple of the block
    float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n) {
        const Entity &en = s_in[threadIdx.x];
        b4 = make_float4((float)en.x, (float)en.y, (float)en.z, (float)en.mass);
    }
    body4[i] = b4;
    if (ext.fill) {
        track_max(ext, max_abs_bits(b4));
        track_max(mass, finite_abs_bits(b4.w));
        const float m0 = (float)s_in[0].mass;
        const bool same = __syncthreads_and(i < n && b4.w == m0 && fabsf(m0) <= 3.4028235e38f);
        if (threadIdx.x == 0 && mass256)
            mass256[blockIdx.x] = same ? m0 : __int_as_float(0x7fc00000);
    }
    if (i >= n) return;
    const Entity en = s_in[threadIdx.x];
    fixed[i] = en.fixed ? 1 : 0;
    m[i] = en.mass;
    if (x) {
        x[i] = en.x;
        y[i] = en.y;
        z[i] = en.z;
        vx[i] = en.vx;
        vy[i] = en.vy;
        vz[i] = en.vz;
        radius[i] = en.radius;
        id[i] = (uint64_t)en.id;
    }
}

// A block's records leave as one contiguous run: out may be host memory.  flags:
// see accumulate_aos_kernel.
__global__ void pack_kernel(Entity *out, int n, const uint8_t *fixed, const double *x,
                            const double *y, const double *z, const double *vx, const double *vy,
                            const double *vz, const double *m, const double *radius,
                            const uint64_t *id, const uint32_t *flags, uint32_t *flags_out)
{
    __shared__ __align__(16) Entity s_out[kThreads];
    if (flags && blockIdx.x == 0 && threadIdx.x < 4) flags_out[threadIdx.x] = flags[threadIdx.x];
    const int base = blockIdx.x * kThreads;
    const int count = min(kThreads, n - base);
    const int i = base + threadIdx.x;
    if (i < n) {
        Entity en;
        memset(&en, 0, sizeof en);
        en.x = x[i];
        en.y = y[i];
        en.z = z[i];
        en.vx = vx[i];
        en.vy = vy[i];
        en.vz = vz[i];
        en.radius = radius[i];
        en.mass = m[i];
        en.id = (uintptr_t)id[i];
        en.fixed = fixed[i] != 0;
        s_out[threadIdx.x] = en;
    }
    __syncthreads();
    block_copy(out + base, s_out, count * (int)sizeof(Entity));
}

// a_i from the partial sums; zero for fixed bodies (never accumulated);
// NaN for a massless body, whose reference value is F/m_i = 0/0.
__device__ __forceinline__ void body_acc(const double *partial, int splits, int n, int i,
                                         bool fixed, double mass, double &ax, double &ay,
                                         double &az)
{
    ax = ay = az = 0.0;
    if (fixed) return;
    if (splits == 1) {
        // 0 + p without an f64 operation: p, and +0 for -0
        auto plus_zero = [](double p) {
            return __double_as_longlong(p) == (long long)(1ull << 63) ? 0.0 : p;
        };
        ax = plus_zero(partial[i]);
        ay = plus_zero(partial[(size_t)n + i]);
        az = plus_zero(partial[2 * (size_t)n + i]);
        if (mass == 0.0) ax = ay = az = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
    // four splits' loads in flight together (summed in split order): one after
    // another they were a chain of L2 round trips, 6 of 11 us at 17 splits
    constexpr int kAhead = 4;
    for (int s0 = 0; s0 < splits; s0 += kAhead) {
        double p[kAhead][3];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (s0 + u < splits)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    p[u][c] = partial[(size_t)((s0 + u) * 3 + c) * n + i];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (s0 + u < splits) {
                ax += p[u][0];
                ay += p[u][1];
                az += p[u][2];
            }
    }
    if (mass == 0.0) ax = ay = az = __longlong_as_double(0x7ff8000000000000LL);
}

// The block's accelerations are read and written back as one contiguous run;
// a fixed body's entry is written back with the bits it was read with.
// flags: four words that the kernels before this one may have raised, copied to
// host memory (flags_out) on the way.
__global__ void accumulate_aos_kernel(const double *__restrict__ mass, const uint8_t *fixed,
                                      const double *partial, int splits, int n,
                                      Acceleration *acc, const uint32_t *flags,
                                      uint32_t *flags_out)
{
    pdl_wait();
    if (flags && blockIdx.x == 0 && threadIdx.x < 4) flags_out[threadIdx.x] = flags[threadIdx.x];
    __shared__ __align__(16) Acceleration s_acc[kThreads];
    const int base = blockIdx.x * kThreads;
    const int count = min(kThreads, n - base);
    block_copy(s_acc, acc + base, count * (int)sizeof(Acceleration));
    __syncthreads();
    const int i = base + threadIdx.x;
    // transformers.rs:139-141: fixed bodies are left untouched
    if (i < n && !fixed[i]) {
        double ax, ay, az;
        body_acc(partial, splits, n, i, false, mass[i], ax, ay, az);
        Acceleration a = s_acc[threadIdx.x];
        a.x = __dadd_rn(a.x, ax);
        a.y = __dadd_rn(a.y, ay);
        a.z = __dadd_rn(a.z, az);
        s_acc[threadIdx.x] = a;
    }
    __syncthreads();
    block_copy(acc + base, s_acc, count * (int)sizeof(Acceleration));
}

__global__ void combine_soa_kernel(const double *__restrict__ mass, const uint8_t *fixed,
                                   const double *partial, int splits, int n, double *acc)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double ax, ay, az;
    body_acc(partial, splits, n, i, fixed[i] != 0, mass[i], ax, ay, az);
    acc[i] = ax;
    acc[n + i] = ay;
    acc[2 * (size_t)n + i] = az;
}

__global__ void verlet_kernel(float4 *body4, const double *mass, const uint8_t *fixed,
                              const double *partial,
                              int splits, int n, double *x, double *y, double *z, double *vx,
                              double *vy, double *vz, double *px, double *py, double *pz,
                              Divisor dt, int initial, Track ext)
{
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t top = 0;
    if (i < n) {
        float4 b = body4[i];
        double xi = x[i], yi = y[i], zi = z[i];
        double vxi = 0.0, vyi = 0.0, vzi = 0.0, pxi = 0.0, pyi = 0.0, pzi = 0.0;
        if (initial) {  // the Taylor step reads the velocities, the others the positions before
            vxi = vx[i];
            vyi = vy[i];
            vzi = vz[i];
        } else {
            pxi = px[i];
            pyi = py[i];
            pzi = pz[i];
        }
        double ax, ay, az;
        body_acc(partial, splits, n, i, fixed[i] != 0, mass[i], ax, ay, az);
        const double dt2 = __dmul_rn(dt.value, dt.value);
        verlet_axis(xi, vxi, pxi, ax, dt, dt2, initial);
        verlet_axis(yi, vyi, pyi, ay, dt, dt2, initial);
        verlet_axis(zi, vzi, pzi, az, dt, dt2, initial);
        x[i] = xi; y[i] = yi; z[i] = zi;
        vx[i] = vxi; vy[i] = vyi; vz[i] = vzi;
        px[i] = pxi; py[i] = pyi; pz[i] = pzi;
        b.x = (float)xi;
        b.y = (float)yi;
        b.z = (float)zi;
        body4[i] = b;
        top = max_abs_bits(b);
    }
    track_max(ext, top);  // (every thread of the block)
}

__global__ void verlet_aos_kernel(const Entity *in, const Entity *prev, Entity *out, Entity *keep,
                                  const Acceleration *acc, int n, Divisor dt, int initial)
{
    __shared__ __align__(16) Entity s_e[kThreads];
    __shared__ __align__(16) Acceleration s_a[kThreads];
    const int base = blockIdx.x * kThreads;
    const int count = min(kThreads, n - base);
    block_copy(s_e, in + base, count * (int)sizeof(Entity));
    block_copy(s_a, acc + base, count * (int)sizeof(Acceleration));
    __syncthreads();
    if (keep) block_copy(keep + base, s_e, count * (int)sizeof(Entity));
    const int i = base + threadIdx.x;
    double x = 0.0, y = 0.0, z = 0.0, vx = 0.0, vy = 0.0, vz = 0.0;
    if (i < n) {
        const Entity &en = s_e[threadIdx.x];
        x = en.x;
        y = en.y;
        z = en.z;
        vx = en.vx;
        vy = en.vy;
        vz = en.vz;
        const Acceleration a = s_a[threadIdx.x];
        const double dt2 = __dmul_rn(dt.value, dt.value);
        double px = 0.0, py = 0.0, pz = 0.0;
        if (!initial) {
            px = prev[i].x;
            py = prev[i].y;
            pz = prev[i].z;
        }
        verlet_axis(x, vx, px, a.x, dt, dt2, initial);
        verlet_axis(y, vy, py, a.y, dt, dt2, initial);
        verlet_axis(z, vz, pz, a.z, dt, dt2, initial);
    }
    __syncthreads();  // every read of s_e (the keep copy) is done
    // Only the six updated fields are rewritten: every other byte of the
    // output record, struct padding included, is the input's.
    if (i < n) {
        Entity &en = s_e[threadIdx.x];
        en.x = x;
        en.y = y;
        en.z = z;
        en.vx = vx;
        en.vy = vy;
        en.vz = vz;
    }
    __syncthreads();
    block_copy(out + base, s_e, count * (int)sizeof(Entity));
}

// euler.rs:29-37: x + vx*dt + 0.5*a*dt^2 ; vx + a*dt for every body.  A fixed
// body has a = 0 (transforms skip it) and still drifts with its velocity.
__global__ void euler_kernel(float4 *body4, const double *mass, const uint8_t *fixed,
                             const double *partial, int splits, int n, double *x, double *y,
                             double *z, double *vx, double *vy, double *vz, Divisor dt, Track ext)
{
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t top = 0;
    if (i < n) {
        float4 b = body4[i];
        double ax, ay, az;
        body_acc(partial, splits, n, i, fixed[i] != 0, mass[i], ax, ay, az);
        const double dt2 = __dmul_rn(dt.value, dt.value);
        double xi = x[i], yi = y[i], zi = z[i];
        double vxi = vx[i], vyi = vy[i], vzi = vz[i];
        double unused = 0.0;
        verlet_axis(xi, vxi, unused, ax, dt, dt2, true);
        verlet_axis(yi, vyi, unused, ay, dt, dt2, true);
        verlet_axis(zi, vzi, unused, az, dt, dt2, true);
        x[i] = xi; y[i] = yi; z[i] = zi;
        vx[i] = vxi; vy[i] = vyi; vz[i] = vzi;
        b.x = (float)xi;
        b.y = (float)yi;
        b.z = (float)zi;
        body4[i] = b;
        top = max_abs_bits(b);
    }
    track_max(ext, top);  // (every thread of the block)
}

// One RK4 stage (rk4.rs:33-178) for body i, given the stage state q (x, y, z,
// vx, vy, vz), its acceleration a, the entity's own state e and the running
// sum S of the k's.  k = (dt v_q, dt a) (rk4.rs:40-46); S accumulates
// k1 + 2 k2 + 2 k3 + k4 left to right, as rk4.rs:160-165 evaluates it.
// Stages 1-3 return the next stage state e + k/2 (stages 1, 2) or e + k
// (stage 3); stage 4 returns the new state e + S/6, or (e, v = 0) for a fixed
// body (rk4.rs:165-171).
__device__ __forceinline__ void rk4_stage(int stage, const double q[6], const double a[3],
                                          const double e[6], double S[6], bool fixed, double dt,
                                          const Divisor &six, double out[6])
{
    double k[6];
    for (int c = 0; c < 3; ++c) {
        k[c] = __dmul_rn(dt, q[3 + c]);
        k[3 + c] = __dmul_rn(dt, a[c]);
    }
    for (int c = 0; c < 6; ++c) {
        if (stage == 1)
            S[c] = k[c];
        else if (stage == 4)
            S[c] = __dadd_rn(S[c], k[c]);
        else
            S[c] = __dadd_rn(S[c], __dmul_rn(2.0, k[c]));
    }
    if (stage < 3) {
        for (int c = 0; c < 6; ++c) out[c] = __dadd_rn(e[c], __dmul_rn(0.5, k[c]));
    } else if (stage == 3) {
        for (int c = 0; c < 6; ++c) out[c] = __dadd_rn(e[c], k[c]);
    } else if (!fixed) {
        for (int c = 0; c < 6; ++c) out[c] = __dadd_rn(e[c], divide(S[c], six));
    } else {
        for (int c = 0; c < 3; ++c) {
            out[c] = e[c];
            out[3 + c] = 0.0;
        }
    }
}

// Device-resident RK4 stage: the stage state is in (x .. vz) and body4; the
// entity's state is saved in `save` at stage 1; S lives in `ksum`.  Writes
// the next stage state (or the new state) back to (x .. vz) and body4, so
// the next force evaluation reads it like any other state.
__global__ void rk4_stage_kernel(float4 *body4, const double *mass, const uint8_t *fixed,
                                 const double *partial, int splits, int n, double *x, double *y,
                                 double *z, double *vx, double *vy, double *vz, double *save,
                                 double *ksum, double dt, int stage, Divisor six, Track ext)
{
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t top = 0;
    if (i < n) {
        const bool fx = fixed[i] != 0;
        double a[3];
        body_acc(partial, splits, n, i, fx, mass[i], a[0], a[1], a[2]);
        double *st[6] = {x, y, z, vx, vy, vz};
        double q[6], e[6], S[6], out[6];
        for (int c = 0; c < 6; ++c) q[c] = st[c][i];
        if (stage == 1) {
            for (int c = 0; c < 6; ++c) {
                e[c] = q[c];
                save[(size_t)c * n + i] = q[c];
            }
        } else {
            for (int c = 0; c < 6; ++c) {
                e[c] = save[(size_t)c * n + i];
                S[c] = ksum[(size_t)c * n + i];
            }
        }
        rk4_stage(stage, q, a, e, S, fx, dt, six, out);
        if (stage < 4)
            for (int c = 0; c < 6; ++c) ksum[(size_t)c * n + i] = S[c];
        for (int c = 0; c < 6; ++c) st[c][i] = out[c];
        float4 b = body4[i];
        b.x = (float)out[0];
        b.y = (float)out[1];
        b.z = (float)out[2];
        body4[i] = b;
        top = max_abs_bits(b);
    }
    track_max(ext, top);  // (every thread of the block)
}

__global__ void euler_aos_kernel(const Entity *in, Entity *out, const Acceleration *acc, int n,
                                 Divisor dt)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Entity en = in[i];
    const Acceleration a = acc[i];
    const double dt2 = __dmul_rn(dt.value, dt.value);
    double unused = 0.0;
    verlet_axis(en.x, en.vx, unused, a.x, dt, dt2, true);
    verlet_axis(en.y, en.vy, unused, a.y, dt, dt2, true);
    verlet_axis(en.z, en.vz, unused, a.z, dt, dt2, true);
    out[i] = en;
}

// RK4 stage over Entity arrays: `ent` the entities, `q` the stage state, f
// its accelerations; writes the next stage state (stages 1-3: the entity with
// x, v replaced, rk4.rs:50-62) or the new state (stage 4) to `out`, which may
// alias q.
__global__ void rk4_aos_stage_kernel(const Entity *ent, const Entity *q_in,
                                     const Acceleration *f, double *ksum, Entity *out, int n,
                                     double dt, int stage, Divisor six)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Entity en = ent[i];
    const Entity qe = q_in[i];
    const Acceleration fa = f[i];
    const double q[6] = {qe.x, qe.y, qe.z, qe.vx, qe.vy, qe.vz};
    const double e[6] = {en.x, en.y, en.z, en.vx, en.vy, en.vz};
    const double a[3] = {fa.x, fa.y, fa.z};
    double S[6] = {0, 0, 0, 0, 0, 0}, r[6];
    if (stage > 1)
        for (int c = 0; c < 6; ++c) S[c] = ksum[(size_t)c * n + i];
    rk4_stage(stage, q, a, e, S, en.fixed, dt, six, r);
    if (stage < 4)
        for (int c = 0; c < 6; ++c) ksum[(size_t)c * n + i] = S[c];
    Entity o = en;
    o.x = r[0]; o.y = r[1]; o.z = r[2];
    o.vx = r[3]; o.vy = r[4]; o.vz = r[5];
    out[i] = o;
}

}  // namespace

int dev_alloc_bytes(void **p, size_t bytes, cudaStream_t stream)
{
    *p = nullptr;
    int device = 0;
    if (cudaGetDevice(&device) == cudaSuccess && device >= 0 && device < 64) {
        // keep freed blocks in the device's default pool for reuse (a
        // setting of this process's pool only)
        static bool pool_set[64] = {false};
        if (!pool_set[device]) {
            cudaMemPool_t pool;
            if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
                uint64_t keep = ~0ull;
                cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
            }
            pool_set[device] = true;
        }
    }
    cudaError_t err = cudaMallocAsync(p, bytes ? bytes : 1, stream);
    if (err != cudaSuccess) {
        *p = nullptr;
        set_error("device allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(err));
        return PHYSIM_ERR_MEMORY;
    }
    return PHYSIM_OK;
}

void dev_free(void *p, cudaStream_t stream)
{
    if (p) cudaFreeAsync(p, stream);
}

namespace {
std::atomic<uint32_t> g_host_access{PHYSIM_HOST_ACCESS_AUTO};
std::atomic<int> g_pageable[64];  // 0 unknown, 1 no, 2 yes
}  // namespace

int host_direct(int device, bool *direct)
{
    *direct = false;
    const uint32_t mode = g_host_access.load(std::memory_order_relaxed);
    if (mode == PHYSIM_HOST_ACCESS_COPY) return PHYSIM_OK;
    PG_CHECK(device >= 0 && device < 64, PHYSIM_ERR_ARGUMENT, "device %d out of range", device);
    int known = g_pageable[device].load(std::memory_order_relaxed);
    if (known == 0) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrPageableMemoryAccessUsesHostPageTables,
                                   device) != cudaSuccess)
            v = 0;
        known = v ? 2 : 1;
        g_pageable[device].store(known, std::memory_order_relaxed);
    }
    PG_CHECK(known == 2 || mode == PHYSIM_HOST_ACCESS_AUTO, PHYSIM_ERR_ARGUMENT,
             "host access DIRECT: device %d does not reach pageable host memory through the "
             "host's page tables",
             device);
    *direct = known == 2;
    return PHYSIM_OK;
}

int download_direct(int device, const void *p, size_t bytes, bool *direct)
{
    PG_TRY(host_direct(device, direct));
    *direct = *direct && ((uintptr_t)p & 7) == 0 && bytes <= (size_t(32) << 20) &&
              populate_pages(p, bytes, true);
    return PHYSIM_OK;
}

void bodies_free(DeviceBodies &b, cudaStream_t stream)
{
    void *ptrs[] = {b.body4, b.fixed, b.x,  b.y,  b.z,      b.vx, b.vy,    b.vz,
                    b.px,    b.py,    b.pz, b.m,  b.radius, b.id, b.aos, b.scale, b.mass256};
    for (void *p : ptrs) dev_free(p, stream);
    b = DeviceBodies();
}

int bodies_reserve(DeviceBodies &b, size_t n, bool with_state, bool with_scale,
                   cudaStream_t stream)
{
    size_t need = pad_bodies(n);
    if (need <= b.cap && (!with_state || b.x) && (!with_scale || b.scale)) {
        b.n = n;
        return PHYSIM_OK;
    }
    bodies_free(b, stream);
    b.cap = need;
    b.n = n;
    PG_TRY(dev_alloc(b.body4, need, stream));
    PG_TRY(dev_alloc(b.fixed, need, stream));
    PG_TRY(dev_alloc(b.aos, need, stream));
    PG_TRY(dev_alloc(b.m, need, stream));
    if (with_scale) {
        PG_TRY(dev_alloc(b.scale, 1, stream));
        PG_CUDA(cudaMemsetAsync(b.scale, 0, sizeof(PairScale), stream));
        PG_TRY(dev_alloc(b.mass256, need / kThreads, stream));
    }
    if (with_state) {
        double **d[] = {&b.x, &b.y, &b.z, &b.vx, &b.vy, &b.vz, &b.px, &b.py, &b.pz, &b.radius};
        for (double **p : d) PG_TRY(dev_alloc(*p, need, stream));
        PG_TRY(dev_alloc(b.id, need, stream));
    }
    return PHYSIM_OK;
}

namespace {

// The tracked halves of the largest |coordinate|; they change places once the
// kernel is launched.
Track next_extent(const DeviceBodies &b)
{
    if (!b.scale) return Track();
    return {&b.scale->ext[b.ext_half ^ 1], &b.scale->ext[b.ext_half]};
}

__global__ void settle_kernel(uint32_t *ext, int eh, uint32_t *mass, int mh)
{
    ext[eh] = ext[eh ^ 1];
    ext[eh ^ 1] = 0u;
    if (mass) {
        mass[mh] = mass[mh ^ 1];
        mass[mh ^ 1] = 0u;
    }
}

// After a kernel that filled the other halves: they are current from here on, or,
// once a caller has captured such a kernel (its graph may be launched any number of
// times, between other steps and uploads), the values move back into the halves
// that its kernels read.
int swap_halves(DeviceBodies &b, bool mass_too, cudaStream_t stream)
{
    PG_CUDA(cudaGetLastError());
    if (!b.scale) return PHYSIM_OK;
    if (!b.swap_in_capture) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        PG_CUDA(cudaStreamIsCapturing(stream, &cs));
        if (cs != cudaStreamCaptureStatusNone) b.halves_fixed = true;
        if (b.halves_fixed) {
            settle_kernel<<<1, 1, 0, stream>>>(b.scale->ext, b.ext_half,
                                               mass_too ? b.scale->mass : nullptr, b.mass_half);
            PG_CUDA(cudaGetLastError());
            return PHYSIM_OK;
        }
    }
    b.ext_half ^= 1;
    if (mass_too) b.mass_half ^= 1;
    return PHYSIM_OK;
}

// Threads per block of the integrators: small states in small blocks, over more
// SMs, as the f64 pipe bounds them (73% of the cycles at 262,148 bodies).  Steps of
// Barnes-Hut simulations with blocks of 64 / 256 (us): 2,000 bodies 37.3 / 38.3,
// 30,000 65.3 / 67.1, rk4 262 / 270; 40,000 70.2 / 70.1, rk4 285 / 282; 100,003 87.2 /
// 87.3, rk4 353 / 350; 400,009 152.9 / 153.2.
int integrator_threads(size_t n) { return n <= 40000 ? 64 : kThreads; }

int integrator_blocks(size_t n)
{
    const size_t t = (size_t)integrator_threads(n);
    return (int)((n + t - 1) / t);
}

}  // namespace

int launch_unpack(DeviceBodies &b, const Entity *aos, size_t n, bool full_state,
                  cudaStream_t stream)
{
    size_t n_pad = pad_bodies(n);
    if (n_pad == 0) return PHYSIM_OK;
    Track mass;
    if (b.scale) mass = {&b.scale->mass[b.mass_half ^ 1], &b.scale->mass[b.mass_half]};
    unpack_kernel<<<blocks_for(n_pad), kThreads, 0, stream>>>(
        aos, (int)n, (int)n_pad, b.body4, b.fixed, full_state ? b.x : nullptr, b.y, b.z, b.vx,
        b.vy, b.vz, b.m, b.radius, b.id, next_extent(b), mass, b.mass256);
    return swap_halves(b, true, stream);
}

int launch_pack(DeviceBodies &b, Entity *out, cudaStream_t stream, const uint32_t *flags,
                uint32_t *flags_out)
{
    if (b.n == 0) return PHYSIM_OK;
    pack_kernel<<<blocks_for(b.n), kThreads, 0, stream>>>(out, (int)b.n, b.fixed, b.x, b.y, b.z,
                                                            b.vx, b.vy, b.vz, b.m, b.radius, b.id,
                                                            flags, flags_out);
    PG_CUDA(cudaGetLastError());
    return PHYSIM_OK;
}

int launch_accumulate_aos(const DeviceBodies &b, const double *partial, int splits,
                          Acceleration *d_acc, cudaStream_t stream, const uint32_t *flags,
                          uint32_t *flags_out)
{
    if (b.n == 0) return PHYSIM_OK;
    // (as dependent launches, this and the small force kernel: 1,002 bodies 57 -> 51 us
    // per pipeline step, 50,021 by quadtree 271 -> 264; the pair sums' reduction gains
    // nothing by it, rk4 of 16,387 1,804 -> 1,824)
    return launch_pdl(accumulate_aos_kernel, blocks_for(b.n), kThreads, stream, b.m, b.fixed,
                      partial, splits, (int)b.n, d_acc, flags, flags_out);
}

int launch_combine_soa(const DeviceBodies &b, const double *partial, int splits,
                       double *acc_soa, cudaStream_t stream)
{
    if (b.n == 0) return PHYSIM_OK;
    combine_soa_kernel<<<blocks_for(b.n), kThreads, 0, stream>>>(b.m, b.fixed, partial,
                                                                   splits, (int)b.n, acc_soa);
    PG_CUDA(cudaGetLastError());
    return PHYSIM_OK;
}

int launch_verlet(DeviceBodies &b, const double *partial, int splits, double dt, bool initial,
                  cudaStream_t stream)
{
    if (b.n == 0) return PHYSIM_OK;
    PG_TRY(launch_pdl(verlet_kernel, integrator_blocks(b.n), integrator_threads(b.n), stream,
                      b.body4, b.m, b.fixed, partial, splits, (int)b.n, b.x, b.y, b.z, b.vx, b.vy,
                      b.vz, b.px, b.py, b.pz, make_divisor(dt), initial ? 1 : 0, next_extent(b)));
    return swap_halves(b, false, stream);
}

int launch_euler(DeviceBodies &b, const double *partial, int splits, double dt,
                 cudaStream_t stream)
{
    if (b.n == 0) return PHYSIM_OK;
    PG_TRY(launch_pdl(euler_kernel, integrator_blocks(b.n), integrator_threads(b.n), stream,
                      b.body4, b.m, b.fixed, partial, splits, (int)b.n, b.x, b.y, b.z, b.vx, b.vy,
                      b.vz, make_divisor(dt), next_extent(b)));
    return swap_halves(b, false, stream);
}

int launch_rk4_stage(DeviceBodies &b, const double *partial, int splits, double dt, int stage,
                     double *save, double *ksum, cudaStream_t stream)
{
    if (b.n == 0) return PHYSIM_OK;
    PG_CHECK(stage >= 1 && stage <= 4, PHYSIM_ERR_ARGUMENT, "rk4 stage %d", stage);
    PG_TRY(launch_pdl(rk4_stage_kernel, integrator_blocks(b.n), integrator_threads(b.n), stream,
                      b.body4, b.m, b.fixed, partial, splits, (int)b.n, b.x, b.y, b.z, b.vx, b.vy,
                      b.vz, save, ksum, dt, stage, make_divisor(6.0), next_extent(b)));
    return swap_halves(b, false, stream);
}

int launch_euler_aos(const Entity *d_in, Entity *d_out, const Acceleration *d_acc, size_t n,
                     double dt, cudaStream_t stream)
{
    if (n == 0) return PHYSIM_OK;
    euler_aos_kernel<<<blocks_for(n), kThreads, 0, stream>>>(d_in, d_out, d_acc, (int)n,
                                                             make_divisor(dt));
    PG_CUDA(cudaGetLastError());
    return PHYSIM_OK;
}

int launch_rk4_aos_stage(const Entity *d_ent, const Entity *d_q, const Acceleration *d_f,
                         double *ksum, Entity *d_out, size_t n, double dt, int stage,
                         cudaStream_t stream)
{
    if (n == 0) return PHYSIM_OK;
    PG_CHECK(stage >= 1 && stage <= 4, PHYSIM_ERR_ARGUMENT, "rk4 stage %d", stage);
    rk4_aos_stage_kernel<<<blocks_for(n), kThreads, 0, stream>>>(d_ent, d_q, d_f, ksum, d_out,
                                                                 (int)n, dt, stage, make_divisor(6.0));
    PG_CUDA(cudaGetLastError());
    return PHYSIM_OK;
}

int launch_verlet_aos(const Entity *in, const Entity *d_prev, Entity *out, Entity *keep,
                      const Acceleration *acc, size_t n, double dt, bool initial,
                      cudaStream_t stream)
{
    if (n == 0) return PHYSIM_OK;
    verlet_aos_kernel<<<blocks_for(n), kThreads, 0, stream>>>(in, d_prev, out, keep, acc, (int)n,
                                                              make_divisor(dt), initial ? 1 : 0);
    PG_CUDA(cudaGetLastError());
    return PHYSIM_OK;
}

}  // namespace pg

void pg::host_prefault(const void *p, size_t bytes, bool write)
{
    (void)populate_pages(p, bytes, write);
}

extern "C" int physim_gpu_set_host_access(uint32_t mode)
{
    PG_CHECK(mode <= PHYSIM_HOST_ACCESS_DIRECT, PHYSIM_ERR_ARGUMENT, "unknown host access mode %u",
             mode);
    pg::g_host_access.store(mode);
    return PHYSIM_OK;
}

extern "C" int physim_gpu_host_access(int32_t device, uint32_t *mode)
{
    PG_CHECK(mode, PHYSIM_ERR_ARGUMENT, "null argument");
    bool direct = false;
    PG_TRY(pg::host_direct(device, &direct));
    *mode = direct ? PHYSIM_HOST_ACCESS_DIRECT : PHYSIM_HOST_ACCESS_COPY;
    return PHYSIM_OK;
}
