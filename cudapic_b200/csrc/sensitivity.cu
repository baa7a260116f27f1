// sensitivity.cu -- voltage sensitivities of time-averaged observables of one
// discharge by a pathwise adjoint, with collision events and random draws
// frozen: forward run with checkpoints, segment-wise recompute with a tape,
// reverse sweep (cudapic_sens_* in include/cudapic.h).
//
// Model: the slot form of the reference step (Rust-CUDA/src/main.rs:1725-1808):
// the same kernels in the same order -- densities, Poisson, electron push,
// ion push every N_SUB-th step, electron collisions with their spawns, ion
// collisions -- with particles kept in their slots.  An absorbed particle is
// marked dead (x = -1) instead of being compacted away, and the spawns of a
// step take the next free slots in the slot order of their parents (a chunk
// count, a scan, a ranked write), so each particle keeps one RNG stream for
// its whole life and a run is a deterministic function of the initial state
// and the voltage: recompute from a checkpoint reproduces the trajectory bit
// for bit.  Deposits are exact integer sums (2^-20 fixed point), the Poisson
// sums FP64, scattering uses the algebraic sines and cosines.
//
// Observables (time averages over the window of K steps):
//   J_P  <j E> electron power averaged over the gap [W m^-3] (C/eduPIC.cc:
//        593-614, 1011-1026, per particle): -e (W/A) / L / K * sum over steps
//        and electrons of (v + f E(x)/2) E(x);
//   J_G  ion flux to the grounded electrode [m^-2 s^-1]: the CIC flux density
//        n v at node N_G-1 (boundary node doubled, as the density), a smooth
//        estimate of the counted flux of C/eduPIC.cc:651-658.
//
// Step kernels: one forward step is three launches -- the field (node sums to
// densities, the solve, the step's marks: one CTA), the electrons (push,
// collisions and the next step's deposit in one pass over the slots) and the
// spawns -- and four more on an ion step.  At 2e5 particles every one of them
// is a few microseconds of latency, so what counts is their number and that
// programmatic dependent launch overlaps each one's launch with the previous
// one's tail (every kernel waits before its first global access).  The
// backward pass recomputes each checkpoint interval once and sweeps the
// adjoints of both observables through it together: they share the tape, the
// records and the collision Jacobians.  2e5 + 2e5 particles, 200 steps:
// forward 3.6 ms, backward 10.2 ms (with seven launches per forward step, no
// overlap and a recompute per observable: 8.5 and 32.7 ms).
//
// Adjoint kernels: push (field gather -> its adjoint scatters into the field
// adjoint, FP64 shared-memory sums), collisions (Jacobians by forward-mode
// tangents of the same scattering arithmetic, applied transposed), spawns
// (a child's adjoint flows back to its parent), the symmetric Poisson solve
// (the same two-scan closed form, in kernels_poisson.cu), deposit (a gather).
// Particle adjoints in f32, the field, density and voltage adjoints in FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "detmath.cuh"
#include "internal.h"
#include "mcc.cuh"
#include "poisson.cuh"
#include "push.cuh"
#include "state_impl.h"
#include "step.cuh"

namespace cudapic {

namespace {

constexpr int SENS_THREADS = 256;
constexpr int SENS_PER_SM = 4;
constexpr uint32_t SENS_CHUNK = 1024;      // spawn-order chunk (one CTA of the spawn write)
constexpr uint32_t NO_SPAWN = 0xFFFFFFFFu;
constexpr uint32_t SPAWN_NOREC = 0xFFFFFFFEu;
constexpr uint32_t NO_SLOT = 0xFFFFFFFFu;
// The kernels that sum over the particles into node histograms: one CTA per SM
// and as many threads as give every particle one (256 to 1024), because each
// CTA ends with an atomic per node.  With four CTAs of 256 per SM, 200 000
// electrons made 240 000 (deposit) and 470 000 (adjoint push) of them a step:
// 13.9 ms per forward and backward pass of 200 steps, now 11.9.
constexpr int SENS_WIDE = 1024;
constexpr uint32_t SENS_MAX_NG = 4096;

// counters block
enum : int { C_NE = 0, C_NI, C_REC_E, C_REC_I, C_ERR, C_N0E, C_N0I, C_PAD, C_COUNT };

struct SensRecE {
    uint32_t p, ev, ce, ci;
    float v[3];
    float a, eta;   // a: cos chi draw 1 - 2u (ev 1, 2) or the energy-sharing draw u (ev 3)
};

struct SensRecI {
    uint32_t p, ev;
    float v[3], t[3];  // pre-collision velocity, target atom velocity
    float c, eta;      // c: cos chi draw (ev 4)
};

struct Planes {
    float *x, *vx, *vy, *vz;
    uint32_t *r[4];
};

// ---------------------------------------------------------------- tangents
// Forward-mode derivative in three directions (d/dvx, d/dvy, d/dvz).
struct D3 {
    float v, d0, d1, d2;
};
__device__ __forceinline__ D3 dc(float c) { return {c, 0.0f, 0.0f, 0.0f}; }
__device__ __forceinline__ D3 operator+(D3 a, D3 b) { return {a.v + b.v, a.d0 + b.d0, a.d1 + b.d1, a.d2 + b.d2}; }
__device__ __forceinline__ D3 operator-(D3 a, D3 b) { return {a.v - b.v, a.d0 - b.d0, a.d1 - b.d1, a.d2 - b.d2}; }
__device__ __forceinline__ D3 operator-(D3 a) { return {-a.v, -a.d0, -a.d1, -a.d2}; }
__device__ __forceinline__ D3 operator*(D3 a, D3 b) {
    return {a.v * b.v, a.d0 * b.v + a.v * b.d0, a.d1 * b.v + a.v * b.d1, a.d2 * b.v + a.v * b.d2};
}
__device__ __forceinline__ D3 operator*(float a, D3 b) { return {a * b.v, a * b.d0, a * b.d1, a * b.d2}; }
__device__ __forceinline__ D3 operator*(D3 a, float b) { return {a.v * b, a.d0 * b, a.d1 * b, a.d2 * b}; }
__device__ __forceinline__ D3 operator/(D3 a, D3 b) {
    const float q = a.v / b.v;
    return {q, (a.d0 - q * b.d0) / b.v, (a.d1 - q * b.d1) / b.v, (a.d2 - q * b.d2) / b.v};
}
__device__ __forceinline__ D3 operator/(D3 a, float b) { return {a.v / b, a.d0 / b, a.d1 / b, a.d2 / b}; }
__device__ __forceinline__ D3 operator-(float a, D3 b) { return {a - b.v, -b.d0, -b.d1, -b.d2}; }
__device__ __forceinline__ D3 operator+(float a, D3 b) { return {a + b.v, b.d0, b.d1, b.d2}; }
__device__ __forceinline__ D3 operator+(D3 a, float b) { return {a.v + b, a.d0, a.d1, a.d2}; }
__device__ __forceinline__ D3 operator-(D3 a, float b) { return {a.v - b, a.d0, a.d1, a.d2}; }
__device__ __forceinline__ float val(float a) { return a; }
__device__ __forceinline__ float val(const D3 &a) { return a.v; }
__device__ __forceinline__ float tsqrt(float a) { return sqrtf(a); }
__device__ __forceinline__ D3 tsqrt(D3 a) {
    const float s = sqrtf(a.v);
    const float k = s > 0.0f ? 0.5f / s : 0.0f;
    return {s, a.d0 * k, a.d1 * k, a.d2 * k};
}
__device__ __forceinline__ float tfabs(float a) { return fabsf(a); }
__device__ __forceinline__ D3 tfabs(D3 a) { return a.v < 0.0f ? -a : a; }
__device__ __forceinline__ float ttan(float a) { return dm::tanf_det(a); }
__device__ __forceinline__ D3 ttan(D3 a) {
    const float t = dm::tanf_det(a.v);
    const float k = 1.0f + t * t;
    return {t, a.d0 * k, a.d1 * k, a.d2 * k};
}
__device__ __forceinline__ float tatan(float a) { return dm::atanf_det(a); }
__device__ __forceinline__ D3 tatan(D3 a) {
    const float k = 1.0f / (1.0f + a.v * a.v);
    return {dm::atanf_det(a.v), a.d0 * k, a.d1 * k, a.d2 * k};
}
template <typename T> __device__ __forceinline__ T tconst(float c);
template <> __device__ __forceinline__ float tconst<float>(float c) { return c; }
template <> __device__ __forceinline__ D3 tconst<D3>(float c) { return dc(c); }

// --------------------------------------------------------------- scattering
struct ScatK {
    float f1, f2;
};

template <typename T>
__device__ __forceinline__ void euler_alg_t(T gx, T gy, T gz, T &st, T &ct, T &sp, T &cp) {
    const T r2 = gy * gy + gz * gz;
    const T r = tsqrt(r2);
    if (val(gx) == 0.0f) {
        st = tconst<T>(1.0f);
        ct = tconst<T>(0.0f);
    } else {
        const T gn = tsqrt(gx * gx + r2);
        st = r / gn;
        ct = gx / gn;
    }
    if (val(gy) == 0.0f) {
        sp = tconst<T>(val(gz) > 0.0f ? 1.0f : -1.0f);
        cp = tconst<T>(0.0f);
    } else {
        sp = gz / r;
        cp = gy / r;
    }
}

template <typename T>
__device__ __forceinline__ void sincos_acos_t(T c, T &s, T &co) {
    const T t = (1.0f - c) * (1.0f + c);
    s = val(t) > 0.0f ? tsqrt(t) : tconst<T>(0.0f);
    co = c;
}

template <typename T>
__device__ __forceinline__ void rot_t(T g, T sc, T cc, float se, float ce, T st, T ct, T sp, T cp, T &ox, T &oy,
                                      T &oz) {
    ox = g * (ct * cc - st * sc * ce);
    oy = g * (st * cp * cc + ct * cp * sc * ce - sp * sc * se);
    oz = g * (st * sp * cc + ct * sp * sc * ce + cp * sc * se);
}

// collision_e (Rust-CUDA/src/main.rs:1035-1165) with the algebraic sines and
// cosines and the draws given (ev 1 elastic / 2 excitation: a = 1 - 2u is
// cos chi; ev 3 ionization: a = the energy-sharing draw u; eta = 2 pi u):
// out = the scattered velocity, child (ev 3) = the new electron.  T = float
// is the forward arithmetic, T = D3 its tangents.
template <typename T>
__device__ void scatter_e_t(const ScatK &k, const T v[3], int ev, float a, float eta, T out[3], T child[3]) {
    const float exc_j = 11.5f * E_CHARGE_F;
    const float ion_j = 15.8f * E_CHARGE_F;
    const T gx = v[0], gy = v[1], gz = v[2];
    T gm = tsqrt(gx * gx + gy * gy + gz * gz);
    const T wx = k.f1 * gx, wy = k.f1 * gy, wz = k.f1 * gz;
    T st, ct, sp, cp;
    euler_alg_t(gx, gy, gz, st, ct, sp, cp);
    T chi_s, chi_c;
    float se, ce;
    if (ev == 1) {
        sincos_acos_t(tconst<T>(a), chi_s, chi_c);
    } else if (ev == 2) {
        T en = 0.5f * E_MASS_F * gm * gm;
        en = tfabs(en - exc_j);
        gm = tsqrt(2.0f * en / E_MASS_F);
        sincos_acos_t(tconst<T>(a), chi_s, chi_c);
    } else {
        T en = 0.5f * E_MASS_F * gm * gm;
        en = tfabs(en - ion_j);
        const T e_new = 10.0f * ttan(a * tatan(en / E_CHARGE_F / 20.0f)) * E_CHARGE_F;
        const T e_orig = tfabs(en - e_new);
        gm = tsqrt(2.0f * e_orig / E_MASS_F);
        const T g_new = tsqrt(2.0f * e_new / E_MASS_F);
        T sc2, cc2, nx, ny, nz;
        sincos_acos_t(tsqrt(e_new / en), sc2, cc2);
        dm::sincosf_det(eta, &se, &ce);
        rot_t(g_new, sc2, cc2, -se, -ce, st, ct, sp, cp, nx, ny, nz);
        child[0] = wx + k.f2 * nx;
        child[1] = wy + k.f2 * ny;
        child[2] = wz + k.f2 * nz;
        sincos_acos_t(tsqrt(e_orig / en), chi_s, chi_c);
    }
    if (ev != 3) dm::sincosf_det(eta, &se, &ce);
    T nx, ny, nz;
    rot_t(gm, chi_s, chi_c, se, ce, st, ct, sp, cp, nx, ny, nz);
    out[0] = wx + k.f2 * nx;
    out[1] = wy + k.f2 * ny;
    out[2] = wz + k.f2 * nz;
}

// collision_i (Rust-CUDA/src/main.rs:1221-1292) with the algebraic sines and
// cosines: ev 4 isotropic (c = cos chi), ev 5 backscatter (chi = pi exactly).
template <typename T>
__device__ void scatter_i_t(const T v[3], const float t[3], int ev, float c, float eta, T out[3]) {
    const T gx = v[0] - t[0], gy = v[1] - t[1], gz = v[2] - t[2];
    const T gg = tsqrt(gx * gx + gy * gy + gz * gz);
    const T wx = 0.5f * (v[0] + t[0]), wy = 0.5f * (v[1] + t[1]), wz = 0.5f * (v[2] + t[2]);
    T st, ct, sp, cp, sc, cc;
    euler_alg_t(gx, gy, gz, st, ct, sp, cp);
    if (ev == 4) {
        sincos_acos_t(tconst<T>(c), sc, cc);
    } else {
        sc = tconst<T>(0.0f);
        cc = tconst<T>(-1.0f);
    }
    float se, ce;
    dm::sincosf_det(eta, &se, &ce);
    T nx, ny, nz;
    rot_t(gg, sc, cc, se, ce, st, ct, sp, cp, nx, ny, nz);
    out[0] = wx + 0.5f * nx;
    out[1] = wy + 0.5f * ny;
    out[2] = wz + 0.5f * nz;
}

__device__ __forceinline__ D3 seed(float v, int k) {
    return {v, k == 0 ? 1.0f : 0.0f, k == 1 ? 1.0f : 0.0f, k == 2 ? 1.0f : 0.0f};
}

// w^T J: the adjoint of the inputs given the adjoint w of the outputs.
__device__ __forceinline__ void apply_jt(const D3 out[3], const float w[3], float r[3]) {
    r[0] = out[0].d0 * w[0] + out[1].d0 * w[1] + out[2].d0 * w[2];
    r[1] = out[0].d1 * w[0] + out[1].d1 * w[1] + out[2].d1 * w[2];
    r[2] = out[0].d2 * w[0] + out[1].d2 * w[1] + out[2].d2 * w[2];
}

__device__ __forceinline__ double block_sum(double v, double *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    return s;
}

// ------------------------------------------------------------------ forward
// The CTA's deposit: 2^-20 fixed-point weights (push.cuh dep_add) in a 32-bit
// shared histogram (five times the rate of 64-bit shared atomics), drained
// into 64-bit sums before a node can overflow.  Dynamic shared memory:
// [n_g] u64, [n_g] u32.  The node sums are exact, so neither the order nor the
// split over CTAs matters.
struct SensDep {
    unsigned long long *acc;
    uint32_t *h;
    uint32_t n_g;
    __device__ __forceinline__ SensDep(unsigned long long *smem, uint32_t n) : acc(smem), n_g(n) {
        h = reinterpret_cast<uint32_t *>(smem + n);
        for (uint32_t k = threadIdx.x; k < n_g; k += blockDim.x) {
            acc[k] = 0ull;
            h[k] = 0u;
        }
        __syncthreads();
    }
    // before round r of the CTA (every thread calls it)
    __device__ __forceinline__ void round(uint32_t r) {
        if (r == 0 || r % (DEP_MAX_PER_COPY / blockDim.x) != 0) return;
        __syncthreads();
        dep_drain(h, 1, n_g, acc, n_g);
        __syncthreads();
    }
    __device__ __forceinline__ void flush(unsigned long long *hist) {
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < n_g; k += blockDim.x) {
            const unsigned long long v = acc[k] + h[k];
            if (v) atomicAdd(&hist[k], v);
        }
    }
};
size_t dep_smem(uint32_t n_g) { return (size_t)n_g * (sizeof(unsigned long long) + sizeof(uint32_t)); }

__global__ void __launch_bounds__(SENS_WIDE)
    sens_deposit_kernel(const float *__restrict__ x, const uint32_t *__restrict__ n_ptr,
                        unsigned long long *__restrict__ hist, const __grid_constant__ cudapic_grid g) {
    extern __shared__ unsigned long long sens_sm[];
    SensDep dep(sens_sm, g.n_g);
    grid_dep_wait();
    const uint32_t n = min(*n_ptr, g.capacity);
    const uint32_t stride = gridDim.x * blockDim.x;
    uint32_t r = 0;
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < n; b += stride, ++r) {
        dep.round(r);
        const uint64_t p = b + threadIdx.x;
        if (p < n) {
            const float xv = x[p];
            if (xv >= 0.0f) dep_add(dep.h, xv, g);
        }
    }
    dep.flush(hist);
}

// One more particle at x into the global node sums (a spawn).
__device__ __forceinline__ void deposit_spawn(unsigned long long *hist, float x, const cudapic_grid &g) {
    const float pos = x * g.inv_dx;
    const int c = cell_of(pos, g.n_g);
    const uint32_t r = min(__float2uint_rn((pos - (float)c) * (float)(1u << DEP_Q)), 1u << DEP_Q);
    atomicAdd(&hist[c], (unsigned long long)((1u << DEP_Q) - r));
    atomicAdd(&hist[c + 1], (unsigned long long)r);
}

// The field of a step, one CTA: marks the slot and record counts at the
// step's start (mark may be null) and the spawn bases, turns the node sums
// into f32 densities (boundary nodes doubled) and clears them, and solves
// by two scans (poisson_body; the drivers solve by one), which the recompute
// and the oracle's model repeat bit for bit.  efield: the step's field (on
// the tape when recording).
template <int PT>
__global__ void __launch_bounds__(POIS_MAX_THREADS)
    sens_field_kernel(uint32_t *__restrict__ cnt, uint32_t *__restrict__ mark, unsigned long long *__restrict__ hist_e,
                      unsigned long long *__restrict__ hist_i, float *__restrict__ dens_e,
                      float *__restrict__ dens_i, int ions, float *__restrict__ pot, float *__restrict__ efield,
                      float pot0, const __grid_constant__ cudapic_grid g) {
    grid_dep_wait();
    if (threadIdx.x < 4 && mark) mark[threadIdx.x] = cnt[threadIdx.x];
    if (threadIdx.x == 0) {
        cnt[C_N0E] = min(cnt[C_NE], g.capacity);
        cnt[C_N0I] = min(cnt[C_NI], g.capacity);
    }
    const double w = g.weight_factor_d * (1.0 / (double)(1u << DEP_Q));
    for (int s = 0; s < (ions ? 2 : 1); ++s) {
        unsigned long long *h = s ? hist_i : hist_e;
        float *d = s ? dens_i : dens_e;
        for (uint32_t k = threadIdx.x; k < g.n_g; k += blockDim.x) {
            float f = (float)((double)h[k] * w);
            if (k == 0 || k == g.n_g - 1) f *= 2.0f;
            d[k] = f;
            h[k] = 0ull;
        }
    }
    __syncthreads();
    poisson_body<double, PT>(dens_e, dens_i, pot, efield, pot0, nullptr, nullptr, g, nullptr, nullptr);
}

// Push of the live ions in place (Rust-CUDA/src/main.rs:596-620); a particle
// leaving [0, L] is marked dead.  obs (may be null) += the observable sum;
// tx / tv (may be null): the tape of x and v before the push.
__global__ void __launch_bounds__(SENS_THREADS)
    sens_push_i_kernel(float *__restrict__ x, float *__restrict__ vx, const uint32_t *__restrict__ n_ptr,
                       const float *__restrict__ E, double *__restrict__ obs, float *__restrict__ tx,
                       float *__restrict__ tv, const __grid_constant__ cudapic_grid g) {
    __shared__ double red[SENS_THREADS / 32];
    grid_dep_wait();
    const uint32_t n = min(*n_ptr, g.capacity);
    const float f = g.factor_i, dt = g.dt_i;
    double acc = 0.0;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const float xv = x[p], v = vx[p];
        if (tx) {
            tx[p] = xv;
            tv[p] = v;
        }
        if (!(xv >= 0.0f)) continue;
        const float pos = xv * g.inv_dx;
        const int c = cell_of(pos, g.n_g);
        const float c2 = pos - (float)c;
        const float ex = (1.0f - c2) * E[c] + c2 * E[c + 1];
        if (c == (int)g.n_g - 2) acc += (double)v * (double)c2;
        const float v1 = v + f * ex;
        const float x1 = xv + v1 * dt;
        vx[p] = v1;
        x[p] = (x1 >= 0.0f && x1 <= g.gap) ? x1 : -1.0f;
    }
    if (obs) {
        const double s = block_sum(acc, red);
        if (threadIdx.x == 0 && s != 0.0) atomicAdd(obs, s);
    }
}

// The electrons of a step in one pass over the slots live before its spawns:
// push (:596-620; tape, observable sum and dead marks as for the ions),
// check_collisions_e (Rust-CUDA/src/main.rs:971-1033; the certain-rejection
// bound of step.cuh first, the same decisions) and the deposit of the new
// positions for the next step.  An ionizing slot leaves its spawn request
// (children's velocities, record index) for the ranked spawn write.
__global__ void __launch_bounds__(SENS_WIDE)
    sens_electrons_kernel(Planes e, uint32_t *__restrict__ cnt, const float *__restrict__ E, double *__restrict__ obs,
                          float *__restrict__ tx, float *__restrict__ tv, unsigned long long *__restrict__ hist,
                          const float *__restrict__ sig_e, float sigma_max, const float *__restrict__ cs,
                          SensRecE *__restrict__ rec, uint32_t rec_cap, uint32_t *__restrict__ spawn_rec,
                          float *__restrict__ spawn_v, uint32_t *__restrict__ chunk_count,
                          const __grid_constant__ cudapic_grid g) {
    extern __shared__ unsigned long long sens_sm[];
    __shared__ double red[SENS_WIDE / 32];
    SensDep dep(sens_sm, g.n_g);
    grid_dep_wait();
    const uint32_t n = min(cnt[C_N0E], g.capacity);
    const uint32_t cap = g.capacity;
    const ScatK k{g.f1, g.f2};
    const float f = g.factor_e, dt = g.dt_e;
    const float rej_k2 = sigma_max * dt * (sigma_max * dt) * 1.0001f;  // may_collide's bound
    double acc = 0.0;
    const uint32_t stride = gridDim.x * blockDim.x;
    uint32_t r = 0;
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < n; b += stride, ++r) {
        dep.round(r);
        const uint32_t p = (uint32_t)b + threadIdx.x;
        if (p >= n) continue;
        const float xv = e.x[p], vo = e.vx[p];
        if (tx) {
            tx[p] = xv;
            tv[p] = vo;
        }
        if (!(xv >= 0.0f)) continue;
        const float vyp = e.vy[p], vzp = e.vz[p];
        Xoshiro128p rs{e.r[0][p], e.r[1][p], e.r[2][p], e.r[3][p]};
        const float pos = xv * g.inv_dx;
        const int c = cell_of(pos, g.n_g);
        const float c2 = pos - (float)c;
        const float ex = (1.0f - c2) * E[c] + c2 * E[c + 1];
        acc += ((double)vo + 0.5 * (double)f * (double)ex) * (double)ex;
        const float v1 = vo + f * ex;
        const float x1 = xv + v1 * dt;
        const bool stays = x1 >= 0.0f && x1 <= g.gap;
        e.x[p] = stays ? x1 : -1.0f;
        float vxn = v1;
        if (stays) {
            dep_add(dep.h, x1, g);
            const float v[3] = {v1, vyp, vzp};
            // test_electron's draw and decision
            const float v2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
            const float u = rs.uniform();
            if (may_collide(u, v2, rej_k2)) {
                const uint32_t idx = energy_index(g.half_me_over_e * v2);
                const float velocity = sqrtf(v2);
                if (collision_draw(u, __ldg(sig_e + idx) * velocity * dt)) {
                    const float t0 = __ldg(cs + idx);
                    const float t1 = t0 + __ldg(cs + CS_RANGES + idx);
                    const float t2 = t1 + __ldg(cs + 2 * CS_RANGES + idx);
                    const float rnd = rs.uniform();
                    int ev;
                    float a;
                    if (rnd < t0 / t2) {
                        ev = 1;
                        a = 1.0f - 2.0f * rs.uniform();
                    } else if (rnd < t1 / t2) {
                        ev = 2;
                        a = 1.0f - 2.0f * rs.uniform();
                    } else {
                        ev = 3;
                        a = rs.uniform();
                    }
                    const float eta = TWO_PI_F * rs.uniform();
                    float out[3], child[3];
                    scatter_e_t<float>(k, v, ev, a, eta, out, child);
                    uint32_t ri = SPAWN_NOREC;
                    if (rec) {
                        ri = atomicAdd(&cnt[C_REC_E], 1u);
                        if (ri < rec_cap) {
                            SensRecE q;
                            q.p = p;
                            q.ev = (uint32_t)ev;
                            q.ce = NO_SLOT;
                            q.ci = NO_SLOT;
                            q.v[0] = v[0];
                            q.v[1] = v[1];
                            q.v[2] = v[2];
                            q.a = a;
                            q.eta = eta;
                            rec[ri] = q;
                        } else {
                            set_dev_err(&cnt[C_ERR], CUDAPIC_DEVERR_RECORDS);
                            ri = SPAWN_NOREC;
                        }
                    }
                    if (ev == 3) {
                        float ia, ib, ic;
                        rs.three_normal(g.normal_range, ia, ib, ic);
                        spawn_v[0 * (size_t)cap + p] = child[0];
                        spawn_v[1 * (size_t)cap + p] = child[1];
                        spawn_v[2 * (size_t)cap + p] = child[2];
                        spawn_v[3 * (size_t)cap + p] = ia;
                        spawn_v[4 * (size_t)cap + p] = ib;
                        spawn_v[5 * (size_t)cap + p] = ic;
                        spawn_rec[p] = ri;
                        atomicAdd(&chunk_count[p / SENS_CHUNK], 1u);
                    }
                    vxn = out[0];
                    e.vy[p] = out[1];
                    e.vz[p] = out[2];
                }
            }
            e.r[0][p] = rs.s0;
            e.r[1][p] = rs.s1;
            e.r[2][p] = rs.s2;
            e.r[3][p] = rs.s3;
        }
        e.vx[p] = vxn;
    }
    dep.flush(hist);
    if (obs) {
        const double s = block_sum(acc, red);
        if (threadIdx.x == 0 && s != 0.0) atomicAdd(obs, s);
    }
}

__device__ __forceinline__ uint32_t block_excl_scan_u32(uint32_t v, uint32_t *wsum, uint32_t &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < nw ? wsum[lane] : 0u;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < nw) wsum[lane] = w;
    }
    __syncthreads();
    const uint32_t excl = incl - v + (warp > 0 ? wsum[warp - 1] : 0u);
    total = wsum[nw - 1];
    __syncthreads();
    return excl;
}

// The spawns of a step in slot order, one CTA of SENS_CHUNK threads per chunk
// with spawns: children at n0 + (spawns of the chunks before) + rank of the
// parent among the chunk's spawning slots, the electron also added to the
// next step's node sums.  Each such CTA sums the counts before its chunk
// itself (spawns are rare: most CTAs read one count and leave), CTA 0 the
// total, with which it advances both counts (capped at the capacity, dropped
// spawns flagged).  `done`: the previous step's counts, cleared for the next.
__global__ void __launch_bounds__(SENS_CHUNK)
    sens_spawn_kernel(Planes e, Planes ion, uint32_t *__restrict__ cnt, const uint32_t *__restrict__ chunk_count,
                      uint32_t *__restrict__ done, uint32_t *__restrict__ spawn_rec,
                      const float *__restrict__ spawn_v, SensRecE *__restrict__ rec,
                      unsigned long long *__restrict__ hist_e, const __grid_constant__ cudapic_grid g) {
    __shared__ uint32_t wsum[32];
    __shared__ uint32_t s_before;
    grid_dep_wait();
    const uint32_t cap = g.capacity;
    const uint32_t n0e = cnt[C_N0E], n0i = cnt[C_N0I];
    const uint32_t nch = (n0e + SENS_CHUNK - 1) / SENS_CHUNK;
    if (blockIdx.x == 0) {
        uint32_t sum = 0;
        for (uint32_t k = threadIdx.x; k < nch; k += blockDim.x) sum += chunk_count[k];
        uint32_t total;
        block_excl_scan_u32(sum, wsum, total);
        if (threadIdx.x == 0) {
            const uint64_t ne = (uint64_t)n0e + total, ni = (uint64_t)n0i + total;
            if (ne > cap) set_dev_err(&cnt[C_ERR], CUDAPIC_DEVERR_SPAWN_E);
            if (ni > cap) set_dev_err(&cnt[C_ERR], CUDAPIC_DEVERR_SPAWN_I);
            cnt[C_NE] = ne > cap ? cap : (uint32_t)ne;
            cnt[C_NI] = ni > cap ? cap : (uint32_t)ni;
        }
    }
    for (uint32_t c = blockIdx.x; c < nch; c += gridDim.x) {
        if (threadIdx.x == 0) done[c] = 0u;
        if (chunk_count[c] == 0) continue;  // uniform in the block
        uint32_t sum = 0;
        for (uint32_t k = threadIdx.x; k < c; k += blockDim.x) sum += chunk_count[k];
        uint32_t before;
        block_excl_scan_u32(sum, wsum, before);
        if (threadIdx.x == 0) s_before = before;
        __syncthreads();
        const uint32_t p = c * SENS_CHUNK + threadIdx.x;
        const uint32_t fl = p < n0e ? spawn_rec[p] : NO_SPAWN;
        const uint32_t flag = fl != NO_SPAWN ? 1u : 0u;
        uint32_t total;
        const uint32_t rank = block_excl_scan_u32(flag, wsum, total);
        if (flag) {
            const uint32_t k = s_before + rank;
            const uint32_t se = n0e + k, si = n0i + k;
            const float xp = e.x[p];
            uint32_t ce = NO_SLOT, ci = NO_SLOT;
            if (se < cap) {
                e.x[se] = xp;
                e.vx[se] = spawn_v[0 * (size_t)cap + p];
                e.vy[se] = spawn_v[1 * (size_t)cap + p];
                e.vz[se] = spawn_v[2 * (size_t)cap + p];
                deposit_spawn(hist_e, xp, g);
                ce = se;
            }
            if (si < cap) {
                ion.x[si] = xp;
                ion.vx[si] = spawn_v[3 * (size_t)cap + p];
                ion.vy[si] = spawn_v[4 * (size_t)cap + p];
                ion.vz[si] = spawn_v[5 * (size_t)cap + p];
                ci = si;
            }
            if (rec && fl != SPAWN_NOREC) {
                rec[fl].ce = ce;
                rec[fl].ci = ci;
            }
            spawn_rec[p] = NO_SPAWN;
        }
        __syncthreads();  // s_before is rewritten for the next chunk
    }
}

// check_collisions_i (Rust-CUDA/src/main.rs:1167-1219) over the live ions,
// this step's spawns included.
__global__ void __launch_bounds__(SENS_THREADS)
    sens_collide_i_kernel(Planes ion, uint32_t *__restrict__ cnt, const float *__restrict__ sig_i,
                          const float *__restrict__ cs, SensRecI *__restrict__ rec, uint32_t rec_cap,
                          const __grid_constant__ cudapic_grid g) {
    grid_dep_wait();
    const uint32_t n = min(cnt[C_NI], g.capacity);
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        if (!(ion.x[p] >= 0.0f)) continue;
        Xoshiro128p rs{ion.r[0][p], ion.r[1][p], ion.r[2][p], ion.r[3][p]};
        const float v[3] = {ion.vx[p], ion.vy[p], ion.vz[p]};
        const IonTest ts = test_ion(v[0], v[1], v[2], rs, GlobalTable{sig_i}, g);
        if (ts.collide) {
            const uint32_t idx = ts.idx;
            const float t0 = __ldg(cs + 3 * CS_RANGES + idx);
            const float t1 = t0 + __ldg(cs + 4 * CS_RANGES + idx);
            const float rnd = rs.uniform();
            int ev;
            float c = 0.0f;
            if (rnd < t0 / t1) {
                ev = 4;
                c = 1.0f - 2.0f * rs.uniform();
            } else {
                ev = 5;
            }
            const float eta = TWO_PI_F * rs.uniform();
            const float t[3] = {ts.vxa, ts.vya, ts.vza};
            float out[3];
            scatter_i_t<float>(v, t, ev, c, eta, out);
            ion.vx[p] = out[0];
            ion.vy[p] = out[1];
            ion.vz[p] = out[2];
            if (rec) {
                const uint32_t ri = atomicAdd(&cnt[C_REC_I], 1u);
                if (ri < rec_cap) {
                    SensRecI r;
                    r.p = p;
                    r.ev = (uint32_t)ev;
                    for (int j = 0; j < 3; ++j) {
                        r.v[j] = v[j];
                        r.t[j] = t[j];
                    }
                    r.c = c;
                    r.eta = eta;
                    rec[ri] = r;
                } else {
                    set_dev_err(&cnt[C_ERR], CUDAPIC_DEVERR_RECORDS);
                }
            }
        }
        ion.r[0][p] = rs.s0;
        ion.r[1][p] = rs.s1;
        ion.r[2][p] = rs.s2;
        ion.r[3][p] = rs.s3;
    }
}

__global__ void sens_fill_kernel(float *__restrict__ p, uint32_t n, float v) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = v;
}

// Tape mark of a segment's end: slot counts and record counters.
__global__ void sens_mark_kernel(const uint32_t *__restrict__ cnt, uint32_t *__restrict__ mark) {
    grid_dep_wait();
    if (threadIdx.x < 4) mark[threadIdx.x] = cnt[threadIdx.x];
}

// ------------------------------------------------------------------ adjoint
// Both observables' adjoints go through the reverse sweep together (SENS_OBS
// sets of planes): the tape, the records and the collision Jacobians are the
// same for both.
constexpr int SENS_OBS = 2;

struct AdjPlanes {
    float *x, *vx, *vy, *vz;
};
struct AdjSet {
    AdjPlanes o[SENS_OBS];
};

__global__ void __launch_bounds__(SENS_THREADS)
    sens_adj_collide_i_kernel(const SensRecI *__restrict__ rec, const uint32_t *__restrict__ mark0,
                              const uint32_t *__restrict__ mark1, uint32_t rec_cap,
                              const __grid_constant__ AdjSet ion) {
    grid_dep_wait();
    // an overflowed tape (flagged by the forward kernel) is read only up to its capacity
    const uint32_t b = min(mark0[C_REC_I], rec_cap), e = min(mark1[C_REC_I], rec_cap);
    for (uint32_t j = b + blockIdx.x * blockDim.x + threadIdx.x; j < e; j += gridDim.x * blockDim.x) {
        const SensRecI r = rec[j];
        D3 v[3], out[3];
        for (int q = 0; q < 3; ++q) v[q] = seed(r.v[q], q);
        scatter_i_t<D3>(v, r.t, (int)r.ev, r.c, r.eta, out);
#pragma unroll
        for (int o = 0; o < SENS_OBS; ++o) {
            const AdjPlanes &a = ion.o[o];
            const float w[3] = {a.vx[r.p], a.vy[r.p], a.vz[r.p]};
            float nv[3];
            apply_jt(out, w, nv);
            a.vx[r.p] = nv[0];
            a.vy[r.p] = nv[1];
            a.vz[r.p] = nv[2];
        }
    }
}

__global__ void __launch_bounds__(SENS_THREADS)
    sens_adj_collide_e_kernel(const SensRecE *__restrict__ rec, const uint32_t *__restrict__ mark0,
                              const uint32_t *__restrict__ mark1, uint32_t rec_cap, const __grid_constant__ AdjSet es,
                              const __grid_constant__ AdjSet is, const __grid_constant__ cudapic_grid g) {
    grid_dep_wait();
    const uint32_t b = min(mark0[C_REC_E], rec_cap), en = min(mark1[C_REC_E], rec_cap);
    const ScatK k{g.f1, g.f2};
    for (uint32_t j = b + blockIdx.x * blockDim.x + threadIdx.x; j < en; j += gridDim.x * blockDim.x) {
        const SensRecE r = rec[j];
        const uint32_t p = r.p;
        // the adjoints gathered before the Jacobian is formed: their latency hides behind it
        float w[SENS_OBS][3], xb[SENS_OBS];
#pragma unroll
        for (int o = 0; o < SENS_OBS; ++o) {
            w[o][0] = es.o[o].vx[p];
            w[o][1] = es.o[o].vy[p];
            w[o][2] = es.o[o].vz[p];
            xb[o] = es.o[o].x[p];
        }
        D3 v[3], out[3], child[3];
        for (int q = 0; q < 3; ++q) v[q] = seed(r.v[q], q);
        scatter_e_t<D3>(k, v, (int)r.ev, r.a, r.eta, out, child);
#pragma unroll
        for (int o = 0; o < SENS_OBS; ++o) {
            const AdjPlanes &e = es.o[o], &ion = is.o[o];
            float nv[3];
            apply_jt(out, w[o], nv);
            if (r.ev == 3 && r.ce != NO_SLOT) {
                const uint32_t s = r.ce;
                const float wc[3] = {e.vx[s], e.vy[s], e.vz[s]};
                float nc[3];
                apply_jt(child, wc, nc);
                for (int q = 0; q < 3; ++q) nv[q] += nc[q];
                xb[o] += e.x[s];
                e.x[s] = e.vx[s] = e.vy[s] = e.vz[s] = 0.0f;
            }
            if (r.ev == 3 && r.ci != NO_SLOT) {
                const uint32_t s = r.ci;
                xb[o] += ion.x[s];
                ion.x[s] = ion.vx[s] = ion.vy[s] = ion.vz[s] = 0.0f;
            }
            e.x[p] = xb[o];
            e.vx[p] = nv[0];
            e.vy[p] = nv[1];
            e.vz[p] = nv[2];
        }
    }
}

// Adjoint of the push (and of the species' observable term, weight wo[o] for
// observable o) of the slots live at the step's start; the field adjoints
// (eb: [SENS_OBS][n_g]) are summed in FP64.
struct ObsWeights {
    float w[SENS_OBS];
};

__global__ void __launch_bounds__(SENS_WIDE)
    sens_adj_push_kernel(const float *__restrict__ tx, const float *__restrict__ tv, const uint32_t *__restrict__ n_ptr,
                         const float *__restrict__ E, float f, float dt, int ions, const ObsWeights wo,
                         const __grid_constant__ AdjSet adj, double *__restrict__ eb,
                         const __grid_constant__ cudapic_grid g, int copies) {
    extern __shared__ double sens_eb[];  // [copies][SENS_OBS][n_g], warp w adds into copy w % copies
    const uint32_t n_g = g.n_g;
    for (uint32_t k = threadIdx.x; k < copies * SENS_OBS * n_g; k += blockDim.x) sens_eb[k] = 0.0;
    double *ebs = sens_eb + (threadIdx.x / 32u % (uint32_t)copies) * SENS_OBS * n_g;
    __syncthreads();
    grid_dep_wait();
    const uint32_t n = min(*n_ptr, g.capacity);
    const float inv_dx = g.inv_dx;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const float x = tx[p];
        const float v = tv[p];
        float a[SENS_OBS], b[SENS_OBS];
#pragma unroll
        for (int o = 0; o < SENS_OBS; ++o) {
            a[o] = adj.o[o].x[p];
            b[o] = adj.o[o].vx[p];
        }
        if (!(x >= 0.0f)) continue;
        const float pos = x * inv_dx;
        const int c = cell_of(pos, n_g);
        const float c2 = pos - (float)c;
        const float e0 = E[c], e1 = E[c + 1];
        const float ex = (1.0f - c2) * e0 + c2 * e1;
        const float dex = (e1 - e0) * inv_dx;
#pragma unroll
        for (int o = 0; o < SENS_OBS; ++o) {
            const float bt = b[o] + dt * a[o];
            float nx = a[o], nv = bt, eg = bt * f;
            if (!ions) {
                nv += wo.w[o] * ex;
                eg += wo.w[o] * (v + f * ex);
            } else if (c == (int)n_g - 2) {
                nv += wo.w[o] * c2;
                nx += wo.w[o] * v * inv_dx;
            }
            nx += eg * dex;
            if (eg != 0.0f) {
                atomicAdd(&ebs[o * n_g + c], (double)eg * (double)(1.0f - c2));
                atomicAdd(&ebs[o * n_g + c + 1], (double)eg * (double)c2);
            }
            adj.o[o].x[p] = nx;
            adj.o[o].vx[p] = nv;
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < SENS_OBS * n_g; k += blockDim.x) {
        double v = sens_eb[k];
        for (int c = 1; c < copies; ++c) v += sens_eb[(uint32_t)c * SENS_OBS * n_g + k];
        if (v != 0.0) atomicAdd(&eb[k], v);
    }
}

// Deposit adjoint: x adjoint += d/dx sum_k db[k] n_k(x) (CIC, boundary nodes
// doubled); db: [SENS_OBS][n_g].
__global__ void __launch_bounds__(SENS_THREADS)
    sens_adj_gather_kernel(const float *__restrict__ tx, const uint32_t *__restrict__ n_ptr,
                           const double *__restrict__ db, const __grid_constant__ AdjSet adj,
                           const __grid_constant__ cudapic_grid g) {
    grid_dep_wait();
    const uint32_t n = min(*n_ptr, g.capacity);
    const double k = g.weight_factor_d / g.dx;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const float x = tx[p];
        if (!(x >= 0.0f)) continue;
        const int c = cell_of(x * g.inv_dx, g.n_g);
        const double b0 = c == 0 ? 2.0 : 1.0, b1 = (c + 1 == (int)g.n_g - 1) ? 2.0 : 1.0;
#pragma unroll
        for (int o = 0; o < SENS_OBS; ++o) {
            const double *d = db + (size_t)o * g.n_g;
            adj.o[o].x[p] += (float)(k * (b1 * d[c + 1] - b0 * d[c]));
        }
    }
}

}  // namespace

}  // namespace cudapic

using namespace cudapic;

struct cudapic_sens {
    cudapic_state *st = nullptr;
    int device = 0;
    cudaStream_t stream = nullptr;
    cudapic_grid g{};
    uint32_t cap = 0, K = 0, S = 0, H = 0, n_seg = 0, n_g = 0, n_sub = 0, n_t = 0;
    uint32_t rec_cap_e = 0, rec_cap_i = 0;
    uint32_t n_init[2] = {0, 0};
    double voltage = 0.0;
    bool have_forward = false;
    Planes cur[2]{}, init[2]{};
    uint32_t *cnt = nullptr;
    unsigned long long *hist = nullptr;  // [2][n_g]
    float *dens = nullptr, *efield = nullptr, *pot = nullptr;
    double *obs = nullptr;               // [2] raw sums
    uint32_t *spawn_rec = nullptr;
    uint32_t *chunk_count[2] = {nullptr, nullptr};  // spawns per chunk, by the parity of the step
    float *spawn_v = nullptr;
    float *ckpt = nullptr;               // [n_seg - 1][2][8][cap] (RNG planes stored bitwise), of segment 1 on:
                                         // segment 0 starts from init
    uint32_t *ckpt_cnt = nullptr;        // [n_seg][C_COUNT]
    float *tx_e = nullptr, *tv_e = nullptr, *tx_i = nullptr, *tv_i = nullptr, *tE = nullptr;
    uint32_t *tmark = nullptr;           // [S + 1][4]
    SensRecE *rec_e = nullptr;
    SensRecI *rec_i = nullptr;
    float *adj = nullptr;                // [SENS_OBS][2][4][cap]
    double *eb = nullptr, *neb = nullptr, *nib_acc = nullptr, *vbar = nullptr;  // [SENS_OBS][n_g], vbar [SENS_OBS]
    std::vector<void *> allocs;
    size_t bytes = 0;
};

namespace {

int sens_alloc(cudapic_sens *s, void **p, size_t bytes) {
    *p = nullptr;
    if (bytes == 0) bytes = 16;
    const cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) return check_cuda(e, "sensitivity allocation");
    s->allocs.push_back(*p);
    s->bytes += bytes;
    return CUDAPIC_OK;
}

template <typename T>
int sens_alloc_t(cudapic_sens *s, T **p, size_t count) {
    void *v = nullptr;
    CUDAPIC_CHECK(sens_alloc(s, &v, count * sizeof(T)));
    *p = static_cast<T *>(v);
    return CUDAPIC_OK;
}

Planes planes_of(float *base, uint32_t cap) {
    Planes p;
    p.x = base;
    p.vx = base + (size_t)cap;
    p.vy = base + 2 * (size_t)cap;
    p.vz = base + 3 * (size_t)cap;
    for (int k = 0; k < 4; ++k) p.r[k] = reinterpret_cast<uint32_t *>(base + (4 + k) * (size_t)cap);
    return p;
}

AdjSet adj_of(const cudapic_sens *s, int sp) {
    AdjSet a;
    for (int o = 0; o < SENS_OBS; ++o) {
        float *b = s->adj + ((size_t)o * 2 + sp) * 4 * s->cap;
        a.o[o] = {b, b + s->cap, b + 2 * (size_t)s->cap, b + 3 * (size_t)s->cap};
    }
    return a;
}

struct WideShape {
    unsigned grid, threads;
};
WideShape wide_shape(uint32_t units) {
    unsigned threads = 256;
    while (threads < SENS_WIDE && (uint64_t)threads * sm_count() < units) threads *= 2;
    return {persistent_grid(1, ((uint64_t)units + threads - 1) / threads), threads};
}
// Copies of the adjoint push's FP64 sums (shared FP64 adds retry when two
// warps meet on a node): four, fewer on large grids.
constexpr int EB_SMEM_MAX = 96 * 1024;  // one copy fits at SENS_MAX_NG
static_assert(sizeof(double) * SENS_OBS * SENS_MAX_NG <= EB_SMEM_MAX, "one copy");
int eb_copies(uint32_t n_g) {
    return (int)std::min<size_t>(4, EB_SMEM_MAX / (sizeof(double) * SENS_OBS * n_g));
}
unsigned grid_n(uint32_t units) { return persistent_grid(SENS_PER_SM, (units + SENS_THREADS - 1) / SENS_THREADS); }

bool ion_step(const cudapic_sens *s, uint32_t t) { return t % s->n_sub == 0; }

float pot0_at(const cudapic_sens *s, uint32_t t) {
    return (float)(s->voltage * std::cos(((double)(t % s->n_t) / (double)s->n_t) * (2.0 * 3.141592653589793)));
}

double cos_at(const cudapic_sens *s, uint32_t t) {
    return std::cos(((double)(t % s->n_t) / (double)s->n_t) * (2.0 * 3.141592653589793));
}

// Observable scales per unit of the raw sums: J_P, J_G.
void obs_scale(const cudapic_sens *s, double *cP, double *cG) {
    const double w_over_a = s->g.weight_factor_d * s->g.dx;
    uint32_t k_i = 0;
    for (uint32_t t = 0; t < s->K; ++t) k_i += ion_step(s, t);
    *cP = -1.60217662e-19 * w_over_a / (double)s->g.gap / (double)s->K;
    *cG = 2.0 * s->g.weight_factor_d / (double)(k_i ? k_i : 1);
}

int launch_field(cudapic_sens *s, float *efield, uint32_t *mark, int ions, float pot0) {
    int threads, pt;
    poisson_shape(s->n_g, threads, pt);
    auto kern = pt == 1 ? sens_field_kernel<1> : pt == 2 ? sens_field_kernel<2> : sens_field_kernel<4>;  // n_g <= 4096
    return launch_kernel("sens_field", kern, 1, threads, sizeof(double) * s->n_g, s->stream, s->cnt, mark, s->hist,
                         s->hist + s->n_g, s->dens, s->dens + s->n_g, ions, s->pot, efield, pot0, s->g);
}

// Before the first step of a run or segment: the node sums of its electrons,
// no spawns counted.
int start_steps(cudapic_sens *s) {
    CUDAPIC_CHECK(check_cuda(cudaMemsetAsync(s->hist, 0, sizeof(unsigned long long) * 2 * s->n_g, s->stream), "sens hist"));
    for (auto *c : s->chunk_count)
        CUDAPIC_CHECK(check_cuda(cudaMemsetAsync(c, 0, sizeof(uint32_t) * (s->cap / SENS_CHUNK + 2), s->stream),
                                 "sens chunks"));
    const WideShape w = wide_shape(s->cap);
    return launch_kernel("sens_deposit", sens_deposit_kernel, w.grid, w.threads, dep_smem(s->n_g), s->stream,
                         s->cur[0].x, s->cnt + C_NE, s->hist, s->g);
}

// One forward step t; rec: record the tape at step j of the segment.
int fwd_step(cudapic_sens *s, uint32_t t, bool rec, uint32_t j) {
    cudaStream_t st = s->stream;
    const cudapic_grid &g = s->g;
    const bool ions = ion_step(s, t);
    const size_t cap = s->cap;
    const unsigned gd = grid_n(s->cap);
    const WideShape w = wide_shape(s->cap);
    if (ions)
        CUDAPIC_CHECK(launch_kernel("sens_deposit", sens_deposit_kernel, w.grid, w.threads, dep_smem(s->n_g), st,
                                    s->cur[1].x, s->cnt + C_NI, s->hist + s->n_g, g));
    float *E = rec ? s->tE + (size_t)j * s->n_g : s->efield;
    CUDAPIC_CHECK(launch_field(s, E, rec ? s->tmark + 4 * j : nullptr, ions ? 1 : 0, pot0_at(s, t)));
    CUDAPIC_CHECK(launch_kernel("sens_electrons", sens_electrons_kernel, w.grid, w.threads, dep_smem(s->n_g), st,
                                s->cur[0], s->cnt, E, rec ? nullptr : s->obs, rec ? s->tx_e + j * cap : nullptr,
                                rec ? s->tv_e + j * cap : nullptr, s->hist, s->st->sigma_tot_e, s->st->sigma_max_e,
                                s->st->cs, rec ? s->rec_e : nullptr, s->rec_cap_e, s->spawn_rec, s->spawn_v,
                                s->chunk_count[t & 1u], g));
    if (ions) {
        const size_t ji = j / s->n_sub;
        CUDAPIC_CHECK(launch_kernel("sens_push_i", sens_push_i_kernel, gd, SENS_THREADS, 0, st, s->cur[1].x,
                                    s->cur[1].vx, s->cnt + C_NI, E, rec ? nullptr : s->obs + 1,
                                    rec ? s->tx_i + ji * cap : nullptr, rec ? s->tv_i + ji * cap : nullptr, g));
    }
    const unsigned nch = (s->cap + SENS_CHUNK - 1) / SENS_CHUNK;
    CUDAPIC_CHECK(launch_kernel("sens_spawn", sens_spawn_kernel, std::min<unsigned>(nch, 4096u), SENS_CHUNK, 0, st,
                                s->cur[0], s->cur[1], s->cnt, s->chunk_count[t & 1u], s->chunk_count[(t & 1u) ^ 1u],
                                s->spawn_rec, s->spawn_v, rec ? s->rec_e : nullptr, s->hist, g));
    if (ions)
        CUDAPIC_CHECK(launch_kernel("sens_collide_i", sens_collide_i_kernel, gd, SENS_THREADS, 0, st, s->cur[1], s->cnt,
                                    s->st->sigma_tot_i, s->st->cs, rec ? s->rec_i : nullptr, s->rec_cap_i, g));
    return CUDAPIC_OK;
}

int copy_planes(cudapic_sens *s, float *dst, const float *src) {
    return check_cuda(cudaMemcpyAsync(dst, src, sizeof(float) * 16 * (size_t)s->cap, cudaMemcpyDeviceToDevice,
                                      s->stream),
                      "sensitivity plane copy");
}

// The planes at the start of segment k.
float *checkpoint_of(const cudapic_sens *s, uint32_t k) {
    return k ? s->ckpt + (size_t)(k - 1) * 16 * s->cap : s->init[0].x;
}

// Reverse step t (segment step j).
int adj_step(cudapic_sens *s, uint32_t t, uint32_t j, const ObsWeights &wP, const ObsWeights &wG) {
    cudaStream_t st = s->stream;
    const cudapic_grid &g = s->g;
    const bool ions = ion_step(s, t);
    const size_t cap = s->cap;
    const uint32_t *m0 = s->tmark + 4 * j, *m1 = s->tmark + 4 * (j + 1);
    const unsigned gd = grid_n(s->cap);
    const AdjSet ae = adj_of(s, 0), ai = adj_of(s, 1);
    if (ions)
        CUDAPIC_CHECK(launch_kernel("sens_adj_collide_i", sens_adj_collide_i_kernel, gd, SENS_THREADS, 0, st, s->rec_i,
                                    m0, m1, s->rec_cap_i, ai));
    CUDAPIC_CHECK(launch_kernel("sens_adj_collide_e", sens_adj_collide_e_kernel, gd, SENS_THREADS, 0, st, s->rec_e, m0,
                                m1, s->rec_cap_e, ae, ai, g));
    const float *E = s->tE + (size_t)j * s->n_g;
    const WideShape w = wide_shape(s->cap);
    const int copies = eb_copies(s->n_g);
    const size_t esm = sizeof(double) * SENS_OBS * copies * s->n_g;
    CUDAPIC_CHECK(launch_kernel("sens_adj_push", sens_adj_push_kernel, w.grid, w.threads, esm, st, s->tx_e + j * cap,
                                s->tv_e + j * cap, m0 + C_NE, E, g.factor_e, g.dt_e, 0, wP, ae, s->eb, g,
                                copies));
    const size_t ji = j / s->n_sub;
    if (ions)
        CUDAPIC_CHECK(launch_kernel("sens_adj_push", sens_adj_push_kernel, w.grid, w.threads, esm, st,
                                    s->tx_i + ji * cap, s->tv_i + ji * cap, m0 + C_NI, E, g.factor_i, g.dt_i, 1, wG,
                                    ai, s->eb, g, copies));
    // the ion-density adjoint gathered at step t + 1 (an ion step) restarts
    CUDAPIC_CHECK(launch_poisson_adjoint(s->eb, s->neb, s->nib_acc, ion_step(s, t + 1) ? 1 : 0, cos_at(s, t), s->vbar,
                                         SENS_OBS, g, st));
    CUDAPIC_CHECK(launch_kernel("sens_adj_gather", sens_adj_gather_kernel, gd, SENS_THREADS, 0, st, s->tx_e + j * cap,
                                m0 + C_NE, (const double *)s->neb, ae, g));
    if (ions)
        CUDAPIC_CHECK(launch_kernel("sens_adj_gather", sens_adj_gather_kernel, gd, SENS_THREADS, 0, st,
                                    s->tx_i + ji * cap, m0 + C_NI, (const double *)s->nib_acc, ai, g));
    return CUDAPIC_OK;
}

int read_err(cudapic_sens *s, uint32_t *err) {
    CUDAPIC_CHECK(check_cuda(cudaMemcpyAsync(err, s->cnt + C_ERR, sizeof(uint32_t), cudaMemcpyDeviceToHost, s->stream),
                             "sensitivity error word"));
    return check_cuda(cudaStreamSynchronize(s->stream), "sensitivity sync");
}

}  // namespace

extern "C" int cudapic_sens_create(cudapic_state *st, uint32_t window_steps, uint32_t checkpoint_every,
                                   uint32_t horizon, cudapic_sens **out) {
    if (!st || !out) return fail(CUDAPIC_ERR_ARG, "sens_create: null pointer");
    *out = nullptr;
    const cudapic_params &p = st->params;
    if (window_steps == 0 || checkpoint_every == 0) return fail(CUDAPIC_ERR_ARG, "sens_create: empty window");
    if (checkpoint_every % p.n_sub || window_steps % checkpoint_every)
        return fail(CUDAPIC_ERR_ARG, "sens_create: the window must be whole checkpoint intervals of whole ion cycles");
    if (horizon % checkpoint_every) return fail(CUDAPIC_ERR_ARG, "sens_create: horizon must be whole checkpoint intervals");
    if (p.n_g > SENS_MAX_NG) return fail(CUDAPIC_ERR_ARG, "sens_create: n_g > 4096");
    if (p.flags & CUDAPIC_FLAG_POISSON_F32_SCAN) return fail(CUDAPIC_ERR_ARG, "sens_create: needs the FP64 Poisson sums");
    DeviceGuard dg(st->device);
    if (!dg.ok) return fail(CUDAPIC_ERR_CUDA, "sens_create: cannot select the state's device");
    auto *s = new cudapic_sens();
    s->st = st;
    s->device = st->device;
    s->stream = st->stream;
    s->g = st->grid;
    s->g.dev_err = nullptr;
    s->g.work = nullptr;
    s->cap = p.capacity;
    s->K = window_steps;
    s->S = checkpoint_every;
    s->H = horizon;
    s->n_seg = window_steps / checkpoint_every;
    s->n_g = p.n_g;
    s->n_sub = p.n_sub;
    s->n_t = p.n_t;
    const size_t cap = s->cap;
    s->rec_cap_e = (uint32_t)std::min<uint64_t>(0xFFFFFFF0ull, cap * s->S / 32 + 65536);
    s->rec_cap_i = (uint32_t)std::min<uint64_t>(0xFFFFFFF0ull, cap * (s->S / s->n_sub) / 8 + 65536);
    auto fail_free = [&](int rc) {
        cudapic_sens_destroy(s);
        return rc;
    };
    int rc = CUDAPIC_OK;
    float *init = nullptr, *cur = nullptr;
    if ((rc = sens_alloc_t(s, &init, 16 * cap)) || (rc = sens_alloc_t(s, &cur, 16 * cap)) ||
        (rc = sens_alloc_t(s, &s->cnt, C_COUNT)) || (rc = sens_alloc_t(s, &s->hist, 2 * (size_t)s->n_g)) ||
        (rc = sens_alloc_t(s, &s->dens, 2 * (size_t)s->n_g)) || (rc = sens_alloc_t(s, &s->efield, s->n_g)) ||
        (rc = sens_alloc_t(s, &s->pot, s->n_g)) || (rc = sens_alloc_t(s, &s->obs, 2)) ||
        (rc = sens_alloc_t(s, &s->spawn_rec, cap)) || (rc = sens_alloc_t(s, &s->spawn_v, 6 * cap)) ||
        (rc = sens_alloc_t(s, &s->chunk_count[0], cap / SENS_CHUNK + 2)) ||
        (rc = sens_alloc_t(s, &s->chunk_count[1], cap / SENS_CHUNK + 2)) ||
        (rc = sens_alloc_t(s, &s->ckpt, (size_t)(s->n_seg - 1) * 16 * cap)) ||
        (rc = sens_alloc_t(s, &s->ckpt_cnt, (size_t)s->n_seg * C_COUNT)) ||
        (rc = sens_alloc_t(s, &s->tx_e, (size_t)s->S * cap)) || (rc = sens_alloc_t(s, &s->tv_e, (size_t)s->S * cap)) ||
        (rc = sens_alloc_t(s, &s->tx_i, (size_t)(s->S / s->n_sub) * cap)) ||
        (rc = sens_alloc_t(s, &s->tv_i, (size_t)(s->S / s->n_sub) * cap)) ||
        (rc = sens_alloc_t(s, &s->tE, (size_t)s->S * s->n_g)) ||
        (rc = sens_alloc_t(s, &s->tmark, 4 * ((size_t)s->S + 1))) ||
        (rc = sens_alloc_t(s, &s->rec_e, s->rec_cap_e)) || (rc = sens_alloc_t(s, &s->rec_i, s->rec_cap_i)) ||
        (rc = sens_alloc_t(s, &s->adj, SENS_OBS * 8 * cap)) || (rc = sens_alloc_t(s, &s->eb, SENS_OBS * (size_t)s->n_g)) ||
        (rc = sens_alloc_t(s, &s->neb, SENS_OBS * (size_t)s->n_g)) ||
        (rc = sens_alloc_t(s, &s->nib_acc, SENS_OBS * (size_t)s->n_g)) || (rc = sens_alloc_t(s, &s->vbar, SENS_OBS)))
        return fail_free(rc);
    // above the 48 KB a launch may take by default (n_g up to 4096)
    if ((rc = check_cuda(cudaFuncSetAttribute(sens_deposit_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)dep_smem(SENS_MAX_NG)), "cudaFuncSetAttribute(sens)")) ||
        (rc = check_cuda(cudaFuncSetAttribute(sens_electrons_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)dep_smem(SENS_MAX_NG)), "cudaFuncSetAttribute(sens)")) ||
        (rc = check_cuda(cudaFuncSetAttribute(sens_adj_push_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              EB_SMEM_MAX),
                         "cudaFuncSetAttribute(sens)")))
        return fail_free(rc);
    for (int sp = 0; sp < 2; ++sp) {
        s->init[sp] = planes_of(init + (size_t)sp * 8 * cap, s->cap);
        s->cur[sp] = planes_of(cur + (size_t)sp * 8 * cap, s->cap);
    }
    // snapshot of the state's particles and RNG streams (the initial state of every run)
    uint32_t ne = 0, ni = 0;
    if ((rc = cudapic_state_counts(st, &ne, &ni))) return fail_free(rc);
    cudapic_buffers b;
    if ((rc = cudapic_state_buffers(st, &b))) return fail_free(rc);
    s->n_init[0] = ne;
    s->n_init[1] = ni;
    cudaStream_t sm = s->stream;
    for (int sp = 0; sp < 2; ++sp) {
        const Planes &d = s->init[sp];
        const float *src[4] = {b.x[sp], b.vx[sp], b.vy[sp], b.vz[sp]};
        float *dst[4] = {d.x, d.vx, d.vy, d.vz};
        for (int k = 0; k < 4; ++k) {
            if ((rc = check_cuda(cudaMemsetAsync(dst[k], 0, sizeof(float) * cap, sm), "sens init")))
                return fail_free(rc);
            // slots past the live count start dead (x = -1)
            if (k == 0 &&
                (rc = launch_kernel("sens_fill", sens_fill_kernel, grid_n(s->cap), SENS_THREADS, 0, sm, dst[0],
                                    s->cap, -1.0f)))
                return fail_free(rc);
            if (s->n_init[sp] &&
                (rc = check_cuda(cudaMemcpyAsync(dst[k], src[k], sizeof(float) * s->n_init[sp], cudaMemcpyDeviceToDevice,
                                                 sm), "sens init copy")))
                return fail_free(rc);
            if ((rc = check_cuda(cudaMemcpyAsync(d.r[k], b.rng[sp][k], sizeof(uint32_t) * cap, cudaMemcpyDeviceToDevice,
                                                 sm), "sens init rng")))
                return fail_free(rc);
        }
    }
    if ((rc = check_cuda(cudaMemsetAsync(s->spawn_rec, 0xFF, sizeof(uint32_t) * cap, sm), "sens spawn flags")) ||
        (rc = check_cuda(cudaStreamSynchronize(sm), "sens create sync")))
        return fail_free(rc);
    *out = s;
    return CUDAPIC_OK;
}

extern "C" int cudapic_sens_forward(cudapic_sens *s, double voltage, double obs[2]) {
    if (!s || !obs) return fail(CUDAPIC_ERR_ARG, "sens_forward: null pointer");
    DeviceGuard dg(s->device);
    s->voltage = voltage;
    s->have_forward = false;
    cudaStream_t st = s->stream;
    const size_t cap = s->cap;
    // start: the snapshot (dead slots beyond the live counts)
    CUDAPIC_CHECK(copy_planes(s, s->cur[0].x, s->init[0].x));
    uint32_t c0[C_COUNT] = {s->n_init[0], s->n_init[1], 0, 0, 0, 0, 0, 0};
    CUDAPIC_CHECK(check_cuda(cudaMemcpyAsync(s->cnt, c0, sizeof(c0), cudaMemcpyHostToDevice, st), "sens counters"));
    CUDAPIC_CHECK(check_cuda(cudaMemsetAsync(s->obs, 0, 2 * sizeof(double), st), "sens obs"));
    PdlScope pdl(s->st->overlap);
    CUDAPIC_CHECK(start_steps(s));
    for (uint32_t t = 0; t < s->K; ++t) {
        if (t % s->S == 0) {
            const uint32_t k = t / s->S;
            if (k) CUDAPIC_CHECK(copy_planes(s, checkpoint_of(s, k), s->cur[0].x));
            CUDAPIC_CHECK(check_cuda(cudaMemcpyAsync(s->ckpt_cnt + (size_t)k * C_COUNT, s->cnt, sizeof(uint32_t) * C_COUNT,
                                                     cudaMemcpyDeviceToDevice, st), "sens checkpoint counters"));
        }
        CUDAPIC_CHECK(fwd_step(s, t, false, 0));
    }
    double raw[2];
    CUDAPIC_CHECK(check_cuda(cudaMemcpyAsync(raw, s->obs, sizeof(raw), cudaMemcpyDeviceToHost, st), "sens obs read"));
    uint32_t err = 0;
    CUDAPIC_CHECK(read_err(s, &err));
    double cP, cG;
    obs_scale(s, &cP, &cG);
    obs[0] = cP * raw[0];
    obs[1] = cG * raw[1];
    s->have_forward = true;
    if (err) return fail(CUDAPIC_ERR_CAPACITY, "sens_forward: device error (spawns beyond the capacity)");
    return CUDAPIC_OK;
}

extern "C" int cudapic_sens_backward(cudapic_sens *s, double grad[2]) {
    if (!s || !grad) return fail(CUDAPIC_ERR_ARG, "sens_backward: null pointer");
    if (!s->have_forward) return fail(CUDAPIC_ERR_STATE, "sens_backward: no forward run");
    DeviceGuard dg(s->device);
    cudaStream_t st = s->stream;
    const size_t cap = s->cap;
    double cP, cG;
    obs_scale(s, &cP, &cG);
    const ObsWeights wP{{(float)cP, 0.0f}}, wG{{0.0f, (float)cG}};
    const size_t adj_bytes = sizeof(float) * SENS_OBS * 8 * cap, node_bytes = sizeof(double) * SENS_OBS * s->n_g;
    CUDAPIC_CHECK(check_cuda(cudaMemsetAsync(s->adj, 0, adj_bytes, st), "sens adjoint"));
    CUDAPIC_CHECK(check_cuda(cudaMemsetAsync(s->eb, 0, node_bytes, st), "sens eb"));
    CUDAPIC_CHECK(check_cuda(cudaMemsetAsync(s->nib_acc, 0, node_bytes, st), "sens nib"));
    CUDAPIC_CHECK(check_cuda(cudaMemsetAsync(s->vbar, 0, SENS_OBS * sizeof(double), st), "sens vbar"));
    PdlScope pdl(s->st->overlap);
    for (int64_t k = (int64_t)s->n_seg - 1; k >= 0; --k) {
        const uint32_t t0 = (uint32_t)k * s->S;
        if (s->H && (t0 + s->S) % s->H == 0)  // a horizon ends after this segment: the adjoint restarts
            CUDAPIC_CHECK(check_cuda(cudaMemsetAsync(s->adj, 0, adj_bytes, st), "sens horizon"));
        // recompute the segment from its checkpoint, recording the tape
        CUDAPIC_CHECK(copy_planes(s, s->cur[0].x, checkpoint_of(s, (uint32_t)k)));
        CUDAPIC_CHECK(check_cuda(cudaMemcpyAsync(s->cnt, s->ckpt_cnt + (size_t)k * C_COUNT, sizeof(uint32_t) * C_COUNT,
                                                 cudaMemcpyDeviceToDevice, st), "sens restore counters"));
        CUDAPIC_CHECK(check_cuda(cudaMemsetAsync(s->cnt + C_REC_E, 0, 2 * sizeof(uint32_t), st), "sens records"));
        CUDAPIC_CHECK(start_steps(s));
        for (uint32_t j = 0; j < s->S; ++j) CUDAPIC_CHECK(fwd_step(s, t0 + j, true, j));
        CUDAPIC_CHECK(launch_kernel("sens_mark", sens_mark_kernel, 1, 32, 0, st, s->cnt, s->tmark + 4 * s->S));
        for (int64_t j = (int64_t)s->S - 1; j >= 0; --j)
            CUDAPIC_CHECK(adj_step(s, t0 + (uint32_t)j, (uint32_t)j, wP, wG));
    }
    CUDAPIC_CHECK(check_cuda(cudaMemcpyAsync(grad, s->vbar, SENS_OBS * sizeof(double), cudaMemcpyDeviceToHost, st),
                             "sens gradient read"));
    uint32_t err = 0;
    CUDAPIC_CHECK(read_err(s, &err));
    if (err & CUDAPIC_DEVERR_RECORDS) return fail(CUDAPIC_ERR_CAPACITY, "sens_backward: collision records overflowed");
    if (err) return fail(CUDAPIC_ERR_CAPACITY, "sens_backward: device error (spawns beyond the capacity)");
    return CUDAPIC_OK;
}

extern "C" int cudapic_sens_info(cudapic_sens *s, uint32_t counts[2], uint32_t *dev_err, uint64_t *device_bytes) {
    if (!s) return fail(CUDAPIC_ERR_ARG, "sens_info: null pointer");
    DeviceGuard dg(s->device);
    uint32_t c[C_COUNT];
    CUDAPIC_CHECK(check_cuda(cudaMemcpyAsync(c, s->cnt, sizeof(c), cudaMemcpyDeviceToHost, s->stream), "sens info"));
    CUDAPIC_CHECK(check_cuda(cudaStreamSynchronize(s->stream), "sens info sync"));
    if (counts) {
        counts[0] = c[C_NE];
        counts[1] = c[C_NI];
    }
    if (dev_err) *dev_err = c[C_ERR];
    if (device_bytes) *device_bytes = s->bytes;
    return CUDAPIC_OK;
}

extern "C" int cudapic_sens_download(cudapic_sens *s, int species, float *x, float *vx, float *vy, float *vz,
                                     uint32_t *rng, uint32_t capacity) {
    if (!s || species < 0 || species > 1 || !x || !vx || !vy || !vz)
        return fail(CUDAPIC_ERR_ARG, "sens_download: bad arguments");
    if (capacity < s->cap) return fail(CUDAPIC_ERR_ARG, "sens_download: host buffers smaller than the capacity");
    DeviceGuard dg(s->device);
    const Planes &p = s->cur[species];
    float *dst[4] = {x, vx, vy, vz};
    const float *src[4] = {p.x, p.vx, p.vy, p.vz};
    for (int k = 0; k < 4; ++k)
        CUDAPIC_CHECK(check_cuda(cudaMemcpyAsync(dst[k], src[k], sizeof(float) * s->cap, cudaMemcpyDeviceToHost, s->stream),
                                 "sens download"));
    if (rng)
        for (int k = 0; k < 4; ++k)
            CUDAPIC_CHECK(check_cuda(cudaMemcpyAsync(rng + (size_t)k * s->cap, p.r[k], sizeof(uint32_t) * s->cap,
                                                     cudaMemcpyDeviceToHost, s->stream), "sens download rng"));
    return check_cuda(cudaStreamSynchronize(s->stream), "sens download sync");
}

extern "C" int cudapic_sens_destroy(cudapic_sens *s) {
    if (!s) return CUDAPIC_OK;
    DeviceGuard dg(s->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    for (void *p : s->allocs) cudaFree(p);
    delete s;
    return CUDAPIC_OK;
}
