// poisson.cuh -- the one-CTA scan-based Poisson solve and field (the body
// of the driver's solve kernels, kernels_poisson.cu, also run by the last
// CTA of the in-place step's scatter pass, kernels_inplace.cu).
//
// Reference: solve_poisson_scan_f32, Rust-CUDA/src/main.rs:408-494.  The
// Dirichlet problem pot[i-1] - 2 pot[i] + pot[i+1] = f_i has unit
// tridiagonal coefficients, so the Thomas recurrences collapse to
//     G_i = sum_{j<=i} j f_j,   r_i = -G_i / ((i+1) i),   pot_i = i sum_{j=i}^{N-2} r_j,
// two inclusive prefix sums, the second over the first (C/eduPIC.cc:461-494
// is the sequential Thomas form of the same system): poisson_body, the
// reference's f32 arithmetic and the sensitivity path's FP64 one.
//
// The FP64 solve of the drivers (poisson_fused) sums by parts: with
// F_i = sum_{j<=i} f_j and 1/(j(j+1)) = 1/j - 1/(j+1),
//     sum_{j=i}^{N-2} r_j = -(G_i / i - G_{N-2}/(N-1) + F_{N-2} - F_i),
//     pot_i = pot_0 - G_i + i (C + F_i),   C = (G_{N-2} - pot_0)/(N-1) - F_{N-2}
// (the f_j here without the boundary value), and the field needs no
// difference of potentials: E_i = -(C + F_i - f_i / 2) / dx inside.  Both sums
// then run in ONE scan, without a division per node, a pass over shared
// memory for the neighbours or the boundary value's load in front of it; one
// block barrier instead of seven.  Latency-bound: the solve kernel takes 2.2 us at N_G = 400,
// 4.3 at 4096 and 14 at 16384 (two scans: 2.8, 7.6 and 62 us).
#pragma once
#include "common.cuh"

namespace cudapic {

constexpr int POIS_MAX_THREADS = 1024;
constexpr int POIS_MAX_PER_THREAD = 16;  // N_G <= 16384

template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
    }
    return v;
}

// Exclusive block scan of one value per thread; also returns the block total.
template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T *wsum, T &total) {
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    T incl = warp_incl_scan(v, lane);
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        T w = lane < nwarps ? wsum[lane] : T(0);
        w = warp_incl_scan(w, lane);
        if (lane < nwarps) wsum[lane] = w;
    }
    __syncthreads();
    T excl = incl - v + (warp > 0 ? wsum[warp - 1] : T(0));
    total = wsum[nwarps - 1];
    __syncthreads();
    return excl;
}

// The solve of one discharge by one CTA (after grid_dep_wait), shared by
// poisson_kernel, the batched solve and the scatter pass of the in-place
// electron step, whose last CTA solves the next step's field
// (kernels_inplace.cu).  The densities are read through L2 (__ldcg): in the
// scatter pass other CTAs of the same launch have just added to them.
// T: arithmetic type of the scans (double or float); PT: nodes per thread.
template <typename T, int PT>
__device__ __forceinline__ void poisson_body(const float *__restrict__ e_density, const float *__restrict__ i_density,
                                             float *__restrict__ pot_out, float *__restrict__ efield_out,
                                             float pot0_arg, const float *__restrict__ pot0_table,
                                             uint32_t *__restrict__ step_counter, const cudapic_grid &g,
                                             float *__restrict__ zero_a, float *__restrict__ zero_b) {
    constexpr int per_thread = PT;
    extern __shared__ unsigned char smem_raw[];
    T *pot_s = reinterpret_cast<T *>(smem_raw);        // n_g
    __shared__ T wsum[32];
    __shared__ T r_total_s;
    __shared__ float pot0_s;

    const int n = (int)g.n_g;
    const int tid = threadIdx.x;
    for (int k = tid; k < n; k += blockDim.x) {  // next-step accumulators of the driver
        if (zero_a) zero_a[k] = 0.0f;
        if (zero_b) zero_b[k] = 0.0f;
    }
    if (tid == 0) {
        float p0 = pot0_arg;
        if (pot0_table) {
            uint32_t t = *step_counter;
            p0 = pot0_table[t % g.n_t];
            *step_counter = t + 1;
        }
        pot0_s = p0;
    }
    __syncthreads();
    const T pot0 = (T)pot0_s;

    // node-dependent constants in the arithmetic type of the solve
    const T e_charge = sizeof(T) == 8 ? (T)1.60217662e-19 : (T)g.e_charge;
    const T alpha = sizeof(T) == 8 ? (T)(-g.dx * g.dx / 8.85418781e-12) : (T)g.alpha;

    const int first = tid * per_thread;
    T rho[PT];
    T G[PT];
    T local = 0;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        if (j < per_thread) {
            const int i = first + j;
            T rh = 0, gi = 0;
            if (i < n) {
                const float di = __ldcg(i_density + i), de = __ldcg(e_density + i);
                if (sizeof(T) == 8)
                    rh = e_charge * ((T)di - (T)de);
                else
                    rh = e_charge * (T)(di - de);
                if (i != 0) {
                    T fi = alpha * rh - (i == 1 ? pot0 : T(0));
                    gi = (T)i * fi;
                }
            }
            rho[j] = rh;
            local += gi;
            G[j] = local;
        }
    }
    T tot;
    T off = block_excl_scan<T>(local, wsum, tot);

    T r[PT];
    T R[PT];
    local = 0;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        if (j < per_thread) {
            const int i = first + j;
            T ri = 0;
            if (i != 0 && i < n - 1) {
                T hi = -(G[j] + off) / ((T)i + T(1));
                ri = hi / (T)i;
            }
            r[j] = ri;
            local += ri;
            R[j] = local;
        }
    }
    off = block_excl_scan<T>(local, wsum, tot);
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        if (j < per_thread && first + j == n - 2) r_total_s = R[j] + off;
    }
    __syncthreads();
    const T r_total = r_total_s;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        if (j < per_thread) {
            const int i = first + j;
            if (i < n) {
                T p;
                if (i == 0) p = pot0;
                else if (i < n - 1) p = (T)i * (r_total - (R[j] + off) + r[j]);
                else p = T(0);
                pot_s[i] = p;
            }
        }
    }
    __syncthreads();
    const T inv_dx = sizeof(T) == 8 ? (T)(1.0 / g.dx) : (T)g.inv_dx;
    const T half_inv_dx = sizeof(T) == 8 ? (T)(0.5 / g.dx) : (T)g.half_inv_dx;
    const T half_dx_over_eps = sizeof(T) == 8 ? (T)(g.dx / (2.0 * 8.85418781e-12)) : (T)g.half_dx_over_eps;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        if (j < per_thread) {
            const int i = first + j;
            if (i < n) {
                T pk = pot_s[i];
                T e;
                if (i == 0) e = (pk - pot_s[1]) * inv_dx - rho[j] * half_dx_over_eps;
                else if (i == n - 1) e = (pot_s[n - 2] - pk) * inv_dx + rho[j] * half_dx_over_eps;
                else e = (pot_s[i - 1] - pot_s[i + 1]) * half_inv_dx;
                pot_out[i] = (float)pk;
                efield_out[i] = (float)e;
            }
        }
    }
}

// The densities of PT consecutive nodes from `first` (0 past n - 1), through
// L2 (see poisson_body); vec: both arrays 16-byte aligned.
template <int PT>
__device__ __forceinline__ void load_nodes(const float *__restrict__ d, int first, int n, bool vec, float (&v)[PT]) {
    if (PT % 4 == 0 && vec && first + PT <= n) {
#pragma unroll
        for (int j = 0; j < PT; j += 4) {
            const float4 q = __ldcg(reinterpret_cast<const float4 *>(d + first + j));
            v[j] = q.x;
            v[j + 1] = q.y;
            v[j + 2] = q.z;
            v[j + 3] = q.w;
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < PT; ++j) v[j] = first + j < n ? __ldcg(d + first + j) : 0.0f;
}

// The solve in FP64 by one scan (see the head of this file); arguments as
// poisson_body's.  PT consecutive nodes per thread, blockDim.x * PT >= n_g.
template <int PT>
__device__ __forceinline__ void poisson_fused(const float *__restrict__ e_density, const float *__restrict__ i_density,
                                              float *__restrict__ pot_out, float *__restrict__ efield_out,
                                              float pot0_arg, const float *__restrict__ pot0_table,
                                              uint32_t *__restrict__ step_counter, const cudapic_grid &g,
                                              float *__restrict__ zero_a, float *__restrict__ zero_b) {
    __shared__ double w_f[32], w_g[32];
    __shared__ float s_pot0;
    const int n = (int)g.n_g;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int first = tid * PT;
    const double e_charge = 1.60217662e-19;
    const double alpha_e = -g.dx * g.dx / 8.85418781e-12 * e_charge;
    const double inv_n1 = 1.0 / (double)(n - 1);  // the divisions ahead of the loads they do not depend on
    const double inv_dx = 1.0 / g.dx;
    const double half_dx_over_eps = g.dx / (2.0 * 8.85418781e-12);
    const bool vec = ((reinterpret_cast<uintptr_t>(e_density) | reinterpret_cast<uintptr_t>(i_density)) & 15u) == 0;
    float de[PT], di[PT];
    load_nodes<PT>(e_density, first, n, vec, de);
    load_nodes<PT>(i_density, first, n, vec, di);
    float p0 = pot0_arg;
    if (tid == 0 && pot0_table) {
        const uint32_t t = *step_counter;
        p0 = pot0_table[t % g.n_t];
        *step_counter = t + 1;
    }
    double f[PT];
    double sum_f = 0.0, sum_g = 0.0;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        const int i = first + j;
        f[j] = i >= 1 && i <= n - 2 ? alpha_e * ((double)di[j] - (double)de[j]) : 0.0;
        sum_f += f[j];
        sum_g += (double)i * f[j];
    }
    // charge densities at the electrodes (the one-sided field differences)
    const double rho_first = e_charge * ((double)di[0] - (double)de[0]);  // used by node 0 only
    double rho_last = 0.0;                                                // used by node n - 1 only
#pragma unroll
    for (int j = 0; j < PT; ++j)
        if (first + j == n - 1) rho_last = e_charge * ((double)di[j] - (double)de[j]);
    double in_f = sum_f, in_g = sum_g;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double a = __shfl_up_sync(0xffffffffu, in_f, o), b = __shfl_up_sync(0xffffffffu, in_g, o);
        if (lane >= o) {
            in_f += a;
            in_g += b;
        }
    }
    if (lane == 31) {
        w_f[warp] = in_f;
        w_g[warp] = in_g;
    }
    if (tid == 0) s_pot0 = p0;
    __syncthreads();
    // next-step accumulators of the driver (never the densities read here)
    for (int k = tid; k < n; k += blockDim.x) {
        if (zero_a) zero_a[k] = 0.0f;
        if (zero_b) zero_b[k] = 0.0f;
    }
    if (warp * 32 * PT >= n) return;  // no node in this warp
    double tf = lane < nwarps ? w_f[lane] : 0.0, tg = lane < nwarps ? w_g[lane] : 0.0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {  // every warp scans the warp totals itself: no second barrier
        const double a = __shfl_up_sync(0xffffffffu, tf, o), b = __shfl_up_sync(0xffffffffu, tg, o);
        if (lane >= o) {
            tf += a;
            tg += b;
        }
    }
    const double all_f = __shfl_sync(0xffffffffu, tf, 31), all_g = __shfl_sync(0xffffffffu, tg, 31);
    const double before_f = __shfl_sync(0xffffffffu, tf, warp > 0 ? warp - 1 : 0);
    const double before_g = __shfl_sync(0xffffffffu, tg, warp > 0 ? warp - 1 : 0);
    double run_f = in_f - sum_f + (warp > 0 ? before_f : 0.0);
    double run_g = in_g - sum_g + (warp > 0 ? before_g : 0.0);
    const double pot0 = (double)s_pot0;
    const double c = (all_g - pot0) * inv_n1 - all_f;
    constexpr int W = PT % 4 == 0 ? 4 : 1;  // nodes per store
    const bool vec_out = W == 4 && ((reinterpret_cast<uintptr_t>(pot_out) | reinterpret_cast<uintptr_t>(efield_out)) & 15u) == 0;
#pragma unroll
    for (int j0 = 0; j0 < PT; j0 += W) {
        float p[W], e[W];
#pragma unroll
        for (int u = 0; u < W; ++u) {
            const int j = j0 + u, i = first + j;
            run_f += f[j];
            run_g += (double)i * f[j];
            double pi = pot0 - run_g + (double)i * (c + run_f), ei = -(c + run_f - 0.5 * f[j]) * inv_dx;
            if (i == 0) {
                pi = pot0;
                ei = -c * inv_dx - rho_first * half_dx_over_eps;
            } else if (i == n - 1) {
                pi = 0.0;
                ei = -(c + run_f) * inv_dx + rho_last * half_dx_over_eps;
            }
            p[u] = (float)pi;
            e[u] = (float)ei;
        }
        // several nodes per thread: scalar stores would be one sector each
        if (vec_out && first + j0 + W <= n) {
            *reinterpret_cast<float4 *>(pot_out + first + j0) = make_float4(p[0], p[W > 1 ? 1 : 0], p[W > 2 ? 2 : 0], p[W > 3 ? 3 : 0]);
            *reinterpret_cast<float4 *>(efield_out + first + j0) = make_float4(e[0], e[W > 1 ? 1 : 0], e[W > 2 ? 2 : 0], e[W > 3 ? 3 : 0]);
        } else {
#pragma unroll
            for (int u = 0; u < W; ++u) {
                if (first + j0 + u < n) {
                    pot_out[first + j0 + u] = p[u];
                    efield_out[first + j0 + u] = e[u];
                }
            }
        }
    }
}

// The solve of a driver or a drop-in call: FP64 sums (T = double) by one
// scan, or the reference's f32 arithmetic.
template <typename T, int PT>
__device__ __forceinline__ void poisson_solve(const float *__restrict__ e_density, const float *__restrict__ i_density,
                                              float *__restrict__ pot_out, float *__restrict__ efield_out,
                                              float pot0_arg, const float *__restrict__ pot0_table,
                                              uint32_t *__restrict__ step_counter, const cudapic_grid &g,
                                              float *__restrict__ zero_a, float *__restrict__ zero_b) {
    if constexpr (sizeof(T) == 8)
        poisson_fused<PT>(e_density, i_density, pot_out, efield_out, pot0_arg, pot0_table, step_counter, g, zero_a,
                          zero_b);
    else
        poisson_body<T, PT>(e_density, i_density, pot_out, efield_out, pot0_arg, pot0_table, step_counter, g, zero_a,
                            zero_b);
}
// Dynamic shared memory of poisson_solve.
template <typename T>
constexpr size_t poisson_solve_smem(uint32_t n_g) {
    return sizeof(T) == 8 ? 0 : (size_t)n_g * sizeof(T);
}

}  // namespace cudapic
