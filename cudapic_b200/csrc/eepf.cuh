// eepf.cuh -- one step's EEPF samples, by the CTAs of the kernel of its own
// (kernels_mcc.cu) or beside the next step's solve (kernels_poisson.cu).
#pragma once
#include "common.cuh"
#include "internal.h"

namespace cudapic {

// accumulate_eepf, Rust-CUDA/src/main.rs:1301-1339: per-block shared
// histogram, one global atomic per non-empty bin and block.  Four consecutive
// positions per thread and round (vec: one 16-byte load; x must be aligned),
// velocities only of the electrons in the window; the centre-energy sums are
// reduced over the block before their two global atomics (one pair per warp
// serialised thousands of atomics on two addresses): 400 000 electrons 9.5 us,
// now 5.3 us.  CTA `block` of `blocks`, whole warps, at most 1024 threads.
__device__ __forceinline__ void eepf_accumulate(const EepfSamples &a, const cudapic_grid &g, bool vec, uint32_t block,
                                                uint32_t blocks) {
    __shared__ uint32_t h[N_EEPF];
    __shared__ double s_sum[32];
    __shared__ uint32_t s_cnt[32];
    for (uint32_t k = threadIdx.x; k < N_EEPF; k += blockDim.x) h[k] = 0;
    __syncthreads();
    grid_dep_wait();
    const uint32_t n = load_count(a.active_e, g.capacity, g.dev_err);
    const float *x = a.x, *vx = a.vx, *vy = a.vy, *vz = a.vz, *efield = a.efield;
    double e_sum = 0.0;
    uint32_t e_cnt = 0;
    auto sample = [&](uint32_t i, float xi) {
        if (xi <= g.min_x || xi >= g.max_x) return;
        const float pos = xi * g.inv_dx;
        const int p = cell_of(pos, g.n_g);
        const float c2 = pos - (float)p;
        const float e_x = (1.0f - c2) * __ldg(efield + p) + c2 * __ldg(efield + p + 1);
        const float mvx = vx[i] - 0.5f * e_x * g.eepf_half_kick;
        const float vyi = vy[i], vzi = vz[i];
        const float v2 = mvx * mvx + vyi * vyi + vzi * vzi;
        const float energy = g.half_me_over_e * v2;
        const float binf = energy / DE_EEPF_F;
        if (binf < (float)N_EEPF) atomicAdd(&h[(uint32_t)binf], 1u);
        e_sum += (double)energy;
        ++e_cnt;
    };
    const uint64_t stride = (uint64_t)blocks * blockDim.x;
    for (uint64_t j = (uint64_t)block * blockDim.x + threadIdx.x; 4u * j < n; j += stride) {
        const uint32_t i0 = (uint32_t)(4u * j);
        float xs[4];
        if (vec && i0 + 4u <= n) {
            const float4 X = *reinterpret_cast<const float4 *>(x + i0);
            xs[0] = X.x;
            xs[1] = X.y;
            xs[2] = X.z;
            xs[3] = X.w;
        } else {
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) xs[u] = i0 + u < n ? x[i0 + u] : g.min_x;  // min_x: not sampled
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) sample(i0 + u, xs[u]);
    }
    if (a.esum) {  // mean energy of the sampled electrons (the report's centre energy)
        for (int o = 16; o > 0; o >>= 1) {
            e_sum += __shfl_down_sync(0xffffffffu, e_sum, o);
            e_cnt += __shfl_down_sync(0xffffffffu, e_cnt, o);
        }
        if ((threadIdx.x & 31) == 0) {
            s_sum[threadIdx.x >> 5] = e_sum;
            s_cnt[threadIdx.x >> 5] = e_cnt;
        }
    }
    __syncthreads();
    if (a.esum && threadIdx.x == 0) {
        unsigned long long c = 0;
        e_sum = 0.0;
        for (int w = 0; w < (int)(blockDim.x / 32); ++w) {
            e_sum += s_sum[w];
            c += s_cnt[w];
        }
        if (c) {
            atomicAdd(a.esum, e_sum);
            atomicAdd(a.ecount, c);
        }
    }
    for (uint32_t k = threadIdx.x; k < N_EEPF; k += blockDim.x)
        if (h[k]) atomicAdd(&a.eepf[k], h[k]);
}

}  // namespace cudapic
