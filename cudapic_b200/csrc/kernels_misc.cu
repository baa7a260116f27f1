// kernels_misc.cu -- RNG seeding (jump), the RNG known-answer wrapper and
// the math self-evaluation entry point.
//
// References: xoshiro128_seed_streams, Rust-CUDA/src/main.rs:1446-1496 (host,
// O(128 n) sequential jumps); xoshiro128p_test_wrapper, :1341-1357.
//
// Seeding on the GPU: xoshiro128+ is linear over GF(2), so stream k = J^k m
// (m = master state, J = the 128x128 bit matrix of one jump); the matrices
// J^(2^l), l = 0..27, are generated at build time (gen_jump_tables.py).
// CTA c produces the streams [k0, k0 + 256 R), k0 = 256 R c:
//  1. one warp forms J^k0 m from the set bits of k0, four matrix columns per
//     lane and an XOR reduction over the warp; meanwhile the other warps
//     build the product table of step 3;
//  2. the CTA doubles that state to 256 consecutive ones (t + 2^l from t with
//     the matrix of level l, one warp per product: 255 products in all);
//  3. each thread then steps by J^256, R - 1 times, storing one state per
//     step: the stores of a warp are consecutive.  The product is 22 table
//     lookups (6 bits of the state each, 128 B of shared memory per row: the
//     16-byte product repeated for 8 lanes, so that the 8 lanes which a
//     128-bit shared load serves together always use different banks).
// Bound by the shared loads: 22 x 4 wavefronts per 32 streams and SM.  A
// product by masked columns (128 x 6 instructions) was bound by instructions
// and stored 16 consecutive streams per thread, uncoalesced: 2 097 155 streams
// took 277 us, now 35 us (byte tables of 64 KB have fewer lookups but about
// 2.7 lanes per bank; nibble tables 32 lookups).
// Bit-identical to the sequential host loop.
#include "common.cuh"
#include "detmath.cuh"
#include "internal.h"
#include "rng.cuh"
#include "tma.cuh"

#include "generated/jump_tables.inc"

namespace cudapic {

constexpr int SEED_THREADS = 256;
constexpr int SEED_WARPS = SEED_THREADS / 32;
constexpr int SEED_LEVEL = 8;             // a thread steps by J^(2^8) = J^SEED_THREADS
constexpr int SEED_GROUPS = 22;           // 6-bit groups of a 128-bit state (the last one: 2 bits)
constexpr uint32_t SEED_ROWS = 21u * 64u + 4u;
constexpr size_t SEED_TABLE_BYTES = (size_t)SEED_ROWS * 128;
static_assert((1 << SEED_LEVEL) == SEED_THREADS, "a step covers the CTA's threads");

__device__ __forceinline__ void xor4(uint4 &a, const uint4 &b) {
    a.x ^= b.x;
    a.y ^= b.y;
    a.z ^= b.z;
    a.w ^= b.w;
}

// The calling lane's four columns (4 lane .. 4 lane + 3) of level l.
__device__ __forceinline__ void seed_columns(int l, int lane, uint4 (&c)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) c[q] = __ldg(&d_jump_pow[l][4 * lane + q]);
}

// Matrix-vector product by one warp (all lanes hold the state s and their
// four columns c); every lane gets the product.
__device__ __forceinline__ uint4 seed_product(const uint4 &s, const uint4 (&c)[4], int lane) {
    const uint32_t word = lane < 16 ? (lane < 8 ? s.x : s.y) : (lane < 24 ? s.z : s.w);
    const uint32_t bits = word >> ((4 * lane) & 31);
    uint4 acc = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint32_t m = 0u - ((bits >> q) & 1u);
        acc.x ^= c[q].x & m;
        acc.y ^= c[q].y & m;
        acc.z ^= c[q].z & m;
        acc.w ^= c[q].w & m;
    }
    acc.x = __reduce_xor_sync(0xffffffffu, acc.x);
    acc.y = __reduce_xor_sync(0xffffffffu, acc.y);
    acc.z = __reduce_xor_sync(0xffffffffu, acc.z);
    acc.w = __reduce_xor_sync(0xffffffffu, acc.w);
    return acc;
}

// Rows first, first + stride, ...: row 64 g + v is the XOR of the columns
// 6 g + i of level SEED_LEVEL over the set bits i of v, repeated 8 times (in
// an order rotated by the lane: conflict-free stores).
__device__ __forceinline__ void seed_fill_table(uint4 *tab, uint32_t first, uint32_t stride, int lane) {
    for (uint32_t row = first; row < SEED_ROWS; row += stride) {
        const uint32_t g = row >> 6, v = row & 63u;
        uint4 e = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (uint32_t i = 0; i < 6; ++i)
            if (v >> i & 1u) xor4(e, __ldg(&d_jump_pow[SEED_LEVEL][6u * g + i]));  // g = 21: v < 4
#pragma unroll
        for (uint32_t r = 0; r < 8; ++r) tab[row * 8u + ((r + (uint32_t)lane) & 7u)] = e;
    }
}

// J^SEED_THREADS s from the table (mine: the table at this lane's copy).
__device__ __forceinline__ uint4 seed_step(const uint4 &s, const uint4 *mine) {
    const uint32_t w[5] = {s.x, s.y, s.z, s.w, 0u};
    uint4 acc = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int g = 0; g < SEED_GROUPS; ++g) {
        const int bit = 6 * g, k = bit >> 5, sh = bit & 31;
        const uint32_t v = __funnelshift_r(w[k], w[k + 1], sh) & 63u;  // the last group reads zeros past bit 127
        xor4(acc, mine[(64u * (uint32_t)g + v) * 8u]);
    }
    return acc;
}

__global__ void __launch_bounds__(SEED_THREADS)
    seed_streams_kernel(uint4 master, uint32_t n, uint32_t per_thread, uint32_t *__restrict__ r0,
                        uint32_t *__restrict__ r1, uint32_t *__restrict__ r2, uint32_t *__restrict__ r3) {
    extern __shared__ __align__(128) unsigned char seed_smem[];
    uint4 *tab = reinterpret_cast<uint4 *>(seed_smem);  // [SEED_ROWS][8] (per_thread > 1)
    __shared__ uint4 st[SEED_THREADS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t k0 = blockIdx.x * (SEED_THREADS * per_thread);  // < n <= 2^28
    if (warp == 0) {
        uint4 s = master, c[4];
        uint32_t left = k0;
        if (left) seed_columns(__ffs(left) - 1, lane, c);
        while (left) {  // the next level's columns are fetched during this level's product
            left &= left - 1u;
            uint4 next[4] = {};
            if (left) seed_columns(__ffs(left) - 1, lane, next);
            s = seed_product(s, c, lane);
#pragma unroll
            for (int q = 0; q < 4; ++q) c[q] = next[q];
        }
        if (lane == 0) st[0] = s;
    } else if (per_thread > 1) {
        seed_fill_table(tab, (uint32_t)(tid - 32), SEED_THREADS - 32, lane);
    }
    uint4 c[4];
    seed_columns(0, lane, c);
#pragma unroll
    for (int l = 0; l < SEED_LEVEL; ++l) {
        uint4 next[4] = {};
        if (l + 1 < SEED_LEVEL) seed_columns(l + 1, lane, next);
        __syncthreads();
        for (int t = warp; t < (1 << l); t += SEED_WARPS) {
            const uint4 p = seed_product(st[t], c, lane);
            if (lane == 0) st[t + (1 << l)] = p;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) c[q] = next[q];
    }
    __syncthreads();
    uint4 s = st[tid];
    const uint4 *mine = tab + (lane & 7);
    uint64_t k = (uint64_t)k0 + tid;
    for (uint32_t r = 0;;) {
        if (k >= n) break;
        r0[k] = s.x;
        r1[k] = s.y;
        r2[k] = s.z;
        r3[k] = s.w;
        if (++r == per_thread) break;
        s = seed_step(s, mine);
        k += SEED_THREADS;
    }
}

__global__ void xoshiro_test_kernel(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3, uint32_t *dest) {
    Xoshiro128p r{s0, s1, s2, s3};
    dest[0] = r.next();
    dest[1] = r.s0;
    dest[2] = r.s1;
    dest[3] = r.s2;
    dest[4] = r.s3;
}

__global__ void math_eval_kernel(int fn, const float *__restrict__ in, const float *__restrict__ in2,
                                 float *__restrict__ out, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = in[i];
    float r;
    switch (fn) {
    case 0: r = dm::expf_det(v); break;
    case 1: r = dm::logf_det(v); break;
    case 2: r = dm::sinf_det(v); break;
    case 3: r = dm::cosf_det(v); break;
    case 4: r = dm::tanf_det(v); break;
    case 5: r = dm::atanf_det(v); break;
    case 6: r = dm::acosf_det(v); break;
    default: r = dm::atan2f_det(v, in2[i]); break;
    }
    out[i] = r;
}

// Self-test of the bounded waits: thread 0 arms an mbarrier for 16 bytes of
// transfer that no copy will deliver, and every thread waits on it with a
// limit of `limit` SM clocks.  The wait runs out and the CTA reports
// CUDAPIC_DEVERR_TIMEOUT into dev_err, the route a stage wait of the
// streaming kernels takes when a bulk copy does not complete.  No copy is
// issued, so nothing is in flight when the kernel returns.
__global__ void wait_timeout_probe_kernel(uint32_t *dev_err, long long limit) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) mbar_arrive_expect_tx(&bar, 16u);
    __syncthreads();
    const bool ok = mbar_wait_bounded(&bar, 0u, limit);
    if (__syncthreads_or(!ok) && threadIdx.x == 0) set_dev_err(dev_err, CUDAPIC_DEVERR_TIMEOUT);
}

int launch_wait_timeout_probe(uint32_t *dev_err, long long limit, cudaStream_t stream) {
    wait_timeout_probe_kernel<<<1, 64, 0, stream>>>(dev_err, limit);
    return check_launch("wait_timeout_probe");
}

}  // namespace cudapic

using namespace cudapic;

extern "C" int cudapic_xoshiro128p_test_wrapper(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3, uint32_t *dest,
                                                cudapic_stream_t stream) {
    CUDAPIC_REQUIRE(dest, "xoshiro128p_test_wrapper: null pointer");
    xoshiro_test_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(s0, s1, s2, s3, dest);
    return check_launch("xoshiro128p_test_wrapper");
}

extern "C" int cudapic_xoshiro128_seed_streams(const uint32_t master[4], uint32_t n, uint32_t *rng0,
                                               uint32_t *rng1, uint32_t *rng2, uint32_t *rng3,
                                               cudapic_stream_t stream) {
    CUDAPIC_REQUIRE(master && rng0 && rng1 && rng2 && rng3, "xoshiro128_seed_streams: null pointer");
    CUDAPIC_REQUIRE((master[0] | master[1] | master[2] | master[3]) != 0u,
                    "xoshiro128_seed_streams: master state must not be all zero");
    CUDAPIC_REQUIRE((uint64_t)n <= (1ull << CUDAPIC_JUMP_LEVELS), "xoshiro128_seed_streams: n > 2^28");
    if (n == 0) return CUDAPIC_OK;
    const uint4 m = make_uint4(master[0], master[1], master[2], master[3]);
    // one CTA per SM, each a contiguous range of 256 x per_thread streams; up
    // to one stream per thread (n <= 256 SMs) nothing is stepped: no table
    const uint32_t step = (uint32_t)sm_count() * SEED_THREADS;
    const uint32_t per_thread = (n + step - 1) / step;
    const uint32_t block = SEED_THREADS * per_thread;
    const size_t smem = per_thread > 1 ? SEED_TABLE_BYTES : 0;
    CUDAPIC_CHECK(kernel_smem((const void *)seed_streams_kernel, smem, "xoshiro128_seed_streams"));
    seed_streams_kernel<<<(n + block - 1) / block, SEED_THREADS, smem, (cudaStream_t)stream>>>(m, n, per_thread, rng0,
                                                                                              rng1, rng2, rng3);
    return check_launch("xoshiro128_seed_streams");
}

extern "C" int cudapic_math_eval(int fn, const float *in, const float *in2, float *out, uint32_t n,
                                 cudapic_stream_t stream) {
    CUDAPIC_REQUIRE(in && out && fn >= 0 && fn <= 7 && (fn != 7 || in2), "math_eval: bad arguments");
    if (n == 0) return CUDAPIC_OK;
    math_eval_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(fn, in, in2, out, n);
    return check_launch("math_eval");
}
