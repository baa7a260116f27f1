// kernels_mcc.cu -- Monte-Carlo collisions of electrons and ions.
//
// Reference: check_collisions_e / collision_e, Rust-CUDA/src/main.rs:971-1165,
// check_collisions_i / collision_i, :1167-1292.  Per electron: energy index
// min(int(E/1 meV + 0.5), 1e6-1), nu = sigma_tot(E) |v|, collide iff
// u < 1 - exp(-nu dt); the type (elastic / excitation / ionization) from
// the cumulative cross-section ratios; Euler-angle rotation of the relative
// velocity; ionization spawns an electron and an ion.  Per ion: a Maxwellian
// target atom (Box-Muller), relative energy, isotropic or backward
// scattering.  The RNG draw order of the reference is kept exactly.
//
// B200 design: HBM-bound streaming (28 B read + 16 B RNG written per
// particle; velocities written only by colliders, ~0.5 % of electrons per
// step at the reference conditions).  Two kernels share the physics:
//  * streaming kernel (default, cudapic_tuning.mcc_variant = 1): one
//    1024-thread CTA per SM, 16-byte loads, a certain rejection that needs no
//    table; what it leaves open goes to warp-private queues drained 32 at a
//    time -- no block barrier in the main loop;
//  * bulk-copy kernel (mcc_variant = 2): tiles of the seven SoA arrays staged
//    by cp.async.bulk on mbarriers, the full test on every particle (its
//    provably exact fast reject skips exp() for almost all), a CTA-wide
//    collider queue.
// Common to both:
//  * particles that the test rejects store their advanced RNG state
//    (coalesced);
//  * a collider keeps its slot and its RNG state before the test; the drain
//    re-runs the deterministic test and scatters it on a full warp (one
//    collider per lane) instead of one lane in 32;
//  * ionization spawns claim slots with one warp-aggregated atomicAdd per
//    counter, bounded by capacity: a spawn that does not fit is dropped and
//    flagged, never written out of bounds (the reference writes unbounded,
//    :1132-1149);
//  * transcendentals from detmath.cuh (bit-reproducible, see there).
#include "common.cuh"
#include "eepf.cuh"
#include "internal.h"
#include "mcc.cuh"
#include "step.cuh"
#include "tma.cuh"

namespace cudapic {

constexpr int MCC_THREADS = 256;

// ------------------------------------------------------------------ bulk-copy kernels

constexpr int MT_U = 2;                       // particles per thread and tile
constexpr int MT_TILE = MCC_THREADS * MT_U;   // 512
constexpr int MT_MAX_STAGES = 4;              // pipeline depth: cudapic_tuning.mcc_stages
constexpr int MT_ARRAYS = 7;                  // vx, vy, vz, rng0..3
constexpr int MT_QFLUSH = 256;                // drain the queue when it holds more
constexpr int MT_QCAP = MT_QFLUSH + MT_TILE;  // never overflows: one tile adds <= 512
constexpr int MT_QWORDS = 5;                  // slot index + the RNG state before the test

size_t mcc_tma_smem_bytes(int stages) {
    return (size_t)stages * MT_ARRAYS * MT_TILE * 4 + (size_t)MT_QCAP * MT_QWORDS * 4 +
           (size_t)stages * sizeof(uint64_t);
}

// ION = false: check_collisions_e; ION = true: check_collisions_i.
// A queued collider keeps only its slot and its RNG state before the test;
// the drain re-runs the (deterministic) test from that state, reading the
// velocity again, and continues into the scattering.
template <bool ION, bool EVENTS>
__global__ void __launch_bounds__(MCC_THREADS, 4)
    check_collisions_tma_kernel(const float *__restrict__ sigma_tot, const float *__restrict__ cs,
                                const uint32_t *__restrict__ active, float *x, float *vx, float *vy, float *vz,
                                uint32_t *rng0, uint32_t *rng1, uint32_t *rng2, uint32_t *rng3, float *ix,
                                float *ivx, float *ivy, float *ivz, uint32_t *alive_e, uint32_t *alive_i,
                                uint8_t *events, const __grid_constant__ cudapic_grid g, int stages,
                                float *dep_e, float *dep_i, unsigned long long *coll, float ion_k) {
    extern __shared__ __align__(128) unsigned char smem[];
    uint32_t *in = reinterpret_cast<uint32_t *>(smem);             // [stages][7][TILE]
    uint32_t *queue = in + stages * MT_ARRAYS * MT_TILE;           // [5][QCAP]
    uint64_t *bar = reinterpret_cast<uint64_t *>(queue + MT_QWORDS * MT_QCAP);
    __shared__ uint32_t s_q;
    __shared__ int s_ready;

    const int tid = threadIdx.x;
    grid_dep_wait();
    const uint32_t n = load_count(active, g.capacity, g.dev_err);
    const uint32_t ntiles = (n + MT_TILE - 1) / MT_TILE;
    const void *src[MT_ARRAYS] = {vx, vy, vz, rng0, rng1, rng2, rng3};

    auto issue = [&](uint32_t tile, int stage) {
        const uint32_t t0 = tile * MT_TILE;
        const uint32_t cnt = min((uint32_t)MT_TILE, n - t0);
        const uint32_t bytes = ((cnt + 3u) & ~3u) * 4u;
        mbar_arrive_expect_tx(&bar[stage], MT_ARRAYS * bytes);
#pragma unroll
        for (int a = 0; a < MT_ARRAYS; ++a)
            bulk_load(in + (stage * MT_ARRAYS + a) * MT_TILE, static_cast<const uint32_t *>(src[a]) + t0, bytes,
                      &bar[stage]);
    };

    const GlobalTable table{sigma_tot};
    // Drains the collider queue: one collider per thread, full warps.
    auto drain = [&]() {
        const uint32_t qn = s_q;
        if (coll && tid == 0 && qn) atomicAdd(coll, (unsigned long long)qn);  // collision events (measurement)
        for (uint32_t q = tid; q < qn; q += MCC_THREADS) {
            const uint32_t i = queue[0 * MT_QCAP + q];
            Xoshiro128p rs{queue[1 * MT_QCAP + q], queue[2 * MT_QCAP + q], queue[3 * MT_QCAP + q],
                           queue[4 * MT_QCAP + q]};
            const float vxi = vx[i], vyi = vy[i], vzi = vz[i];
            uint32_t ev;
            if (ION) {
                const IonTest t = test_ion(vxi, vyi, vzi, rs, table, g);
                ev = collide_ion(i, t.idx, vxi, vyi, vzi, t.vxa, t.vya, t.vza, rs, cs, vx, vy, vz, g);
            } else {
                const Test t = test_electron(vxi, vyi, vzi, rs, table, g);
                ev = collide_electron(0u, i, t.idx, vxi, vyi, vzi, rs, cs, x, vx, vy, vz, ix, ivx, ivy, ivz, alive_e,
                                      alive_i, g, dep_e, dep_i);
            }
            rng0[i] = rs.s0;
            rng1[i] = rs.s1;
            rng2[i] = rs.s2;
            rng3[i] = rs.s3;
            if (EVENTS) events[i] = (uint8_t)ev;
        }
        __syncthreads();
        if (tid == 0) s_q = 0;
        __syncthreads();
    };

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) mbar_init(&bar[s], 1);
        fence_mbar_init();
        s_q = 0;
    }
    __syncthreads();
    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            const uint32_t tile = blockIdx.x + (uint32_t)s * gridDim.x;
            if (tile < ntiles) issue(tile, s);
        }
    }

    uint32_t it = 0;
    for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
        const int s = (int)(it % (uint32_t)stages);
        const uint32_t parity = (it / (uint32_t)stages) & 1u;
        if (tid == 0) {
            const int ok = mbar_wait_bounded(&bar[s], parity) ? 1 : 0;
            if (!ok) set_dev_err(g.dev_err, CUDAPIC_DEVERR_TIMEOUT);
            s_ready = ok;
        }
        __syncthreads();
        if (!s_ready) return;
        const uint32_t t0 = tile * MT_TILE;
        const uint32_t cnt = min((uint32_t)MT_TILE, n - t0);
        const uint32_t *b = in + s * MT_ARRAYS * MT_TILE;
#pragma unroll
        for (int u = 0; u < MT_U; ++u) {
            const uint32_t j = (uint32_t)u * MCC_THREADS + tid;
            if (j < cnt) {
                const uint32_t i = t0 + j;
                const uint32_t q0 = b[3 * MT_TILE + j], q1 = b[4 * MT_TILE + j], q2 = b[5 * MT_TILE + j],
                               q3 = b[6 * MT_TILE + j];
                Xoshiro128p rs{q0, q1, q2, q3};
                const float vxi = __uint_as_float(b[0 * MT_TILE + j]);
                const float vyi = __uint_as_float(b[1 * MT_TILE + j]);
                const float vzi = __uint_as_float(b[2 * MT_TILE + j]);
                bool collide;
                if (ION) collide = ion_collides(vxi, vyi, vzi, rs, table, g, ion_k);
                else collide = test_electron(vxi, vyi, vzi, rs, table, g).collide;
                if (collide) {
                    const uint32_t q = atomicAdd(&s_q, 1u);
                    queue[0 * MT_QCAP + q] = i;
                    queue[1 * MT_QCAP + q] = q0;
                    queue[2 * MT_QCAP + q] = q1;
                    queue[3 * MT_QCAP + q] = q2;
                    queue[4 * MT_QCAP + q] = q3;
                } else {
                    rng0[i] = rs.s0;
                    rng1[i] = rs.s1;
                    rng2[i] = rs.s2;
                    rng3[i] = rs.s3;
                    if (EVENTS) events[i] = 0;
                }
            }
        }
        __syncthreads();  // stage consumed; queue count visible
        if (tid == 0) {
            const uint32_t next = tile + (uint32_t)stages * gridDim.x;
            if (next < ntiles) issue(next, s);
        }
        if (s_q > (uint32_t)MT_QFLUSH) drain();
    }
    __syncthreads();
    if (s_q > 0) drain();
}

// ------------------------------------------------------------------ streaming kernel
//
// One 1024-thread CTA per SM, no bulk copies and no block barrier in the main
// loop; a warp takes tiles of 128 particles, four consecutive ones per lane
// (16-byte loads where the planes are aligned and the group whole):
//  * the certain rejection decides for nearly every particle without the
//    table, a square root, a division or the target atom: electrons by
//    may_collide's bound (step.cuh), ions by ion_collides' bound with the
//    square root taken out (ion_surely_passes).  Both need the largest entry
//    of the table the particle can meet: given by the caller (the bounded ion
//    entry, the drivers), or found here, over the first MS_TABLE entries, by
//    the CTAs of a cluster (half of the entries each, while the first
//    tiles are on their way into L2); particles that
//    could meet a higher entry's energy are not decided by it;
//  * undecided particles go to a queue private to their warp (slot and RNG
//    state before the test); whenever it holds 32 the warp takes 32 of them,
//    one per lane, through the full test and, colliding, the scattering --
//    only __syncwarp, no block-wide synchronisation.  A tile with many of them
//    takes the full test first and queues its colliders (MS_DENSE_E).
// Bound by memory (44 B per particle).  With the first 32768 entries copied to
// every SM's shared memory and the full test on every particle (128 KB per
// CTA and launch, scalar loads, a square root and a division each) 2 000 001
// electrons took 30.3 us, now 25.5; 4 194 304 ions 49.4, now 40.1 (bounded); 1000
// of either 8.0, now 6.7 and 4.7 (kernel alone).  Prefetching every tile and not
// only the first into L2 gave nothing more.

constexpr int MS_THREADS = 1024;
constexpr int MS_WARPS = MS_THREADS / 32;
constexpr int MS_ROW = 4;                       // particles per lane and tile
constexpr int MS_TILE = 32 * MS_ROW;
constexpr int MS_QCAP = 32 + MS_TILE;           // a warp drains at 32; one tile adds <= 128
constexpr size_t MS_SMEM = (size_t)MS_WARPS * 5 * MS_QCAP * sizeof(uint32_t);
constexpr int MS_CLUSTER = 2;                   // the largest that still reaches every SM (4 leaves some idle)
constexpr uint32_t MS_TABLE = 32768;            // entries whose maximum a launch looks for
constexpr float MS_TABLE_EV = 32.7f;            // energies below have an index below MS_TABLE
// Undecided particles of a tile beyond which all of its undecided take the
// full test where they are: a queue's particles are gathered again, 32 at a
// time, which pays for a few of 128 and not for a hot or strongly collisional
// population.  2 000 001 electrons of 3 / 30 / 1000 eV (a call, 10 Pa) took 31 /
// 82 / 118 us by the queue alone, now 28 / 38 / 38 (34 / 43 / 40 with the full
// test on every particle, its table in shared memory); ions of 500 eV at 100 Pa,
// bounded, 77, now 48 (52).  Between the two forms the calls cross at a quarter
// to a half of a tile.  That full test stays ahead where nearly every particle
// is tested and scatters: 30 eV at 100 / 1000 Pa 55 / 121 us, here 59 / 138.
constexpr int MS_DENSE_E = 32, MS_DENSE_I = 48;

// The larger of two floats, NaN (the canonical one, 0x7fffffff) if either is.
__device__ __forceinline__ float max_nan(float a, float b) {
    float m;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
    return m;
}

template <bool ION, bool EVENTS, bool BOUNDED>
__global__ void __launch_bounds__(MS_THREADS, 1)
    check_collisions_stream_kernel(const float *__restrict__ sigma_tot, const float *__restrict__ cs,
                                   const uint32_t *__restrict__ active, float *x, float *vx, float *vy, float *vz,
                                   uint32_t *rng0, uint32_t *rng1, uint32_t *rng2, uint32_t *rng3, float *ix,
                                   float *ivx, float *ivy, float *ivz, uint32_t *alive_e, uint32_t *alive_i,
                                   uint8_t *events, const __grid_constant__ cudapic_grid g, int vec, float *dep_e,
                                   float *dep_i, unsigned long long *coll, float ion_k) {
    extern __shared__ __align__(16) uint32_t ms_smem[];
    __shared__ uint32_t s_max[MS_WARPS], s_top;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    uint32_t *wq = ms_smem + (size_t)warp * 5 * MS_QCAP;  // [5][QCAP]
    const unsigned lt = lanemask_lt();
    const float dt = ION ? g.dt_i : g.dt_e;
    grid_dep_wait();
    const uint32_t n = load_count(active, g.capacity, g.dev_err);

    // largest energy-indexed entry the certain rejection may assume, and the
    // largest v.v it then holds for
    float k = ion_k;  // BOUNDED: max(sigma_tot) dt, rounded up
    float v2_max = INFINITY;
    if (!BOUNDED) {
        const uint32_t j = (blockIdx.x + (uint32_t)warp * gridDim.x) * MS_TILE + (uint32_t)lane * MS_ROW;
        if (j < n && (lane & 1) == 0) {  // one request per 32-byte sector of the warp's first tile
            for (const void *p : {(const void *)(vx + j), (const void *)(vy + j), (const void *)(vz + j),
                                  (const void *)(rng0 + j), (const void *)(rng1 + j), (const void *)(rng2 + j),
                                  (const void *)(rng3 + j)})
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
        }
        cg::cluster_group cluster = cg::this_cluster();
        constexpr uint32_t part = MS_TABLE / MS_CLUSTER;
        const float *mine = sigma_tot + cluster.block_rank() * part;
        // the largest of +0 and the entries: an entry below zero (or -0) never
        // lets a particle collide, a NaN stays and makes a bound that decides nothing
        float largest = 0.0f;
#pragma unroll
        for (uint32_t q = 0; q < part / MS_THREADS; ++q) largest = max_nan(largest, __ldg(mine + q * MS_THREADS + tid));
        uint32_t top = __float_as_uint(largest);  // non-negative or the canonical NaN: ordered as integers
        top = __reduce_max_sync(0xffffffffu, top);
        if (lane == 0) s_max[warp] = top;
        __syncthreads();
        if (warp == 0) {
            top = __reduce_max_sync(0xffffffffu, s_max[lane]);
            if (lane == 0) s_top = top;
        }
        cluster.sync();
        top = __reduce_max_sync(0xffffffffu, lane < MS_CLUSTER ? *cluster.map_shared_rank(&s_top, lane) : 0u);
        cluster.sync();  // no CTA leaves while its maximum is read
        const float sigma_max = __uint_as_float(top);
        k = ION ? sigma_max * dt * 1.00001f : sigma_max * dt;
        if (ION) {  // |g| <= |v| + 9.2 sigma for every target atom: its energy below MS_TABLE_EV
            const float v_max = sqrtf(MS_TABLE_EV / g.half_mu_over_e) - 9.21f * g.normal_range;
            v2_max = v_max > 0.0f ? v_max * v_max * 0.9999f : -1.0f;
        } else {
            v2_max = MS_TABLE_EV / g.half_me_over_e;
        }
    }
    const float k2 = k * k * 1.0001f;                 // the bound on (nu dt)^2 / v.v
    const float c = ion_bound_offset(k, g.normal_range);  // ions: beside it
    const GlobalTable table{sigma_tot};
    // the four particles of a lane: neighbours for the vector loads, else 32
    // apart, so that the scalar loads of a warp meet
    const uint32_t di = vec ? 1u : 32u;

    auto drain = [&](uint32_t first, uint32_t count) {  // lanes < count take entries first + lane
        bool hit = false;
        if ((uint32_t)lane < count) {
            const uint32_t q = first + lane;
            const uint32_t i = wq[0 * MS_QCAP + q];
            Xoshiro128p rs{wq[1 * MS_QCAP + q], wq[2 * MS_QCAP + q], wq[3 * MS_QCAP + q], wq[4 * MS_QCAP + q]};
            const float vxi = vx[i], vyi = vy[i], vzi = vz[i];
            uint32_t ev = 0;
            if (ION) {
                const IonTest t = test_ion(vxi, vyi, vzi, rs, table, g);
                hit = t.collide;
                if (hit) ev = collide_ion(i, t.idx, vxi, vyi, vzi, t.vxa, t.vya, t.vza, rs, cs, vx, vy, vz, g);
            } else {
                const Test t = test_electron(vxi, vyi, vzi, rs, table, g);
                hit = t.collide;
                if (hit)
                    ev = collide_electron(0u, i, t.idx, vxi, vyi, vzi, rs, cs, x, vx, vy, vz, ix, ivx, ivy, ivz, alive_e,
                                          alive_i, g, dep_e, dep_i);
            }
            rng0[i] = rs.s0;
            rng1[i] = rs.s1;
            rng2[i] = rs.s2;
            rng3[i] = rs.s3;
            if (EVENTS) events[i] = (uint8_t)ev;
        }
        if (coll) {  // collision events (measurement)
            const unsigned hits = __ballot_sync(0xffffffffu, hit);
            if (lane == 0 && hits) atomicAdd(coll, (unsigned long long)__popc(hits));
        }
        __syncwarp();
    };

    auto passes = [&](Xoshiro128p &rs, float v2) {  // the certain rejection; rs past the test's draws
        bool p;
        if (ION) {
            rs.next();  // the target atom's four draws
            rs.next();
            rs.next();
            rs.next();
            p = ion_surely_passes(rs.uniform(), v2, k2, c);
        } else {
            p = !may_collide(rs.uniform(), v2, k2);
        }
        return p && (BOUNDED || v2 < v2_max);
    };

    uint32_t qn = 0;  // entries in this warp's queue (warp-uniform)
    // A thread for each particle: one per lane, so that every warp has some of
    // the colliders.  A warp scatters 32 at a time, one lot after the other, and
    // with tiles of 128 three quarters of the warps have none: 1000 / 20 000 /
    // 120 000 electrons of 30 eV at 1000 Pa, a call, 33.3 / 33.0 / 36.1 us, now
    // 20.8 / 21.3 / 24.1; of 3 eV at 10 Pa 16.2 / 17.1 / 19.4, now 16.8 / 17.0 /
    // 17.9.
    const bool one = n <= gridDim.x * MS_THREADS;
    if (one) {
        const uint32_t i = (blockIdx.x + (uint32_t)warp * gridDim.x) * 32u + (uint32_t)lane;
        float vxi = 0.0f, vyi = 0.0f, vzi = 0.0f;
        Xoshiro128p r0{};
        if (i < n) {
            vxi = vx[i], vyi = vy[i], vzi = vz[i];
            r0 = Xoshiro128p{rng0[i], rng1[i], rng2[i], rng3[i]};
        }
        Xoshiro128p rs = r0;
        const bool undecided = !passes(rs, vxi * vxi + vyi * vyi + vzi * vzi) && i < n;
        if (i < n && !undecided) {
            rng0[i] = rs.s0;
            rng1[i] = rs.s1;
            rng2[i] = rs.s2;
            rng3[i] = rs.s3;
            if (EVENTS) events[i] = 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, undecided);
        if (undecided) {
            const uint32_t q = __popc(m & lt);
            wq[0 * MS_QCAP + q] = i;
            wq[1 * MS_QCAP + q] = r0.s0;
            wq[2 * MS_QCAP + q] = r0.s1;
            wq[3 * MS_QCAP + q] = r0.s2;
            wq[4 * MS_QCAP + q] = r0.s3;
        }
        qn = __popc(m);
    }
    // ions: this warp met a tile beyond MS_DENSE_I; its further tiles skip the bound (50 eV at 100 Pa, unbounded,
    // 54 us with it, 51 without; for electrons the flag cost 2 to 8 %)
    bool dense = false;
    // tile t to CTA t mod gridDim: every SM gets the same number to within one
    const uint32_t tiles = one ? 0u : (uint32_t)(((uint64_t)n + MS_TILE - 1) / MS_TILE);
    for (uint32_t t = blockIdx.x + (uint32_t)warp * gridDim.x; t < tiles; t += gridDim.x * MS_WARPS) {
        const uint32_t i0 = t * MS_TILE + (uint32_t)lane * (vec ? MS_ROW : 1u);
        const bool whole = vec && n - min(n, i0) >= MS_ROW;
        uint32_t s[4][MS_ROW];
        float v[3][MS_ROW];
        if (whole) {
            const float4 a = *reinterpret_cast<const float4 *>(vx + i0), b = *reinterpret_cast<const float4 *>(vy + i0);
            const float4 d = *reinterpret_cast<const float4 *>(vz + i0);
            const uint4 e = *reinterpret_cast<const uint4 *>(rng0 + i0), f = *reinterpret_cast<const uint4 *>(rng1 + i0);
            const uint4 h = *reinterpret_cast<const uint4 *>(rng2 + i0), w = *reinterpret_cast<const uint4 *>(rng3 + i0);
            v[0][0] = a.x, v[0][1] = a.y, v[0][2] = a.z, v[0][3] = a.w;
            v[1][0] = b.x, v[1][1] = b.y, v[1][2] = b.z, v[1][3] = b.w;
            v[2][0] = d.x, v[2][1] = d.y, v[2][2] = d.z, v[2][3] = d.w;
            s[0][0] = e.x, s[0][1] = e.y, s[0][2] = e.z, s[0][3] = e.w;
            s[1][0] = f.x, s[1][1] = f.y, s[1][2] = f.z, s[1][3] = f.w;
            s[2][0] = h.x, s[2][1] = h.y, s[2][2] = h.z, s[2][3] = h.w;
            s[3][0] = w.x, s[3][1] = w.y, s[3][2] = w.z, s[3][3] = w.w;
        } else {
#pragma unroll
            for (uint32_t u = 0; u < MS_ROW; ++u) {
                const bool in = i0 + u * di < n;
                v[0][u] = in ? vx[i0 + u * di] : 0.0f;
                v[1][u] = in ? vy[i0 + u * di] : 0.0f;
                v[2][u] = in ? vz[i0 + u * di] : 0.0f;
                s[0][u] = in ? rng0[i0 + u * di] : 0u;
                s[1][u] = in ? rng1[i0 + u * di] : 0u;
                s[2][u] = in ? rng2[i0 + u * di] : 0u;
                s[3][u] = in ? rng3[i0 + u * di] : 0u;
            }
        }
        uint32_t open = 0xfu;  // bit u: not decided by the bound (its state stays before the test)
        if (!whole) {
#pragma unroll
            for (uint32_t u = 0; u < MS_ROW; ++u)
                if (i0 + u * di >= n) open &= ~(1u << u);
        }
        if (!dense) {
#pragma unroll
            for (int u = 0; u < MS_ROW; ++u) {
                const float v2 = v[0][u] * v[0][u] + v[1][u] * v[1][u] + v[2][u] * v[2][u];
                Xoshiro128p rs{s[0][u], s[1][u], s[2][u], s[3][u]};
                if (passes(rs, v2)) {
                    s[0][u] = rs.s0;
                    s[1][u] = rs.s1;
                    s[2][u] = rs.s2;
                    s[3][u] = rs.s3;
                    open &= ~(1u << u);
                }
            }
        }
        if (ION) {
            dense = dense || __reduce_add_sync(0xffffffffu, __popc(open)) > MS_DENSE_I;
            if (dense) settle_ions(open, v, s, table, g);
        } else if (__reduce_add_sync(0xffffffffu, __popc(open)) > MS_DENSE_E) {
            settle_electrons(open, v, s, table, g);
        }
        if (whole) {  // open ones keep their state until their drain
            *reinterpret_cast<uint4 *>(rng0 + i0) = make_uint4(s[0][0], s[0][1], s[0][2], s[0][3]);
            *reinterpret_cast<uint4 *>(rng1 + i0) = make_uint4(s[1][0], s[1][1], s[1][2], s[1][3]);
            *reinterpret_cast<uint4 *>(rng2 + i0) = make_uint4(s[2][0], s[2][1], s[2][2], s[2][3]);
            *reinterpret_cast<uint4 *>(rng3 + i0) = make_uint4(s[3][0], s[3][1], s[3][2], s[3][3]);
        } else {
#pragma unroll
            for (uint32_t u = 0; u < MS_ROW; ++u) {
                if (i0 + u * di >= n) continue;
                rng0[i0 + u * di] = s[0][u];
                rng1[i0 + u * di] = s[1][u];
                rng2[i0 + u * di] = s[2][u];
                rng3[i0 + u * di] = s[3][u];
            }
        }
        if (EVENTS) {
#pragma unroll
            for (uint32_t u = 0; u < MS_ROW; ++u)
                if (i0 + u * di < n) events[i0 + u * di] = 0;  // an open one's own event follows with its drain
        }
        if (__ballot_sync(0xffffffffu, open != 0)) {
#pragma unroll
            for (int u = 0; u < MS_ROW; ++u) {
                const unsigned m = __ballot_sync(0xffffffffu, open >> u & 1u);
                if (open >> u & 1u) {
                    const uint32_t q = qn + __popc(m & lt);
                    wq[0 * MS_QCAP + q] = i0 + (uint32_t)u * di;
                    wq[1 * MS_QCAP + q] = s[0][u];
                    wq[2 * MS_QCAP + q] = s[1][u];
                    wq[3 * MS_QCAP + q] = s[2][u];
                    wq[4 * MS_QCAP + q] = s[3][u];
                }
                qn += __popc(m);
            }
            __syncwarp();
            while (qn >= 32) {  // full-warp drains from the top of the queue
                qn -= 32;
                drain(qn, 32);
            }
        }
    }
    __syncwarp();
    if (qn) drain(0, qn);
}

// accumulate_eepf as a launch of its own (eepf.cuh).
constexpr int EEPF_THREADS = 512;

__global__ void __launch_bounds__(EEPF_THREADS)
    accumulate_eepf_kernel(const EepfSamples a, const __grid_constant__ cudapic_grid g, int vec) {
    eepf_accumulate(a, g, vec != 0, blockIdx.x, gridDim.x);
}

namespace {

bool tma_ready(uint32_t capacity, std::initializer_list<const void *> ptrs) {
    if (capacity % 4u) return false;
    for (const void *p : ptrs)
        if (!aligned16(p)) return false;
    return true;
}

template <bool ION, bool EVENTS>
int launch_tma(const float *sigma_tot, const float *cs, const uint32_t *active, float *x, float *vx, float *vy,
               float *vz, uint32_t *r0, uint32_t *r1, uint32_t *r2, uint32_t *r3, float *ix, float *ivx, float *ivy,
               float *ivz, uint32_t *alive_e, uint32_t *alive_i, uint8_t *events, const cudapic_grid &g,
               cudaStream_t stream, float *dep_e, float *dep_i, unsigned long long *coll, float ion_k) {
    auto kern = check_collisions_tma_kernel<ION, EVENTS>;
    const cudapic_tuning t = tuning();
    const int stages = std::min(std::max(t.mcc_stages, 2), MT_MAX_STAGES);
    const size_t smem = mcc_tma_smem_bytes(stages);
    int per_sm = 0;
    CUDAPIC_CHECK(kernel_blocks((const void *)kern, MCC_THREADS, smem, &per_sm, "occupancy(check_collisions)"));
    per_sm = std::min(std::max(per_sm, 1), t.mcc_ctas_per_sm);
    const uint64_t tiles_max = ((uint64_t)g.capacity + MT_TILE - 1) / MT_TILE;
    const unsigned grid = persistent_grid(per_sm, tiles_max);
    return launch_kernel(ION ? "check_collisions_i" : "check_collisions_e", kern, dim3(grid), dim3(MCC_THREADS), smem,
                         stream, sigma_tot, cs, active, x, vx, vy, vz, r0, r1, r2, r3, ix, ivx, ivy, ivz, alive_e,
                         alive_i, events, g, stages, dep_e, dep_i, coll, ion_k);
}

template <bool ION, bool EVENTS, bool BOUNDED>
int launch_stream_t(const float *sigma_tot, const float *cs, const uint32_t *active, float *x, float *vx, float *vy,
                    float *vz, uint32_t *r0, uint32_t *r1, uint32_t *r2, uint32_t *r3, float *ix, float *ivx,
                    float *ivy, float *ivz, uint32_t *alive_e, uint32_t *alive_i, uint8_t *events,
                    const cudapic_grid &g, cudaStream_t stream, float *dep_e, float *dep_i,
                    unsigned long long *coll, float ion_k) {
    auto kern = check_collisions_stream_kernel<ION, EVENTS, BOUNDED>;
    const char *name = ION ? "check_collisions_i" : "check_collisions_e";
    CUDAPIC_CHECK(kernel_smem((const void *)kern, MS_SMEM, name));
    bool vec = true;
    for (const void *p : {(const void *)vx, (const void *)vy, (const void *)vz, (const void *)r0, (const void *)r1,
                          (const void *)r2, (const void *)r3})
        vec = vec && aligned16(p);
    constexpr unsigned cl = BOUNDED ? 1 : MS_CLUSTER;  // the unbounded kernel finds its bound in clusters
    unsigned grid = persistent_grid(1, ((uint64_t)g.capacity + MS_TILE - 1) / MS_TILE);
    grid = grid / cl * cl ? grid / cl * cl : cl;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(MS_THREADS);
    cfg.dynamicSmemBytes = MS_SMEM;
    cfg.stream = stream;
    cfg.attrs = attr;
    if (!BOUNDED) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = cl;
        attr[cfg.numAttrs].val.clusterDim.y = 1;
        attr[cfg.numAttrs].val.clusterDim.z = 1;
        ++cfg.numAttrs;
    }
    if (pdl_enabled()) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
        ++cfg.numAttrs;
    }
    CUDAPIC_CHECK(check_cuda(cudaLaunchKernelEx(&cfg, kern, sigma_tot, cs, active, x, vx, vy, vz, r0, r1, r2, r3, ix, ivx,
                                                ivy, ivz, alive_e, alive_i, events, g, (int)vec, dep_e, dep_i, coll,
                                                ion_k), name));
    return check_launch(name);
}

// A finite ion_k is the caller's bound for the ion test; electrons and ions
// without one find theirs in the launch.
template <bool ION, bool EVENTS, typename... Args>
int launch_stream(float ion_k, Args... args) {
    if constexpr (ION) {
        if (ion_k < INFINITY) return launch_stream_t<ION, EVENTS, true>(args..., ion_k);
    }
    return launch_stream_t<ION, EVENTS, false>(args..., ion_k);
}

// Variant choice: the bulk-copy kernel needs 16-byte aligned planes and a
// capacity that is a multiple of 4; the streaming kernel takes anything.
template <bool ION>
int launch_collisions(const float *sigma_tot, const float *cs, const uint32_t *active, float *x, float *vx,
                      float *vy, float *vz, uint32_t *r0, uint32_t *r1, uint32_t *r2, uint32_t *r3, float *ix,
                      float *ivx, float *ivy, float *ivz, uint32_t *alive_e, uint32_t *alive_i, uint8_t *events,
                      const cudapic_grid &g, cudaStream_t stream, float *dep_e, float *dep_i,
                      unsigned long long *coll, float ion_k = INFINITY) {
    const bool bulk = tuning().mcc_variant == 2 && tma_ready(g.capacity, {vx, vy, vz, r0, r1, r2, r3});
    if (bulk) {
        if (events)
            return launch_tma<ION, true>(sigma_tot, cs, active, x, vx, vy, vz, r0, r1, r2, r3, ix, ivx, ivy, ivz,
                                         alive_e, alive_i, events, g, stream, dep_e, dep_i, coll, ion_k);
        return launch_tma<ION, false>(sigma_tot, cs, active, x, vx, vy, vz, r0, r1, r2, r3, ix, ivx, ivy, ivz,
                                      alive_e, alive_i, nullptr, g, stream, dep_e, dep_i, coll, ion_k);
    }
    if (events)
        return launch_stream<ION, true>(ion_k, sigma_tot, cs, active, x, vx, vy, vz, r0, r1, r2, r3, ix, ivx, ivy, ivz,
                                        alive_e, alive_i, events, g, stream, dep_e, dep_i, coll);
    return launch_stream<ION, false>(ion_k, sigma_tot, cs, active, x, vx, vy, vz, r0, r1, r2, r3, ix, ivx, ivy, ivz,
                                     alive_e, alive_i, (uint8_t *)nullptr, g, stream, dep_e, dep_i, coll);
}

}  // namespace

int launch_collisions_e(const float *total_cs_e, const float *cs, const uint32_t *active_e, float *x, float *vx,
                        float *vy, float *vz, uint32_t *rng0, uint32_t *rng1, uint32_t *rng2, uint32_t *rng3,
                        float *i_x, float *i_vx, float *i_vy, float *i_vz, uint32_t *alive_e, uint32_t *alive_i,
                        uint8_t *events, const cudapic_grid &g, cudaStream_t stream, float *dep_e, float *dep_i,
                        unsigned long long *coll) {
    return launch_collisions<false>(total_cs_e, cs, active_e, x, vx, vy, vz, rng0, rng1, rng2, rng3, i_x, i_vx, i_vy,
                                    i_vz, alive_e, alive_i, events, g, stream, dep_e, dep_i, coll);
}

int launch_collisions_i(const float *total_cs_i, const float *cs, const uint32_t *active_i, float *vx, float *vy,
                        float *vz, uint32_t *rng0, uint32_t *rng1, uint32_t *rng2, uint32_t *rng3, uint8_t *events,
                        const cudapic_grid &g, cudaStream_t stream, unsigned long long *coll, float ion_k) {
    return launch_collisions<true>(total_cs_i, cs, active_i, nullptr, vx, vy, vz, rng0, rng1, rng2, rng3, nullptr,
                                   nullptr, nullptr, nullptr, nullptr, nullptr, events, g, stream, nullptr, nullptr,
                                   coll, ion_k);
}

float ion_reject_k(float sigma_max_i, const cudapic_grid &g) {
    if (!(sigma_max_i > 0.0f) || !(g.dt_i > 0.0f) || !std::isfinite(sigma_max_i)) return INFINITY;
    const double k = (double)sigma_max_i * (double)g.dt_i * (1.0 + 1e-5);
    return std::nextafter((float)k, INFINITY);
}

int launch_eepf(const EepfSamples &a, const cudapic_grid &g, cudaStream_t stream) {
    const unsigned grid = persistent_grid(2, ((uint64_t)g.capacity + 4 * EEPF_THREADS - 1) / (4 * EEPF_THREADS));
    return launch_kernel("accumulate_eepf", accumulate_eepf_kernel, dim3(grid), dim3(EEPF_THREADS), 0, stream, a, g,
                         (int)aligned16(a.x));
}

}  // namespace cudapic

using namespace cudapic;

#define CUDAPIC_E_ARGS_NONNULL                                                                              \
    (total_cs_e && cs && active_e && x && vx && vy && vz && rng0 && rng1 && rng2 && rng3 && i_x && i_vx && \
     i_vy && i_vz && alive_e && alive_i)

extern "C" int cudapic_check_collisions_e(const float *total_cs_e, const float *cs, const uint32_t *active_e,
                                          float *x, float *vx, float *vy, float *vz, uint32_t *rng0,
                                          uint32_t *rng1, uint32_t *rng2, uint32_t *rng3, float *i_x, float *i_vx,
                                          float *i_vy, float *i_vz, uint32_t *alive_e, uint32_t *alive_i,
                                          const cudapic_grid *grid, cudapic_stream_t stream) {
    CUDAPIC_CHECK(validate_grid(grid));
    CUDAPIC_REQUIRE(CUDAPIC_E_ARGS_NONNULL, "check_collisions_e: null pointer");
    return launch_collisions_e(total_cs_e, cs, active_e, x, vx, vy, vz, rng0, rng1, rng2, rng3, i_x, i_vx, i_vy,
                               i_vz, alive_e, alive_i, nullptr, *grid, (cudaStream_t)stream);
}

extern "C" int cudapic_check_collisions_e_events(const float *total_cs_e, const float *cs,
                                                 const uint32_t *active_e, float *x, float *vx, float *vy,
                                                 float *vz, uint32_t *rng0, uint32_t *rng1, uint32_t *rng2,
                                                 uint32_t *rng3, float *i_x, float *i_vx, float *i_vy,
                                                 float *i_vz, uint32_t *alive_e, uint32_t *alive_i,
                                                 uint8_t *events, const cudapic_grid *grid,
                                                 cudapic_stream_t stream) {
    CUDAPIC_CHECK(validate_grid(grid));
    CUDAPIC_REQUIRE(CUDAPIC_E_ARGS_NONNULL && events, "check_collisions_e_events: null pointer");
    return launch_collisions_e(total_cs_e, cs, active_e, x, vx, vy, vz, rng0, rng1, rng2, rng3, i_x, i_vx, i_vy,
                               i_vz, alive_e, alive_i, events, *grid, (cudaStream_t)stream);
}

extern "C" int cudapic_check_collisions_e_deposit(const float *total_cs_e, const float *cs,
                                                  const uint32_t *active_e, float *x, float *vx, float *vy,
                                                  float *vz, uint32_t *rng0, uint32_t *rng1, uint32_t *rng2,
                                                  uint32_t *rng3, float *i_x, float *i_vx, float *i_vy,
                                                  float *i_vz, uint32_t *alive_e, uint32_t *alive_i,
                                                  float *e_next_density, float *i_next_density,
                                                  const cudapic_grid *grid, cudapic_stream_t stream) {
    CUDAPIC_CHECK(validate_grid(grid));
    CUDAPIC_REQUIRE(CUDAPIC_E_ARGS_NONNULL, "check_collisions_e_deposit: null pointer");
    return launch_collisions_e(total_cs_e, cs, active_e, x, vx, vy, vz, rng0, rng1, rng2, rng3, i_x, i_vx, i_vy,
                               i_vz, alive_e, alive_i, nullptr, *grid, (cudaStream_t)stream, e_next_density,
                               i_next_density);
}

extern "C" int cudapic_check_collisions_i(const float *total_cs_i, const float *cs, const uint32_t *active_i,
                                          float *vx, float *vy, float *vz, uint32_t *rng0, uint32_t *rng1,
                                          uint32_t *rng2, uint32_t *rng3, const cudapic_grid *grid,
                                          cudapic_stream_t stream) {
    CUDAPIC_CHECK(validate_grid(grid));
    CUDAPIC_REQUIRE(total_cs_i && cs && active_i && vx && vy && vz && rng0 && rng1 && rng2 && rng3,
                    "check_collisions_i: null pointer");
    return launch_collisions_i(total_cs_i, cs, active_i, vx, vy, vz, rng0, rng1, rng2, rng3, nullptr, *grid,
                               (cudaStream_t)stream);
}

extern "C" int cudapic_check_collisions_i_events(const float *total_cs_i, const float *cs,
                                                 const uint32_t *active_i, float *vx, float *vy, float *vz,
                                                 uint32_t *rng0, uint32_t *rng1, uint32_t *rng2, uint32_t *rng3,
                                                 uint8_t *events, const cudapic_grid *grid,
                                                 cudapic_stream_t stream) {
    CUDAPIC_CHECK(validate_grid(grid));
    CUDAPIC_REQUIRE(total_cs_i && cs && active_i && vx && vy && vz && rng0 && rng1 && rng2 && rng3 && events,
                    "check_collisions_i_events: null pointer");
    return launch_collisions_i(total_cs_i, cs, active_i, vx, vy, vz, rng0, rng1, rng2, rng3, events, *grid,
                               (cudaStream_t)stream);
}

extern "C" int cudapic_check_collisions_i_bounded(const float *total_cs_i, const float *cs,
                                                  const uint32_t *active_i, float *vx, float *vy, float *vz,
                                                  uint32_t *rng0, uint32_t *rng1, uint32_t *rng2, uint32_t *rng3,
                                                  float sigma_max_i, uint8_t *events, const cudapic_grid *grid,
                                                  cudapic_stream_t stream) {
    CUDAPIC_CHECK(validate_grid(grid));
    CUDAPIC_REQUIRE(total_cs_i && cs && active_i && vx && vy && vz && rng0 && rng1 && rng2 && rng3,
                    "check_collisions_i_bounded: null pointer");
    CUDAPIC_REQUIRE(sigma_max_i >= 0.0f, "check_collisions_i_bounded: sigma_max_i must be the largest entry of total_cs_i");
    return launch_collisions_i(total_cs_i, cs, active_i, vx, vy, vz, rng0, rng1, rng2, rng3, events, *grid,
                               (cudaStream_t)stream, nullptr, ion_reject_k(sigma_max_i, *grid));
}

extern "C" int cudapic_accumulate_eepf(const float *x, const float *vx, const float *vy, const float *vz,
                                       const float *efield, const uint32_t *active_e, uint32_t *eepf,
                                       const cudapic_grid *grid, cudapic_stream_t stream) {
    CUDAPIC_CHECK(validate_grid(grid));
    CUDAPIC_REQUIRE(x && vx && vy && vz && efield && active_e && eepf, "accumulate_eepf: null pointer");
    return launch_eepf(EepfSamples{x, vx, vy, vz, efield, active_e, eepf, nullptr, nullptr}, *grid,
                       (cudaStream_t)stream);
}
