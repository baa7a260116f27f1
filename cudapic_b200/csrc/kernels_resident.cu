// kernels_resident.cu -- whole ion cycles of a small discharge in one launch.
//
// Reference: the per-step loop, Rust-CUDA/src/main.rs:1725-1808, as the fused
// driver runs it (state.cpp): solve, [ion push], in-place electron step,
// [ion collisions], and at the end of every N_SUB steps the compaction of the
// electrons.  At 1e4 particles a step of the driver is two launches that
// each do a microsecond of work behind five of latency (launch, counts, field,
// particles and densities through L2, the collider list, the completion
// ticket).  Here one thread-block cluster keeps the grid AND the electrons in
// shared memory and steps the discharge without leaving the kernel:
//  * every CTA owns a share of the electrons (position, velocity, RNG state
//    and the slot whose stream that is: 36 B) and runs the driver's step on
//    them: push, absorption, collision test, deposit (2^-20 fixed point,
//    push.cuh), then its own colliders from a list, the whole CTA together;
//    a spawned electron joins its parent's CTA with the stream of a freed
//    entry or of the next slot of the state's counter;
//  * the CTAs exchange their 64-bit node sums through distributed shared
//    memory, one cluster barrier per step (the sums alternate between two
//    buffers), and every CTA solves the field itself (the one-scan solve of
//    poisson.cuh): no launch, no ticket, and the density sums are exact.
//    With the electrons in global memory the barrier's release waited for a
//    step's stores (2 us) and a round of loads and stores cost another two;
//  * holes are closed within the CTA once per ion cycle.  The CTAs write their
//    electrons back, compact, and share them out again when one could
//    overflow in the next step or the slots not given out might not suffice
//    for it, and at the end;
//  * ions stay in global memory (touched once per ion cycle): pushed and
//    compacted to the other side, tested in place; the push appends at the
//    one of the two ion counters that the spawns then claim from.
// The cluster's barrier is the hardware's: nothing spins.  Particle planes,
// counters, densities and RNG planes are left as the driver's own steps leave
// them, so runs may mix both.
// Measured (N_G = 400, reference discharge; us per step alone / per step with
// three discharges in flight), here against the launched steps: 1300
// electrons 5.4 / 1.8 against 10.0 / 3.9, 13 700 electrons 6.5 / 2.2 against
// 11.3 / 4.2, 27 500 electrons (16 CTAs) 7.7 / 2.6 against 12.4 / 4.3.  What is
// left is latency: reading the peers' sums (0.6 us), the barrier with the
// wait for the slowest CTA (1 us), one chain of scattering (1 us), the solve.
#include <cooperative_groups.h>

#include <algorithm>

#include "batch_internal.h"
#include "internal.h"
#include "mcc.cuh"
#include "push.cuh"
#include "resident.h"
#include "step.cuh"

namespace cudapic {

namespace {

constexpr int RS_THREADS = 512;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_U = 2;                            // electrons per thread and round
constexpr int RS_ROW = 4;                          // ions per thread and round (16-byte accesses)
constexpr int RS_ROUND = RS_THREADS * RS_ROW;
constexpr int RS_COPIES = 4;                       // deposit histogram copies (RS_WARPS / 4 warps each)
constexpr int RS_PT = 2;                           // nodes per thread of the solve
constexpr uint32_t RS_MAX_NG = RS_THREADS * RS_PT;
constexpr uint32_t RS_ION_EPOCH = DEP_MAX_PER_COPY / (RS_ROUND / RS_COPIES);  // ion rounds between drains
constexpr uint32_t RS_NO_SLOT = 0xffffffffu;       // an entry without a stream (its spawn found no slot)
// Entries of a CTA, and how many may be filled when a step begins: each
// electron can spawn one in the step, and the step's deposits (electrons and
// spawns, at most 2^20 each on a node) then fit the 32-bit node sums.
constexpr uint32_t RS_ENTRIES = 4096;
constexpr uint32_t RS_FILL = RS_ENTRIES / 2 - 1;
static_assert(2 * RS_FILL <= DEP_MAX_PER_COPY, "32-bit node sums");

constexpr size_t resident_smem(uint32_t ef_pad) {
    return (size_t)ef_pad * (2 * 8 + (2 + 2 + RS_COPIES) * 4) + (size_t)RS_ENTRIES * (9 * 4 + 2 * 2);
}

struct ResidentSmem {
    unsigned long long *acc_i;           // [ef_pad] 64-bit ion sums of this CTA
    unsigned long long *exch_i;          // [ef_pad] published ion sums (once per ion cycle)
    uint32_t *exch[2];                   // [ef_pad] published electron sums, by the step's parity
    float *ef, *dens_i;                  // [ef_pad] field; ion density of the cycle
    uint32_t *hist;                      // [RS_COPIES][ef_pad]
    float *x, *vx, *vy, *vz;             // [RS_ENTRIES] electrons (x = CUDAPIC_DEAD_X: absorbed)
    uint32_t *r[4], *slot;               // [RS_ENTRIES] RNG state and the slot whose stream it is
    uint16_t *list[2];                   // [RS_ENTRIES] colliders; holes and movers of the compaction
    __device__ __forceinline__ ResidentSmem(unsigned char *smem, uint32_t ef_pad) {
        acc_i = reinterpret_cast<unsigned long long *>(smem);
        exch_i = acc_i + ef_pad;
        exch[0] = reinterpret_cast<uint32_t *>(exch_i + ef_pad);
        exch[1] = exch[0] + ef_pad;
        ef = reinterpret_cast<float *>(exch[1] + ef_pad);
        dens_i = ef + ef_pad;
        hist = reinterpret_cast<uint32_t *>(dens_i + ef_pad);
        x = reinterpret_cast<float *>(hist + RS_COPIES * ef_pad);
        vx = x + RS_ENTRIES;
        vy = vx + RS_ENTRIES;
        vz = vy + RS_ENTRIES;
        r[0] = reinterpret_cast<uint32_t *>(vz + RS_ENTRIES);
        r[1] = r[0] + RS_ENTRIES;
        r[2] = r[1] + RS_ENTRIES;
        r[3] = r[2] + RS_ENTRIES;
        slot = r[3] + RS_ENTRIES;
        list[0] = reinterpret_cast<uint16_t *>(slot + RS_ENTRIES);
        list[1] = list[0] + RS_ENTRIES;
    }
};

// Counters of the CTA in shared memory.
struct ResidentCount {
    uint32_t queued;         // colliders listed
    uint32_t filled;         // entries in use (live and absorbed)
    uint32_t claims, ions;   // slots claimed and ions gained this step
    uint32_t live, holes, movers;
};

// Spawns of this CTA (mcc.cuh): the electron takes the next entry, with its
// stream where the entry has one, else with that of the next slot; the ion a
// slot of the ion planes.  Both go into the CTA's own sums.
struct SpawnResident {
    const ResidentSmem &sm;
    ResidentCount &n;
    const ResidentArgs &a;
    uint32_t *h;                  // the warp's electron histogram copy
    uint32_t with_stream;         // entries that came with a stream
    const ResidentPlanes &ions;
    uint32_t *ctr_i;
    const cudapic_grid &g;
    __device__ __forceinline__ void electron(float x, float vx, float vy, float vz) const {
        const uint32_t k = atomicAdd(&n.filled, 1u);  // < entries: a step starts with at most half of them filled
        if (k >= with_stream || sm.slot[k] == RS_NO_SLOT) {
            uint32_t slot;
            if (!claim_slot(a.n_e, g.capacity, slot)) {
                sm.x[k] = CUDAPIC_DEAD_X;
                sm.slot[k] = RS_NO_SLOT;
                set_dev_err(g.dev_err, CUDAPIC_DEVERR_SPAWN_E);
                return;
            }
            atomicAdd(&n.claims, 1u);
            sm.slot[k] = slot;
#pragma unroll
            for (int w = 0; w < 4; ++w) sm.r[w][k] = __ldcg(a.rng_e[w] + slot);
        }
        sm.x[k] = x;
        sm.vx[k] = vx;
        sm.vy[k] = vy;
        sm.vz[k] = vz;
        dep_add(h, x, g);
    }
    __device__ __forceinline__ void ion(float x, float vx, float vy, float vz) const {
        uint32_t slot;
        if (!claim_slot(ctr_i, g.capacity, slot)) {
            set_dev_err(g.dev_err, CUDAPIC_DEVERR_SPAWN_I);
            return;
        }
        atomicAdd(&n.ions, 1u);
        ions.x[slot] = x;
        ions.vx[slot] = vx;
        ions.vy[slot] = vy;
        ions.vz[slot] = vz;
        const float pos = x * g.inv_dx;
        const int p = cell_of(pos, g.n_g);
        const uint32_t r = min(__float2uint_rn((pos - (float)p) * (float)(1u << DEP_Q)), 1u << DEP_Q);
        atomicAdd(&sm.acc_i[p], (unsigned long long)((1u << DEP_Q) - r));
        atomicAdd(&sm.acc_i[p + 1], (unsigned long long)r);
    }
};

// The cluster's sums of the nodes k0, k0 + 1 (k0 even) from the CTAs'
// published words, through distributed shared memory.
template <int C, typename T>
__device__ __forceinline__ void sum_nodes(const cg::cluster_group &cluster, T *published, uint32_t k0,
                                          unsigned long long (&s)[RS_PT]) {
    struct alignas(RS_PT * sizeof(T)) Pair {
        T v[RS_PT];
    };
#pragma unroll
    for (unsigned c = 0; c < C; ++c) {
        const Pair p = *reinterpret_cast<const Pair *>(cluster.map_shared_rank(published, c) + k0);
        s[0] += p.v[0];
        s[1] += p.v[1];
    }
}

// The calling lane's CTA's published word (0 beyond the cluster).
template <int C>
__device__ __forceinline__ uint32_t peer_word(const cg::cluster_group &cluster, uint32_t *published, int lane) {
    return lane < C ? *cluster.map_shared_rank(published, lane) : 0u;
}

__device__ __forceinline__ void prefetch_l1(const float *p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// The published counts over the cluster (one warp): sums of claims, ions and
// filled entries, and the largest fill.
template <int C>
__device__ __forceinline__ void gather_counts(const cg::cluster_group &cluster, uint32_t *published, uint32_t *sum,
                                              int lane) {
    const uint32_t claims = peer_word<C>(cluster, published, lane), ions = peer_word<C>(cluster, published + 1, lane);
    const uint32_t filled = peer_word<C>(cluster, published + 2, lane);
    const uint32_t a = __reduce_add_sync(0xffffffffu, claims), b = __reduce_add_sync(0xffffffffu, ions);
    const uint32_t c = __reduce_add_sync(0xffffffffu, filled), d = __reduce_max_sync(0xffffffffu, filled);
    if (lane == 0) {
        sum[0] = a;
        sum[1] = b;
        sum[2] = c;
        sum[3] = d;
    }
}

// Node sum -> f32 density, as dep_flush (boundary nodes doubled).
__device__ __forceinline__ float node_density(unsigned long long a, uint32_t k, double w, uint32_t n_g) {
    float v = (float)((double)a * w);
    if (k == 0 || k == n_g - 1) v *= 2.0f;
    return v;
}

// Four consecutive words of an ion plane, through L2 (other CTAs write slots too).
__device__ __forceinline__ float4 ld4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }

// Equal shares of [0, n), multiples of 4.
__device__ __forceinline__ void share(uint32_t n, unsigned rank, unsigned count, uint32_t &beg, uint32_t &end) {
    const uint32_t chunk = ((n + count - 1) / count + 3u) & ~3u;
    beg = min(n, rank * chunk);
    end = min(n, beg + chunk);
}

// Appends the kept rows of a warp's four at *counter (one atomic per warp).
__device__ __forceinline__ void append_rows(uint32_t keep, unsigned lt, uint32_t *counter, uint32_t (&slot)[RS_ROW]) {
    uint32_t total = 0;
#pragma unroll
    for (int u = 0; u < RS_ROW; ++u) {
        const unsigned m = __ballot_sync(0xffffffffu, keep >> u & 1u);
        slot[u] = total + __popc(m & lt);
        total += __popc(m);
    }
    uint32_t base = 0;
    if (total && (threadIdx.x & 31) == 0) base = atomicAdd(counter, total);
    base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
    for (int u = 0; u < RS_ROW; ++u) slot[u] += base;
}

// The slots [beg, end) of the planes become entries 0 .. end - beg.
__device__ __forceinline__ void load_entries(const ResidentSmem &sm, const ResidentArgs &a, uint32_t beg, uint32_t end) {
    for (uint32_t k = threadIdx.x; k < end - beg; k += RS_THREADS) {
        sm.x[k] = __ldcg(a.e.x + beg + k);
        sm.vx[k] = __ldcg(a.e.vx + beg + k);
        sm.vy[k] = __ldcg(a.e.vy + beg + k);
        sm.vz[k] = __ldcg(a.e.vz + beg + k);
#pragma unroll
        for (int w = 0; w < 4; ++w) sm.r[w][k] = __ldcg(a.rng_e[w] + beg + k);
        sm.slot[k] = beg + k;
    }
}

// Closes the holes of the `filled` entries: live ones from the end move into
// them (position and velocity; streams stay with their entries).  Returns the
// number of live entries; every thread of the CTA calls it.
__device__ __forceinline__ uint32_t close_holes(const ResidentSmem &sm, ResidentCount &n, uint32_t filled) {
    __syncthreads();
    if (threadIdx.x == 0) n.live = n.holes = n.movers = 0u;
    __syncthreads();
    uint32_t mine = 0;
    for (uint32_t k = threadIdx.x; k < filled; k += RS_THREADS) mine += slot_dead(sm.x[k]) ? 0u : 1u;
    mine = __reduce_add_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&n.live, mine);
    __syncthreads();
    const uint32_t live = n.live;
    if (live == filled) return live;
    for (uint32_t k = threadIdx.x; k < filled; k += RS_THREADS) {
        const bool dead = slot_dead(sm.x[k]);
        if (dead && k < live) sm.list[0][atomicAdd(&n.holes, 1u)] = (uint16_t)k;
        if (!dead && k >= live) sm.list[1][atomicAdd(&n.movers, 1u)] = (uint16_t)k;
    }
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < n.holes; t += RS_THREADS) {  // as many movers as holes
        const uint32_t d = sm.list[0][t], s = sm.list[1][t];
        sm.x[d] = sm.x[s];
        sm.vx[d] = sm.vx[s];
        sm.vy[d] = sm.vy[s];
        sm.vz[d] = sm.vz[s];
        if (sm.slot[d] == RS_NO_SLOT) {  // the hole of a spawn without a slot: the electron keeps its stream
            sm.slot[d] = sm.slot[s];
            sm.slot[s] = RS_NO_SLOT;
#pragma unroll
            for (int w = 0; w < 4; ++w) sm.r[w][d] = sm.r[w][s];
        }
    }
    __syncthreads();
    return live;
}

}  // namespace

// Writes the CTA's `live` entries back to the planes, compact over the
// cluster (each CTA behind those of lower rank), and every entry's RNG state
// to its slot; *n_e becomes the total, which is returned.  Ends with a
// cluster barrier: everything is visible.
template <int C>
__device__ __forceinline__ uint32_t store_entries(const cg::cluster_group &cluster, const ResidentSmem &sm,
                                                  const ResidentArgs &a, uint32_t *s_live, uint32_t live,
                                                  uint32_t with_stream) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) *s_live = live;
    cluster.sync();
    const uint32_t peer = peer_word<C>(cluster, s_live, lane);
    const uint32_t first = __reduce_add_sync(0xffffffffu, lane < (int)cluster.block_rank() ? peer : 0u);
    const uint32_t total = __reduce_add_sync(0xffffffffu, peer);
    for (uint32_t k = threadIdx.x; k < live; k += RS_THREADS) {
        a.e.x[first + k] = sm.x[k];
        a.e.vx[first + k] = sm.vx[k];
        a.e.vy[first + k] = sm.vy[k];
        a.e.vz[first + k] = sm.vz[k];
    }
    for (uint32_t k = threadIdx.x; k < with_stream; k += RS_THREADS) {
        const uint32_t slot = sm.slot[k];
        if (slot == RS_NO_SLOT) continue;
#pragma unroll
        for (int w = 0; w < 4; ++w) a.rng_e[w][slot] = sm.r[w][k];
    }
    if (cluster.block_rank() == 0 && threadIdx.x == 0) *a.n_e = total;
    cluster.sync();
    return total;
}

template <int C>
__global__ void __launch_bounds__(RS_THREADS, 1)
    discharge_resident_kernel(const __grid_constant__ ResidentArgs a, const __grid_constant__ cudapic_grid g,
                              uint32_t steps, uint32_t ef_pad) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ ResidentCount cnt;
    __shared__ uint32_t s_pub[2][3], s_live;  // published: claims, ions gained, entries filled; live entries
    __shared__ uint32_t s_sum[4];             // over the cluster: claims, ions gained, entries filled; most filled
    __shared__ double w_f[RS_WARPS], w_g[RS_WARPS];
    __shared__ double s_k[4];  // the solve's constants: FP64 divisions, once
    const ResidentSmem sm(smem, ef_pad);
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned rank = cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = lanemask_lt();
    const uint32_t n_g = g.n_g;
    uint32_t *h = sm.hist + (uint32_t)(warp % RS_COPIES) * ef_pad;
    const double w_node = g.weight_factor_d * (1.0 / (double)(1u << DEP_Q));
    const float factor = g.factor_e, dt = g.dt_e, sigma_max = a.sigma_max;
    const float rej_k2 = sigma_max * dt * (sigma_max * dt) * 1.0001f;  // may_collide's bound

    for (uint32_t k = tid; k < ef_pad; k += RS_THREADS) {
        sm.acc_i[k] = 0ull;
        sm.dens_i[k] = k < n_g ? a.i_collected[k] : 0.0f;  // current from the first step, an ion step, on
#pragma unroll
        for (int c = 0; c < RS_COPIES; ++c) sm.hist[(uint32_t)c * ef_pad + k] = 0u;
    }
    uint32_t n_i = load_count(a.n_i, g.capacity, g.dev_err);
    uint32_t claimed = load_count(a.n_e, g.capacity, g.dev_err);  // slots given out: [0, claimed)
    const uint32_t t0 = *a.step_counter;
    uint32_t *ctr_i = a.n_i, *free_i = a.alive_i;  // free: zero until used
    int si = 0;                    // live ion side, relative to a's
    uint32_t work = 0;
    uint32_t beg, end;
    share(claimed, rank, C, beg, end);
    uint32_t filled = end - beg, with_stream = filled;
    load_entries(sm, a, beg, end);
    if (tid == 0) {
        cnt = ResidentCount{};
        cnt.filled = filled;
        s_k[0] = -g.dx * g.dx / 8.85418781e-12 * 1.60217662e-19;  // density to f_i
        s_k[1] = 1.0 / (double)(n_g - 1);
        s_k[2] = 1.0 / g.dx;
        s_k[3] = g.dx / (2.0 * 8.85418781e-12) * 1.60217662e-19;  // density to the one-sided field correction
    }
    cluster.sync();                // every CTA runs and has read the counters

    for (uint32_t j = 0; j < steps; ++j) {
        const uint32_t par = j & 1u;
        const bool ion_step = j % a.n_sub == 0, cycle_end = (j + 1) % a.n_sub == 0;

        // ---- densities of the present particles, and the field (poisson.cuh)
        float de[RS_PT];
        double f[RS_PT], sum_f = 0.0, sum_g = 0.0;
        const uint32_t k0 = (uint32_t)tid * RS_PT;  // this thread's nodes; ef_pad is a multiple of RS_PT
        const float pot0_f = a.pot0_table[(t0 + j) % g.n_t];
        if (j != 0 && warp == RS_WARPS - 1) gather_counts<C>(cluster, s_pub[par ^ 1u], s_sum, lane);  // of the last step
        unsigned long long ns[RS_PT] = {0ull, 0ull};
        if (j != 0 && k0 < n_g) {
            sum_nodes<C>(cluster, sm.exch[par ^ 1u], k0, ns);
            if (ion_step) {  // the sums collected over the last ion cycle
                unsigned long long ni[RS_PT] = {0ull, 0ull};
                sum_nodes<C>(cluster, sm.exch_i, k0, ni);
#pragma unroll
                for (int q = 0; q < RS_PT; ++q)
                    if (k0 + q < n_g) sm.dens_i[k0 + q] = node_density(ni[q], k0 + q, w_node, n_g);
            }
        }
#pragma unroll
        for (int q = 0; q < RS_PT; ++q) {
            const uint32_t k = k0 + q;
            de[q] = 0.0f;
            f[q] = 0.0;
            if (k < n_g) {
                de[q] = j == 0 ? __ldcg(a.e_dens_in + k) : node_density(ns[q], k, w_node, n_g);
                if (k >= 1 && k <= n_g - 2) f[q] = s_k[0] * ((double)sm.dens_i[k] - (double)de[q]);
            }
            sum_f += f[q];
            sum_g += (double)k * f[q];
        }
        double in_f = sum_f, in_g = sum_g;
        if ((uint32_t)warp * 32u * RS_PT < n_g) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double p = __shfl_up_sync(0xffffffffu, in_f, o), q = __shfl_up_sync(0xffffffffu, in_g, o);
                if (lane >= o) {
                    in_f += p;
                    in_g += q;
                }
            }
        }
        if (lane == 31) {
            w_f[warp] = in_f;
            w_g[warp] = in_g;
        }
        __syncthreads();
        bool reshare = false;
        if (j != 0) {
            claimed += s_sum[0];
            if ((j - 1) % a.n_sub != 0) n_i += s_sum[1];  // an ion step counted its ions itself
            // A new share-out when an entry or a slot could be missing in this
            // step (the same numbers, hence the same decision, in every CTA).
            // Slots of electrons absorbed in earlier cycles are only given out
            // again by their own CTA or by a share-out, so it comes while the
            // slots not given out yet are fewer than the electrons, each of
            // which may spawn one, and others are bound like that: on an ion
            // step (the entries counted still include the last cycle's absorbed)
            // or with more slots given out than entries filled.  (Only below a
            // quarter, on ion steps: 3 % faster where the capacity is 1.5 to 2.3
            // times the electrons, but growth above that within a cycle lost
            // spawns while slots were free.)
            const bool bound = ion_step || claimed > s_sum[2];
            reshare = s_sum[3] > RS_FILL || (bound && g.capacity - claimed < s_sum[2]);
        }
        if ((uint32_t)warp * 32u * RS_PT < n_g) {
            double tf = lane < RS_WARPS ? w_f[lane] : 0.0, tg = lane < RS_WARPS ? w_g[lane] : 0.0;
#pragma unroll
            for (int o = 1; o < RS_WARPS; o <<= 1) {
                const double p = __shfl_up_sync(0xffffffffu, tf, o), q = __shfl_up_sync(0xffffffffu, tg, o);
                if (lane >= o) {
                    tf += p;
                    tg += q;
                }
            }
            const double all_f = __shfl_sync(0xffffffffu, tf, RS_WARPS - 1), all_g = __shfl_sync(0xffffffffu, tg, RS_WARPS - 1);
            const double before_f = __shfl_sync(0xffffffffu, tf, warp > 0 ? warp - 1 : 0);
            const double before_g = __shfl_sync(0xffffffffu, tg, warp > 0 ? warp - 1 : 0);
            double run_f = in_f - sum_f + (warp > 0 ? before_f : 0.0);
            double run_g = in_g - sum_g + (warp > 0 ? before_g : 0.0);
            const double pot0 = (double)pot0_f;
            const double cst = (all_g - pot0) * s_k[1] - all_f, inv_dx = s_k[2];
            const bool out = j + 1 == steps && rank == 0;
#pragma unroll
            for (int q = 0; q < RS_PT; ++q) {
                const uint32_t k = k0 + q;
                if (k >= n_g) continue;
                run_f += f[q];
                run_g += (double)k * f[q];
                double p = pot0 - run_g + (double)k * (cst + run_f), e = -(cst + run_f - 0.5 * f[q]) * inv_dx;
                const double edge = ((double)sm.dens_i[k] - (double)de[q]) * s_k[3];
                if (k == 0) {
                    p = pot0;
                    e = -cst * inv_dx - edge;
                } else if (k == n_g - 1) {
                    p = 0.0;
                    e = -(cst + run_f) * inv_dx + edge;
                }
                sm.ef[k] = (float)e;
                if (out) {
                    a.pot[k] = (float)p;
                    a.efield[k] = (float)e;
                }
            }
        }
        __syncthreads();
        if (reshare) {
            filled = close_holes(sm, cnt, filled);
            claimed = store_entries<C>(cluster, sm, a, &s_live, filled, with_stream);
            share(claimed, rank, C, beg, end);
            filled = with_stream = end - beg;
            load_entries(sm, a, beg, end);
            if (tid == 0) cnt.filled = filled;
            __syncthreads();
        }

        // ---- ion push and compaction to the other side (move_and_compact with the deposit)
        if (ion_step) {
            uint32_t ib, ie;
            share(n_i, rank, C, ib, ie);
            work += tid == 0 ? ie - ib : 0u;
            const ResidentPlanes &src = a.i[si], &dst = a.i[si ^ 1];
            uint32_t r = 0;
            for (uint32_t b = ib; b < ie; b += RS_ROUND, ++r) {
                if (r != 0 && r % RS_ION_EPOCH == 0) {
                    __syncthreads();
                    dep_drain(sm.hist, RS_COPIES, ef_pad, sm.acc_i, n_g);
                    __syncthreads();
                }
                const uint32_t s0 = b + (uint32_t)tid * RS_ROW;
                float4 IX = {}, IVX = {}, IVY = {}, IVZ = {};
                if (s0 < ie) {
                    IX = ld4(src.x + s0);
                    IVX = ld4(src.vx + s0);
                    IVY = ld4(src.vy + s0);
                    IVZ = ld4(src.vz + s0);
                }
                float px[RS_ROW] = {IX.x, IX.y, IX.z, IX.w}, pv[RS_ROW] = {IVX.x, IVX.y, IVX.z, IVX.w};
                const float py[RS_ROW] = {IVY.x, IVY.y, IVY.z, IVY.w}, pz[RS_ROW] = {IVZ.x, IVZ.y, IVZ.z, IVZ.w};
                uint32_t keep = 0, slot[RS_ROW];
#pragma unroll
                for (int u = 0; u < RS_ROW; ++u) {
                    if (s0 + (uint32_t)u >= ie) continue;
                    const PushResult pr = push_one(px[u], pv[u], sm.ef, g.factor_i, g.dt_i, g);
                    px[u] = pr.x;
                    pv[u] = pr.vx;
                    if (pr.keep) keep |= 1u << u;
                }
                append_rows(keep, lt, free_i, slot);
                // other CTAs' spawns of this step already claim from the same counter
                uint32_t kept = 0;
#pragma unroll
                for (int u = 0; u < RS_ROW; ++u) {
                    if (!(keep >> u & 1u)) continue;
                    if (slot[u] >= g.capacity) {
                        set_dev_err(g.dev_err, CUDAPIC_DEVERR_SPAWN_I);
                        continue;
                    }
                    ++kept;
                    dst.x[slot[u]] = px[u];
                    dst.vx[slot[u]] = pv[u];
                    dst.vy[slot[u]] = py[u];
                    dst.vz[slot[u]] = pz[u];
                    dep_add(h, px[u], g);
                }
                kept = __reduce_add_sync(0xffffffffu, kept);
                if (lane == 0 && kept) atomicAdd(&cnt.ions, kept);
            }
            __syncthreads();
            dep_drain(sm.hist, RS_COPIES, ef_pad, sm.acc_i, n_g);
            __syncthreads();
            si ^= 1;
            uint32_t *const t = ctr_i;
            ctr_i = free_i;
            free_i = t;
        }
        const ResidentPlanes &ions = a.i[si];

        // ---- electrons: push, test, deposit; colliders listed, then scattered
        for (uint32_t b = 0; b < filled; b += RS_THREADS * RS_U) {
            float px[RS_U], pv[RS_U], py[RS_U], pz[RS_U], rnd[RS_U];
            uint32_t kept = 0, may = 0;
#pragma unroll
            for (int u = 0; u < RS_U; ++u) {
                const uint32_t k = b + (uint32_t)(u * RS_THREADS) + tid;
                px[u] = k < filled ? sm.x[k] : CUDAPIC_DEAD_X;
                pv[u] = py[u] = pz[u] = 0.0f;
                if (slot_dead(px[u])) continue;
                pv[u] = sm.vx[k];
                py[u] = sm.vy[k];
                pz[u] = sm.vz[k];
                ++work;
                const PushResult pr = push_one_c(px[u], pv[u], sm.ef, factor, dt, g.inv_dx, n_g, g.gap, g);
                if (pr.keep) {
                    kept |= 1u << u;
                    px[u] = pr.x;
                    pv[u] = pr.vx;
                    dep_add(h, pr.x, g);
                    sm.vx[k] = pr.vx;
                }
                sm.x[k] = pr.keep ? pr.x : CUDAPIC_DEAD_X;
            }
#pragma unroll
            for (int u = 0; u < RS_U; ++u) {
                const uint32_t k = b + (uint32_t)(u * RS_THREADS) + tid;
                rnd[u] = 0.0f;
                if (!(kept >> u & 1u)) continue;
                Xoshiro128p rs{sm.r[0][k], sm.r[1][k], sm.r[2][k], sm.r[3][k]};
                const float v2 = pv[u] * pv[u] + py[u] * py[u] + pz[u] * pz[u];
                rnd[u] = rs.uniform();
                if (may_collide(rnd[u], v2, rej_k2)) may |= 1u << u;
                sm.r[0][k] = rs.s0;
                sm.r[1][k] = rs.s1;
                sm.r[2][k] = rs.s2;
                sm.r[3][k] = rs.s3;
            }
            if (may) {  // the exact test where the bound cannot decide
#pragma unroll
                for (int u = 0; u < RS_U; ++u) {
                    if (!(may >> u & 1u)) continue;
                    const float v2 = pv[u] * pv[u] + py[u] * py[u] + pz[u] * pz[u];
                    const float velocity = sqrtf(v2);
                    const uint32_t idx = energy_index(g.half_me_over_e * v2);
                    const float st = __ldg(a.sigma_tot_e + idx);
                    // the scattering's table entries on their way to L1 beside the test's
                    prefetch_l1(a.cs + idx);
                    prefetch_l1(a.cs + CS_RANGES + idx);
                    prefetch_l1(a.cs + 2 * CS_RANGES + idx);
                    if (collision_draw(rnd[u], st * velocity * dt))
                        sm.list[0][atomicAdd(&cnt.queued, 1u)] = (uint16_t)(b + (uint32_t)(u * RS_THREADS) + tid);
                }
            }
        }
        __syncthreads();
        const uint32_t queued = cnt.queued;
        const SpawnResident spawn{sm, cnt, a, h, with_stream, ions, ctr_i, g};
        for (uint32_t q = tid; q < queued; q += RS_THREADS) {
            const uint32_t k = sm.list[0][q];
            const float vxi = sm.vx[k], vyi = sm.vy[k], vzi = sm.vz[k];
            Xoshiro128p rs{sm.r[0][k], sm.r[1][k], sm.r[2][k], sm.r[3][k]};
            const float v2 = vxi * vxi + vyi * vyi + vzi * vzi;
            collide_electron_body<true, true>(k, energy_index(g.half_me_over_e * v2), vxi, vyi, vzi, rs, a.cs, sm.x,
                                              sm.vx, sm.vy, sm.vz, g, spawn, sm.x[k]);
            sm.r[0][k] = rs.s0;
            sm.r[1][k] = rs.s1;
            sm.r[2][k] = rs.s2;
            sm.r[3][k] = rs.s3;
        }
        __syncthreads();

        // ---- publish this CTA's sums and counts; one barrier per step
        for (uint32_t k = tid; k < n_g; k += RS_THREADS) {
            uint32_t v = 0u;
#pragma unroll
            for (int c = 0; c < RS_COPIES; ++c) {
                v += sm.hist[(uint32_t)c * ef_pad + k];
                sm.hist[(uint32_t)c * ef_pad + k] = 0u;
            }
            sm.exch[par][k] = v;
            if (cycle_end) {
                sm.exch_i[k] = sm.acc_i[k];
                sm.acc_i[k] = 0ull;
            }
        }
        filled = cnt.filled;
        with_stream = max(with_stream, filled);
        if (tid == 0) {
            s_pub[par][0] = cnt.claims;
            s_pub[par][1] = cnt.ions;
            s_pub[par][2] = filled;
            cnt.claims = cnt.ions = cnt.queued = 0u;
        }
        cluster.sync();

        // ---- ion collisions (the ions of this step, its spawns included)
        if (ion_step) {
            if (warp == RS_WARPS - 1) gather_counts<C>(cluster, s_pub[par], s_sum, lane);
            __syncthreads();
            n_i = s_sum[1];  // the survivors and the spawns of this step
            __syncthreads();
            if (rank == 0 && tid == 0) *free_i = 0u;  // next used an ion cycle from now
            uint32_t ib, ie;
            share(n_i, rank, C, ib, ie);
            const GlobalTable table{a.sigma_tot_i};
            for (uint32_t i = ib + tid; i < ie; i += RS_THREADS) {
                const Xoshiro128p r0{__ldcg(a.rng_i[0] + i), __ldcg(a.rng_i[1] + i), __ldcg(a.rng_i[2] + i),
                                     __ldcg(a.rng_i[3] + i)};
                const float vxi = __ldcg(ions.vx + i), vyi = __ldcg(ions.vy + i), vzi = __ldcg(ions.vz + i);
                Xoshiro128p rs = r0;
                if (ion_collides(vxi, vyi, vzi, rs, table, g, a.ion_k)) {
                    rs = r0;
                    const IonTest t = test_ion(vxi, vyi, vzi, rs, table, g);
                    collide_ion(i, t.idx, vxi, vyi, vzi, t.vxa, t.vya, t.vza, rs, a.cs, ions.vx, ions.vy, ions.vz, g);
                }
                a.rng_i[0][i] = rs.s0;
                a.rng_i[1][i] = rs.s1;
                a.rng_i[2][i] = rs.s2;
                a.rng_i[3][i] = rs.s3;
            }
        }

        if (cycle_end) {
            filled = close_holes(sm, cnt, filled);
            __syncthreads();
            if (tid == 0) cnt.filled = filled;
            __syncthreads();
        }
    }

    // ---- the state as the driver's steps leave it: electrons, counts, collected densities
    store_entries<C>(cluster, sm, a, &s_live, filled, with_stream);
    if (rank == 0) {
        if (warp == RS_WARPS - 1) gather_counts<C>(cluster, s_pub[(steps - 1) & 1u], s_sum, lane);
        for (uint32_t k0 = (uint32_t)tid * RS_PT; k0 < n_g; k0 += RS_THREADS * RS_PT) {
            unsigned long long s[RS_PT] = {0ull, 0ull}, t[RS_PT] = {0ull, 0ull};
            sum_nodes<C>(cluster, sm.exch[(steps - 1) & 1u], k0, s);
            sum_nodes<C>(cluster, sm.exch_i, k0, t);
#pragma unroll
            for (int q = 0; q < RS_PT; ++q) {
                const uint32_t k = k0 + q;
                if (k >= n_g) continue;
                a.e_dens_out[k] = node_density(s[q], k, w_node, n_g);
                a.i_collected_out[k] = node_density(t[q], k, w_node, n_g);
                a.i_current_out[k] = sm.dens_i[k];
            }
        }
        __syncthreads();
        if (tid == 0) {
            *a.n_i = n_i + s_sum[1];  // the last step is not an ion step (n_sub >= 2)
            *a.alive_i = 0u;
            *a.step_counter = t0 + steps;
        }
    }
    add_work(g.work, work);
    cluster.sync();  // rank 0 has read the other CTAs' sums
}

namespace {

// CTAs of the cluster for a capacity (0: none fits): a share-out never fills
// more than RS_FILL entries (shares are rounded up to 4 slots).  The capacity
// counts and not the population, which may grow to it inside the kernel.  The
// line is the room of the largest cluster and not where the launched steps get
// faster: 27 500 electrons in 32 688 slots take 7.7 us per step (2.6 with three
// discharges in flight), launched, in 32 692 slots, 12.4 (4.3).
int resident_cluster(const cudapic_grid &g) {
    const uint64_t need = (uint64_t)g.capacity + 64;
    return need <= 8 * RS_FILL ? 8 : need <= 16 * RS_FILL ? 16 : 0;
}

uint32_t resident_ef_pad(const cudapic_grid &g) { return (g.n_g + 3u) & ~3u; }

// A cluster's launch; the caller's `attr` outlives it.
template <int C>
cudaLaunchConfig_t resident_config(const cudapic_grid &g, cudaStream_t stream, cudaLaunchAttribute &attr) {
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = C;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(RS_THREADS);
    cfg.dynamicSmemBytes = resident_smem(resident_ef_pad(g));
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cfg;
}

template <int C>
bool resident_launchable_t(const cudapic_grid &g, cudaStream_t stream) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = resident_config<C>(g, stream, attr);
    auto kern = discharge_resident_kernel<C>;
    int clusters = 0;
    const bool ok = cfg.dynamicSmemBytes <= (size_t)max_smem_optin() &&
                    kernel_smem((const void *)kern, cfg.dynamicSmemBytes, "resident steps") == CUDAPIC_OK &&
                    // beyond the portable size of 8
                    (C <= 8 || cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
                    cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters >= 1;
    if (!ok) cudaGetLastError();
    return ok;
}

template <int C>
int launch_resident_t(const ResidentArgs &a, const cudapic_grid &g, uint32_t steps, cudaStream_t stream) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = resident_config<C>(g, stream, attr);
    return check_cuda(cudaLaunchKernelEx(&cfg, discharge_resident_kernel<C>, a, g, steps, resident_ef_pad(g)),
                      "launch resident steps");
}

}  // namespace

bool resident_fits(const cudapic_grid &g, uint32_t n_sub) {
    return g.n_g <= RS_MAX_NG && n_sub >= 2 && !(g.flags & CUDAPIC_FLAG_POISSON_F32_SCAN) && resident_cluster(g) != 0;
}

bool resident_launchable(const cudapic_grid &g, cudaStream_t stream) {
    return resident_cluster(g) == 8 ? resident_launchable_t<8>(g, stream) : resident_launchable_t<16>(g, stream);
}

int launch_resident(const ResidentArgs &a, const cudapic_grid &g, uint32_t steps, cudaStream_t stream) {
    return resident_cluster(g) == 8 ? launch_resident_t<8>(a, g, steps, stream)
                                    : launch_resident_t<16>(a, g, steps, stream);
}

}  // namespace cudapic
