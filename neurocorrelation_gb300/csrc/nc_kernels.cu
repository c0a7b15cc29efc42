// nc_kernels.cu — the NeuCor step on sm_103a.
//
// One simulation step t of every packed net is two launches:
//
//   k_neuron_step
//     a. plasticity deferred from step t-1 (src/NeuCor.cpp:740-761):
//        post-spike branch for every neuron that fired at t-1 (its whole in-synapse
//        row, eight lanes a row), then the arrival branch for every spike that arrived
//        at t-1 (Synapse::run, src/NeuCor.cpp:718-726)
//     b. Neuron::run at t (src/NeuCor.cpp:619-641): charge_insynapses folds the
//        terms of spikes that arrived at t-1..t-KC in ascending source order (the
//        ring bits are in CSC order, so the fold follows std::map order), charge_passive,
//        charge_thresholdCheck with the forced-fire requests, AP
//     c. background fire draws for t+1 (src/NeuCor.cpp:604-607)
//     d. fired bits; the last warp to have read the step counters advances them
//
//   k_spike_launch (one warp per up to 8 neurons' fired bits)
//     Synapse::fire (src/NeuCor.cpp:727-738) on each out-synapse: drop if busy,
//     capture fl(fl(0.2f*52)*w) times deltaT (the fold forms the contribution term from
//     it), mark the ring bit of the arrival step.
//
// The CPU restatement runs neurons in ascending id, each update firing at once.
// Two rules make the split launches produce the same bits:
//   * a synapse freed by its target's update at t (src/NeuCor.cpp:697) is free for
//     a launch at t only when the target's id is not above the source's
//     (free iff t - last_arrival >= KC + [target > source]);
//   * when the target also fired at t and precedes the source, the captured weight
//     includes the target's post-spike plasticity of t, computed on the fly.
// Plasticity of step t is written by the next k_neuron_step (or k_stdp_flush), so
// every launch at t reads weights as of the end of t-1.
//
// Floating point: built with --fmad=false so every multiply and add rounds on its
// own, as in the reference's x86-64 build.  The reference's transcendentals
// (powf, exp) are host-built tables indexed by step differences.
#include "nc_engine.cuh"
#include "nc_device.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

namespace {

using namespace nc_dev;

// Programmatic dependent launch: the step's two kernels are scheduled while the one before
// drains and wait here before they read anything it writes.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Post-spike branch of the plasticity of step `prev` (src/NeuCor.cpp:650-655, 740-761):
// the whole in-row of every neuron of the tile that fired at prev.  Groups of eight lanes
// take a row each, a quad per lane and up to four quads in flight (all lanes call).
__device__ void postfire_rows(const NcPools& P, const NcNetDesc& D, uint32_t fired, int lane, int64_t s0, int64_t s1,
                              int32_t prev)
{
    const float* tab_pre = P.tables + D.table_base;
    const int32_t tpl = D.tab_pre_len;
    const Rates R = rates_of(D);
    const bool inh = !D.nonneg_terms;
    const float post0 = R.post * 0.0f;
    while (fired) {
        // the next four rows, one per group
        int row = -1;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const int j = fired ? __ffs(fired) - 1 : -1;
            fired &= fired - 1u;
            if (lane >> 3 == g) row = j;
        }
        const int64_t a = __shfl_sync(kFull, s0, row < 0 ? 0 : row), e = __shfl_sync(kFull, s1, row < 0 ? 0 : row);
        const int32_t nq = row < 0 ? 0 : (int32_t)((e - a) >> 2);
        for (int32_t q0 = lane & 7; q0 < nq; q0 += 32) {
            float4 w[4];
            int4 ta[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (q0 + 8 * u >= nq) continue;
                w[u] = *((const float4*)(P.w + a) + q0 + 8 * u);
                ta[u] = *((const int4*)(P.t_arr + a) + q0 + 8 * u);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (q0 + 8 * u >= nq) continue;
                const int64_t s = a + 4 * (int64_t)(q0 + 8 * u);
                const uint32_t ih = inh ? __ldg(P.inh + (s >> 5)) >> (s & 31) : 0u;
                float* wv = &w[u].x;
                const int32_t* tv = &ta[u].x;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const bool neg = (ih >> k) & 1u;
                    const float tr = trace_at_u(tab_pre, tpl, prev, tv[k]);
                    wv[k] = clamp_weight(wv[k] + (R.pre * tr - post0) * R.lr, neg ? -1.0f : 0.0f, neg ? 0.0f : 1.0f);
                }
                *((float4*)P.w + (s >> 2)) = w[u];
            }
        }
    }
    __syncwarp();
}

// Arrival branch of the plasticity of step `prev` (Synapse::run, src/NeuCor.cpp:718-726:
// lastSpikeArrival = now, so traceS = 0) for one lane's in-row; used when the
// plasticity is flushed outside the step.
__device__ void arrival_row(const NcPools& P, const NcNetDesc& D, int64_t s0, int32_t r0, int32_t r1, int32_t lf,
                            int32_t prev)
{
    const float* tab_post = P.tables + D.table_base + D.tab_pre_len;
    const uint32_t* slot = P.ring + D.ring_base + (int64_t)(prev & D.ring_mask) * D.ring_words;
    const float trT = trace_at(tab_post, D.tab_post_len, prev, lf);
    const Rates R = rates_of(D);
    for (int32_t wi = r0; wi < r1; ++wi) {
        uint32_t bits = slot[wi];
        if (!bits) continue;
        const int64_t cs = s0 + (int64_t)(wi - r0) * 32;
        const uint32_t ih = inh_bits32(P, cs);
        while (bits) {
            int b[8];
            pop8(&bits, b);
            float wv[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (b[k] >= 0) wv[k] = P.w[cs + b[k]];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (b[k] < 0) continue;
                P.t_arr[cs + b[k]] = prev;
                P.w[cs + b[k]] = plasticity(wv[k], (ih >> b[k]) & 1u, 0.0f, trT, R);
            }
        }
    }
}

// Four consecutive ring words of a row, over the steps t-1 .. t-KC.
struct RowBits {
    uint32_t win[4];  // arrived t-KC .. t-1: in the fold
    uint32_t arr[4];  // arrived t-1
    uint32_t old;     // bit q: word q of slot t-KC, released by this step, is not empty
};

// Loads the words [wi, min(wi + 4, r1)) of every slot of the window, four slots at a time so
// that their latencies overlap.
__device__ __forceinline__ void row_bits(RowBits& B, const uint32_t* ring, int64_t rw, int32_t ring_mask, int32_t wi,
                                         int32_t r1, int32_t t, int32_t kc)
{
    B.old = 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q) B.win[q] = B.arr[q] = 0u;
    for (int32_t k0 = 1; k0 <= kc && t - k0 >= 1; k0 += 4) {
        uint32_t x[4][4];
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            const int32_t k = k0 + d;
            const bool in = k <= kc && t - k >= 1;
            const uint32_t* row = ring + (int64_t)((t - k) & ring_mask) * rw + wi;
#pragma unroll
            for (int q = 0; q < 4; ++q) x[d][q] = in && wi + q < r1 ? row[q] : 0u;
        }
#pragma unroll
        for (int d = 0; d < 4; ++d)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                B.win[q] |= x[d][q];
                if (k0 + d == 1) B.arr[q] = x[d][q];
                if (k0 + d == kc && x[d][q]) B.old |= 1u << q;
            }
    }
}

// Pops up to kB set bits of the four words m (ascending, -1 when exhausted) into b; base is
// the bit number of m[0]'s first bit (an empty word costs a slot).
template <int kB>
__device__ __forceinline__ void pop_words(uint32_t (&m)[4], int& base, int (&b)[kB])
{
#pragma unroll
    for (int k = 0; k < kB; ++k) {
        if (m[0] == 0u) {
            m[0] = m[1];
            m[1] = m[2];
            m[2] = m[3];
            m[3] = 0u;
            base += 32;
        }
        b[k] = m[0] ? base + __ffs((int)m[0]) - 1 : -1;
        m[0] &= m[0] - 1u;
    }
}
__device__ __forceinline__ bool any_words(const uint32_t (&m)[4]) { return (m[0] | m[1] | m[2] | m[3]) != 0u; }

constexpr int kBatch = 8;  // charges, or weights, of a row gathered together

// One warp per warp_rows (8, 16 or 32) neurons of one net; blocks of any size, no block
// barrier.  The chain of dependent loads bounds it (about 800 cycles each and more for what
// is not in L2), so:
//   - what neither the spike launch of the step before nor a kernel between two steps writes
//     (everything but charges, ring bits, arrival steps and fire requests) is read, and the
//     draws are made, before the wait.  A flush writes stdp_done too: the step after one waits
//     for it as a whole (launch_neuron_step);
//   - the ring words of the whole window come in one go, then the gathers of the arrivals'
//     weights and of the sum's charges together;
//   - a small network gives a warp fewer neurons, so that a warp has fewer fired rows and a
//     shorter longest sum.
// Measured with the spike launch, a step (with a list of the fired neurons between the two
// kernels before): 50k x 80 at 1.7 Hz 26.9 -> 13.6 us, 8k x 50 with inhibitory synapses at
// 100 Hz 41.7 -> 20.2 us, 60k x 100 at 333 Hz 125 -> 85 us.
__global__ void __launch_bounds__(256, NC_NEURON_MIN_BLOCKS) k_neuron_step(NcPools P)
{
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const int rows = P.warp_rows;
    const int parts = 32 / rows;  // warps per tile
    bool waited = false;
    int n_tiles = P.n_tiles;
    if (P.n_tiles_dev) {
        wait_previous();
        waited = true;
        n_tiles = *P.n_tiles_dev;
    }
    const int units = n_tiles * parts, warps = gridDim.x * wpb;
    const int me = blockIdx.x * wpb + (threadIdx.x >> 5);
    for (int u = me; u < units; u += warps) {
        const NcTile tile = P.tiles[u / parts];
        const NcNetDesc& D = P.nets[tile.net];
        const int32_t first = tile.first + (u % parts) * rows, j = first + lane;
        const bool live = lane < rows && j < D.n;
        const int32_t pj = D.neuron_base + j;
        const int32_t pb = D.ptr_base + j;
        const int64_t word = D.word_base + (first >> 5);
        const int shift = first & 31;
        const uint32_t mask = (rows == 32 ? ~0u : (1u << rows) - 1u) << shift;
        uint32_t* ring = P.ring + D.ring_base;
        const int64_t rw = D.ring_words;
        const int32_t ring_mask = D.ring_mask, kc = D.kc;
        // (mutable state past the L1: it may hold what an earlier kernel left)
        const int32_t t = __ldcg(&D.t), done_to = __ldcg(&D.stdp_done);
        const bool act = __ldcg(&D.active) && t <= __ldcg(&D.t_end);
        const int32_t prev = t - 1;
        int64_t s0 = 0, s1 = 0;
        int32_t r0 = 0, r1 = 0, cid = j;
        int32_t lf = NC_NEVER;
        float pot = 0.0f;
        if (live) {
            lf = __ldcg(P.lf + pj);
            pot = __ldcg(P.pot + pj);
            s0 = __ldg(P.in_ptr + pb);
            s1 = __ldg(P.in_ptr + pb + 1);
            r0 = __ldg(P.ring_off + pb);
            r1 = __ldg(P.ring_off + pb + 1);
            if (D.permuted) cid = __ldg(P.orig_id + pj);
        }
        const uint32_t was = (__ldcg(P.fired + (int64_t)(prev & 1) * P.total_words + word) & mask) >> shift;
        // input requests, and the background target for step t+1 (src/NeuCor.cpp:604-607),
        // drawn per caller id
        bool forced = false;
        uint32_t bg = ~0u;
        if (live && act) {
            if (D.n_groups) forced = input_request(P, D, cid, t);
            if (D.bg_period > 0) {
                uint32_t o[4];
                philox((uint32_t)cid, (uint32_t)t, NC_STREAM_BACKGROUND, 0u, D, o);
                if (o[0] % (uint32_t)D.bg_period == 0u) {
                    bg = o[1] % (uint32_t)D.n;
                    if (D.permuted) bg = (uint32_t)__ldg(P.slot_of + D.neuron_base + bg);
                }
            }
        }
        if (!waited) {
            wait_previous();
            release_next();
            waited = true;
        }
        // the last unit's counters are read (the condition needs them): say so
        unsigned arrived = 0u;
        const bool last_unit = u + warps >= units;
        if (!act && !last_unit) continue;
        if (last_unit && lane == 0) arrived = atomicAdd(P.done_ctr, min(t, done_to) > NC_NEVER ? 1u : 0u);
        if (act) {
            const bool stdp = prev >= 1 && done_to < prev;
            // fire requests: kernels between two steps set them, so not before the wait
            const uint32_t fw = (__ldcg(P.forced + (int64_t)(t & 1) * P.total_words + word) & mask) >> shift;
            const uint32_t uw = (__ldcg(P.ufire + (int64_t)(t & 1) * P.total_words + word) & mask) >> shift;
            forced = forced || ((fw >> lane) & 1u);
            RowBits B;
            row_bits(B, ring, rw, ring_mask, r0, r1, t, kc);
            if (bg != ~0u)
                atomicOr(P.forced + (int64_t)((t + 1) & 1) * P.total_words + D.word_base + (bg >> 5), 1u << (bg & 31));
            if (stdp && was) postfire_rows(P, D, was, lane, s0, s1, prev);

            // charge_insynapses (src/NeuCor.cpp:688-700): terms of spikes that arrived
            // t-1 .. t-KC, ascending source id.  The arrival branch of the deferred
            // plasticity rides along: the spikes that arrived at prev are the ring bits of
            // slot prev.  Inside its AP (t - lastFire < KC) a neuron's potential comes from
            // the AP table whatever the sum is, and it cannot cross the threshold, so only
            // its sum is skipped; so is the rest of it once a neuron of a net with no
            // negative term is certain to fire (fires_at).
            const bool can = lf == NC_NEVER || t - lf >= kc;
            const bool stop = D.nonneg_terms != 0;
            const float leak = D.leak;
            bool settled = !can || (stop && fires_at(pot, leak));
            const TermFactor F = term_factor(D);
            const float trT = trace_at_u(P.tables + D.table_base + D.tab_pre_len, D.tab_post_len, prev, lf);
            const Rates R = rates_of(D);
            const float chg = (R.pre * 0.0f - R.post * trT) * R.lr;
            for (int32_t wi = r0; wi < r1;) {
                const int64_t sb = s0 + (int64_t)(wi - r0) * 32;
                int ba0 = 0, bw0 = 0;
                if (!stdp) B.arr[0] = B.arr[1] = B.arr[2] = B.arr[3] = 0u;
                if (settled) B.win[0] = B.win[1] = B.win[2] = B.win[3] = 0u;
                int bw[kBatch];
                float xv[kBatch];
                pop_words(B.win, bw0, bw);
#pragma unroll
                for (int k = 0; k < kBatch; ++k) xv[k] = bw[k] >= 0 ? P.x[sb + bw[k]] : -0.0f;
                while (any_words(B.arr)) {
                    int ba[kBatch];
                    float wv[kBatch];
                    uint32_t neg = 0u;
                    pop_words(B.arr, ba0, ba);
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        if (ba[k] < 0) continue;
                        wv[k] = P.w[sb + ba[k]];
                        if (!stop) neg |= inh_bit(P, sb + ba[k]) ? 1u << k : 0u;
                    }
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        if (ba[k] < 0) continue;
                        const bool n = (neg >> k) & 1u;
                        P.t_arr[sb + ba[k]] = prev;
                        P.w[sb + ba[k]] = clamp_weight(wv[k] + chg, n ? -1.0f : 0.0f, n ? 0.0f : 1.0f);
                    }
                }
                while (true) {
                    // the next batch's charges are gathered while this one is summed
                    const bool more = any_words(B.win);
                    float xn[kBatch];
                    if (more) {
                        pop_words(B.win, bw0, bw);
#pragma unroll
                        for (int k = 0; k < kBatch; ++k) xn[k] = bw[k] >= 0 ? P.x[sb + bw[k]] : -0.0f;
                    }
                    if (!settled) pot = fold_terms(pot, xv, F);
                    if (stop && !settled) settled = fires_at(pot, leak);
                    if (!more || settled) break;
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) xv[k] = xn[k];
                }
                // the spikes that arrived KC steps ago are released (AP_fireTime = 0)
                if (t - kc >= 1) {
                    uint32_t* orow = ring + (int64_t)((t - kc) & ring_mask) * rw + wi;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if ((B.old >> q) & 1u) orow[q] = 0u;
                }
                wi += 4;
                if (wi < r1) row_bits(B, ring, rw, ring_mask, wi, r1, t, kc);
            }
            bool fired = false;
            if (live) {
                // charge_passive (src/NeuCor.cpp:677-680)
                pot = (pot - -70.0f) * leak + -70.0f;
                // charge_thresholdCheck (src/NeuCor.cpp:682-686); vesicles stay positive.  An
                // input firer's Neuron::fire has no threshold or refractory test
                fired = ((uw >> lane) & 1u) || ((-55.0f < pot || forced) && can);
                if (fired) {
                    lf = t;
                    P.lf[pj] = t;
                    atomicAdd(P.firings + pj, 1u);  // (nothing waits for a value)
                }
                // AP (src/NeuCor.cpp:706-714)
                if (lf != NC_NEVER && t - lf < kc) pot = __ldg(P.tables + D.ap_base + (t - lf));
                P.pot[pj] = pot;
            }
            // bytes (8 neurons) of the bitsets: a warp may own part of a word
            const uint32_t fmask = __ballot_sync(kFull, fired);
            if (8 * lane < rows && first + 8 * lane < D.n) {
                const int64_t b = 4 * (D.word_base + (int64_t)(first >> 5)) + (shift >> 3) + lane;
                const uint8_t v = (uint8_t)(fmask >> (8 * lane));
                ((uint8_t*)(P.fired + (int64_t)(t & 1) * P.total_words))[b] = v;
                if ((fw >> (8 * lane)) & 0xffu) ((uint8_t*)(P.forced + (int64_t)(t & 1) * P.total_words))[b] = 0;
                if ((uw >> (8 * lane)) & 0xffu) ((uint8_t*)(P.ufire + (int64_t)(t & 1) * P.total_words))[b] = 0;
                if (D.raster_len > 0 && t >= D.raster_t0 && t - D.raster_t0 < D.raster_len)
                    ((uint8_t*)(D.raster + (int64_t)(t - D.raster_t0) * D.n_words))[(first >> 3) + lane] = v;
            }
        }
        if (last_unit && __shfl_sync(kFull, arrived, 0) == (unsigned)min(units, warps) - 1u) advance_steps<kEvent>(P, lane);
    }
    if (units == 0 && blockIdx.x == 0 && threadIdx.x < 32) {  // nets without neurons still step
        if (!waited) wait_previous();
        advance_steps<kEvent>(P, lane);
    }
}

// A warp's counts of the net it works on (nl, nd per lane), added when it passes to another.
struct LaunchCounts {
    int net = -1;
    unsigned fires = 0, nl = 0, nd = 0;
    __device__ __forceinline__ void turn_to(const NcPools& P, int n, int lane)
    {
        if (n == net) return;
        if (net >= 0) {
            nl = __reduce_add_sync(kFull, nl);
            nd = __reduce_add_sync(kFull, nd);
            if (lane == 0) {
                unsigned long long* st = P.nets[net].stats;
                atomicAdd(st + 0, (unsigned long long)fires);
                atomicAdd(st + 1, (unsigned long long)nl);
                atomicAdd(st + 2, (unsigned long long)nd);
            }
        }
        net = n;
        fires = nl = nd = 0;
    }
};

// The out-synapses of the neurons whose bits are set in `fired` (all lanes call).  start: row
// start of the unit's neuron `lane`.
__device__ __forceinline__ void launch_unit(const NcPools& P, const NcNetDesc& D, uint32_t fired, int32_t t,
                                            int64_t start, int lane, LaunchCounts& C)
{
    C.fires += __popc(fired);
    const uint32_t* fired_t = P.fired + (int64_t)(t & 1) * P.total_words + D.word_base;
    const float* tab_pre = P.tables + D.table_base;
    uint32_t* ring = P.ring + D.ring_base;
    // the descriptor's fields in registers: it lives in global memory, where every
    // store below could alias it
    const int32_t kc = D.kc, tpl = D.tab_pre_len, ring_mask = D.ring_mask;
    const int64_t syn_base = D.syn_base, ring_words = D.ring_words;
    const float dt = D.dt, c52 = D.c52;
    const Rates R = rates_of(D);
    for (; fired; fired &= fired - 1u) {
        const int i = __ffs((int)fired) - 1;
        const int64_t k0 = __shfl_sync(kFull, start, i), k1 = __shfl_sync(kFull, start, i + 1);
        for (int64_t kb = k0; kb < k1; kb += 128) {
            uint4 o[4];
            int32_t la[4];
            bool ok[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int64_t k = kb + lane + 32 * v;
                ok[v] = k < k1;
                if (ok[v]) {
                    o[v] = __ldg((const uint4*)P.out + k);
                    la[v] = P.last_arr[k];
                }
            }
            float wv[4];
            uint32_t fw[4];
            bool acc[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                // freed by the target's update at t only if the target's id is not above
                acc[v] = ok[v] && (la[v] == NC_NEVER || t - la[v] >= kc + (int32_t)((o[v].w >> 14) & 1u));
                fw[v] = 0u;
                if (acc[v]) {
                    wv[v] = P.w[syn_base + o[v].x];
                    // target id below the source's: its update ran first
                    if ((o[v].w >> 15) & 1u) fw[v] = fired_t[o[v].y >> 5] >> (o[v].y & 31);
                }
                C.nl += acc[v] ? 1u : 0u;
                C.nd += ok[v] && !acc[v] ? 1u : 0u;
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                if (!acc[v]) continue;
                const int64_t k = kb + lane + 32 * v;
                const int64_t s = syn_base + o[v].x;
                float w = wv[v];
                if (fw[v] & 1u)
                    w = plasticity(w, inh_bit(P, s), trace_at(tab_pre, tpl, t, P.t_arr[s]), 0.0f, R);
                // AP_depolFac = 0.2f; *= 52.0; *= weight  (src/NeuCor.cpp:729-731)
                P.x[s] = dt * (c52 * w);
                const int32_t d = (int32_t)(o[v].w & 0x3fffu);
                P.last_arr[k] = t + d;
                atomicOr(ring + (int64_t)((t + d) & ring_mask) * ring_words + (o[v].z >> 5), 1u << (o[v].z & 31));
            }
        }
    }
}

// Synapse::fire (src/NeuCor.cpp:727-738) on the out-synapses of the neurons that fired at t,
// a warp per launch_rows (1 to 8) neurons' fired bits (a unit), all lanes on a fired neuron's
// out-synapses, four in flight each.  Its chain of loads bounds it: the fired byte (of both
// parities, beside the step counter), the 16-byte out-synapse records, the weights and the
// fired words of targets that came first.
//   kMany: a warp has several units (many_units), and a lane looks at the fired byte of one of
//   its next 32: one after the other, a quiet network of 2M neurons took 83 us for them, 26 so.
//   With one unit a warp the row starts are read before the wait: 0.9 us less (50k x 80 quiet).
template <bool kMany>
__global__ void __launch_bounds__(256, NC_LAUNCH_MIN_BLOCKS) k_spike_launch(NcPools P)
{
    __shared__ int s_net[8];
    __shared__ unsigned s_acc[8][3];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int nwb = blockDim.x >> 5;
    bool waited = false;
    int n_tiles = P.n_tiles;
    if (P.n_tiles_dev) {
        wait_previous();
        waited = true;
        n_tiles = *P.n_tiles_dev;
    }
    const int rows = P.launch_rows, parts = 32 / rows;
    const int units = parts * n_tiles;
    LaunchCounts C;
    const int warps = gridDim.x * nwb;
    for (int base = blockIdx.x * nwb + wib; base < units; base += (kMany ? 32 : 1) * warps) {
        const int mine = base + (kMany ? lane * warps : 0);
        int32_t net = -1, first = 0;
        int64_t byte = 0, start = 0;
        if (mine < units) {
            const NcTile tile = P.tiles[mine / parts];
            const NcNetDesc& D = P.nets[tile.net];
            first = tile.first + (mine % parts) * rows;
            if (first < D.n) {
                net = tile.net;
                byte = 4 * (D.word_base + (int64_t)(first >> 5)) + ((first & 31) >> 3);
                if (!kMany && lane <= min(rows, D.n - first)) start = __ldg(P.out_ptr + D.ptr_base + first + lane);
            }
        }
        if (!kMany && net < 0) continue;
        if (!waited) {
            wait_previous();
            release_next();
            waited = true;
        }
        uint32_t fired = 0u;
        int32_t t = 0;
        if (net >= 0) {
            // both parities' bytes beside the counter that picks one
            const uint32_t f0 = __ldcg((const uint8_t*)P.fired + byte);
            const uint32_t f1 = __ldcg((const uint8_t*)(P.fired + P.total_words) + byte);
            t = __ldcg(&P.nets[net].t) - 1;
            fired = ((t & 1 ? f1 : f0) >> (first & 7)) & ((1u << rows) - 1u);
            if (fired && !__ldcg(&P.nets[net].live)) fired = 0u;
        }
        if (!kMany) {
            if (!fired) continue;
            C.turn_to(P, net, lane);
            launch_unit(P, P.nets[net], fired, t, start, lane, C);
            continue;
        }
        for (unsigned todo = __ballot_sync(kFull, fired != 0u); todo; todo &= todo - 1u) {
            const int who = __ffs((int)todo) - 1;
            const int32_t n = __shfl_sync(kFull, net, who), f = __shfl_sync(kFull, first, who);
            const NcNetDesc& D = P.nets[n];
            if (lane <= min(rows, D.n - f)) start = __ldg(P.out_ptr + D.ptr_base + f + lane);
            C.turn_to(P, n, lane);
            launch_unit(P, D, __shfl_sync(kFull, fired, who), __shfl_sync(kFull, t, who), start, lane, C);
        }
    }
    if (!waited) wait_previous();
    // per-block reduction of the counters, per net
    if (!__syncthreads_or(C.net >= 0)) return;
    C.nl = __reduce_add_sync(kFull, C.nl);
    C.nd = __reduce_add_sync(kFull, C.nd);
    if (lane == 0) {
        s_net[wib] = C.net;
        s_acc[wib][0] = C.fires;
        s_acc[wib][1] = C.nl;
        s_acc[wib][2] = C.nd;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 0; w < nwb; ++w) {
            const int n = s_net[w];
            if (n < 0) continue;
            unsigned long long c[3] = {s_acc[w][0], s_acc[w][1], s_acc[w][2]};
            for (int v = w + 1; v < nwb; ++v) {
                if (s_net[v] != n) continue;
#pragma unroll
                for (int k = 0; k < 3; ++k) c[k] += s_acc[v][k];
                s_net[v] = -1;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (c[k]) atomicAdd(P.nets[n].stats + k, c[k]);
        }
    }
}

// Applies the plasticity deferred from the last simulated step (before read-back).
__global__ void __launch_bounds__(256) k_stdp_flush(NcPools P)
{
    const int lane = threadIdx.x & 31;
    const int gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (gw >= P.n_tiles) return;
    const NcTile tile = P.tiles[gw];
    const NcNetDesc& D = P.nets[tile.net];
    const int32_t prev = D.t - 1;
    if (!D.active || prev < 1 || D.stdp_done >= prev) return;
    const int32_t j = tile.first + lane;
    const bool live = j < D.n;
    const int32_t pb = D.ptr_base + j;
    int32_t lf = NC_NEVER;
    int64_t s0 = 0, s1 = 0;
    int32_t r0 = 0, r1 = 0;
    if (live) {
        lf = P.lf[D.neuron_base + j];
        s0 = P.in_ptr[pb];
        s1 = P.in_ptr[pb + 1];
        r0 = P.ring_off[pb];
        r1 = P.ring_off[pb + 1];
    }
    postfire_rows(P, D, P.fired[(int64_t)(prev & 1) * P.total_words + D.word_base + (tile.first >> 5)], lane, s0, s1,
                  prev);
    if (live && r1 > r0) arrival_row(P, D, s0, r0, r1, lf, prev);
}

__global__ void k_mark_flushed(NcPools P)
{
    for (int n = threadIdx.x; n < P.n_nets; n += blockDim.x) {
        NcNetDesc* D = P.nets + n;
        if (D->active && D->stdp_done < D->t - 1) D->stdp_done = D->t - 1;
    }
}

// Background draws made at step 0 for step 1 (the first NeuCor::run, src/NeuCor.cpp:604-607).
__global__ void k_background_prologue(NcPools P, int net)
{
    const NcNetDesc& D = P.nets[net];
    const int32_t j = blockIdx.x * blockDim.x + threadIdx.x;  // caller id
    if (j >= D.n || D.bg_period <= 0) return;
    uint32_t o[4];
    philox((uint32_t)j, 0u, NC_STREAM_BACKGROUND, 0u, D, o);
    if (o[0] % (uint32_t)D.bg_period == 0u) {
        uint32_t tgt = o[1] % (uint32_t)D.n;
        if (D.permuted) tgt = (uint32_t)P.slot_of[D.neuron_base + tgt];
        atomicOr(P.forced + (int64_t)(1 & 1) * P.total_words + D.word_base + (tgt >> 5), 1u << (tgt & 31));
    }
}

__global__ void k_fill_words(uint32_t* a, int64_t count, uint32_t v)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < count; k += (int64_t)gridDim.x * blockDim.x)
        a[k] = v;
}

// Forced fire requests for the net's next step (Neuron::scheduleFire).
__global__ void k_force_bits(NcPools P, int net, const int32_t* ids, int count)
{
    const NcNetDesc& D = P.nets[net];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const int32_t j = ids[k];
    atomicOr(P.forced + (int64_t)(D.t & 1) * P.total_words + D.word_base + (j >> 5), 1u << (j & 31));
}

}  // namespace

namespace nc {

static int check_launch()
{
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Launches fn<<<grid, block, 0, s>>>(P), as a programmatic dependent launch unless `whole`.
static int launch_dependent(void (*fn)(NcPools), int grid, int block, void* stream, const NcPools& P, bool whole = false)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = whole ? 0 : 1;
    if (cudaLaunchKernelEx(&cfg, fn, P) != cudaSuccess) return -1;
    return check_launch();
}

// Blocks of `threads` threads of the neuron step that the current device holds at once (cached
// per device and block size; 0 when it does not say).
int event_resident_blocks(int threads)
{
    static std::atomic<int> cache[64][9];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::atomic<int>& c = cache[dev][threads / 32];
    int n = c.load(std::memory_order_relaxed);
    if (n == 0) {
        int sms = 0, per_sm = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_neuron_step, threads, 0) != cudaSuccess)
            return 0;
        n = sms * per_sm;
        c.store(n, std::memory_order_relaxed);
    }
    return n;
}

int launch_neuron_step(const NcPools& P, const LaunchShape& L, bool whole, void* stream)
{
    const int64_t warps = (int64_t)P.n_tiles * (32 / P.warp_rows);
    int64_t blocks = (warps + L.neuron_block / 32 - 1) / (L.neuron_block / 32);
    // at most a wave: a warp goes on to its next tile sooner than a block takes the place of
    // another (2M neurons, 13 waves: 151 us a step, 134 so; 500k busy 312 either way)
    const int resident = event_resident_blocks(L.neuron_block);
    if (resident > 0) blocks = std::min<int64_t>(blocks, resident);
    return launch_dependent(k_neuron_step, (int)std::max<int64_t>(1, blocks), L.neuron_block, stream, P, whole);
}

bool many_units(int n_tiles, const NcPools& P, const LaunchShape& L)
{
    // two units a warp: 100k neurons (1.3 a warp) 25.2 us a step one after the other and 26.1
    // with lanes, 200k (2.6) 31.3 and 29.6, 500k (6.4) 57 and 46
    return (int64_t)n_tiles * (32 / P.launch_rows) > 2 * (int64_t)L.launch_blocks * (L.launch_block / 32);
}

int launch_spike_launch(const NcPools& P, const LaunchShape& L, bool many, void* stream)
{
    return launch_dependent(many ? k_spike_launch<true> : k_spike_launch<false>, L.launch_blocks,
                            L.launch_block, stream, P);
}

int launch_stdp_flush(const NcPools& P, const LaunchShape& L, void* stream)
{
    const int warps_per_block = L.neuron_block / 32;
    const int blocks = (P.n_tiles + warps_per_block - 1) / warps_per_block;
    if (blocks > 0) k_stdp_flush<<<blocks, L.neuron_block, 0, (cudaStream_t)stream>>>(P);
    k_mark_flushed<<<1, 256, 0, (cudaStream_t)stream>>>(P);
    return check_launch();
}

int launch_fill_words(uint32_t* a, int64_t count, uint32_t v, void* stream)
{
    if (count <= 0) return 0;
    const int64_t blocks = (count + 1023) / 1024;
    k_fill_words<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, (cudaStream_t)stream>>>(a, count, v);
    return check_launch();
}

int launch_background_prologue(const NcPools& P, int net, int n_neurons, void* stream)
{
    const int blocks = (n_neurons + 255) / 256;
    if (blocks > 0) k_background_prologue<<<blocks, 256, 0, (cudaStream_t)stream>>>(P, net);
    return check_launch();
}

int launch_force_bits(const NcPools& P, int net, const int32_t* d_ids, int count, void* stream)
{
    if (count <= 0) return 0;
    k_force_bits<<<(count + 255) / 256, 256, 0, (cudaStream_t)stream>>>(P, net, d_ids, count);
    return check_launch();
}

}  // namespace nc
