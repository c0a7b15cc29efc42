// nc_device.cuh — device helpers shared by the step kernels: the reference's
// plasticity and trace arithmetic, the ordered `float += double` fold, the input draws
// and bit iteration.
#pragma once
#include "nc_engine.cuh"

#include <cstddef>

namespace nc_dev {

constexpr unsigned kFull = 0xffffffffu;

static __device__ __forceinline__ float trace_at(const float* tab, int len, int32_t now, int32_t then)
{
    if (then == NC_NEVER) return 0.0f;  // lastSpikeArrival = -inf / lastFire = NaN
    const int32_t k = now - then;
    return k < len ? __ldg(tab + k) : 0.0f;
}

static __device__ __forceinline__ bool inh_bit(const NcPools& P, int64_t s)
{
    return (__ldg(P.inh + (s >> 5)) >> (s & 31)) & 1u;
}

// The 32 inhibitory bits of synapses s .. s+31 (s need not be word-aligned; the pool
// keeps one spare word at its end).
static __device__ __forceinline__ uint32_t inh_bits32(const NcPools& P, int64_t s)
{
    const int64_t w0 = s >> 5;
    return __funnelshift_r(__ldg(P.inh + w0), __ldg(P.inh + w0 + 1), (uint32_t)(s & 31));
}

// The learning constants a kernel holds in registers (read from the descriptor once:
// the descriptor lives in global memory, where every store could alias it).
struct Rates {
    float pre, post, lr;
};
static __device__ __forceinline__ Rates rates_of(const NcNetDesc& D) { return Rates{D.pre_factor, D.post_factor, D.lr}; }

// Synapse::synapticPlasticity weight update and clamp (src/NeuCor.cpp:757-761);
// fmin/fmax keep the C library's generic semantics.
static __device__ __forceinline__ float plasticity(float w, bool inh, float traceS, float traceT, const Rates& R)
{
    const float weightChange = R.pre * traceS - R.post * traceT;
    float v = w + weightChange * R.lr;
    if (!inh) {
        const float m = (v <= 1.0f) ? v : 1.0f;
        v = (m >= 0.0f) ? m : 0.0f;
    } else {
        const float m = (v <= 0.0f) ? v : 0.0f;
        v = (m >= -1.0f) ? m : -1.0f;
    }
    return v;
}

// The clamp of synapticPlasticity (src/NeuCor.cpp:757-761): hi = 1, lo = 0 for an excitatory
// synapse, hi = 0, lo = -1 for an inhibitory one.  fminf is the compare and select of the
// upper bound (a NaN becomes hi); the lower one keeps a negative zero, as the reference's.
static __device__ __forceinline__ float clamp_weight(float v, float lo, float hi)
{
    const float m = fminf(v, hi);
    return (m >= lo) ? m : lo;
}

// trace_at with one unsigned compare: a step counter `then` of NC_NEVER (INT32_MIN) puts
// now - then at 2^31 or above, past any table.
static __device__ __forceinline__ float trace_at_u(const float* tab, int len, int32_t now, int32_t then)
{
    const uint32_t k = (uint32_t)now - (uint32_t)then;
    return k < (uint32_t)len ? __ldg(tab + k) : 0.0f;
}

static __device__ __forceinline__ float plasticity(float w, bool inh, float traceS, float traceT, const NcNetDesc& D)
{
    return plasticity(w, inh, traceS, traceT, rates_of(D));
}

// The charge_insynapses term of a captured charge x = deltaT*AP_depolFac,
// x*0.9943*exp(0.3702*deltaT) (src/NeuCor.cpp:695).
static __device__ __forceinline__ double make_term(float x, double e_term)
{
    return __dmul_rn(__dmul_rn((double)x, 0.9943), e_term);
}

// The factor of every term of a net, 0.9943*exp(0.3702*deltaT), as a float and the float
// of what it leaves (within 2^-49 of it together), and the binary64 factor of the exact form.
struct TermFactor {
    float hi, lo;
    double e_term;
};
static __device__ __forceinline__ TermFactor term_factor(const NcNetDesc& D)
{
    return TermFactor{D.term_hi, D.term_lo, D.e_term};
}

// `p += term` of the charge x (src/NeuCor.cpp:695: a binary64 sum rounded to float) on float
// arithmetic alone, by Ziv's rounding test: the term as a float pair th + tl within 2^-46 of
// itself, p + th exactly as s + e (Knuth's TwoSum), and s + (e + tl) rounded from either end
// of an interval that holds the exact sum, the binary64 rounding included.  Where both ends
// round to the same float that float is the result; otherwise `ok` is cleared and the
// caller redoes its batch exactly (6 in a million terms of ordinary networks; sums near
// zero, infinities and NaN always).  An FP64 instruction takes a scheduler 64 cycles here
// and a dependent add about 300: a batch of 8 took 2,400 cycles in a chain of binary64 adds
// and takes 400 so.  (tests/test_fold_add.py compares the same arithmetic on the CPU.)
static __device__ __forceinline__ float add_term(float p, float x, const TermFactor& F, bool& ok)
{
    const float th = x * F.hi;
    const float tl = __fmaf_rn(x, F.hi, -th) + x * F.lo;
    const float s = p + th;
    const float bb = s - p;
    const float e = (p - (s - bb)) + (th - bb);
    const float r = e + tl;
    // half the interval: eight times the errors of r, tl and the binary64 rounding of the sum
    const float base = __fmaf_rn(fabsf(s), 0x1p-50f, __fmaf_rn(fabsf(th), 0x1p-43f, 0x1p-120f));
    const float d = __fmaf_rn(fabsf(r), 0x1p-21f, base);
    const float a = s + (r + d);
    ok = ok && a == s + (r - d);
    return a;
}

// The exact form of fold_terms, on binary64.  Kept out of line: a rare redo.
static __device__ __noinline__ float fold_exact(float p, float x0, float x1, float x2, float x3, float x4, float x5,
                                                float x6, float x7, double e_term)
{
    const float x[8] = {x0, x1, x2, x3, x4, x5, x6, x7};
#pragma unroll
    for (int k = 0; k < 8; ++k)
        p = __double2float_rn(__dadd_rn((double)p, make_term(x[k], e_term)));
    return p;
}

// Folds the terms of the charges x[0..8) into p, in order.  An absent term is the charge
// -0.0, which adds the term -0.0 and changes no p.
static __device__ __forceinline__ float fold_terms(float p, const float (&x)[8], const TermFactor& F)
{
    const float p0 = p;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 8; ++k) p = add_term(p, x[k], F, ok);
    if (__builtin_expect(!ok, 0)) p = fold_exact(p0, x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7], F.e_term);
    return p;
}

// Whether a neuron out of its AP with potential `pot` (its sum so far) fires:
// charge_passive and the threshold test of charge_thresholdCheck (src/NeuCor.cpp:677-686),
// with the step kernels' own operations.  When no term of the net can be negative the sum
// only grows (rounding keeps the order) and so does this result, so a fold may stop once
// it holds: the neuron fires whatever the remaining terms are, and its potential is then
// replaced by the AP table (src/NeuCor.cpp:706-714).
static __device__ __forceinline__ bool fires_at(float pot, float leak)
{
    return -55.0f < (pot - -70.0f) * leak + -70.0f;
}

static __device__ __forceinline__ void philox(uint32_t a, uint32_t b, uint32_t stream, uint32_t c, const NcNetDesc& D,
                                       uint32_t out[4])
{
    nc_philox(a, b, stream, c, D.key0, D.key1, out);
}

#ifndef NC_GROUP_RANGE
#define NC_GROUP_RANGE 1
#endif
// Whether input neuron j requests a fire at step t (Poisson groups).
static __device__ bool input_request(const NcPools& P, const NcNetDesc& D, int32_t j, int32_t t)
{
    // most neurons are in no group: one range test instead of a walk over the groups
    if (NC_GROUP_RANGE && (j < D.group_lo || j >= D.group_hi)) return false;
    uint32_t o[4];
    for (int g = 0; g < D.n_groups; ++g) {
        const NcGroupDev G = P.groups[D.group_base + g];
        if (j < G.first || j >= G.first + G.count) continue;
        const uint32_t m = (uint32_t)(j - G.first);
        if (!G.correlated) {
            philox((uint32_t)G.index, (uint32_t)t, NC_STREAM_INDEPENDENT, m, D, o);
            if (o[0] < G.thresh) return true;
            continue;
        }
        for (int32_t src = t - G.jitter; src <= t + G.jitter; ++src) {
            if (src < 0) continue;
            philox((uint32_t)G.index, (uint32_t)src, NC_STREAM_SOURCE, 0u, D, o);
            if (!(o[0] < G.thresh)) continue;
            philox((uint32_t)G.index, (uint32_t)src, NC_STREAM_JITTER, m, D, o);
            const int32_t off = (int32_t)(o[0] % (uint32_t)(2 * G.jitter + 1)) - G.jitter;
            if (src + off == t) return true;
        }
    }
    return false;
}

// Once every block (or warp) of a launch has read the step counters, one warp moves those of
// nets 0 .. n-1 on: kStep counts the dense step, kEvent the event form's neuron step (and notes
// the nets it advanced: live), kFlush notes that the launches and plasticity of every active
// net's last step are done.
enum Advance { kStep, kEvent, kFlushed };

// c: t, t_end, stdp_done, tsum; f: active, live, dt_again
template <Advance kHow>
static __device__ __forceinline__ void advance_net(NcNetDesc* D, unsigned long long* stats, int4 c, int4 f)
{
    const bool go = f.x && (kHow == kFlushed ? c.z < c.x - 1 : c.x <= c.y);
    if (kHow == kEvent && f.y != (int32_t)go) D->live = go;
    if (!go) return;
    if (c.z < c.x - 1) c.z = c.x - 1;
    if (kHow != kFlushed) {
        atomicAdd(stats + 3, 1ull);
        c.x += 1;
        c.w = __float_as_int(__fadd_rn(__int_as_float(c.w), __int_as_float(f.z)));  // currentTime = targetTime (src/NeuCor.cpp:616)
    }
    *(int4*)D = c;
}

// Many nets: a lane's loads of eight nets, two of 16 bytes from one sector each, are under way
// together: one after the other, with each net's constants from a second line, 2,000 nets of 20
// neurons took 89 us a step dense and 86 in the event form, 25 and 26 now.  Out of line: its
// registers are not the step's.
template <Advance kHow>
static __device__ __noinline__ void advance_many(NcNetDesc* nets, unsigned long long* stats, int n_nets, int lane)
{
    constexpr int kU = 8;
    for (int n0 = lane; n0 < n_nets; n0 += 32 * kU) {
        int4 c[kU], f[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int4* D = (const int4*)(nets + min(n0 + 32 * u, n_nets - 1));
            c[u] = __ldcg(D);
            f[u] = __ldcg(D + 1);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int n = n0 + 32 * u;
            if (n < n_nets) advance_net<kHow>(nets + n, stats + 4 * (int64_t)n, c[u], f[u]);
        }
    }
}

template <Advance kHow>
static __device__ __forceinline__ void advance_steps(const NcPools& P, int lane)
{
    static_assert(offsetof(NcNetDesc, t) == 0 && offsetof(NcNetDesc, t_end) == 4 && offsetof(NcNetDesc, stdp_done) == 8 &&
                      offsetof(NcNetDesc, tsum) == 12 && offsetof(NcNetDesc, active) == 16 &&
                      offsetof(NcNetDesc, live) == 20 && offsetof(NcNetDesc, dt_again) == 24,
                  "counters");
    const int n_nets = P.n_nets_dev ? __ldcg(P.n_nets_dev) : P.n_nets;
    if (n_nets > 32) {
        advance_many<kHow>(P.nets, P.stats, n_nets, lane);
    } else if (lane < n_nets) {
        const int4* D = (const int4*)(P.nets + lane);
        advance_net<kHow>(P.nets + lane, P.stats + 4 * lane, __ldcg(D), __ldcg(D + 1));
    }
    if (lane == 0) *P.done_ctr = 0u;
}

// Pops up to 8 set bits of *m in ascending order into b[] (-1 when exhausted).
static __device__ __forceinline__ void pop8(uint32_t* m, int b[8])
{
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        b[k] = *m ? __ffs(*m) - 1 : -1;
        *m &= *m - 1u;
    }
}

}  // namespace nc_dev
