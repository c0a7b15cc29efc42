// nc_host.cpp — host-side construction: synapse table layout, reference-arithmetic
// tables, and the network builders.  Compiled with -ffp-contract=off: every float
// expression here mirrors a reference expression and must round the same way.
#include "nc_host.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <thread>

namespace nc {

float step_ms(int64_t k, float dt) { return (float)k * dt; }

float get_dist(const float* a, const float* b)
{
    // sqrtf(powf(x-c.x,2)+powf(y-c.y,2)+powf(z-c.z,2)); GCC folds powf(v,2) to v*v
    const float dx = a[0] - b[0], dy = a[1] - b[1], dz = a[2] - b[2];
    return sqrtf(dx * dx + dy * dy + dz * dz);
}

int32_t delay_steps(float length, float dt)
{
    // AP_fireTime = length*AP_speed (AP_speed = 2.0, src/NeuCor.cpp:485,733), in
    // whole steps rounded to nearest, at least one step
    const float ms = length * 2.0f;
    const float q = floorf(ms / dt + 0.5f);
    if (!(q >= 1.0f)) return 1;
    if (q > 32767.0f) return -1;
    return (int32_t)q;
}

uint32_t rate_threshold(float rate_hz, float dt)
{
    const double prob = (double)rate_hz * (double)dt / 1000.0;
    if (!(prob > 0.0)) return 0u;
    const double v = prob * 4294967296.0;
    if (v >= 4294967295.0) return 4294967295u;
    return (uint32_t)v;
}

float ap_value(float x)
{
    // Neuron::AP with x = (float)currentT - lastFire; member values from the Neuron
    // constructor (src/NeuCor.cpp:376-385)
    const float AP_h = 100.0f, AP_depolW = 0.3f, AP_polW = 0.6f, AP_deltaPol = 1.16f;
    const float AP_depolFac = 0.2f, AP_deltaStart = 1.0f, baselevel = -70.0f, threshold = -55.0f;
    const float a = x - AP_deltaStart;
    const float b = x - AP_deltaStart - AP_deltaPol;
    const double v = AP_h * (exp(-(a * a) / (2.0 * AP_depolW * AP_depolW)) -
                             exp(-(b * b) / (2.0 * AP_polW * AP_polW)) * AP_depolFac) +
                     baselevel + (threshold - baselevel) * fmax(1.0 - (double)x, 0.0);
    return (float)v;
}

// Morton code of a position quantised to 10 bits per axis over the bounding box.
static uint32_t morton3(uint32_t x, uint32_t y, uint32_t z)
{
    auto spread = [](uint32_t v) {
        v &= 0x3ffu;
        v = (v | (v << 16)) & 0x30000ffu;
        v = (v | (v << 8)) & 0x300f00fu;
        v = (v | (v << 4)) & 0x30c30c3u;
        v = (v | (v << 2)) & 0x9249249u;
        return v;
    };
    return spread(x) | (spread(y) << 1) | (spread(z) << 2);
}

static void storage_order(NetHost& h, const float* xyz, int32_t order_kind)
{
    const int32_t n = h.n;
    h.orig_id.resize((size_t)n);
    h.slot_of.resize((size_t)n);
    for (int32_t i = 0; i < n; ++i) h.orig_id[(size_t)i] = i;
    if (order_kind == NC_ORDER_SPATIAL && xyz && n > 1) {
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        for (int32_t i = 0; i < n; ++i)
            for (int a = 0; a < 3; ++a) {
                const double v = xyz[3 * (size_t)i + a];
                if (std::isfinite(v)) {
                    lo[a] = std::min(lo[a], v);
                    hi[a] = std::max(hi[a], v);
                }
            }
        std::vector<uint32_t> code((size_t)n);
        for (int32_t i = 0; i < n; ++i) {
            uint32_t q[3];
            for (int a = 0; a < 3; ++a) {
                const double v = xyz[3 * (size_t)i + a];
                const double span = hi[a] - lo[a];
                double f = (std::isfinite(v) && span > 0) ? (v - lo[a]) / span : 0.0;
                f = std::min(1.0, std::max(0.0, f));
                q[a] = (uint32_t)(f * 1023.0);
            }
            code[(size_t)i] = morton3(q[0], q[1], q[2]);
        }
        // by code, equal ones by id: three stable passes over ten bits each (a comparison sort
        // took 1.5 of the 4 ms that building 20k x 60 on the device takes, 8.6 ms of 15 at
        // 100k x 100)
        std::vector<int32_t> other((size_t)n);
        for (int shift = 0; shift < 30; shift += 10) {
            int32_t at[1025] = {0};
            for (int32_t i = 0; i < n; ++i) at[(code[(size_t)i] >> shift & 1023u) + 1]++;
            for (int b = 0; b < 1024; ++b) at[b + 1] += at[b];
            for (int32_t id : h.orig_id) other[(size_t)at[code[(size_t)id] >> shift & 1023u]++] = id;
            h.orig_id.swap(other);
        }
    }
    h.permuted = false;
    for (int32_t s = 0; s < n; ++s) {
        h.slot_of[(size_t)h.orig_id[(size_t)s]] = s;
        if (h.orig_id[(size_t)s] != s) h.permuted = true;
    }
}

// Trace table powf(decay, k*dt) for k = 0.. until it underflows to zero, with the
// reference's "a trace of exactly 1 counts as 0" rule (src/NeuCor.cpp:744-745).
static bool trace_table(float decay, float dt, std::vector<float>& out, int32_t& len)
{
    const int64_t cap = 1 << 22;
    len = 0;
    for (int64_t k = 0; k < cap; ++k) {
        const float raw = powf(decay, step_ms(k, dt));
        if (raw == 0.0f) {
            len = (int32_t)k;
            return true;
        }
        out.push_back(raw == 1.0f ? 0.0f : raw);
    }
    return false;
}

bool inhibitory_flag(const NetHost& h, int64_t c) { return (h.inh_bits[(size_t)(c >> 5)] >> (c & 31)) & 1u; }

// Whether the m-th synapse appended to an outSynapses vector that ends with `size`
// elements was copied by a reallocation: reserve(5) (src/NeuCor.cpp:374), then
// libstdc++ doubles the capacity of a full vector.
static bool grown_copy(int64_t m, int64_t size)
{
    int64_t cap = 5;
    while (cap <= m) cap *= 2;
    return size > cap;
}

KnnGrid knn_grid(int32_t n, int32_t k, float density)
{
    KnnGrid G;
    G.side = (float)std::cbrt((double)n / (double)density);
    // uniform grid, cells of about k/8 points
    const double cell_target = std::cbrt(std::max(1.0, (double)k / 8.0) / (double)density);
    G.g = std::max(1, (int32_t)std::floor((double)G.side / cell_target));
    G.g = std::min(G.g, 1024);
    G.h = G.side / (float)G.g;
    return G;
}

// The synapses, as indexes into the input, by target slot and in each target's row by the
// caller's source id, repeats in input order: two counting sorts, the first left out where
// the input is in source order already (a kNN network's is).  start: n + 1 row starts.
template <class Index>
static std::unique_ptr<Index[]> rows_of_targets(const NetHost& h, int64_t n_syn, const int32_t* from, const int32_t* to,
                                                bool by_source, const std::vector<int64_t>& start)
{
    std::unique_ptr<Index[]> first, order(new Index[(size_t)n_syn]);
    if (!by_source) {
        std::vector<int64_t> at((size_t)h.n + 1, 0);
        for (int64_t k = 0; k < n_syn; ++k) at[(size_t)from[k] + 1]++;
        for (int32_t i = 0; i < h.n; ++i) at[(size_t)i + 1] += at[(size_t)i];
        first.reset(new Index[(size_t)n_syn]);
        for (int64_t k = 0; k < n_syn; ++k) first[(size_t)at[(size_t)from[k]]++] = (Index)k;
    }
    std::vector<int64_t> at(start.begin(), start.end() - 1);
    for (int64_t q = 0; q < n_syn; ++q) {
        const int64_t k = by_source ? q : (int64_t)first[(size_t)q];
        order[(size_t)at[(size_t)h.slot_of[(size_t)to[k]]]++] = (Index)k;
    }
    return order;
}

// The in-synapse rows (CSC): the first of repeated (source, target) pairs is kept
// (createSynapse, src/NeuCor.cpp:189-191).  above: delay and same-step order flags of every
// position, as in the upper part of a key; row_end: end of each row's synapses.
template <class Index>
static int fill_rows(NetHost& h, const Index* order, const std::vector<int64_t>& start, const int32_t* from,
                     const float* weight, const float* length, std::vector<uint32_t>& above,
                     std::vector<int64_t>& row_end, std::string& err)
{
    const int32_t n = h.n, pad = pad_slot(n);
    int64_t size = 0;  // were no pair repeated
    for (int32_t j = 0; j < n; ++j)
        size = (size + start[(size_t)j + 1] - start[(size_t)j] + row_align(j) - 1) / row_align(j) * row_align(j);
    h.csc_pre.resize((size_t)size);
    h.w.resize((size_t)size);
    above.resize((size_t)size);
    int32_t* pre = h.csc_pre.data();
    float* w = h.w.data();
    int64_t c = 0;
    for (int32_t j = 0; j < n; ++j) {
        h.in_ptr[(size_t)j] = c;
        const int32_t dst = h.orig_id[(size_t)j];
        const float* at = &h.xyz[3 * (size_t)dst];
        int32_t last_pre = -1;
        for (int64_t q = start[(size_t)j]; q < start[(size_t)j + 1]; ++q) {
            const int64_t k = (int64_t)order[q];
            const int32_t src = from[k];
            if (src == last_pre) continue;
            last_pre = src;
            h.input_to_csc[(size_t)k] = c;
            pre[c] = h.slot_of[(size_t)src];
            const float len = length ? length[k] : get_dist(&h.xyz[3 * (size_t)src], at);
            const int32_t d = delay_steps(len, h.dt);
            if (d < 0 || d > kMaxDelay) { err = "synapse delay exceeds 16383 steps"; return NC_ERR_INVALID; }
            h.max_delay = std::max(h.max_delay, d);
            // the same-step order rules compare the caller's ids of target and source
            above[(size_t)c] = (uint32_t)d << NC_KEY_DELAY_SHIFT | (dst > src ? NC_KEY_AFTER : 0u) |
                               (dst < src ? NC_KEY_BEFORE : 0u);
            w[c++] = weight[k];
        }
        row_end[(size_t)j] = c;
        h.s += c - h.in_ptr[(size_t)j];
        for (; c & (row_align(j) - 1); ++c) {
            pre[c] = pad;
            above[(size_t)c] = 0u;
            w[c] = 0.0f;
        }
    }
    h.in_ptr[(size_t)n] = c;
    h.sp = c;
    h.csc_pre.resize((size_t)c);
    h.w.resize((size_t)c);
    above.resize((size_t)c);
    return NC_OK;
}

int build_net(int32_t n, const float* xyz, int64_t n_syn, const int32_t* from, const int32_t* to,
              const float* weight, const float* length, const uint8_t* inhibitory, const nc_params& p,
              NetHost& h, std::string& err, bool rows_only)
{
    if (p.inhibitory_rule != NC_INHIBITORY_COPY_LOSS && p.inhibitory_rule != NC_INHIBITORY_SIGN) {
        err = "unknown inhibitory rule";
        return NC_ERR_INVALID;
    }
    if (n < 0 || n_syn < 0) { err = "negative size"; return NC_ERR_INVALID; }
    if (n >= (1 << 30)) { err = "too many neurons"; return NC_ERR_INVALID; }
    if (n_syn > 0 && (!from || !to || !weight)) { err = "null synapse array"; return NC_ERR_INVALID; }
    if (n_syn > 0 && !length && !xyz) { err = "need synapse lengths or neuron positions"; return NC_ERR_INVALID; }
    if (!(p.run_speed > 0.0f) || !std::isfinite(p.run_speed)) { err = "run_speed must be > 0"; return NC_ERR_INVALID; }
    if (!(p.presynaptic_trace_decay > 0.0f && p.presynaptic_trace_decay < 1.0f) ||
        !(p.postsynaptic_trace_decay > 0.0f && p.postsynaptic_trace_decay < 1.0f)) {
        err = "trace decays must lie in (0, 1)";
        return NC_ERR_INVALID;
    }
    bool by_source = true, negative = false;
    for (int64_t k = 0; k < n_syn; ++k) {
        by_source = by_source && (k == 0 || from[k - 1] <= from[k]);
        negative = negative || weight[k] < 0.0f;
        if (from[k] < 0 || from[k] >= n || to[k] < 0 || to[k] >= n) { err = "synapse endpoint out of range"; return NC_ERR_INVALID; }
        if (std::isnan(weight[k])) { err = "NaN weight"; return NC_ERR_INVALID; }
    }

    h = NetHost();
    h.n = n;
    h.n_input = n_syn;
    h.p = p;
    h.dt = p.run_speed;
    h.kc = 1;
    while (!(2.0f < step_ms(h.kc, h.dt))) h.kc++;
    {
        const int period = (int)(600.0f / h.dt);  // std::max(1, static_cast<int>(600.0f / runSpeed))
        h.bg_period = p.background_firing ? std::max(1, period) : 0;
    }
    h.leak = powf(0.5f, h.dt);                          // powf(recharge, deltaT)
    h.c52 = (float)((double)0.2f * 52.0);               // AP_depolFac = 0.2f; AP_depolFac *= 52.0
    h.e_term = exp(0.3702 * (double)h.dt);              // exp(0.3702*deltaT)
    h.xyz.assign(3 * (size_t)n, 0.0f);
    if (xyz) std::memcpy(h.xyz.data(), xyz, sizeof(float) * 3 * (size_t)n);
    if (p.storage_order != NC_ORDER_SPATIAL && p.storage_order != NC_ORDER_ID) {
        err = "unknown storage order";
        return NC_ERR_INVALID;
    }
    if (p.step_mode != NC_STEP_DENSE && p.step_mode != NC_STEP_EVENT && p.step_mode != NC_STEP_AUTO) {
        err = "unknown step mode";
        return NC_ERR_INVALID;
    }
    storage_order(h, xyz, p.storage_order);

    std::vector<int64_t> start((size_t)n + 1, 0), row_end((size_t)n, 0);
    for (int64_t k = 0; k < n_syn; ++k) start[(size_t)h.slot_of[(size_t)to[k]] + 1]++;
    for (int32_t j = 0; j < n; ++j) start[(size_t)j + 1] += start[(size_t)j];
    h.input_to_csc.assign((size_t)n_syn, -1);
    h.in_ptr.assign((size_t)n + 1, 0);
    std::vector<uint32_t> above;
    int rc = NC_OK;
    if (n_syn < (1ll << 32)) {
        auto order = rows_of_targets<uint32_t>(h, n_syn, from, to, by_source, start);
        rc = fill_rows(h, order.get(), start, from, weight, length, above, row_end, err);
    } else {
        auto order = rows_of_targets<int64_t>(h, n_syn, from, to, by_source, start);
        rc = fill_rows(h, order.get(), start, from, weight, length, above, row_end, err);
    }
    if (rc != NC_OK) return rc;
    if (h.s >= (1ll << 31) || h.sp >= (1ll << 32)) { err = "too many synapses in one network"; return NC_ERR_INVALID; }

    // ring words per target: one bit per in-synapse
    h.ring_off.assign((size_t)n + 1, 0);
    for (int32_t j = 0; j < n; ++j) {
        const int64_t fan = row_end[(size_t)j] - h.in_ptr[j];
        const int64_t words = (fan + 31) / 32;
        if ((int64_t)h.ring_off[j] + words >= (1ll << 27)) { err = "network too large for one ring slot"; return NC_ERR_INVALID; }
        h.ring_off[j + 1] = h.ring_off[j] + (int32_t)words;
    }
    h.ring_words = h.ring_off[n];
    h.ring_slots = 1;
    while (h.ring_slots < h.max_delay + h.kc + 1) h.ring_slots <<= 1;

    // tables: presynaptic trace, postsynaptic trace, AP shape
    h.tables.clear();
    if (!trace_table(p.presynaptic_trace_decay, h.dt, h.tables, h.tab_pre_len) ||
        !trace_table(p.postsynaptic_trace_decay, h.dt, h.tables, h.tab_post_len)) {
        err = "trace table does not underflow";
        return NC_ERR_INVALID;
    }
    h.ap_len = h.kc;
    for (int32_t k = 0; k < h.kc; ++k) h.tables.push_back(ap_value(step_ms(k, h.dt)));

    choose_key(h);
    const bool dense = p.step_mode != NC_STEP_EVENT;
    if (dense) {
        h.key.resize((size_t)(h.sp * key_words(h)));
        h.qrow.resize((size_t)(h.sp / 4));
        for (int64_t c = 0; c < h.sp; ++c)
            h.key[(size_t)c] = (uint32_t)h.csc_pre[(size_t)c] << h.key_shift | (h.wide ? 0u : above[(size_t)c]);
        if (h.wide) std::copy(above.begin(), above.end(), h.key.begin() + (size_t)h.sp);
        for (int32_t j = 0; j < n; ++j)
            for (int64_t q = h.in_ptr[j] / 4; q < h.in_ptr[j + 1] / 4; ++q) h.qrow[(size_t)q] = (uint8_t)(j & 31);
    }

    // Synapse::inhibitory: setWeight's sign (src/NeuCor.cpp:576-579), lost by synapses
    // the vector growth copied (rule COPY_LOSS), or the caller's own flags
    h.inh_bits.assign((size_t)((h.sp + 31) / 32), 0u);
    if (negative) {
        // each source's synapses in creation order (Neuron::outSynapses)
        std::vector<int64_t> size((size_t)n, 0), made((size_t)n, 0);
        for (int64_t k = 0; k < n_syn; ++k) size[(size_t)from[k]] += h.input_to_csc[(size_t)k] >= 0 ? 1 : 0;
        for (int64_t k = 0; k < n_syn; ++k) {
            const int64_t c = h.input_to_csc[(size_t)k];
            if (c < 0) continue;
            const int64_t m = made[(size_t)from[k]]++;
            if (!(weight[k] < 0.0f)) continue;
            if (p.inhibitory_rule == NC_INHIBITORY_COPY_LOSS && grown_copy(m, size[(size_t)from[k]])) continue;
            h.inh_bits[(size_t)(c >> 5)] |= 1u << (c & 31);
        }
    }
    if (inhibitory) {
        for (int64_t k = 0; k < n_syn; ++k) {
            const int64_t c = h.input_to_csc[(size_t)k];
            if (c < 0) continue;
            if (inhibitory[k]) h.inh_bits[(size_t)(c >> 5)] |= 1u << (c & 31);
            else h.inh_bits[(size_t)(c >> 5)] &= ~(1u << (c & 31));
        }
    }

    // CSR: each source's out-synapses in creation order
    const bool event = p.step_mode != NC_STEP_DENSE;
    if (event || !rows_only) {
        h.csc_delay.resize((size_t)h.sp);
        for (int64_t c = 0; c < h.sp; ++c) h.csc_delay[(size_t)c] = (int32_t)(above[(size_t)c] >> NC_KEY_DELAY_SHIFT);
        h.out_ptr.assign((size_t)n + 1, 0);
        for (int32_t j = 0; j < n; ++j)
            for (int64_t c = h.in_ptr[j]; c < row_end[(size_t)j]; ++c) h.out_ptr[(size_t)h.csc_pre[c] + 1]++;
        for (int32_t i = 0; i < n; ++i) h.out_ptr[i + 1] += h.out_ptr[i];
        h.out_post.assign((size_t)h.s, 0);
        h.out_csc.assign((size_t)h.s, 0);
        h.out_delay.assign((size_t)h.s, 0);
        if (event) h.out_ringpos.assign((size_t)h.s, 0);
        std::vector<int64_t> fill(h.out_ptr.begin(), h.out_ptr.end() - 1);
        for (int64_t k = 0; k < n_syn; ++k) {
            const int64_t c = h.input_to_csc[(size_t)k];
            if (c < 0) continue;
            const int32_t i = h.csc_pre[(size_t)c], j = h.slot_of[(size_t)to[k]];
            const int64_t q = fill[i]++;
            const int64_t b = c - h.in_ptr[j];
            h.out_post[(size_t)q] = j;
            h.out_csc[(size_t)q] = (int32_t)(uint32_t)c;
            const uint32_t flags = (to[k] > from[k] ? 1u << kAfterBit : 0u) | (to[k] < from[k] ? 1u << kBeforeBit : 0u);
            h.out_delay[(size_t)q] = (int16_t)(uint16_t)((uint32_t)h.csc_delay[(size_t)c] | flags);
            if (!event) continue;
            h.out_ringpos[(size_t)q] = ((uint32_t)(h.ring_off[j] + (int32_t)(b >> 5)) << 5) | (uint32_t)(b & 31);
        }
    }

    // Every term a launch can add is >= 0 when no synapse is inhibitory and no weight is
    // negative: plasticity keeps an excitatory weight in [0, 1] (src/NeuCor.cpp:757-761)
    // and no call changes a weight after creation.
    h.nonneg_terms = true;
    for (uint32_t b : h.inh_bits) h.nonneg_terms = h.nonneg_terms && b == 0u;
    for (float x : h.w) h.nonneg_terms = h.nonneg_terms && x >= 0.0f;

    if (dense) {
        for (size_t w = 0; w < h.inh_bits.size(); ++w)
            for (uint32_t m = h.inh_bits[w]; m; m &= m - 1u) {
                int b = 0;
                while (!((m >> b) & 1u)) ++b;
                h.key[(h.wide ? (size_t)h.sp : 0) + 32 * w + (size_t)b] |= NC_KEY_INH;
            }
    }
    return NC_OK;
}

void choose_key(NetHost& h)
{
    auto bits = [](uint32_t v) {
        int32_t b = 0;
        while (b < 32 && v >> b) ++b;
        return b;
    };
    // one word per synapse holds slot, flags and delay, and one the last two arrivals, unless
    // the delay needs more bits than the slot leaves or an age that still matters (a trace
    // not yet underflowed, the fold window) could pass NC_AGE_OLD
    const int32_t slot_bits = std::max(1, bits((uint32_t)pad_slot(h.n)));
    h.wide = slot_bits + NC_KEY_DELAY_SHIFT + bits((uint32_t)h.max_delay) > 32 || h.tab_pre_len > NC_AGE_OLD ||
             h.kc + 1 > NC_AGE_OLD;
    h.key_shift = h.wide ? 0 : 32 - slot_bits;
}

std::vector<NcOut> out_records(const NetHost& h)
{
    std::vector<NcOut> out((size_t)h.s);
    for (size_t q = 0; q < out.size(); ++q)
        out[q] = NcOut{(uint32_t)h.out_csc[q], h.out_post[q], h.out_ringpos[q], (uint16_t)h.out_delay[q]};
    return out;
}

void plan_rows(const std::vector<RowNet>& nets, int blocks, std::vector<NcRowTile>& tiles,
               std::vector<int32_t>& start)
{
    // a run of 8 neurons weighs its quads and a little for the neurons themselves
    constexpr int64_t kNeuronWeight = 2;
    int64_t total = 0, done = 0;
    for (const RowNet& r : nets) total += r.h->sp / 4 + kNeuronWeight * r.h->n;
    tiles.clear();
    start.assign(1, 0);
    int32_t splits = 0;
    for (const RowNet& r : nets) {
        const NetHost& h = *r.h;
        bool open = false;  // the last tile may grow
        auto reach = [&](int64_t block) {
            while ((int64_t)start.size() <= block) {
                start.push_back((int32_t)tiles.size());
                open = false;
            }
        };
        for (int32_t f = 0; f < h.n; f += 8) {
            const int32_t count = std::min(h.n - f, 8);
            const int64_t a = h.in_ptr[(size_t)f] / 4, quads = h.in_ptr[(size_t)(f + count)] / 4 - a;
            const int64_t weight = quads + kNeuronWeight * count;
            const NcRowTile run{(uint32_t)(r.syn_base / 4 + a), (int32_t)quads, r.net, f, r.neuron_base + f,
                                r.ptr_base + f, count, 0};
            const int64_t first = std::min<int64_t>(blocks - 1, (int64_t)((double)done * blocks / total));
            // a run of several shares (rows of many in-synapses) is split over as many blocks, from the
            // one it begins in: where one row is most of it, over all that it reaches into (there are
            // few such runs); where its rows are even, so that no two runs' parts fall to one block
            int64_t parts = 1;
            if (quads > kSplitQuads) {
                int64_t longest = 0;
                for (int32_t j = f; j < f + count; ++j)
                    longest = std::max(longest, h.in_ptr[(size_t)j + 1] / 4 - h.in_ptr[(size_t)j] / 4);
                if (2 * longest > quads && weight * blocks > 2 * total) parts = (weight * blocks + total - 1) / total;
                else if (quads > kSplitEvenQuads) parts = (4 * weight * blocks + total) / (4 * total);
                parts = std::min<int64_t>({parts, quads / kPartQuads, blocks - first});
            }
            if (parts > 1) {
                ++splits;
                int64_t from = 0;
                for (int64_t p = 0; p < parts; ++p) {
                    reach(first + p);
                    // (parts begin on a 128-byte line of the streams)
                    const int64_t to = p + 1 == parts ? quads : quads * (p + 1) / parts / 8 * 8;
                    NcRowTile t = run;
                    t.q0 += (uint32_t)from;
                    t.nq = (int32_t)(to - from);
                    t.part = (int32_t)(parts << 16) | splits;
                    tiles.push_back(t);
                    from = to;
                }
                open = false;
                done += weight;
                continue;
            }
            // the block its middle falls to
            reach(std::min<int64_t>(blocks - 1, (int64_t)((done + 0.5 * weight) * blocks / total)));
            done += weight;
            if (open && tiles.back().count + count <= NC_TILE_ROWS) {
                tiles.back().nq += run.nq;
                tiles.back().count += count;
            } else {
                tiles.push_back(run);
                open = true;
            }
        }
    }
    while ((int)start.size() <= blocks) start.push_back((int32_t)tiles.size());
}

bool has_parts(const std::vector<NcRowTile>& tiles)
{
    return std::any_of(tiles.begin(), tiles.end(), [](const NcRowTile& t) { return t.part != 0; });
}

int set_groups(NetHost& h, int32_t n_groups, const nc_group* groups, std::string& err)
{
    if (n_groups < 0 || (n_groups > 0 && !groups)) { err = "bad group array"; return NC_ERR_INVALID; }
    std::vector<NcGroupDev> out;
    for (int32_t g = 0; g < n_groups; ++g) {
        const nc_group& G = groups[g];
        if (G.first < 0 || G.count < 0 || G.jitter < 0 || G.jitter > 1000 || (int64_t)G.first + G.count > h.n ||
            !(G.rate_hz >= 0.0f)) {
            err = "input group out of range";
            return NC_ERR_INVALID;
        }
        out.push_back(NcGroupDev{G.first, G.count, rate_threshold(G.rate_hz, h.dt), G.correlated ? 1 : 0,
                                 G.jitter, g});
    }
    h.groups = out;
    return NC_OK;
}

}  // namespace nc

// ------------------------------------------------------------------ C ABI
extern "C" int nc_philox4x32_10(const uint32_t ctr[4], const uint32_t key[2], uint32_t out[4])
{
    if (!ctr || !key || !out) return NC_ERR_INVALID;
    nc_philox(ctr[0], ctr[1], ctr[2], ctr[3], key[0], key[1], out);
    return NC_OK;
}

namespace nc {

int build_knn(int32_t n, int32_t k, float density, uint64_t seed, int32_t threads, float* xyz, int32_t* syn_from,
              int32_t* syn_to, float* syn_weight)
{
    if (n < 0 || k < 0 || !(density > 0.0f) || !xyz || ((int64_t)n * k > 0 && (!syn_from || !syn_to || !syn_weight)))
        return NC_ERR_INVALID;
    if (n > 0 && k >= n) return NC_ERR_INVALID;
    const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
    const KnnGrid grid = knn_grid(n, k, density);
    const float side = grid.side;
    for (int32_t i = 0; i < n; ++i) {
        uint32_t o[4];
        nc_philox((uint32_t)i, 0u, kStreamPosition, 0u, k0, k1, o);
        xyz[3 * (size_t)i + 0] = unit24(o[0]) * side;
        xyz[3 * (size_t)i + 1] = unit24(o[1]) * side;
        xyz[3 * (size_t)i + 2] = unit24(o[2]) * side;
    }
    if (k == 0 || n == 0) return NC_OK;
    const int32_t g = grid.g;
    const float h = grid.h;
    auto cell_of = [&](float v) { return std::min(g - 1, std::max(0, (int32_t)(v / h))); };
    std::vector<int32_t> cstart((size_t)g * g * g + 1, 0), cell((size_t)n);
    for (int32_t i = 0; i < n; ++i) {
        const int32_t c = (cell_of(xyz[3 * (size_t)i]) * g + cell_of(xyz[3 * (size_t)i + 1])) * g +
                          cell_of(xyz[3 * (size_t)i + 2]);
        cell[i] = c;
        cstart[(size_t)c + 1]++;
    }
    for (size_t c = 0; c + 1 < cstart.size(); ++c) cstart[c + 1] += cstart[c];
    // the points by cell, with their positions: a run of cells along z is a run of memory
    struct Point {
        float p[3];
        int32_t id;
    };
    std::vector<Point> points((size_t)n);
    {
        std::vector<int32_t> fill(cstart.begin(), cstart.end() - 1);
        for (int32_t i = 0; i < n; ++i) {
            const float* p = &xyz[3 * (size_t)i];
            points[(size_t)fill[(size_t)cell[(size_t)i]]++] = Point{{p[0], p[1], p[2]}, i};
        }
    }
    // Shells of cells of growing Chebyshev radius r.  Once k candidates are known, only points
    // up to the k-th distance so far (`far`) can be among the k nearest.  A candidate is its
    // distance's bits, which order as the distance does, above its id.
    auto worker = [&](int32_t lo, int32_t hi) {
        std::vector<uint64_t> cand;
        for (int32_t i = lo; i < hi; ++i) {
            const float* pi = &xyz[3 * (size_t)i];
            const int32_t cx = cell_of(pi[0]), cy = cell_of(pi[1]), cz = cell_of(pi[2]);
            cand.clear();
            float far2 = INFINITY;  // no less than the square of any distance up to `far`
            auto visit = [&](int32_t x, int32_t y, int32_t z0, int32_t z1) {
                const size_t row = ((size_t)x * g + y) * g;
                for (int32_t q = cstart[row + z0], e = cstart[row + z1 + 1]; q < e; ++q) {
                    const Point& pt = points[(size_t)q];
                    const float dx = pi[0] - pt.p[0], dy = pi[1] - pt.p[1], dz = pi[2] - pt.p[2];
                    if (dx * dx + dy * dy + dz * dz > far2 || pt.id == i) continue;
                    const float d = get_dist(pi, pt.p);
                    uint32_t bits;
                    std::memcpy(&bits, &d, sizeof(bits));
                    cand.push_back((uint64_t)bits << 32 | (uint32_t)pt.id);
                }
            };
            for (int32_t r = 0;; ++r) {
                const int32_t z0 = std::max(0, cz - r), z1 = std::min(g - 1, cz + r);
                for (int32_t x = std::max(0, cx - r); x <= std::min(g - 1, cx + r); ++x)
                    for (int32_t y = std::max(0, cy - r); y <= std::min(g - 1, cy + r); ++y) {
                        if (std::max(std::abs(x - cx), std::abs(y - cy)) == r) {
                            visit(x, y, z0, z1);
                            continue;
                        }
                        if (cz - r >= 0) visit(x, y, cz - r, cz - r);
                        if (cz + r < g) visit(x, y, cz + r, cz + r);
                    }
                const bool all = r >= g;
                if ((int32_t)cand.size() >= k) {
                    // every unvisited point is at least r*h away
                    std::nth_element(cand.begin(), cand.begin() + (k - 1), cand.end());
                    const uint32_t bits = (uint32_t)(cand[(size_t)k - 1] >> 32);
                    float far;
                    std::memcpy(&far, &bits, sizeof(far));
                    if (all || far < (float)r * h) break;
                    far2 = far * far * (1.0f + 0x1p-20f) + 0x1p-100f;
                    cand.resize((size_t)k);  // those beyond stay beyond
                } else if (all) {
                    break;
                }
            }
            std::sort(cand.begin(), cand.begin() + k);  // the k nearest, by distance and id
            uint32_t o[4] = {0u, 0u, 0u, 0u};
            for (int32_t m = 0; m < k; ++m) {
                const size_t q = (size_t)i * k + m;
                syn_from[q] = i;
                syn_to[q] = (int32_t)(uint32_t)cand[(size_t)m];
                if ((m & 3) == 0) nc_philox((uint32_t)i, (uint32_t)(m >> 2), kStreamWeight, 0u, k0, k1, o);
                syn_weight[q] = unit24(o[m & 3]);
            }
        }
    };
    // chunks of points, taken in turn (a chunk is some milliseconds' worth at most)
    constexpr int32_t kChunk = 128;
    threads = std::max(1, std::min(std::min(threads, 64), (n + kChunk - 1) / kChunk));
    std::atomic<int32_t> next{0};
    auto chunks = [&] {
        for (int64_t lo = (int64_t)kChunk * next++; lo < n; lo = (int64_t)kChunk * next++)
            worker((int32_t)lo, (int32_t)std::min<int64_t>(n, lo + kChunk));
    };
    std::vector<std::thread> pool;
    for (int32_t t = 1; t < threads; ++t) pool.emplace_back(chunks);
    chunks();
    for (auto& th : pool) th.join();
    return NC_OK;
}

}  // namespace nc

extern "C" int nc_build_knn(int32_t n, int32_t k, float density, uint64_t seed, float* xyz, int32_t* syn_from,
                            int32_t* syn_to, float* syn_weight)
{
    return nc::build_knn(n, k, density, seed, (int32_t)std::max(1u, std::thread::hardware_concurrency()), xyz, syn_from,
                         syn_to, syn_weight);
}

namespace {
float randomUnit() { return static_cast<float>(rand()) / static_cast<float>(RAND_MAX); }
}  // namespace

extern "C" int nc_reference_positions(int32_t n, float* xyz)
{
    if (n < 0 || (n > 0 && !xyz)) return NC_ERR_INVALID;
    // createNeuron with NaN positions while totalGenNeurons = n (src/NeuCor.cpp:154-170)
    float spawnSize = 2.0f;
    if (n != 0) spawnSize = powf((float)((unsigned)n / (1.3333 * 3.1459 * 8)), (float)0.33333) * 2.0;
    for (int32_t i = 0; i < n; ++i) {
        float x, y, z;
        do {
            x = (randomUnit() - 0.5f) * spawnSize;
            y = (randomUnit() - 0.5f) * spawnSize;
            z = (randomUnit() - 0.5f) * spawnSize;
        } while ((double)x * x + (double)y * y + (double)z * z > (spawnSize / 2.0) * (spawnSize / 2.0));
        xyz[3 * (size_t)i] = x;
        xyz[3 * (size_t)i + 1] = y;
        xyz[3 * (size_t)i + 2] = z;
    }
    return NC_OK;
}

extern "C" int nc_reference_connection_count(int32_t n, const float* xyz, int64_t* n_synapses)
{
    if (n < 0 || !n_synapses || (n > 0 && !xyz)) return NC_ERR_INVALID;
    int64_t s = 0;
    for (int32_t i = 0; i < n; ++i)
        for (int32_t j = 0; j < n; ++j)
            if (nc::get_dist(&xyz[3 * (size_t)i], &xyz[3 * (size_t)j]) < 1.0 && j != i) ++s;
    *n_synapses = s;
    return NC_OK;
}

extern "C" int nc_reference_connections(int32_t n, const float* xyz, int32_t* syn_from, int32_t* syn_to,
                                        float* syn_weight, int64_t capacity)
{
    if (n < 0 || (n > 0 && !xyz)) return NC_ERR_INVALID;
    int64_t s = 0;
    // Neuron::makeConnections for every neuron in order (src/NeuCor.cpp:418-444); each new
    // Synapse draws its weight (src/NeuCor.cpp:471-473)
    for (int32_t i = 0; i < n; ++i) {
        for (int32_t j = 0; j < n; ++j) {
            const float distance = nc::get_dist(&xyz[3 * (size_t)i], &xyz[3 * (size_t)j]);
            if (!(distance < 1.0 && j != i)) continue;
            if (s >= capacity || !syn_from || !syn_to || !syn_weight) return NC_ERR_INVALID;
            float weight = randomUnit() * 0.8f + 0.2f;
            if (randomUnit() < 0.2f) weight = -weight;
            syn_from[s] = i;
            syn_to[s] = j;
            syn_weight[s] = weight;
            ++s;
        }
    }
    return NC_OK;
}
