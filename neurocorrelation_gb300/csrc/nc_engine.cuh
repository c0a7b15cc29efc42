// nc_engine.cuh — data layout shared by the step kernels and the host engine.
//
// One engine advances one or more independent networks ("nets") packed into
// pooled device arrays.  A single network (nc_create) is an engine with one net;
// the batched and served forms pack many.  Every net keeps its own step counter,
// constants, input groups and draw key, and no array is shared between nets, so a
// net computes the same bits alone or packed with others.
//
// Per net, in HBM:
//   neurons   pot, lf (last fire step), firings, act_start     SoA, pool-indexed
//   in_ptr    CSC row starts (n+1): in-synapses of target j, ascending source id
//             — the order of the reference's std::map inSynapses (src/NeuCor.h:212).
//             Every row is padded to a multiple of 4 positions (a quad) with synapses
//             that no source drives, so a quad belongs to one target and one thread
//             moves it with 16-byte accesses.
//   w, x      per in-synapse (CSC order): weight, and deltaT*AP_depolFac of the last
//             accepted launch (the contribution term is formed from it when summed)
//   dense form   key, state per in-synapse, qrow per quad (see NcPools)
//   event form   t_arr (last arrival step) and inh (one bit: Synapse::inhibitory) per
//                in-synapse; out_ptr CSR row starts (n+1) and per out-synapse (CSR
//                order) an NcOut and the last accepted arrival step
//   Neurons sit in device slots (Morton order of positions by default); every rule
//   that depends on ids uses the caller's ids (orig_id, the order flags, the
//   in-synapse order).
//   ring      R slots x W words: bit b of target j's words in slot a mod R set when
//             the spike on j's b-th in-synapse arrives at step a
//   fired / forced   two parities of one bit per neuron
#pragma once
#include <cstdint>
#include <vector_types.h>

#include <vector>

#ifdef __CUDACC__
#define NC_HD __host__ __device__
#else
#define NC_HD
#endif

#define NC_NEVER INT32_MIN

// Device error codes (NcPools::dev_err).
#define NC_DEV_ERR_FIRER_LOOP 2u     // an input firer's schedule did not advance (capped)
#define NC_DEV_ERR_BARRIER 4u        // a grid barrier of the fused multi-step launch gave up

// Draw streams (third Philox counter word).
#define NC_STREAM_BACKGROUND 1u
#define NC_STREAM_SOURCE 2u
#define NC_STREAM_JITTER 3u
#define NC_STREAM_INDEPENDENT 4u

struct NcGroupDev {
    int32_t first;
    int32_t count;
    uint32_t thresh;     // Bernoulli threshold of the per-step probability, on a 32-bit draw
    int32_t correlated;
    int32_t jitter;
    int32_t index;       // group index within its net (first Philox counter word)
};

// What a step writes comes first, in a cache line of its own: the rest may be read, and stay
// in L1, before a launch's wait for the step before it.
struct alignas(128) NcNetDesc {
    int32_t t;            // step processed by the next launch (>= 1)
    int32_t t_end;        // last step to simulate (inclusive)
    int32_t stdp_done;    // last step whose deferred plasticity has been applied
    float tsum;           // NeuCor::currentTime after t-1 steps: the float sum of t-1 runSpeeds
    int32_t active;       // 0: skipped by the kernels
    int32_t live;         // event form: the last neuron step advanced the net (its fires launch)
    float dt_again;       // dt, for what moves the counters on
    int32_t pad;
    alignas(128) int32_t n; // neurons
    int32_t neuron_base;  // pool index of neuron 0
    int32_t ptr_base;     // pool index of in_ptr/out_ptr/ring_off entry 0 (n+1 entries)
    int32_t word_base;    // pool index of this net's first bitset word
    int32_t n_words;      // ceil(n/32)
    int64_t syn_base;     // pool index of synapse 0 (CSC and CSR arrays; a multiple of 32)
    int64_t ring_base;    // pool word index of ring slot 0
    int32_t ring_words;   // words per slot
    int32_t ring_mask;    // slots - 1
    int32_t kc;           // smallest k >= 1 with 2.0f < k*dt (AP_cutoff, src/NeuCor.cpp:385)
    int32_t bg_period;    // max(1, int(600/dt)); 0 = background off
    uint32_t key0, key1;  // Philox key
    int32_t table_base;   // pool index of the trace tables
    int32_t tab_pre_len;  // presynaptic trace table length
    int32_t tab_post_len; // postsynaptic trace table length
    int32_t ap_base;      // pool index of the AP shape table (kc entries)
    int32_t group_base;
    int32_t n_groups;
    int32_t raster_len;   // recorded steps capacity (0 = off)
    int32_t raster_t0;    // first recorded step
    int32_t permuted;     // neurons are stored in a different order than the caller's ids
    float dt;
    float leak;           // powf(0.5f, dt)  (src/NeuCor.cpp:678)
    float c52;            // float(0.2f * 52.0) (src/NeuCor.cpp:729-730)
    float lr, pre_factor, post_factor;
    double e_term;        // 0.9943 is applied separately; this is exp(0.3702*dt) (src/NeuCor.cpp:695)
    float term_hi, term_lo; // both factors as one: a float and the float of what it leaves
    uint32_t* raster;     // device raster rows of n_words words
    unsigned long long* stats; // the net's four counters (NcPools::stats)
    int64_t n_syn;        // synapses (out-synapse entries)
    int64_t wide;         // dense form: 0, or the offset of the second range (NcPools::key)
    int32_t nonneg_terms; // 1: no launch can add a negative term (no inhibitory synapse, no
                          // negative weight), so a neuron's sum only grows within a step
    int32_t group_lo;     // caller ids [group_lo, group_hi) hold every input group's members
    int32_t group_hi;
    int32_t key_shift;    // dense form: first bit of the source's slot in a key
};

// Dense form: how a synapse's last two arrivals are kept.  A launch is accepted only after
// the previous spike has arrived (src/NeuCor.cpp:697, 728), so the last arrival of a
// synapse is its last accepted one once that has arrived and the one before it until
// then.  One 32-bit word holds both: bits 16-31 the accepted arrival step modulo 2^16,
// bits 0-15 its distance from the arrival before.  With prev the step whose spikes are
// being delivered, age = prev - arrival is negative while the spike travels (delays are
// below 2^14).  Ages grow by one a step and every step visits every synapse: every
// NC_AGE_PERIOD steps those past NC_AGE_LIMIT are set back to NC_AGE_OLD, an age at which
// they already count as never launched (free, outside the fold window, trace underflowed
// to zero), so that 16 bits never wrap.
#define NC_AGE_PERIOD 1024
#define NC_AGE_LIMIT 30000
#define NC_AGE_OLD 21808
// The age of a synapse whose state word is s.
NC_HD inline int32_t nc_state_age(uint32_t s, int32_t prev)
{
    return (int32_t)((((uint32_t)prev << 16) | 0xffffu) - s) >> 16;
}
// The state of a synapse whose accepted spike arrives at prev - age, gap steps after the
// arrival before it.
NC_HD inline uint32_t nc_state_word(int32_t prev, int32_t age, int32_t gap)
{
    return ((uint32_t)(prev - age) << 16) | (uint32_t)gap;
}
// Never launched, for a network whose next step is 1.
NC_HD inline uint32_t nc_state_never() { return nc_state_word(0, NC_AGE_OLD, 0); }
// The same for a network that keeps whole step counters (NcNetDesc::wide).
#define NC_WIDE_NEVER (-(1 << 30))

// The smallest id range holding the members of groups g[0..n) (empty when n is 0).
inline void nc_group_range(const NcGroupDev* g, int n, int32_t& lo, int32_t& hi)
{
    lo = 0;
    hi = 0;
    for (int k = 0; k < n; ++k) {
        if (g[k].count <= 0) continue;
        const int32_t a = g[k].first, b = g[k].first + g[k].count;
        if (lo == hi) {
            lo = a;
            hi = b;
        } else {
            lo = a < lo ? a : lo;
            hi = b > hi ? b : hi;
        }
    }
}

struct NcTile {          // event form: 32 consecutive neurons of one net
    int32_t net;
    int32_t first;       // local id of the first neuron (multiple of 32)
};

struct alignas(16) NcRowTile {  // dense form: up to NC_TILE_ROWS consecutive neurons and their rows
    uint32_t q0;         // pool index of the first quad of its rows
    int32_t nq;          // quads
    int32_t net;
    int32_t first;       // local id of the first neuron (a multiple of 8)
    int32_t neuron;      // pool index of the first neuron
    int32_t ptr;         // pool index of its row start
    int32_t count;       // neurons
    int32_t part;        // 0: all quads of its neurons; otherwise one of (part >> 16) tiles of the same
                         // neurons, which count on NcPools::split_ctr[(part & 0xffff) - 1]
};

constexpr int NC_TILE_ROWS = 32;  // neurons of a dense tile at most: one per lane

struct alignas(16) NcOut {  // event form, per out-synapse
    uint32_t csc;        // its in-synapse position, relative to syn_base
    int32_t post;        // target's device slot
    uint32_t ringpos;    // (word within a ring slot) << 5 | bit
    uint32_t delay;      // bits 0-13; bit 14/15: the target's caller id is above/below the source's
};

struct NcFirer {         // periodic input firer (InputFirer, src/NeuCor.cpp:305-345)
    int32_t net;
    float last;          // InputFirer::lastFire, ms
    float rate;          // its entry of the rate array, Hz
    int32_t near_begin;  // neuron slots firer_near[near_begin .. near_end)
    int32_t near_end;
    int32_t first;       // set before the net's first step: the run call at time 0 evaluates it too
};

// Low bits of a key.
#define NC_KEY_AFTER 1u    // the target's caller id is above the source's
#define NC_KEY_BEFORE 2u   // it is below
#define NC_KEY_INH 4u      // Synapse::inhibitory
#define NC_KEY_DELAY_SHIFT 3

struct NcPools {
    // neurons
    float* pot;
    int32_t* lf;
    uint32_t* firings;
    int32_t* act_start;
    int32_t* orig_id;    // device slot -> caller's id (local to the net)
    int32_t* slot_of;    // caller's id -> device slot (local to the net)
    // per-neuron pointers (n+1 per net)
    int64_t* in_ptr;     // absolute CSC index
    int64_t* out_ptr;    // absolute CSR index
    int32_t* ring_off;   // word offset within a slot
    // in-synapses (CSC); every net's synapse base is a multiple of 32
    float* w;
    float* x;            // deltaT*AP_depolFac of the last accepted launch (src/NeuCor.cpp:695, 729-731)
    // out-synapses (CSR)
    NcOut* out;
    int32_t* last_arr;
    uint32_t* inh;       // event form, CSC: Synapse::inhibitory, one bit per synapse
    int32_t* t_arr;      // event form, CSC: last arrival step
    // dense form: in-synapse (CSC) order, one quad of four per thread.
    //   key    NC_KEY_* flags, the delay in steps and, from bit key_shift up, the source's
    //          device slot (a padding position: a slot past the last, whose fired bit is
    //          never set)
    //   state  last accepted arrival and its distance from the one before (nc_state_age)
    // A net whose slots and delays do not fit one word, or whose trace outlasts
    // NC_AGE_OLD steps, takes a second range of both (wide = its offset): key holds the
    // slot alone and key[wide + s] the flags and delay; state the whole arrival step and
    // state[wide + s] the one before it.
    uint32_t* key;
    uint32_t* state;
    float* pst;          // per neuron: its trace at its last step (src/NeuCor.cpp:671-675)
    uint8_t* qrow;       // per quad: low 5 bits of its target's slot
    uint8_t* nib;        // per quad: window bits of tiles too large for shared memory
    NcRowTile* rtiles;   // in the order of the blocks that run them
    int32_t* rstart;     // first tile of each of row_blocks blocks (row_blocks + 1 entries)
    int32_t row_blocks;
    int32_t split;       // dense step: some tiles are split
    uint32_t* split_ctr; // parts of a split tile that are streamed (a counter each, row_blocks of them)
    int32_t stage;       // dense step: captured charges of the sums pass through shared memory (dense_stages)
    // ring and bitsets
    uint32_t* ring;
    uint32_t* fired;     // 2 parities x total_words
    uint32_t* forced;    // 2 parities x total_words
    uint32_t* ufire;     // 2 parities x total_words: input-firer fires (no threshold, no refractory)
    NcFirer* firers;
    int32_t n_firers;
    int32_t* firer_near;
    int64_t total_words;
    // constants
    float* tables;
    NcGroupDev* groups;
    NcNetDesc* nets;
    int32_t n_nets;
    unsigned long long* stats; // 4 counters a net: fires, launched, dropped, steps
    NcTile* tiles;
    int32_t n_tiles;
    int32_t* n_tiles_dev; // when set, the tile count is read from device memory (served engine)
    int32_t* n_nets_dev;  // when set, the nets from *n_nets_dev on are not active (served engine)
    int32_t warp_rows;   // event form: neurons per warp of the neuron step: 8, 16 or 32
    int32_t launch_rows; // and of the spike launch: 1, 2, 4 or 8
    // engine
    uint32_t* done_ctr;  // blocks (event form: warps) that have read the step counters
    uint32_t* dev_err;   // nonzero: a bounded device wait gave up (NC_DEV_ERR_*)
};

// ------------------------------------------------------------------ Philox
// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11).
NC_HD inline void nc_philox(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0,
                                          uint32_t k1, uint32_t out[4])
{
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int r = 0; r < 10; ++r) {
        if (r) {
            k0 += 0x9E3779B9u;
            k1 += 0xBB67AE85u;
        }
#ifdef __CUDA_ARCH__
        const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
#else
        const uint64_t p0 = (uint64_t)0xD2511F53u * c0, p1 = (uint64_t)0xCD9E8D57u * c2;
        const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
        const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
#endif
        const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0;
        c1 = lo1;
        c2 = n2;
        c3 = lo0;
    }
    out[0] = c0;
    out[1] = c1;
    out[2] = c2;
    out[3] = c3;
}

// Kernel launchers (nc_kernels.cu).
namespace nc {
// Resident 256-thread blocks per SM the event form's neuron step is held to: 128 registers
// (at 80 it spills: 100k-neuron step 112 -> 89 us without).
#ifndef NC_NEURON_MIN_BLOCKS
#define NC_NEURON_MIN_BLOCKS 2
#endif
#ifndef NC_DENSE_BLOCK
#define NC_DENSE_BLOCK 96  // threads per block of the dense step: one warp sums, the others stream
#endif
#ifndef NC_EVENT_BLOCK
#define NC_EVENT_BLOCK 64  // threads per block of the event form's neuron step
#endif
#ifndef NC_LAUNCH_MIN_BLOCKS
#define NC_LAUNCH_MIN_BLOCKS 4
#endif
#ifndef NC_LAUNCH_BLOCKS
#define NC_LAUNCH_BLOCKS 16  // 128-thread blocks per SM of the spike launch's grid
#endif

struct LaunchShape {
    int neuron_block;    // threads per block of the neuron update or of the dense step (multiple of 32)
    int launch_blocks;   // blocks of the spike-launch kernel
    int launch_block;    // threads per block of the spike-launch kernel
    int dense_blocks = 0; // dense form: blocks of the step (0: one wave, or one per tile)
    int fused_ticks = 0;  // dense form: steps per fused cooperative launch (0: one launch
                          // per step, replayed through CUDA graphs)
};
// whole: it waits for the kernel before it as a whole.  For the step after a kernel that writes
// what the step reads before its own wait (potentials, last fires, fired bits, or the counters:
// launch_stdp_flush does).
int launch_neuron_step(const NcPools& P, const LaunchShape& L, bool whole, void* stream);
// Blocks of the neuron step that fit on the current device at once; asked before a capture.
int event_resident_blocks(int threads);
// many: the warps have several units each (many_units of the live tiles).
int launch_spike_launch(const NcPools& P, const LaunchShape& L, bool many, void* stream);
bool many_units(int n_tiles, const NcPools& P, const LaunchShape& L);
int launch_stdp_flush(const NcPools& P, const LaunchShape& L, void* stream);
// Dense form (nc_dense.cu): one step in one launch, and the plasticity flush (the launches
// and plasticity of the last step's fires) before read-back.
int launch_step_dense(const NcPools& P, const LaunchShape& L, bool back, void* stream);
// Blocks of `threads` threads of the dense step that fit on the current device at once (0:
// the device cannot run it); called before a stream capture, where it may not be asked.
int dense_resident_blocks(int threads);
bool dense_stages(const std::vector<NcRowTile>& tiles, const std::vector<int32_t>& start, int threads);
// `ticks` whole dense steps of every net in one cooperative launch (no periodic input
// firers); bar: two zero-initialised words of device memory for its grid barrier.
int launch_fused_dense(const NcPools& P, int32_t ticks, const LaunchShape& L, unsigned* bar, void* stream);
// Conversion of net `net`'s per-synapse arrival state between the forms (nc_form.cu),
// after the current form's plasticity flush.  ring_words: the words of the whole ring
// pool (cleared first).
int launch_form_to_event(const NcPools& P, int net, int64_t n_syn, int64_t ring_words, void* stream);
int launch_form_to_dense(const NcPools& P, int net, int64_t n_syn, void* stream);
int launch_flush_dense(const NcPools& P, const LaunchShape& L, void* stream);
// count words of a set to v.
int launch_fill_words(uint32_t* a, int64_t count, uint32_t v, void* stream);
int launch_background_prologue(const NcPools& P, int net, int n_neurons, void* stream);
int launch_force_bits(const NcPools& P, int net, const int32_t* d_ids, int count, void* stream);
// Input firers (nc_inputs.cu), launched before a step's kernels: each firer's schedule
// for the run call that starts at its net's step t; fires land in the ufire bits of
// step t+1 (and, before the first step, those of the time-0 call in step 1's).
int launch_input_firers(const NcPools& P, bool early, void* stream);
// Mean potential of each detector's near neurons (caller ids; near_ptr has count+1 entries).
int launch_detector_voltages(const NcPools& P, int32_t neuron_base, const int32_t* near, const int32_t* near_ptr,
                             int32_t count, float* out, void* stream);
// Read-backs in the caller's order, into device buffers (nc_read.cu): n neurons from
// caller's id `first` on, rows of a raster.
int launch_gather(const float* src, const uint32_t* index, int64_t count, float* out, void* stream);
int launch_potact(const NcPools& P, int32_t neuron_base, int32_t first, int32_t n, int64_t t, float dt, float* out, void* stream);
int launch_last_fire(const NcPools& P, int32_t neuron_base, int32_t first, int32_t n, float dt, float* out, void* stream);
int launch_raster_bytes(const uint32_t* in, uint8_t* out, const int32_t* slot_of, int32_t n, int32_t n_words,
                        int32_t rows, void* stream);
}  // namespace nc
