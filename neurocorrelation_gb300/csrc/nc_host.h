// nc_host.h — host-side network description (built once, uploaded to the GPU).
#pragma once
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/neucor_gb300.h"
#include "nc_engine.cuh"

namespace nc {

// One network laid out for the step kernels (see nc_engine.cuh), all indices
// relative to the network.
struct NetHost {
    int32_t n = 0;
    int64_t s = 0;        // synapses kept
    int64_t sp = 0;       // in-synapse (CSC) positions: s and the padding of the rows to quads
    int64_t n_input = 0;  // synapses given
    nc_params p{};
    float dt = 1.0f;
    int32_t kc = 3;
    int32_t ring_slots = 1;
    int32_t ring_words = 0;
    int32_t bg_period = 0;
    int32_t max_delay = 1;
    float leak = 0.5f, c52 = 0.0f;
    double e_term = 0.0;
    std::vector<float> xyz;                 // caller's id order
    std::vector<int32_t> orig_id;           // device slot -> caller's id
    std::vector<int32_t> slot_of;           // caller's id -> device slot
    bool permuted = false;
    // Below, neurons are device slots.  The in-synapses of a target are sorted by the
    // caller's source id, each row padded to a multiple of 4 positions; out_delay packs the delay (bits 0-13) and whether the target's
    // caller id is above (bit 14) or below (bit 15) the source's.
    std::vector<int64_t> in_ptr, out_ptr;   // n+1
    std::vector<int32_t> ring_off;          // n+1
    std::vector<float> w;                   // CSC
    std::vector<uint32_t> inh_bits;         // CSC, bit per synapse: Synapse::inhibitory
    std::vector<int32_t> csc_pre, csc_delay;
    // dense form: key of every in-synapse (NcPools::key; when wide, of sp slots and then
    // of sp flags and delays), row of every quad
    std::vector<uint32_t> key;
    std::vector<uint8_t> qrow;
    int32_t key_shift = 0;
    bool wide = false;
    std::vector<int32_t> out_post, out_csc; // out_csc: below 2^32, read as unsigned
    std::vector<int16_t> out_delay;
    std::vector<uint32_t> out_ringpos;
    std::vector<int64_t> input_to_csc;      // -1 for ignored duplicates
    std::vector<float> tables;              // pre trace | post trace | AP shape
    int32_t tab_pre_len = 0, tab_post_len = 0, ap_len = 0;
    std::vector<NcGroupDev> groups;
    bool nonneg_terms = true;               // no inhibitory synapse and no negative weight
};

// Source slot of a padding position: past the net's last slot, in the spare word of its
// fired bits (nothing ever sets it).
inline int32_t pad_slot(int32_t n) { return (n + 31) / 32 * 32; }
// Rows end at a multiple of 4 positions, and every eighth at one of 32: tiles start at
// multiples of 8 neurons, so a warp's 16-byte accesses start on a 128-byte line.
inline int64_t row_align(int32_t j) { return (j & 7) == 7 ? 32 : 4; }
// Chooses key_shift and wide from the net's size, longest delay and tables.
void choose_key(NetHost& h);
// Whether the dense form's arrays hold whole step counters and a second range of keys
// (NcPools::key); the words they take per position.
inline int64_t key_words(const NetHost& h) { return h.wide ? 2 : 1; }
// 0.9943*exp(0.3702*dt) as a float and the float of what it leaves.
inline void term_pair(const NetHost& h, float& hi, float& lo)
{
    const double k = 0.9943 * h.e_term;
    hi = (float)k;
    lo = (float)(k - (double)hi);
}
// Initial state word (never launched) of the net's positions.
inline uint32_t initial_state(const NetHost& h) { return h.wide ? (uint32_t)NC_WIDE_NEVER : nc_state_never(); }
// A run of up to 1,536 quads, 24 rounds of a block's threads, is as fast whole: with a row of
// 1,999 in-synapses 8.4 us a step whole and 15.0 split, of 3,999 12.9 and 14.7, of 7,999 20.4 and
// 14.0.  So is one of up to 2,560 in rows of much the same length (every neuron of 1,000 driving
// every other, inhibitory, quiet 28.9 and 30.7, of 1,500 50.6 and 38.9).
constexpr int64_t kSplitQuads = 1536, kSplitEvenQuads = 2560;
constexpr int64_t kPartQuads = 256;   // of a part, at least
// The row tiles of an engine's nets, and the first tile of each of `blocks` blocks (blocks
// + 1 entries): consecutive runs of neurons with an even share of the quads each, cut at
// multiples of 8 neurons and into tiles of at most NC_TILE_ROWS; 8 neurons with many more quads
// than a share (and kSplitQuads) are split over several blocks (NcRowTile::part).  At most two
// tiles a block more than the nets' own.
struct RowNet {              // a net and its pool indexes
    const NetHost* h;
    int32_t net;
    int64_t syn_base;
    int32_t neuron_base, ptr_base;
};
void plan_rows(const std::vector<RowNet>& nets, int blocks, std::vector<NcRowTile>& tiles,
               std::vector<int32_t>& start);
bool has_parts(const std::vector<NcRowTile>& tiles);
// The net's out-synapse records (event form).
std::vector<NcOut> out_records(const NetHost& h);
// Builds the layout; returns NC_OK or an NC_ERR_* code with `err` set.  rows_only: without the
// out-synapses (csc_delay, out_*) where the form of the step does not need them.
int build_net(int32_t n, const float* xyz, int64_t n_syn, const int32_t* from, const int32_t* to,
              const float* weight, const float* length, const uint8_t* inhibitory, const nc_params& p,
              NetHost& out, std::string& err, bool rows_only = false);
bool inhibitory_flag(const NetHost& h, int64_t csc);
int set_groups(NetHost& net, int32_t n_groups, const nc_group* groups, std::string& err);

// Reference arithmetic helpers shared by build and read-back.
float get_dist(const float* a, const float* b);      // coord3::getDist, src/NeuCor.h:16-18
int32_t delay_steps(float length, float dt);          // -1 when it does not fit int16
constexpr int32_t kMaxDelay = (1 << 14) - 1;          // delay bits of out_delay
constexpr int kAfterBit = 14, kBeforeBit = 15;
// Scatters a device-slot-ordered array into the caller's id order.
template <class T>
void to_caller_order(const NetHost& h, const T* slots, T* out)
{
    for (int32_t i = 0; i < h.n; ++i) out[i] = slots[h.slot_of[(size_t)i]];
}
uint32_t rate_threshold(float rate_hz, float dt);

// kNN networks (nc_build_knn, and its device counterpart in nc_build.cu): positions
// uniform in a cube of side (n/density)^(1/3) from Philox stream kStreamPosition,
// weights from kStreamWeight, neighbours searched over a uniform grid of g^3 cells.
constexpr uint32_t kStreamPosition = 10u;
constexpr uint32_t kStreamWeight = 11u;
NC_HD inline float unit24(uint32_t r) { return (float)(r >> 8) * 0x1p-24f; }
struct KnnGrid {
    float side;
    int32_t g;
    float h;
};
KnnGrid knn_grid(int32_t n, int32_t k, float density);
// nc_build_knn on `threads` threads.
int build_knn(int32_t n, int32_t k, float density, uint64_t seed, int32_t threads, float* xyz, int32_t* syn_from,
              int32_t* syn_to, float* syn_weight);
float ap_value(float x);                              // Neuron::AP, src/NeuCor.cpp:706-714
float step_ms(int64_t k, float dt);                   // k steps as a float time difference

}  // namespace nc
