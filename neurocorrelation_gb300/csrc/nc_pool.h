// nc_pool.h — device engine: packs one or more networks into pooled HBM arrays and
// advances them with the step kernels, replaying captured CUDA graphs.
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "nc_host.h"

namespace nc {

struct NetSlot {       // host view of one packed net
    int32_t n = 0;
    int64_t s = 0;
    int32_t kc = 3;
    float dt = 1.0f;
    int32_t n_words = 0;
    int64_t syn_base = 0;
    int64_t n_input = 0, index_base = 0;  // synapses given, the first one's place in the index
    int32_t neuron_base = 0, ptr_base = 0, word_base = 0, group_cap = 0, group_base = 0;
};

class Engine {
public:
    Engine() = default;
    ~Engine();
    Engine(const Engine&) = delete;
    Engine& operator=(const Engine&) = delete;

    // Packs the nets (all starting at step 1) and uploads them.  group_capacity is
    // the number of input-group entries reserved per net.
    // device_synapses: the in-synapse streams (dense form) are written on the device by
    // the caller (nc_build.cu); only the row starts come from the host description.
    int build(const std::vector<const NetHost*>& nets, int group_capacity, std::string& err,
              const std::vector<int32_t>* horizons = nullptr, bool device_synapses = false);
    void set_launch(const LaunchShape& shape, int ticks_per_graph);
    // Runs `ticks` engine steps (every active net advances one step per tick).
    int step(int64_t ticks, std::string& err);
    // Same, timed with CUDA events on the engine stream.
    int step_timed(int64_t ticks, float* ms, std::string& err);
    // Mean device time of one neuron-update and one spike-launch launch over `ticks`
    // individually timed ticks (these ticks also advance the nets).
    // (dense form: the step kernel, and 0)
    int time_kernels(int ticks, float* neuron_ms, float* launch_ms, std::string& err);
    // (nothing is launched when nothing has been stepped since the last one)
    int flush_plasticity(std::string& err);
    // Steps are launched that this object does not see (nc_run_noalloc's may be replayed).
    void steps_unseen() { unseen_ = true; }
    // Read-backs of a net's neurons and weights in the caller's order (nc_read.cu): gathered
    // into the engine's scratch a part at a time and copied to the host.
    int read_potentials(int net, float* out, std::string& err);
    int read_potact(int net, int64_t t, float* out_2n, std::string& err);
    int read_last_fire(int net, float* out, std::string& err);
    // (needs index(net))
    int read_weights(int net, float* out, std::string& err);
    int read_raster(int net, const uint32_t* d_raster, int32_t rows, uint8_t* out, std::string& err);
    int sync(std::string& err);
    // The CSC position of each of a net's given synapses (~0: not kept) on the device, made with
    // the pools; null when there was no memory for them: the weights are then reordered on the
    // host.  device_synapses: written by the caller.
    uint32_t* index(int net) const { return index_ ? index_ + slots[(size_t)net].index_base : nullptr; }

    int set_groups(int net, const std::vector<NcGroupDev>& groups, std::string& err);
    int set_rates(int net, float lr, float pre_factor, float post_factor, std::string& err);
    int force_fire(int net, const int32_t* ids, int count, std::string& err);
    int set_raster(int net, uint32_t* d_raster, int32_t t0, int32_t len, std::string& err);
    int read_stats(int net, unsigned long long out[4], std::string& err);
    int read_desc(int net, NcNetDesc* out, std::string& err);

    template <class T>
    int download(T* host, const T* dev, size_t count, std::string& err);

    NcPools P{};
    LaunchShape L{};
    std::vector<NetSlot> slots;
    cudaStream_t stream = nullptr;
    int device = 0;
    int graph_ticks = 32;
    bool dense = true;  // the form the next steps run in: NC_STEP_DENSE (nc_dense.cu) or event
    bool both = false;  // NC_STEP_AUTO: the tables of both forms are on the device
    // Switches a single-net engine built with both forms' tables to the other form
    // between steps (flushes the current form's deferred plasticity, converts the
    // per-synapse arrival state, drops the captured graph).
    int set_form(bool to_dense, std::string& err);
    // Launches one tick of the engine's form on `s` (no graph), the input firers' schedule
    // included.
    int launch_tick(cudaStream_t s);
    // Periodic input firers (replaces the set), their state read and written back; the
    // next step's run-call schedule sees every change.
    int set_firers(const std::vector<NcFirer>& firers, const std::vector<int32_t>& near, std::string& err);
    int read_firers(std::vector<NcFirer>& out, std::string& err);
    int write_firers(const std::vector<NcFirer>& in, std::string& err);

private:
    int capture_graph(std::string& err);
    void release_graph();
    template <class T>
    T* alloc(size_t count, std::string& err);
    // Read-back scratch on the device, allocated with the pools: a net's largest read-back,
    // or kScratchMax of it at a time.
    static constexpr size_t kScratchMax = 64 << 20;
    void* scratch_ = nullptr;
    uint32_t* index_ = nullptr;
    bool shared_tables_ = false;  // the GPU uses the host's page tables: it can write ordinary host memory
    size_t scratch_bytes_ = 0;
    bool flushed_ = false, unseen_ = false;
    bool counters_written_ = false;  // by a flush, since the last step that was launched
    std::vector<void*> allocs_;
    char* block_ = nullptr;      // what is left of the last block of small arrays
    size_t block_left_ = 0;
    cudaGraphExec_t graph_ = nullptr;
    void* firers_buf_ = nullptr;
    void* near_buf_ = nullptr;
    int32_t* d_ids_ = nullptr;
    int ids_cap_ = 0;
    bool back_ = false;          // direction of the last dense step's sweep
    unsigned* d_bar_ = nullptr;  // grid barrier of the fused launch (arrivals, generation)
    int64_t ring_words_total_ = 0;
};

// Blocks of `threads` threads that the rows of `neurons` neurons, `quads` in all, are shared out
// to: one wave, or a block for each 8 neurons (more where their rows are long).
int dense_blocks(int64_t neurons, int64_t quads, int threads);
// Neurons per warp of the event form's kernels, for an engine of so many 32-neuron tiles.
void event_rows(int64_t tiles, int sms, NcPools& P);
std::string cuda_msg(const char* what, cudaError_t e);
// Records the calling thread's last error (nc_last_error) and returns `code`.
int set_last_error(int code, const std::string& msg);

}  // namespace nc
