// nc_pool.cu — the device engine (see nc_pool.h).
#include "nc_pool.h"

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <string>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23  // Linux 5.14; older kernels refuse it
#endif

namespace nc {

std::string cuda_msg(const char* what, cudaError_t e)
{
    return std::string(what) + ": " + cudaGetErrorString(e);
}

#define NC_CK(call)                                                  \
    do {                                                             \
        cudaError_t e_ = (call);                                     \
        if (e_ != cudaSuccess) {                                     \
            err = cuda_msg(#call, e_);                               \
            return e_ == cudaErrorMemoryAllocation ? NC_ERR_NOMEM : NC_ERR_CUDA; \
        }                                                            \
    } while (0)

Engine::~Engine()
{
    release_graph();
    if (stream) cudaStreamSynchronize(stream);
    if (firers_buf_) cudaFree(firers_buf_);
    if (near_buf_) cudaFree(near_buf_);
    if (d_ids_) cudaFree(d_ids_);
    for (void* p : allocs_) cudaFree(p);
    if (stream) cudaStreamDestroy(stream);
}

template <class T>
T* Engine::alloc(size_t count, std::string& err)
{
    // Small arrays share blocks: an allocation takes some 40 us and its release as much.  They lie
    // 2 KiB apart: 512 bytes apart, as the allocator packs them, a step's loads meet in few slices
    // of L2 (a step of three neurons 5.1 us, the sphere of 750 6.9, 1k x 50 6.7; 2 KiB apart 5.0,
    // 6.7 and 6.6; 4 to 64 KiB 4.9 to 5.5, 6.7 to 6.9, 6.5 to 6.7).  A block is eight times the array
    // that begins it, and 64 KiB at least: a network of three neurons takes one or two (two of
    // 2 MiB with the arrays 64 KiB apart).
    constexpr size_t kSmallest = 64 << 10, kLargest = 2 << 20, kApart = 2 << 10;
    const size_t bytes = (std::max<size_t>(1, count) * sizeof(T) + kApart - 1) / kApart * kApart;
    const bool shared = bytes <= kLargest / 8;
    if (shared && bytes <= block_left_) {
        void* p = block_;
        block_ += bytes;
        block_left_ -= bytes;
        return (T*)p;
    }
    void* p = nullptr;
    const size_t size = shared ? std::max(kSmallest, 8 * bytes) : std::max<size_t>(1, count) * sizeof(T);
    cudaError_t e = cudaMalloc(&p, size);
    if (e != cudaSuccess) {
        err = cuda_msg("cudaMalloc", e);
        return nullptr;
    }
    allocs_.push_back(p);
    if (shared) {
        block_ = (char*)p + bytes;
        block_left_ = size - bytes;
    }
    e = cudaMemsetAsync(p, 0, size, stream);
    if (e != cudaSuccess) {
        err = cuda_msg("cudaMemsetAsync", e);
        return nullptr;
    }
    return (T*)p;
}

template <class T>
int Engine::download(T* host, const T* dev, size_t count, std::string& err)
{
    if (count == 0) return NC_OK;
    NC_CK(cudaMemcpyAsync(host, dev, count * sizeof(T), cudaMemcpyDeviceToHost, stream));
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

template int Engine::download<float>(float*, const float*, size_t, std::string&);
template int Engine::download<int32_t>(int32_t*, const int32_t*, size_t, std::string&);
template int Engine::download<uint32_t>(uint32_t*, const uint32_t*, size_t, std::string&);
template int Engine::download<int16_t>(int16_t*, const int16_t*, size_t, std::string&);
template int Engine::download<int64_t>(int64_t*, const int64_t*, size_t, std::string&);
template int Engine::download<double>(double*, const double*, size_t, std::string&);

#define NC_ALLOC(ptr, T, count)                  \
    do {                                         \
        ptr = alloc<T>((count), err);            \
        if (!ptr) return NC_ERR_NOMEM;           \
    } while (0)

template <class T>
static cudaError_t upload(T* dev, const std::vector<T>& host, size_t offset, cudaStream_t s)
{
    if (host.empty()) return cudaSuccess;
    return cudaMemcpyAsync(dev + offset, host.data(), host.size() * sizeof(T), cudaMemcpyHostToDevice, s);
}

template <class T>
static cudaError_t upload_part(T* dev, const std::vector<T>& host, int64_t at, int64_t from, int64_t count,
                               cudaStream_t s)
{
    if (count <= 0) return cudaSuccess;
    return cudaMemcpyAsync(dev + at, host.data() + from, (size_t)count * sizeof(T), cudaMemcpyHostToDevice, s);
}

void event_rows(int64_t tiles, int sms, NcPools& P)
{
    // 8k neurons: 26.0 us a step with a warp per 32, 23.8 with one per 8; 50k (1,563 tiles):
    // 15.0 against 27.2
    P.warp_rows = tiles <= 2 * (int64_t)sms ? 8 : tiles <= 4 * (int64_t)sms ? 16 : 32;
    // as few neurons per warp of the spike launch as fill its grid once: their fires are
    // served one after the other
    P.launch_rows = 8;
    while (P.launch_rows > 1 && tiles * 32 / (P.launch_rows / 2) <= (int64_t)sms * NC_LAUNCH_BLOCKS * 4)
        P.launch_rows /= 2;
}

int dense_blocks(int64_t neurons, int64_t quads, int threads)
{
    // fewer blocks than a wave where there are fewer runs of 8 neurons: one for each, or as many
    // for each as its rows are split into (every neuron of 3,000 driving every other 63 -> 46 us
    // a step, with inhibitory synapses 248 -> 222)
    const int64_t most = dense_resident_blocks(threads), runs = std::max<int64_t>(1, (neurons + 7) / 8);
    const int64_t parts = quads / runs > kSplitEvenQuads ? std::min(2 * quads / runs / kSplitEvenQuads, most / runs) : 1;
    return (int)std::max<int64_t>(1, std::min(most, runs * std::max<int64_t>(1, parts)));
}

void Engine::set_launch(const LaunchShape& shape, int ticks_per_graph)
{
    release_graph();
    L = shape;
    if (!dense || both) event_resident_blocks(L.neuron_block);
    graph_ticks = ticks_per_graph;
}

int Engine::build(const std::vector<const NetHost*>& nets, int group_capacity, std::string& err,
                  const std::vector<int32_t>* horizons, bool device_synapses)
{
    NC_CK(cudaGetDevice(&device));
    NC_CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    int sms = 0;
    NC_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    int pageable = 0, tables_shared = 0;
    NC_CK(cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, device));
    NC_CK(cudaDeviceGetAttribute(&tables_shared, cudaDevAttrPageableMemoryAccessUsesHostPageTables, device));
    shared_tables_ = pageable && tables_shared;
    dense = nets.empty() || nets[0]->p.step_mode != NC_STEP_EVENT;
    both = !nets.empty() && nets[0]->p.step_mode == NC_STEP_AUTO;
    const bool event_tables = !dense || both;
    L.launch_block = 128;
    L.launch_blocks = std::max(1, sms * NC_LAUNCH_BLOCKS);

    // pool sizes
    int64_t neurons = 0, ptrs = 0, words = 0, syn = 0, ring = 0, tables = 0, tiles = 0, inputs = 0;
    const int ngroups_each = std::max(group_capacity, 1);
    slots.clear();
    std::vector<NcNetDesc> desc;
    for (size_t q = 0; q < nets.size(); ++q) {
        const NetHost& h = *nets[q];
        NetSlot sl;
        sl.n = h.n;
        sl.s = h.s;
        sl.kc = h.kc;
        sl.dt = h.dt;
        sl.n_words = (h.n + 31) / 32;
        sl.neuron_base = (int32_t)neurons;
        sl.ptr_base = (int32_t)ptrs;
        sl.word_base = (int32_t)words;
        sl.syn_base = syn;
        sl.n_input = h.n_input;
        sl.index_base = inputs;
        inputs += h.n_input;
        sl.group_cap = ngroups_each;
        sl.group_base = (int32_t)(q * ngroups_each);
        NcNetDesc d;
        std::memset(&d, 0, sizeof(d));
        d.t = 1;
        d.t_end = horizons ? (*horizons)[q] : (1 << 30);
        d.stdp_done = 0;
        d.n = h.n;
        d.neuron_base = sl.neuron_base;
        d.ptr_base = sl.ptr_base;
        d.word_base = sl.word_base;
        d.n_words = sl.n_words;
        d.syn_base = syn;
        d.ring_base = ring;
        d.ring_words = h.ring_words;
        d.ring_mask = h.ring_slots - 1;
        d.kc = h.kc;
        d.bg_period = h.bg_period;
        d.key0 = (uint32_t)h.p.seed;
        d.key1 = (uint32_t)(h.p.seed >> 32);
        d.table_base = (int32_t)tables;
        d.tab_pre_len = h.tab_pre_len;
        d.tab_post_len = h.tab_post_len;
        d.ap_base = (int32_t)(tables + h.tab_pre_len + h.tab_post_len);
        d.group_base = sl.group_base;
        d.n_groups = (int32_t)std::min<size_t>(h.groups.size(), (size_t)ngroups_each);
        nc_group_range(h.groups.data(), d.n_groups, d.group_lo, d.group_hi);
        d.active = 1;
        d.permuted = h.permuted ? 1 : 0;
        d.nonneg_terms = h.nonneg_terms ? 1 : 0;
        d.dt = d.dt_again = h.dt;
        d.leak = h.leak;
        d.c52 = h.c52;
        d.lr = h.p.learning_rate;
        d.pre_factor = h.p.presynaptic_factor;
        d.post_factor = h.p.postsynaptic_factor;
        d.e_term = h.e_term;
        term_pair(h, d.term_hi, d.term_lo);
        d.n_syn = h.s;
        d.key_shift = h.key_shift;
        const int64_t range = (h.sp + 31) / 32 * 32;  // keeps every net's inhibitory bits word-aligned
        d.wide = dense && h.wide ? range : 0;
        desc.push_back(d);
        slots.push_back(sl);
        neurons += h.n;
        ptrs += h.n + 1;
        words += sl.n_words + 1;  // a spare word: the fired bits of the rows' padding
        syn += d.wide ? 2 * range : range;
        if (event_tables) ring += (int64_t)h.ring_slots * h.ring_words;
        tables += (int64_t)h.tables.size();
        tiles += sl.n_words;
        if (h.groups.size() > (size_t)ngroups_each) {
            err = "more input groups than reserved";
            return NC_ERR_INVALID;
        }
    }
    if (neurons >= (1ll << 31) || tables >= (1ll << 31) || words >= (1ll << 31)) {
        err = "pool too large";
        return NC_ERR_INVALID;
    }

    NC_ALLOC(P.pot, float, neurons);
    NC_ALLOC(P.lf, int32_t, neurons);
    NC_ALLOC(P.firings, uint32_t, neurons);
    NC_ALLOC(P.act_start, int32_t, neurons);
    NC_ALLOC(P.orig_id, int32_t, neurons);
    NC_ALLOC(P.slot_of, int32_t, neurons);
    NC_ALLOC(P.in_ptr, int64_t, ptrs);
    NC_ALLOC(P.w, float, syn);
    NC_ALLOC(P.x, float, syn);
    if (dense) {
        NC_ALLOC(P.key, uint32_t, syn);
        NC_ALLOC(P.state, uint32_t, syn);
        NC_ALLOC(P.qrow, uint8_t, syn / 4);
        NC_ALLOC(P.pst, float, neurons);
        NC_ALLOC(P.nib, uint8_t, syn / 4 + 8);  // read in 8-byte words
    }
    L.neuron_block = dense ? NC_DENSE_BLOCK : NC_EVENT_BLOCK;
    if (event_tables) {
        event_resident_blocks(L.neuron_block);
        NC_ALLOC(P.inh, uint32_t, (syn + 31) / 32 + 1);  // one spare word for 32-bit windows
        NC_ALLOC(P.t_arr, int32_t, syn);
        NC_ALLOC(P.out_ptr, int64_t, ptrs);
        NC_ALLOC(P.ring_off, int32_t, ptrs);
        NC_ALLOC(P.out, NcOut, syn);
        NC_ALLOC(P.last_arr, int32_t, syn);
        NC_ALLOC(P.ring, uint32_t, ring);
        ring_words_total_ = ring;
    }
    P.total_words = std::max<int64_t>(words, 1);
    NC_ALLOC(P.fired, uint32_t, 2 * P.total_words);
    NC_ALLOC(P.forced, uint32_t, 2 * P.total_words);
    NC_ALLOC(P.ufire, uint32_t, 2 * P.total_words);
    NC_ALLOC(P.tables, float, tables);
    NC_ALLOC(P.groups, NcGroupDev, nets.size() * ngroups_each);
    NC_ALLOC(P.nets, NcNetDesc, nets.size());
    if (event_tables) NC_ALLOC(P.tiles, NcTile, tiles);
    NC_ALLOC(P.done_ctr, uint32_t, 1);
    NC_ALLOC(P.dev_err, uint32_t, 1);
    NC_ALLOC(d_bar_, unsigned, 2);
    NC_ALLOC(P.stats, unsigned long long, 4 * nets.size());
    for (const NetHost* h : nets)
        scratch_bytes_ = std::max(scratch_bytes_, std::max(sizeof(float) * (size_t)h->n_input, 8 * (size_t)h->n));
    scratch_bytes_ = std::max<size_t>(256, std::min(scratch_bytes_, kScratchMax));
    NC_ALLOC(scratch_, char, scratch_bytes_);
    P.n_nets = (int32_t)nets.size();
    P.n_tiles = event_tables ? (int32_t)tiles : 0;
    event_rows(tiles, sms, P);

    // contents
    std::vector<NcTile> tile_host;
    std::vector<RowNet> row_nets;
    for (size_t q = 0; q < nets.size(); ++q) {
        const NetHost& h = *nets[q];
        const NetSlot& sl = slots[q];
        NcNetDesc& d = desc[q];
        d.stats = P.stats + 4 * q;
        std::vector<float> pot((size_t)h.n, -70.0f);  // setPotential(baselevel)
        std::vector<int32_t> lf((size_t)h.n, NC_NEVER);
        NC_CK(upload(P.pot, pot, sl.neuron_base, stream));
        NC_CK(upload(P.lf, lf, sl.neuron_base, stream));
        NC_CK(upload(P.orig_id, h.orig_id, sl.neuron_base, stream));
        NC_CK(upload(P.slot_of, h.slot_of, sl.neuron_base, stream));
        std::vector<int64_t> inp(h.in_ptr), outp(h.out_ptr);
        for (auto& v : inp) v += sl.syn_base;
        for (auto& v : outp) v += sl.syn_base;
        NC_CK(upload(P.in_ptr, inp, sl.ptr_base, stream));
        row_nets.push_back(RowNet{&h, (int32_t)q, sl.syn_base, sl.neuron_base, sl.ptr_base});
        std::vector<int32_t> never;
        std::vector<NcOut> out;
        if (dense && launch_fill_words(P.state + sl.syn_base, d.wide + h.sp, initial_state(h), stream)) {
            err = cuda_msg("initial states", cudaGetLastError());
            return NC_ERR_CUDA;
        }
        if (!device_synapses) {
            NC_CK(upload(P.w, h.w, sl.syn_base, stream));
            if (dense) {
                for (int64_t part = 0; part < key_words(h); ++part)
                    NC_CK(upload_part(P.key, h.key, sl.syn_base + part * d.wide, part * h.sp, h.sp, stream));
                NC_CK(upload(P.qrow, h.qrow, sl.syn_base / 4, stream));
            }
            if (event_tables) {
                never.assign((size_t)h.sp, NC_NEVER);
                NC_CK(upload(P.inh, h.inh_bits, sl.syn_base / 32, stream));
                NC_CK(upload(P.t_arr, never, sl.syn_base, stream));
                NC_CK(upload(P.out_ptr, outp, sl.ptr_base, stream));
                NC_CK(upload(P.ring_off, h.ring_off, sl.ptr_base, stream));
                NC_CK(upload_part(P.last_arr, never, sl.syn_base, 0, h.s, stream));
                out = out_records(h);
                NC_CK(upload(P.out, out, sl.syn_base, stream));
            }
        }
        NC_CK(upload(P.tables, h.tables, d.table_base, stream));
        if (!h.groups.empty()) NC_CK(upload(P.groups, h.groups, sl.group_base, stream));
        if (event_tables)
            for (int32_t f = 0; f < h.n; f += 32) tile_host.push_back(NcTile{(int32_t)q, f});
        // the vectors above must stay alive until the copies finish
        NC_CK(cudaStreamSynchronize(stream));
    }
    NC_CK(upload(P.nets, desc, 0, stream));
    NC_CK(upload(P.tiles, tile_host, 0, stream));
    if (dense) {
        std::vector<NcRowTile> rows;
        std::vector<int32_t> start;
        int64_t quads = 0;
        for (const NetHost* h : nets) quads += h->sp / 4;
        P.row_blocks = dense_blocks(neurons, quads, L.neuron_block);
        plan_rows(row_nets, P.row_blocks, rows, start);
        // sums that run to their last term (inhibitory or negative synapses) gain from it: the
        // sphere of 750 6.3 -> 5.9 us a step, 20k x 100 20.7 -> 19.0 (at the limit: networks of that
        // size whose largest tile has some quads more are not staged); those that stop early, after
        // a batch or two, do not (1k x 50 6.5 either way, 30k x 73 14.7 and 14.9)
        bool all_sum = true;
        for (const NetHost* h : nets) all_sum = all_sum && !h->nonneg_terms;
        P.stage = all_sum && dense_stages(rows, start, L.neuron_block) ? 1 : 0;
        NC_ALLOC(P.rtiles, NcRowTile, rows.size());
        NC_ALLOC(P.rstart, int32_t, start.size());
        NC_ALLOC(P.split_ctr, uint32_t, P.row_blocks);
        P.split = has_parts(rows) ? 1 : 0;
        NC_CK(upload(P.rtiles, rows, 0, stream));
        NC_CK(upload(P.rstart, start, 0, stream));
        NC_CK(cudaStreamSynchronize(stream));
    }
    // The positions of the given synapses, for the read-back of the weights: with the network's
    // other arrays, so that no read-back allocates.  (Last: where memory is short the host
    // reorders instead.)
    index_ = alloc<uint32_t>((size_t)inputs, err);
    if (!index_) {
        cudaGetLastError();
        err.clear();
    }
    for (size_t q = 0; index_ && !device_synapses && q < nets.size(); ++q) {
        const std::vector<uint32_t> index(nets[q]->input_to_csc.begin(), nets[q]->input_to_csc.end());  // -1 becomes ~0
        NC_CK(upload(index_, index, (size_t)slots[q].index_base, stream));
        NC_CK(cudaStreamSynchronize(stream));
    }
    NC_CK(cudaStreamSynchronize(stream));
    for (size_t q = 0; q < nets.size(); ++q) {
        if (launch_background_prologue(P, (int)q, nets[q]->n, stream) != 0) {
            err = cuda_msg("background prologue", cudaGetLastError());
            return NC_ERR_CUDA;
        }
    }
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

void Engine::release_graph()
{
    if (graph_) cudaGraphExecDestroy(graph_);
    graph_ = nullptr;
}

int Engine::capture_graph(std::string& err)
{
    release_graph();
    cudaGraph_t g = nullptr;
    NC_CK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
    int rc = 0;
    for (int k = 0; k < graph_ticks && rc == 0; ++k) rc |= launch_tick(stream);
    cudaError_t e = cudaStreamEndCapture(stream, &g);
    if (rc != 0 || e != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        err = cuda_msg("graph capture", e != cudaSuccess ? e : cudaGetLastError());
        return NC_ERR_CUDA;
    }
    e = cudaGraphInstantiate(&graph_, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        graph_ = nullptr;
        err = cuda_msg("cudaGraphInstantiate", e);
        return NC_ERR_CUDA;
    }
    return NC_OK;
}

int Engine::step(int64_t ticks, std::string& err)
{
    if (ticks <= 0) return NC_OK;
    flushed_ = false;
    if (dense && L.fused_ticks > 0 && P.n_firers == 0) {
        // several whole steps per cooperative launch
        while (ticks > 0) {
            const int32_t m = (int32_t)std::min<int64_t>(ticks, L.fused_ticks);
            if (launch_fused_dense(P, m, L, d_bar_, stream)) {
                err = cuda_msg("fused step launch", cudaGetLastError());
                return NC_ERR_CUDA;
            }
            ticks -= m;
        }
        return NC_OK;
    }
    if (ticks >= graph_ticks && graph_ticks > 0) {
        if (!graph_) {
            const int rc = capture_graph(err);
            if (rc) return rc;
        }
        while (ticks >= graph_ticks) {
            NC_CK(cudaGraphLaunch(graph_, stream));
            ticks -= graph_ticks;
        }
    }
    for (int64_t k = 0; k < ticks; ++k) {
        if (launch_tick(stream)) {
            err = cuda_msg("step launch", cudaGetLastError());
            return NC_ERR_CUDA;
        }
    }
    return NC_OK;
}

int Engine::launch_tick(cudaStream_t s)
{
    int rc = P.n_firers > 0 ? launch_input_firers(P, dense, s) : 0;  // the step's run-call schedule first
    const bool whole = counters_written_;
    counters_written_ = false;
    rc |= dense ? launch_step_dense(P, L, back_ = !back_, s) : (launch_neuron_step(P, L, whole, s) | launch_spike_launch(P, L, many_units(P.n_tiles, P, L), s));
    return rc;
}

int Engine::set_firers(const std::vector<NcFirer>& firers, const std::vector<int32_t>& near, std::string& err)
{
    release_graph();  // the captured ticks change
    NC_CK(cudaStreamSynchronize(stream));
    if (firers_buf_) cudaFree(firers_buf_);
    if (near_buf_) cudaFree(near_buf_);
    firers_buf_ = nullptr;
    near_buf_ = nullptr;
    P.firers = nullptr;
    P.firer_near = nullptr;
    P.n_firers = 0;
    if (firers.empty()) return NC_OK;
    NC_CK(cudaMalloc(&firers_buf_, sizeof(NcFirer) * firers.size()));
    NC_CK(cudaMalloc(&near_buf_, sizeof(int32_t) * std::max<size_t>(near.size(), 1)));
    NC_CK(cudaMemcpyAsync(firers_buf_, firers.data(), sizeof(NcFirer) * firers.size(), cudaMemcpyHostToDevice, stream));
    if (!near.empty())
        NC_CK(cudaMemcpyAsync(near_buf_, near.data(), sizeof(int32_t) * near.size(), cudaMemcpyHostToDevice, stream));
    P.firers = (NcFirer*)firers_buf_;
    P.firer_near = (int32_t*)near_buf_;
    P.n_firers = (int32_t)firers.size();
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

int Engine::read_firers(std::vector<NcFirer>& out, std::string& err)
{
    out.resize((size_t)P.n_firers);
    if (P.n_firers == 0) return NC_OK;
    NC_CK(cudaMemcpyAsync(out.data(), P.firers, sizeof(NcFirer) * out.size(), cudaMemcpyDeviceToHost, stream));
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

int Engine::write_firers(const std::vector<NcFirer>& in, std::string& err)
{
    if ((int32_t)in.size() != P.n_firers) {
        err = "firer count mismatch";
        return NC_ERR_INVALID;
    }
    if (P.n_firers == 0) return NC_OK;
    NC_CK(cudaMemcpyAsync(P.firers, in.data(), sizeof(NcFirer) * in.size(), cudaMemcpyHostToDevice, stream));
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

int Engine::step_timed(int64_t ticks, float* ms, std::string& err)
{
    cudaEvent_t a, b;
    NC_CK(cudaEventCreate(&a));
    NC_CK(cudaEventCreate(&b));
    NC_CK(cudaEventRecord(a, stream));
    int rc = step(ticks, err);
    if (rc == NC_OK) {
        NC_CK(cudaEventRecord(b, stream));
        NC_CK(cudaEventSynchronize(b));
        NC_CK(cudaEventElapsedTime(ms, a, b));
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    return rc;
}

int Engine::time_kernels(int ticks, float* neuron_ms, float* launch_ms, std::string& err)
{
    // the dense form's step is one kernel: its time, and 0
    flushed_ = false;
    const int marks = dense ? 2 : 3;
    std::vector<cudaEvent_t> ev((size_t)marks * (size_t)std::max(ticks, 0));
    for (auto& e : ev) NC_CK(cudaEventCreate(&e));
    for (int k = 0; k < ticks; ++k) {
        cudaEvent_t* at = &ev[(size_t)(marks * k)];
        if (P.n_firers > 0 && launch_input_firers(P, dense, stream)) {
            err = "launch";
            return NC_ERR_CUDA;
        }
        NC_CK(cudaEventRecord(at[0], stream));
        const bool whole = counters_written_;
        counters_written_ = false;
        if (dense ? launch_step_dense(P, L, back_ = !back_, stream) : launch_neuron_step(P, L, whole, stream)) {
            err = "launch";
            return NC_ERR_CUDA;
        }
        NC_CK(cudaEventRecord(at[1], stream));
        if (dense) continue;
        if (launch_spike_launch(P, L, many_units(P.n_tiles, P, L), stream)) {
            err = "launch";
            return NC_ERR_CUDA;
        }
        NC_CK(cudaEventRecord(at[2], stream));
    }
    NC_CK(cudaStreamSynchronize(stream));
    double sa = 0, sb = 0;
    for (int k = 0; k < ticks; ++k) {
        const cudaEvent_t* at = &ev[(size_t)(marks * k)];
        float x = 0, y = 0;
        NC_CK(cudaEventElapsedTime(&x, at[0], at[1]));
        if (!dense) NC_CK(cudaEventElapsedTime(&y, at[1], at[2]));
        sa += x;
        sb += y;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    *neuron_ms = ticks ? (float)(sa / ticks) : 0.0f;
    *launch_ms = ticks ? (float)(sb / ticks) : 0.0f;
    return NC_OK;
}

int Engine::flush_plasticity(std::string& err)
{
    if (flushed_ && !unseen_) return NC_OK;
    if (dense ? launch_flush_dense(P, L, stream) : launch_stdp_flush(P, L, stream)) {
        err = cuda_msg("plasticity flush", cudaGetLastError());
        return NC_ERR_CUDA;
    }
    flushed_ = counters_written_ = true;
    return NC_OK;
}

// Has the pages of a buffer that is about to be filled made present and writable, where it is
// ordinary host memory (and says whether they are).  A page that is not there yet costs the
// host less than it costs the GPU, whose page tables are the host's: with a copy into fresh
// pages, 400 KB 39 us instead of 151, 2 MB 99 instead of 218, and nothing where the GPU is
// still at work on the steps before (a byte written to each page, before: 40 MB 1,590 us, 1,480
// now).  The contents stay as they are until the result is there; what cannot be written is
// left to the copy to report.
static bool bring_in(void* out, size_t bytes)
{
    cudaPointerAttributes at;
    if (!bytes || cudaPointerGetAttributes(&at, out) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (at.type != cudaMemoryTypeUnregistered) return false;
    if (bytes <= 4096) {  // a page or two, nearly always there: a store of what is there saves the system calls
        __atomic_fetch_or((char*)out, 0, __ATOMIC_RELAXED);
        __atomic_fetch_or((char*)out + bytes - 1, 0, __ATOMIC_RELAXED);
        return true;
    }
    static const uintptr_t page = (uintptr_t)std::max<long>(4096, sysconf(_SC_PAGESIZE));
    const uintptr_t from = (uintptr_t)out / page * page;
    const size_t length = (uintptr_t)out + bytes - from;
    constexpr size_t kChunk = 1024;
    unsigned char there[kChunk];
    for (size_t a = 0; a < length; a += kChunk * page) {
        const size_t m = std::min(length - a, kChunk * page);
        // (many pages that are there are only looked at: 40 MB 4 us instead of 80)
        bool all = m >= 16 * page && mincore((void*)(from + a), m, there) == 0;
        for (size_t k = 0; all && k * page < m; ++k) all = there[k] & 1;
        if (!all && madvise((void*)(from + a), m, MADV_POPULATE_WRITE) != 0) return false;
    }
    return true;
}

// Results of up to this many bytes are written by their kernel straight into the caller's
// memory: a read of 64 KB takes 17 us instead of 22, of 256 KB 20 instead of 25 (pages there; 35
// and 46 instead of 41 and 53 into fresh ones).  The line dates from when pages could not be
// populated: into absent ones 800 KB took 404 us instead of 183.  Populated, direct writes lead at
// every size measured (1 MB 29 us instead of 35, 40 MB 235 instead of 291).
constexpr size_t kDirectMax = 256 << 10;

// Runs `launch(first, count, buffer)` for `items` items of per_item bytes: into out itself, or
// into the scratch buffer, as many at a time as it holds, with a copy of each part to out.
// shared_tables: the GPU uses the host's page tables.
template <class F>
static int read_parts(int64_t items, size_t per_item, bool shared_tables, void* buf, size_t buf_bytes, void* out,
                      cudaStream_t stream, F&& launch, std::string& err)
{
    const size_t bytes = items > 0 ? (size_t)items * per_item : 0;
    if (shared_tables && bytes <= kDirectMax && ((uintptr_t)out & 15) == 0 && bring_in(out, bytes)) {
        if (launch(0, items, out)) {
            err = cuda_msg("read-back", cudaGetLastError());
            return NC_ERR_CUDA;
        }
        NC_CK(cudaStreamSynchronize(stream));
        return NC_OK;
    }
    const int64_t part = std::max<int64_t>(1, (int64_t)(buf_bytes / std::max<size_t>(per_item, 1)));
    for (int64_t a = 0; a < items && per_item; a += part) {
        const int64_t m = std::min(part, items - a);
        char* to = (char*)out + a * (int64_t)per_item;
        if (launch(a, m, buf)) {
            err = cuda_msg("read-back", cudaGetLastError());
            return NC_ERR_CUDA;
        }
        if (shared_tables) bring_in(to, (size_t)m * per_item);
        NC_CK(cudaMemcpyAsync(to, buf, (size_t)m * per_item, cudaMemcpyDeviceToHost, stream));
    }
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

int Engine::read_potentials(int net, float* out, std::string& err)
{
    const NetSlot& sl = slots[(size_t)net];
    // slot_of is a permutation of 0 .. n-1: an index of the same bits
    return read_parts(sl.n, sizeof(float), shared_tables_, scratch_, scratch_bytes_, out, stream,
                      [&](int64_t a, int64_t m, void* buf) {
                          return launch_gather(P.pot + sl.neuron_base,
                                               (const uint32_t*)P.slot_of + sl.neuron_base + a, m, (float*)buf, stream);
                      },
                      err);
}

int Engine::read_potact(int net, int64_t t, float* out_2n, std::string& err)
{
    const NetSlot& sl = slots[(size_t)net];
    return read_parts(sl.n, 2 * sizeof(float), shared_tables_, scratch_, scratch_bytes_, out_2n, stream,
                      [&](int64_t a, int64_t m, void* buf) {
                          return launch_potact(P, sl.neuron_base, (int32_t)a, (int32_t)m, t, sl.dt, (float*)buf, stream);
                      },
                      err);
}

int Engine::read_last_fire(int net, float* out, std::string& err)
{
    const NetSlot& sl = slots[(size_t)net];
    return read_parts(sl.n, sizeof(float), shared_tables_, scratch_, scratch_bytes_, out, stream,
                      [&](int64_t a, int64_t m, void* buf) {
                          return launch_last_fire(P, sl.neuron_base, (int32_t)a, (int32_t)m, sl.dt, (float*)buf, stream);
                      },
                      err);
}

int Engine::read_weights(int net, float* out, std::string& err)
{
    const float* w = P.w + slots[(size_t)net].syn_base;
    const uint32_t* at = index(net);
    return read_parts(slots[(size_t)net].n_input, sizeof(float), shared_tables_, scratch_, scratch_bytes_, out, stream,
                      [&](int64_t a, int64_t m, void* buf) { return launch_gather(w, at + a, m, (float*)buf, stream); },
                      err);
}

int Engine::read_raster(int net, const uint32_t* d_raster, int32_t rows, uint8_t* out, std::string& err)
{
    const NetSlot& sl = slots[(size_t)net];
    return read_parts(rows, ((size_t)sl.n + 7) / 8, shared_tables_, scratch_, scratch_bytes_, out, stream,
                      [&](int64_t a, int64_t m, void* buf) {
                          return launch_raster_bytes(d_raster + a * sl.n_words, (uint8_t*)buf, P.slot_of + sl.neuron_base,
                                                     sl.n, sl.n_words, (int32_t)m, stream);
                      },
                      err);
}

int Engine::set_form(bool to_dense, std::string& err)
{
    if (to_dense == dense) return NC_OK;
    if (!both || slots.size() != 1) {
        err = "this network holds the tables of one form only (create it with NC_STEP_AUTO)";
        return NC_ERR_UNSUPPORTED;
    }
    int rc = flush_plasticity(err);
    if (rc != NC_OK) return rc;
    rc = to_dense ? launch_form_to_dense(P, 0, slots[0].s, stream)
                  : launch_form_to_event(P, 0, slots[0].s, ring_words_total_, stream);
    if (rc) {
        err = cuda_msg("form switch", cudaGetLastError());
        return NC_ERR_CUDA;
    }
    release_graph();
    dense = to_dense;
    return sync(err);
}

int Engine::sync(std::string& err)
{
    NC_CK(cudaStreamSynchronize(stream));
    uint32_t dev_err = 0;
    NC_CK(cudaMemcpy(&dev_err, P.dev_err, sizeof(dev_err), cudaMemcpyDeviceToHost));
    if (dev_err) {
        err = "a device wait gave up (code " + std::to_string(dev_err) + ")";
        return NC_ERR_TIMEOUT;
    }
    return NC_OK;
}

template <class F>
static cudaError_t put_field(NcNetDesc* d_nets, int net, size_t offset, const F& value, cudaStream_t s)
{
    return cudaMemcpyAsync((char*)(d_nets + net) + offset, &value, sizeof(F), cudaMemcpyHostToDevice, s);
}

int Engine::set_groups(int net, const std::vector<NcGroupDev>& groups, std::string& err)
{
    if ((int)groups.size() > slots[net].group_cap) {
        err = "too many input groups for this engine";
        return NC_ERR_INVALID;
    }
    if (!groups.empty())
        NC_CK(cudaMemcpyAsync(P.groups + slots[net].group_base, groups.data(), groups.size() * sizeof(NcGroupDev),
                              cudaMemcpyHostToDevice, stream));
    const int32_t ng = (int32_t)groups.size();
    int32_t range[2];
    nc_group_range(groups.data(), ng, range[0], range[1]);
    static_assert(offsetof(NcNetDesc, group_hi) == offsetof(NcNetDesc, group_lo) + sizeof(int32_t), "range");
    NC_CK(cudaMemcpyAsync((char*)(P.nets + net) + offsetof(NcNetDesc, group_lo), range, sizeof(range),
                          cudaMemcpyHostToDevice, stream));
    NC_CK(put_field(P.nets, net, offsetof(NcNetDesc, n_groups), ng, stream));
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

int Engine::set_rates(int net, float lr, float pre_factor, float post_factor, std::string& err)
{
    // plasticity still pending from the last step belongs to the old rates
    const int rc = flush_plasticity(err);
    if (rc != NC_OK) return rc;
    NC_CK(put_field(P.nets, net, offsetof(NcNetDesc, lr), lr, stream));
    NC_CK(put_field(P.nets, net, offsetof(NcNetDesc, pre_factor), pre_factor, stream));
    NC_CK(put_field(P.nets, net, offsetof(NcNetDesc, post_factor), post_factor, stream));
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

int Engine::force_fire(int net, const int32_t* ids, int count, std::string& err)
{
    if (count <= 0) return NC_OK;
    if (count > ids_cap_) {
        if (d_ids_) {
            NC_CK(cudaStreamSynchronize(stream));
            cudaFree(d_ids_);
            d_ids_ = nullptr;
        }
        const int cap = std::max(count, 1024);
        NC_CK(cudaMalloc(&d_ids_, sizeof(int32_t) * cap));
        ids_cap_ = cap;
    }
    NC_CK(cudaMemcpyAsync(d_ids_, ids, sizeof(int32_t) * count, cudaMemcpyHostToDevice, stream));
    if (launch_force_bits(P, net, d_ids_, count, stream)) {
        err = cuda_msg("force bits", cudaGetLastError());
        return NC_ERR_CUDA;
    }
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

int Engine::set_raster(int net, uint32_t* d_raster, int32_t t0, int32_t len, std::string& err)
{
    NC_CK(put_field(P.nets, net, offsetof(NcNetDesc, raster), d_raster, stream));
    NC_CK(put_field(P.nets, net, offsetof(NcNetDesc, raster_t0), t0, stream));
    NC_CK(put_field(P.nets, net, offsetof(NcNetDesc, raster_len), len, stream));
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

int Engine::read_stats(int net, unsigned long long out[4], std::string& err)
{
    NC_CK(cudaMemcpyAsync(out, P.stats + 4 * net, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, stream));
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

int Engine::read_desc(int net, NcNetDesc* out, std::string& err)
{
    NC_CK(cudaMemcpyAsync(out, P.nets + net, sizeof(NcNetDesc), cudaMemcpyDeviceToHost, stream));
    NC_CK(cudaStreamSynchronize(stream));
    return NC_OK;
}

}  // namespace nc
