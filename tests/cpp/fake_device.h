// A CUDA device of host memory, for checks of the library's host code without a GPU.
//
// Linked with the host parts of the library (nc_api.cu, nc_pool.cu, nc_batch.cu, nc_serve.cu,
// nc_noalloc.cu as C++, and nc_host.cpp) in place of the CUDA runtime and of the kernels'
// launchers.  It does what the runtime promises and no more:
//   - work on a stream is done as it is issued; work on the legacy default stream, which
//     waits for none of the library's streams and none for it, is done `legacy_delay` items
//     of other streams later, or when the caller waits for it;
//   - device memory holds garbage until it is written;
//   - reads out of range are counted (`faults`) and not made.
// A step writes the raster row of its step (every bit set) and moves the step counter on;
// gathers are made; other kernels do nothing.
#pragma once
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <limits>
#include <map>
#include <mutex>
#include <vector>

#include "nc_net.h"

namespace fake {

std::recursive_mutex mu;
std::map<char*, size_t> memory;     // device allocations
size_t held = 0;                    // their bytes
int64_t mallocs = 0;                // calls of cudaMalloc
int64_t fail_malloc_at = -1;        // the call that fails (counted from 0)
size_t fail_malloc_from = ~(size_t)0;  // allocations of so many bytes and more fail
int faults = 0;
int legacy_delay = 0;
int gathers_to_fail = 0, graphs_to_fail = 0;
bool flush_open = false;  // the event form's flush was launched, and nothing has waited for it
int early_steps = 0;      // steps that may read what it writes before it is done

struct Late {
    int left;
    std::function<void()> work;
};
std::vector<Late> late;

void all_late()
{
    for (auto& l : late) l.work();
    late.clear();
}

// an item of another stream
void other_stream()
{
    for (size_t k = 0; k < late.size();) {
        if (late[k].left-- > 0) {
            ++k;
            continue;
        }
        late[k].work();
        late.erase(late.begin() + k);
    }
}

bool device_range(const void* p, size_t bytes)
{
    auto it = memory.upper_bound((char*)p);
    if (it == memory.begin()) return false;
    --it;
    return (char*)p + bytes <= it->first + it->second;
}

// graph capture: what a captured launch does, kept for its replays
std::vector<std::function<void()>>* capturing = nullptr;
using Graph = std::vector<std::function<void()>>;

int launch(std::function<void()> work)
{
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (capturing) {
        capturing->push_back(std::move(work));
        return 0;
    }
    work();
    other_stream();
    return 0;
}

void step(const NcPools& P)
{
    for (int32_t n = 0; n < P.n_nets; ++n) {
        NcNetDesc& D = P.nets[n];
        if (!D.active || D.t > D.t_end) continue;
        if (D.raster_len > 0 && D.t >= D.raster_t0 && D.t - D.raster_t0 < D.raster_len) {
            uint32_t* row = D.raster + (int64_t)(D.t - D.raster_t0) * D.n_words;
            if (device_range(row, 4 * (size_t)D.n_words)) std::memset(row, 0xff, 4 * (size_t)D.n_words);
            else ++faults;
        }
        D.t += 1;
    }
}

}  // namespace fake

#define FAKE_LOCK std::lock_guard<std::recursive_mutex> lk_(fake::mu)

// The runtime (C linkage, as cuda_runtime_api.h declares it).
extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t bytes)
{
    FAKE_LOCK;
    if (fake::mallocs++ == fake::fail_malloc_at || bytes >= fake::fail_malloc_from) return cudaErrorMemoryAllocation;
    char* q = (char*)std::malloc(bytes ? bytes : 1);
    std::memset(q, 0xa5, bytes);
    fake::memory[q] = bytes;
    fake::held += bytes;
    *p = q;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    FAKE_LOCK;
    if (!p) return cudaSuccess;
    fake::all_late();
    fake::held -= fake::memory[(char*)p];
    fake::memory.erase((char*)p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* at, const void* p)
{
    FAKE_LOCK;
    at->type = fake::device_range(p, 1) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind, cudaStream_t)
{
    FAKE_LOCK;
    std::memcpy(to, from, bytes);
    fake::other_stream();
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t bytes, cudaStream_t)
{
    FAKE_LOCK;
    std::memset(p, v, bytes);
    fake::other_stream();
    return cudaSuccess;
}
// On the legacy stream: pageable memory is read at once, and may reach the device later.
cudaError_t cudaMemcpy(void* to, const void* from, size_t bytes, cudaMemcpyKind kind)
{
    FAKE_LOCK;
    if (kind == cudaMemcpyDeviceToHost) {
        fake::all_late();
        std::memcpy(to, from, bytes);
        return cudaSuccess;
    }
    std::vector<char> staged((const char*)from, (const char*)from + bytes);
    fake::late.push_back({fake::legacy_delay, [to, staged] { std::memcpy(to, staged.data(), staged.size()); }});
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t bytes)
{
    FAKE_LOCK;
    fake::late.push_back({fake::legacy_delay, [=] { std::memset(p, v, bytes); }});
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)1, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return fake::flush_open = false, cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.0f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    FAKE_LOCK;
    fake::capturing = new fake::Graph;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g)
{
    FAKE_LOCK;
    *g = (cudaGraph_t)fake::capturing;
    fake::capturing = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long)
{
    *e = (cudaGraphExec_t) new fake::Graph(*(fake::Graph*)g);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return delete (fake::Graph*)g, cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return delete (fake::Graph*)e, cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t)
{
    FAKE_LOCK;
    if (fake::graphs_to_fail > 0 && fake::graphs_to_fail-- > 0) return cudaErrorLaunchFailure;
    for (auto& w : *(fake::Graph*)e) fake::launch(w);
    return cudaSuccess;
}
}  // extern "C"

// The kernels' launchers.
namespace nc {
int dense_resident_blocks(int) { return 152 * 8; }
bool dense_stages(const std::vector<NcRowTile>&, const std::vector<int32_t>&, int) { return false; }
int launch_step_dense(const NcPools& P, const LaunchShape&, bool, void*)
{
    return fake::launch([P] { fake::step(P); });
}
int launch_neuron_step(const NcPools& P, const LaunchShape&, bool whole, void*)
{
    if (!fake::capturing) {
        fake::early_steps += fake::flush_open && !whole;
        fake::flush_open = false;
    }
    return fake::launch([P] { fake::step(P); });
}
int event_resident_blocks(int) { return 152 * 8; }
bool many_units(int, const NcPools&, const LaunchShape&) { return false; }
int launch_spike_launch(const NcPools&, const LaunchShape&, bool, void*) { return fake::launch([] {}); }
int launch_fused_dense(const NcPools& P, int32_t ticks, const LaunchShape&, unsigned*, void*)
{
    return fake::launch([P, ticks] {
        for (int32_t k = 0; k < ticks; ++k) fake::step(P);
    });
}
int launch_stdp_flush(const NcPools&, const LaunchShape&, void*)
{
    fake::flush_open = true;
    return fake::launch([] {});
}
int launch_flush_dense(const NcPools&, const LaunchShape&, void*) { return fake::launch([] {}); }
int launch_form_to_event(const NcPools&, int, int64_t, int64_t, void*) { return fake::launch([] {}); }
int launch_form_to_dense(const NcPools&, int, int64_t, void*) { return fake::launch([] {}); }
int launch_background_prologue(const NcPools&, int, int, void*) { return fake::launch([] {}); }
int launch_force_bits(const NcPools&, int, const int32_t*, int, void*) { return fake::launch([] {}); }
int launch_input_firers(const NcPools&, bool, void*) { return fake::launch([] {}); }
int launch_potact(const NcPools&, int32_t, int32_t, int32_t, int64_t, float, float*, void*) { return fake::launch([] {}); }
int launch_last_fire(const NcPools&, int32_t, int32_t, int32_t, float, float*, void*) { return fake::launch([] {}); }
int launch_fill_words(uint32_t* a, int64_t count, uint32_t v, void*)
{
    return fake::launch([=] {
        for (int64_t k = 0; k < count; ++k) a[k] = v;
    });
}
int launch_detector_voltages(const NcPools& P, int32_t base, const int32_t* near, const int32_t* near_ptr, int32_t count,
                             float* out, void*)
{
    return fake::launch([=] {
        for (int32_t d = 0; d < count; ++d) {
            if (!fake::device_range(out + d, 4) || !fake::device_range(near_ptr + d, 8) || near_ptr[d] < 0 || near_ptr[d + 1] < near_ptr[d] ||
                !fake::device_range(near + near_ptr[d], 4 * (size_t)(near_ptr[d + 1] - near_ptr[d]))) {
                ++fake::faults;
                continue;
            }
            out[d] = 0.0f;
            for (int32_t k = near_ptr[d]; k < near_ptr[d + 1]; ++k) out[d] += P.pot[base + P.slot_of[base + near[k]]];
            out[d] /= (float)(near_ptr[d + 1] - near_ptr[d]);
        }
    });
}
int launch_gather(const float* src, const uint32_t* index, int64_t count, float* out, void*)
{
    if (fake::gathers_to_fail > 0 && fake::gathers_to_fail-- > 0) return -1;
    return fake::launch([=] {
        for (int64_t k = 0; k < count; ++k) {
            if (index[k] != ~0u && !fake::device_range(src + index[k], 4)) ++fake::faults;
            else out[k] = index[k] == ~0u ? std::numeric_limits<float>::quiet_NaN() : src[index[k]];
        }
    });
}
int launch_raster_bytes(const uint32_t* in, uint8_t* out, const int32_t*, int32_t n, int32_t n_words, int32_t rows, void*)
{
    return fake::launch([=] {
        const int32_t row = (n + 7) / 8;
        for (int32_t r = 0; r < rows; ++r) std::memcpy(out + (int64_t)r * row, in + (int64_t)r * n_words, (size_t)row);
    });
}
int build_knn_device(int32_t, int32_t, float, uint64_t, const nc_params&, nc_net*, std::string&) { return NC_ERR_UNSUPPORTED; }
}  // namespace nc
