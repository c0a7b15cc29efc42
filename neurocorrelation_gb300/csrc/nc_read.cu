// nc_read.cu — read-back kernels: device state (slot and CSC order) into the caller's
// order, in a device buffer that one copy takes to the caller's memory.
//
// Before, every read-back copied the state as it lies and reordered it on the host, a
// random read per element: 35 ms for the weights of 10M synapses and 23 ms for the
// potentials and activities of 2M neurons, against 0.3 ms for the copies alone on this
// machine (pageable host memory over C2C).  A gather on the device moves a 32-byte sector
// per element at HBM speed.
#include "nc_engine.cuh"

#include <cuda_runtime.h>

namespace {

constexpr int kThreads = 256;

// The read-backs are programmatic dependent launches: they are scheduled while the step (or
// flush) before them drains, and wait here before they read anything (a step and two
// read-backs of three neurons 39.4 -> 36.3 us).
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
int launch_dependent(void (*fn)(P...), dim3 grid, void* stream, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, fn, args...) != cudaSuccess) return -1;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

unsigned blocks_for(int64_t items) { return (unsigned)((items + kThreads - 1) / kThreads); }

// out[k] = src[index[k]]; NaN where the index is ~0 (a synapse that was not kept).
__global__ void k_gather(const float* src, const uint32_t* index, int64_t count, float* out)
{
    wait_previous();
    const int64_t k = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (k >= count) return;
    const uint32_t c = __ldg(index + k);
    out[k] = c == ~0u ? __int_as_float(0x7fc00000) : src[c];
}

// [potential, activity] of every neuron in the caller's order.  Activity:
// setActivity(firings/(((float) currentT-activityStartTime)/10.0)) at the last update
// (src/NeuCor.cpp:640), 0 before the first one.
__global__ void k_potact(const float* pot, const uint32_t* firings, const int32_t* start, const int32_t* slot_of,
                         int32_t n, int64_t t, float dt, float2* out)
{
    wait_previous();
    const int32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const int32_t s = __ldg(slot_of + i);
    float act = 0.0f;
    const int32_t from = start[s];
    if (t >= 1 && t > from) {
        const float ms = __fsub_rn(__fmul_rn((float)t, dt), __fmul_rn((float)from, dt));
        act = __double2float_rn(__ddiv_rn((double)firings[s], __ddiv_rn((double)ms, 10.0)));
    }
    out[i] = make_float2(pot[s], act);
}

// Last fire of every neuron in ms, NaN for none, in the caller's order.
__global__ void k_last_fire(const int32_t* lf, const int32_t* slot_of, int32_t n, float dt, float* out)
{
    wait_previous();
    const int32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    const int32_t t = lf[__ldg(slot_of + i)];
    out[i] = t == NC_NEVER ? __int_as_float(0x7fc00000) : __fmul_rn((float)t, dt);
}

// Raster rows of n_words words in slot order to rows of row_bytes bytes in the caller's
// order: a thread takes one byte of kRows rows, so a neuron's slot is read once for them.
constexpr int kRows = 8;
__global__ void k_raster_bytes(const uint32_t* in, uint8_t* out, const int32_t* slot_of, int32_t n, int32_t n_words,
                               int32_t row_bytes, int32_t rows)
{
    wait_previous();
    const int32_t b = blockIdx.x * kThreads + threadIdx.x;
    if (b >= row_bytes) return;
    const int32_t r0 = blockIdx.y * kRows;
    int32_t slot[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) slot[k] = 8 * b + k < n ? __ldg(slot_of + 8 * b + k) : -1;
    for (int32_t r = r0; r < min(rows, r0 + kRows); ++r) {
        const uint32_t* row = in + (int64_t)r * n_words;
        uint32_t v = 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (slot[k] >= 0) v |= ((row[slot[k] >> 5] >> (slot[k] & 31)) & 1u) << k;
        out[(int64_t)r * row_bytes + b] = (uint8_t)v;
    }
}

}  // namespace

namespace nc {

int launch_gather(const float* src, const uint32_t* index, int64_t count, float* out, void* stream)
{
    if (count <= 0) return 0;
    return launch_dependent(k_gather, dim3(blocks_for(count)), stream, src, index, count, out);
}

int launch_potact(const NcPools& P, int32_t neuron_base, int32_t first, int32_t n, int64_t t, float dt, float* out, void* stream)
{
    if (n <= 0) return 0;
    return launch_dependent(k_potact, dim3(blocks_for(n)), stream, (const float*)(P.pot + neuron_base),
                            (const uint32_t*)(P.firings + neuron_base), (const int32_t*)(P.act_start + neuron_base),
                            (const int32_t*)(P.slot_of + neuron_base + first), n, t, dt, (float2*)out);
}

int launch_last_fire(const NcPools& P, int32_t neuron_base, int32_t first, int32_t n, float dt, float* out, void* stream)
{
    if (n <= 0) return 0;
    return launch_dependent(k_last_fire, dim3(blocks_for(n)), stream, (const int32_t*)(P.lf + neuron_base),
                            (const int32_t*)(P.slot_of + neuron_base + first), n, dt, out);
}

int launch_raster_bytes(const uint32_t* in, uint8_t* out, const int32_t* slot_of, int32_t n, int32_t n_words,
                        int32_t rows, void* stream)
{
    const int32_t row_bytes = (n + 7) / 8;
    if (row_bytes <= 0) return 0;
    // (a grid's second dimension is at most 65,535)
    for (int32_t r = 0; r < rows; r += 65535 * kRows) {
        const int32_t m = rows - r < 65535 * kRows ? rows - r : 65535 * kRows;
        if (launch_dependent(k_raster_bytes, dim3(blocks_for(row_bytes), (unsigned)((m + kRows - 1) / kRows)), stream,
                             in + (int64_t)r * n_words, out + (int64_t)r * row_bytes, slot_of, n, n_words, row_bytes, m))
            return -1;
    }
    return 0;
}

}  // namespace nc
