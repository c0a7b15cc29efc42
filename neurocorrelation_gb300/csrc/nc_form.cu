// nc_form.cu — switching a single network between the two forms of the step kernels
// (NC_STEP_AUTO).  Both forms keep the same neuron state, weights, captured charges and
// fired bitsets; they differ in how a synapse's last launch and arrival are kept:
//   dense form  state[c]     per in-synapse (CSC order): the accepted arrival and its
//                            distance from the one before (nc_state_age);
//   event form  last_arr[k]  per out-synapse (CSR order) and t_arr[c] per in-synapse, plus
//                            the ring bits of the spikes still needed by a fold (arrived
//                            t-KC .. t-1) or in flight.
// A switch happens between steps, after the current form's plasticity flush (every
// launch and every plasticity update of step t-1 done, stdp_done = t-1); the next step
// t then skips its deferred part in either form, so the conversion below is all that
// changes.  An arrival that no longer matters (NC_AGE_OLD) becomes "never" and back.
#include "nc_engine.cuh"

#include <cuda_runtime.h>

namespace {

// Dense -> event: last_arr and t_arr of every synapse from its state, and the ring bits of
// the spikes that arrived t-KC .. t-1 or arrive later (the ring was cleared before).
__global__ void k_form_to_event(NcPools P, int net)
{
    const NcNetDesc& D = P.nets[net];
    const int32_t prev = D.t - 1, kc = D.kc;
    const int64_t sb = D.syn_base;
    uint32_t* ring = P.ring + D.ring_base;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < D.n_syn; k += (int64_t)gridDim.x * blockDim.x) {
        const NcOut o = P.out[sb + k];
        const int64_t c = sb + o.csc;
        const uint32_t s = P.state[c];
        const int32_t age = D.wide ? prev - (int32_t)s : nc_state_age(s, prev);
        // steps since the last arrival: the plasticity of prev is done
        const int32_t since = age >= 0 ? age : (D.wide ? prev - (int32_t)P.state[D.wide + c] : age + (int32_t)(s & 0xffffu));
        const int32_t old = D.wide ? prev - NC_WIDE_NEVER : NC_AGE_OLD;
        P.last_arr[sb + k] = age >= old ? NC_NEVER : prev - age;
        P.t_arr[c] = since >= old ? NC_NEVER : prev - since;
        if (age < kc) {
            atomicOr(ring + (int64_t)((prev - age) & D.ring_mask) * D.ring_words + (o.ringpos >> 5),
                     1u << (o.ringpos & 31));
        }
    }
}

// Event -> dense: the state of every synapse from its last_arr and t_arr.
__global__ void k_form_to_dense(NcPools P, int net)
{
    const NcNetDesc& D = P.nets[net];
    const int32_t prev = D.t - 1;
    const int64_t sb = D.syn_base;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < D.n_syn; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = sb + P.out[sb + k].csc;
        const int32_t la = P.last_arr[sb + k], ta = P.t_arr[c];
        if (D.wide) {
            P.state[c] = (uint32_t)(la == NC_NEVER ? NC_WIDE_NEVER : la);
            P.state[D.wide + c] = (uint32_t)(ta == NC_NEVER ? NC_WIDE_NEVER : ta);
            continue;
        }
        // the arrival before an accepted one still on its way is the last arrival
        const int32_t age = la == NC_NEVER || prev - la > NC_AGE_OLD ? NC_AGE_OLD : prev - la;
        const int32_t since = ta == NC_NEVER || prev - ta > NC_AGE_OLD ? NC_AGE_OLD : prev - ta;
        P.state[c] = nc_state_word(prev, age, age < 0 ? since - age : 0);
    }
}

int grid_for(int64_t items, int per_block)
{
    const int64_t b = (items + per_block - 1) / per_block;
    return (int)(b < 1 ? 1 : (b > 65536 ? 65536 : b));
}

}  // namespace

namespace nc {

int launch_form_to_event(const NcPools& P, int net, int64_t n_syn, int64_t ring_words, void* stream)
{
    const cudaStream_t s = (cudaStream_t)stream;
    if (cudaMemsetAsync(P.ring, 0, sizeof(uint32_t) * (size_t)ring_words, s) != cudaSuccess) return -1;
    k_form_to_event<<<grid_for(n_syn, 256), 256, 0, s>>>(P, net);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_form_to_dense(const NcPools& P, int net, int64_t n_syn, void* stream)
{
    const cudaStream_t s = (cudaStream_t)stream;
    k_form_to_dense<<<grid_for(n_syn, 256), 256, 0, s>>>(P, net);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace nc
