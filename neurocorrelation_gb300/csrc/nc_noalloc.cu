// nc_noalloc.cu — nc_run_noalloc (neucor_gb300.h): the simulation step for callers
// that cannot let the library allocate device memory once their network is set up.
//
// Some callers own every byte of device memory themselves: a simulation service that
// reserves a fixed budget per GPU up front and admits work against it, or a host
// program (a renderer, a game or robotics engine embedding the simulator) whose own
// allocator has carved up the GPU.  A cudaMalloc made behind their back can fail when
// the memory is spoken for, or silently break their accounting.  nc_run instantiates
// CUDA graphs (which allocate) on first use; nc_run_noalloc launches the same kernels
// directly.  Nothing is allocated: the network's own arrays are the inputs and outputs,
// and no kernel needs scratch.
#include <cuda_runtime.h>

#include <string>

#include "nc_net.h"

extern "C" int nc_run_noalloc(nc_net* net, int32_t n_steps, void* stream)
{
    if (!net) return nc::set_last_error(NC_ERR_INVALID, "null handle");
    if (n_steps < 0) return nc::set_last_error(NC_ERR_INVALID, "negative step count");
    if (net->step + n_steps >= (1ll << 30)) return nc::set_last_error(NC_ERR_INVALID, "step counter limit reached");
    cudaError_t e = cudaSetDevice(net->eng.device);
    if (e != cudaSuccess) return nc::set_last_error(NC_ERR_CUDA, nc::cuda_msg("cudaSetDevice", e));
    cudaStream_t s = stream ? (cudaStream_t)stream : net->eng.stream;
    // (the size of a scratch array that the event form once needed; callers are promised the refusal)
    if (!net->eng.dense && net->host.n > NC_NOALLOC_MAX_NEURONS)
        return nc::set_last_error(NC_ERR_INVALID, "nc_run_noalloc serves event-form networks of at most " +
                                                      std::to_string(NC_NOALLOC_MAX_NEURONS) + " neurons; this one has " +
                                                      std::to_string(net->host.n) + " (use nc_run)");
    for (int32_t k = 0; k < n_steps; ++k)
        if (net->eng.launch_tick(s))
            return nc::set_last_error(NC_ERR_CUDA, nc::cuda_msg("nc_run_noalloc launch", cudaGetLastError()));
    net->step += n_steps;
    for (int32_t k = 0; k < n_steps; ++k) net->time = net->time + net->host.dt;
    // the launches above are not tracked by the handle once issued: later calls on the
    // handle read the step counter and simulated time back from the device
    net->counters_on_device = true;
    net->eng.steps_unseen();
    return NC_OK;
}
