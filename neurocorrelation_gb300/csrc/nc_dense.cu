// nc_dense.cu — the dense form of the NeuCor step: one kernel per step.
//
// The event form (nc_kernels.cu) pushes every launched spike from its source into the
// target's CSC row: scattered writes and ring atomics per synaptic event.  When a large
// share of neurons fires every step (the kNN / U[0,1]-weight networks saturate near one
// fire per refractory period), nearly every in-row is touched every step anyway, and
// streaming the rows in order is cheaper than scattering into them.
//
//   k_dense_step, step t, prev = t-1: a block works through the tiles (up to 32
//   consecutive neurons and their in-rows) of its even share of the quads; its last warp
//   is the neuron warp, the others stream.
//     rows (neuron warp): whether each neuron fired at prev, and the weight change an
//       arrival at prev makes (its trace at prev), into shared memory;
//     synapses (stream warps), a quad (four positions of one row) per thread: Synapse::fire
//       of those whose source fired at prev (src/NeuCor.cpp:727-738): dropped while busy,
//       otherwise it captures deltaT * fl(fl(0.2f*52)*w) and its arrival; the plasticity of
//       prev (src/NeuCor.cpp:740-761): post-spike branch on the rows of neurons that fired
//       at prev, arrival branch on synapses whose spike arrived at prev; and four window
//       bits, "arrived in t-KC .. t-1", into a byte of shared memory;
//     neurons (neuron warp, while the others stream the next tile): charge_insynapses in
//       ascending source order from the window bits, charge_passive, threshold, AP, input
//       requests and background draws, fired bits.
//   The kernel boundary between two steps is the only point where neurons meet: the
//   fired bits of t are read by the tiles of t+1.
//   k_dense_fused: several steps in one cooperative launch, a grid barrier after each
//   (batched engines).
//
// Launches of the fires of prev happen at the start of step t instead of the end of
// step prev; nothing between those points reads what they write (a spike launched at
// prev arrives at t at the earliest and joins the fold from t+1), so the results are the
// event form's bit for bit.  The launch decision reads the same rule: accepted iff
// prev - last_arrival >= KC + [target caller id > source caller id], and the captured
// weight includes the target's post-spike plasticity of prev when the target fired at
// prev and its caller id is below the source's.  A flush (before read-back) streams
// early; the step then finds it done (stdp_done) and only gathers the window bits.
//
// What bounds it, and why this shape.  The step streams 12.25 bytes a synapse (key, state,
// weight; a row byte per quad) and writes what changed; on networks past the L2 cache that
// is 23 bytes a synapse of DRAM traffic at 5.8 TB/s (2M x 200: 2,815 -> 1,597 us a step),
// on smaller ones instruction issue and, below some 10k neurons, the chain of dependent
// loads and the boundary between two launches.  The two passes before it (synapses, then
// neurons) read 22 bytes a synapse, took 184 warp instructions per 32 synapses against 75,
// and exchanged window bits, captured terms and traces through memory.  100k x 100: 92 -> 45
// us; 1k x 50: 18.0 -> 6.6; 20k x 100 with inhibitory synapses: 45.8 -> 19; 30k x 73 at dt
// 0.5: 33 -> 14.8.
//   - Rows padded to quads: a thread's four synapses share their target's values, and move
//     with one 16-byte access per array; every eighth row ends on a 128-byte line.
//   - A run of 8 neurons with more quads than two blocks' shares is split over several blocks;
//     the last of them to be done with its part updates the neurons (100k x 10 with one row of
//     99,999 in-synapses 176 -> 18 us, with inhibitory synapses 373 -> 49; 200k x 25 with skewed
//     rows 152 -> 47).
//   - A warp of its own sums, so the others never wait for a sum: with block barriers
//     between the two halves the 100k x 100 step took 78 us (48 then).
//   - 96 threads (two stream warps to a neuron warp), 80 registers, 8 blocks an SM, the
//     rest of shared memory left to the L1 (all of it for shared memory: 57 -> 66 us).
//     128 threads: 49 us against 48, and 19.6 against 16.5 on 30k x 73, whose shares get
//     uneven; 64 registers spill (60 us).
#include "nc_device.cuh"
#include "nc_engine.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <vector>

namespace {

using namespace nc_dev;

constexpr int kMaxThreads = 256;
// Quads whose window bits fit in the block's shared memory (a tile of 32 rows of 256
// synapses); a tile with more keeps them in its slice of NcPools::nib.
constexpr int kNibCap = 2048;
// Quads under way per thread, the current one included (cp.async into the thread's own
// slots of shared memory).  Two leave the memory idle (400k x 100: 215 us a step against
// 180), four take L1 from the gathers of fired bits (188).
constexpr int kRing = 3;
// Quads of a tile whose captured charges fit in a block's shared memory beside the ring.
constexpr int kStageQuads = 640;

// What a step's tiles are: whole; whole, one to a block, with their captured charges staged in
// shared memory (NcPools::stage); some of them split over blocks (NcPools::split).  Kernels of
// their own: the step's 80 registers hold one kind.
enum Kind { kWhole, kStaged, kSplit };

struct RowState {
    float chg;      // weight change of an arrival at prev, before the clamp
    uint32_t tf;    // bit 0: the neuron fired at prev; bit 1: its sum counts (it is out of its AP)
};

struct BlockShared {
    RowState row[2][NC_TILE_ROWS];               // of two tiles: one streamed, one summed
    __align__(16) uint8_t nib[2][kNibCap];       // window bits of their quads
    int ok;
};

constexpr int kRingBytes = kRing * (3 * 16 + 4);  // dynamic shared memory per stream thread
size_t dyn_bytes(int threads, bool stage) { return (size_t)threads * kRingBytes + (stage ? 16 * kStageQuads : 0); }

// Named barriers between the neuron warp and the stream warps, two of each: `ready` once a
// tile's rows are in shared memory and its window bits may be written, `full` once they are.
// (Constant ids: with an id in a register a block reserves all 16 barriers, and an SM then
// holds 4 blocks.)
template <int kId>
__device__ __forceinline__ void bar_sync_id()
{
    asm volatile("bar.sync %0, %1;" ::"n"(kId), "r"(blockDim.x) : "memory");
}
template <int kId>
__device__ __forceinline__ void bar_arrive_id()
{
    asm volatile("bar.arrive %0, %1;" ::"n"(kId), "r"(blockDim.x) : "memory");
}
template <int kId>
__device__ __forceinline__ void bar_sync(int b)  // barrier kId + b, b = 0 or 1
{
    if (b) bar_sync_id<kId + 1>();
    else bar_sync_id<kId>();
}
template <int kId>
__device__ __forceinline__ void bar_arrive(int b)
{
    if (b) bar_arrive_id<kId + 1>();
    else bar_arrive_id<kId>();
}
constexpr int kBarReady = 1, kBarFull = 3;

// Programmatic dependent launch: a step's blocks may be scheduled while the previous step
// drains; they read what no step writes, and wait here for the rest until it has
// completed and its writes are visible.  (A kernel launched without the attribute passes
// the wait at once.)
__device__ __forceinline__ void wait_previous_step() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next step's blocks be scheduled as this one's leave (it waits in turn).
__device__ __forceinline__ void release_next_step() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void async16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// The same, into L2 lines that are evicted after the others (`policy`).
__device__ __forceinline__ void async16_kept(uint32_t dst, const void* src, uint64_t policy)
{
    asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy)
                 : "memory");
}
__device__ __forceinline__ uint64_t keep_half()
{
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 0.5;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void async4(uint32_t dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// waits for all but the kRing groups committed last, and for all
__device__ __forceinline__ void async_wait_first() { asm volatile("cp.async.wait_group %0;" ::"n"(kRing) : "memory"); }
__device__ __forceinline__ void async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 2) : "memory"); }

// *p where `in` is not zero, -0.0 elsewhere: a predicated load, so that nothing waits for the
// value before it is used.  kShared: p points into shared memory.
template <bool kShared>
__device__ __forceinline__ float load_or_absent(const float* p, uint32_t in)
{
    float v;
    if (kShared)
        asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.f32 %0, 0f80000000;\n\t@q ld.shared.f32 %0, [%1];\n\t}"
            : "=f"(v)
            : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(in));
    else
        asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.f32 %0, 0f80000000;\n\t@q ld.global.f32 %0, [%1];\n\t}"
            : "=f"(v)
            : "l"(p), "r"(in));
    return v;
}

// The window bits of one row, taken eight at a time.  nib: the tile's window bits, four to a
// byte; q0, nq: the row's quads; x0: the tile's captured charges.  Eight bytes are packed to a
// word of 32 synapses; a batch looks at the 32 from the first bit left on, across words.
template <bool kShared>
struct WindowBits {
    const unsigned long long* words;
    const float* x;        // charge of the first bit of `cur`
    uint32_t cur, nxt;
    int from;              // first bit left, 0..31
    int w, nw;             // next word to read, words
    uint32_t last;
    __device__ __forceinline__ uint32_t word()
    {
        uint32_t v = 0u;
        if (w < nw) {
            const unsigned long long b = words[w++];
            const uint32_t lo = (uint32_t)b, hi = (uint32_t)(b >> 32);
            v = __byte_perm(lo | lo >> 4, hi | hi >> 4, 0x6420);
            if (w == nw) v &= last;
        }
        return v;
    }
    __device__ __forceinline__ WindowBits(const uint8_t* nib, int q0, int nq, const float* x0)
    {
        const int skip = (int)((uintptr_t)(nib + q0) & 7);  // quads of the first word before the row
        words = (const unsigned long long*)(nib + q0 - skip);
        x = x0 + 4 * (int64_t)(q0 - skip);
        w = 0;
        nw = (skip + nq + 7) >> 3;
        last = ((skip + nq) & 7) ? (1u << (4 * ((skip + nq) & 7))) - 1u : ~0u;
        from = 0;
        cur = word() & (~0u << (4 * skip));
        nxt = word();
    }
    // The charges of the next eight bits, absent ones as -0.0; whether there are any.  (All
    // branches come first, so that the rest runs between the terms of a sum.)
    __device__ __forceinline__ bool next(float (&to)[8])
    {
        uint32_t m;
        while (true) {
            m = from < 32 ? __funnelshift_r(cur, nxt, from) : 0u;
            if (m != 0u || !(nxt | (uint32_t)(w < nw))) break;
            if (from >= 32) from -= 32;
            cur = nxt;
            nxt = word();
            x += 32;
        }
        const bool any = m != 0u;
        const float* xm = x + from;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            to[k] = load_or_absent<kShared>(xm + __ffs((int)m) - 1, m);
            m &= m - 1u;
        }
        from += m ? __ffs((int)m) - 1 : 32;
        return any;
    }
    // The same for windows of few bits: the next eight wherever they lie, a branch at each.
    __device__ __forceinline__ bool next_of_few(float (&to)[8])
    {
        bool any = false;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            uint32_t m = from < 32 ? cur >> from : 0u;
            while (m == 0u && (nxt | (uint32_t)(w < nw))) {
                cur = nxt;
                nxt = word();
                x += 32;
                from = 0;
                m = cur;
            }
            const int b = from + __ffs((int)m) - 1;
            to[k] = load_or_absent<kShared>(x + b, m);
            any = any || m != 0u;
            from = m ? b + 1 : 32;
        }
        return any;
    }
};

// charge_insynapses (src/NeuCor.cpp:688-700) of one row: the terms of the spikes that
// arrived t-1 .. t-KC, in ascending source id, folded into pot.  x0: the tile's charges, in
// global memory or (kShared) staged in shared memory by the stream warps, which copy those of
// quads with window bits behind their own work: a batch then waits for its bits and its sum,
// not for L2 as well.  The bits are streamed in
// batches of 8 terms across word boundaries, so that a warp's batch count is its busiest
// lane's, not a sum of per-word maxima.  A batch takes some 1,100 cycles, a gather from L2 and a
// serial sum; with the bits of 64-bit words taken one by one, and a branch at each for the next
// word, it took 2,500, and 20k x 100 with inhibitory synapses 25.8 us a step (21.7 now).  A
// batch gathered ahead of the sum gains half a microsecond where sums are long and costs 2 to
// 5% where they stop early (more registers, and charges that are not needed).
//
// When no term of the net can be negative (nonneg_terms), the running sum only grows
// (each `float += double` rounds a larger value, and rounding keeps the order), and so
// does charge_passive's result.  Once that result crosses the threshold the neuron fires
// whatever the remaining terms are, and its potential is then replaced by the AP table
// (src/NeuCor.cpp:682-686, 706-714): the fold stops there and returns the partial sum,
// which leads the update to the same decision.
template <bool kShared, bool kFew = false>
__device__ __forceinline__ float fold_row(const uint8_t* nib, int q0, int nq, const float* x0, float pot, float leak,
                                          const TermFactor& F, bool stop)
{
    if (nq <= 0) return pot;
    WindowBits<kShared> at(nib, q0, nq, x0);
    float xv[8];
    while (kFew ? at.next_of_few(xv) : at.next(xv)) {
        pot = fold_terms(pot, xv, F);
        if (stop && fires_at(pot, leak)) break;
    }
    return pot;
}

// fold_row by a whole warp (all lanes call, with the same values, and get the sum), for rows
// long enough to be split over blocks: the window bits of 1,024 synapses at a time are listed in
// shared memory (`list`, 1,024 entries) and the charges gathered 32 at once, so that empty
// stretches cost a load per 1,024 synapses and a term its place in the sum alone.  One lane took
// 188 us for a row of 100k in-synapses of which 600 were in the window.
__device__ __noinline__ float fold_long_row(const uint8_t* nib, int64_t q0, int nq, const float* x, float pot, float leak,
                                            float hi, float lo, double e_term, bool stop, uint16_t* list)
{
    const int lane = threadIdx.x & 31;
    const int skip = (int)((uintptr_t)(nib + q0) & 7);  // quads of the first word before the row
    const unsigned long long* words = (const unsigned long long*)(nib + q0 - skip);
    const int nw = (skip + nq + 7) >> 3;
    x += 4 * (q0 - skip);
    const TermFactor F{hi, lo, e_term};
    unsigned long long next = lane < nw ? __ldcg(words + lane) : 0ull;
    for (int w0 = 0; w0 < nw; w0 += 32, x += 1024) {
        const int w = w0 + lane;
        const uint32_t b0 = (uint32_t)next, b1 = (uint32_t)(next >> 32);
        uint32_t m = __byte_perm(b0 | b0 >> 4, b1 | b1 >> 4, 0x6420);
        if (w == 0) m &= ~0u << (4 * skip);
        if (w == nw - 1 && ((skip + nq) & 7)) m &= (1u << (4 * ((skip + nq) & 7))) - 1u;
        if (w >= nw) m = 0u;
        next = w + 32 < nw ? __ldcg(words + w + 32) : 0ull;
        int at = __popc(m);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, at, o);
            if (lane >= o) at += y;
        }
        const int total = __shfl_sync(kFull, at, 31);
        for (at -= __popc(m); m; m &= m - 1u) list[at++] = (uint16_t)(32 * lane + __ffs((int)m) - 1);
        __syncwarp();
        for (int k0 = 0; k0 < total; k0 += 32) {
            const float xv = k0 + lane < total ? x[list[k0 + lane]] : -0.0f;
            for (int k = 0; k < min(32, total - k0); k += 8) {
                float t[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) t[u] = __shfl_sync(kFull, xv, k + u);
                pot = fold_terms(pot, t, F);
                if (stop && fires_at(pot, leak)) return pot;
            }
        }
        __syncwarp();
    }
    return pot;
}

// The sums of a split tile, whose window bits lie in global memory (all lanes call): lane j's row is the
// nq quads (0: no sum) from q0 on.  A few long rows are summed one after the other, by the whole
// warp, which takes half as long for a term; rows of much the same length side by side, a lane
// each, from shared memory (`buf`, kNibCap bytes) that the warp fills a piece of every row at a
// time (one word after the other from L2: 160 us in the case below).
__device__ __noinline__ float fold_split_rows(const uint8_t* nib, const float* x, int64_t q0, int nq, float pot, float leak,
                                             float hi, float lo, double e_term, bool stop, uint8_t* buf)
{
    const int lane = threadIdx.x & 31;
    const int longest = __reduce_max_sync(kFull, nq), all = __reduce_add_sync(kFull, nq);
    if (all <= 2 * longest) {
        for (unsigned todo = __ballot_sync(kFull, nq > 0); todo; todo &= todo - 1u) {
            const int j = __ffs((int)todo) - 1;
            const float sum = fold_long_row(nib, __shfl_sync(kFull, q0, j), __shfl_sync(kFull, nq, j), x,
                                            __shfl_sync(kFull, pot, j), leak, hi, lo, e_term, stop, (uint16_t*)buf);
            if (lane == j) pot = sum;
        }
        return pot;
    }
    const TermFactor F{hi, lo, e_term};
    uint8_t* lane_of = buf + kNibCap - 32;  // the lanes of the rows left
    unsigned todo;
    for (int done = 0, piece; (todo = __ballot_sync(kFull, nq > done)) != 0u; done += piece) {
        // a row's piece, with up to 7 quads before it in its first word
        // (a short one first: most sums of a busy network stop in it)
        const int rows = __popc(todo), stride = min((kNibCap - 32) / rows & ~7, done || !stop ? kNibCap : 56);
        const int words = stride >> 3, total = words * rows;
        piece = stride - 8;
        const int64_t at = q0 + done;
        const int skip = (int)((uintptr_t)(nib + at) & 7), mine = __popc(todo & ((1u << lane) - 1u));
        if (nq > done) lane_of[mine] = (uint8_t)lane;
        __syncwarp();
        int bits = 0;
        for (int k0 = 0; k0 < total; k0 += 128) {
            unsigned long long v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = min(k0 + 32 * u + lane, total - 1), row = lane_of[k / words], w = k % words;
                const int64_t from = __shfl_sync(kFull, at - skip, row);
                const int left = __shfl_sync(kFull, skip + nq - done, row);
                v[u] = 8 * w < left ? __ldcg((const unsigned long long*)(nib + from) + w) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = k0 + 32 * u + lane;
                if (k < total) *((unsigned long long*)buf + k) = v[u];
                if (k < total) bits += __popcll(v[u]);
            }
        }
        // a batch looks at 32 synapses: with fewer than 3 of each in the window, the next eight are
        // looked for instead (every neuron of 3,000 driving every other, inhibitory, quiet: 83 -> 73
        // us a step, 120 with the rows whole)
        const bool few = __reduce_add_sync(kFull, bits) < 3 * total;
        __syncwarp();
        if (nq > done) {
            const uint8_t* row = buf + stride * mine + skip;
            const int n = min(piece, nq - done);
            pot = few ? fold_row<false, true>(row, 0, n, x + 4 * at, pot, leak, F, stop)
                      : fold_row<false>(row, 0, n, x + 4 * at, pot, leak, F, stop);
            if (stop && fires_at(pot, leak)) nq = 0;
        }
        __syncwarp();
    }
    return pot;
}

// Whether this block is the last of those that stream the parts of a split tile (the neuron
// warp calls, after its stream warps have arrived): it updates the neurons, the others' window
// bits are there to read.
__device__ __forceinline__ bool last_part(const NcPools& P, int32_t part, int lane)
{
    unsigned n = 0u;
    if (lane == 0) {
        uint32_t* ctr = P.split_ctr + (part & 0xffff) - 1;
        __threadfence();
        n = atomicAdd(ctr, 1u) + 1u;
        if (n == (unsigned)part >> 16) *ctr = 0u;
        __threadfence();
    }
    __syncwarp();  // what lane 0 has seen, all lanes read
    return __shfl_sync(kFull, n, 0) == (unsigned)part >> 16;
}

// What a net's quads share.
struct TileConst {
    const uint32_t* fprev;   // fired bits of prev
    const float* tab_pre;    // presynaptic trace table
    int32_t tab_pre_len;
    int32_t prev, kc;
    int32_t key_shift;
    float dt, c52;
    float post0;             // postsynaptic factor * 0: the absent trace of a post-spike update
    float pre, lr;
    bool refresh;            // set old ages back in this step (NC_AGE_PERIOD)
    int64_t wide;
};

// Quad Q (pool index) of a row: launches and plasticity of prev.  Returns the
// quad's window bits.  Branches are per quad (the row fired; something to store); the four
// synapses run side by side on selects, so that their gathers are under way together.
// f: bit 0 of each, its source fired at prev.  kInh: the net has inhibitory synapses.
template <bool kWide, bool kInh>
__device__ __forceinline__ uint32_t quad_update(const NcPools& P, const TileConst& C, uint32_t Q, const RowState row,
                                                const uint4 key, const uint4 st, const uint4 w, const uint32_t (&f)[4],
                                                unsigned& nl, unsigned& nf)
{
    uint32_t h[4], s[4] = {st.x, st.y, st.z, st.w}, bf[4];
    const uint32_t k[4] = {key.x, key.y, key.z, key.w};
    const float w0[4] = {__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w)};
    if (kWide) {
        const uint4 hi4 = __ldg((const uint4*)(P.key + C.wide) + Q);
        const uint4 before4 = *((const uint4*)(P.state + C.wide) + Q);
        h[0] = hi4.x, h[1] = hi4.y, h[2] = hi4.z, h[3] = hi4.w;
        bf[0] = before4.x, bf[1] = before4.y, bf[2] = before4.z, bf[3] = before4.w;
    }
    const uint32_t dmask = kWide ? ~0u : (1u << C.key_shift) - 1u;
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (!kWide) h[u] = k[u];
    // steps since the accepted arrival, negative while the spike travels
    int32_t age[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) age[u] = kWide ? C.prev - (int32_t)s[u] : nc_state_age(s[u], C.prev);
    float lo[4], hi[4], w1[4], w2[4], cap[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const bool inh = kInh && (h[u] & NC_KEY_INH) != 0u;
        lo[u] = inh ? -1.0f : 0.0f;
        hi[u] = inh ? 0.0f : 1.0f;
        w1[u] = cap[u] = w0[u];
    }
    if (row.tf & 1u) {
        // post-spike branch: the trace since the last arrival before prev
        float tr[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int32_t since =
                age[u] > 0 ? age[u] : (kWide ? C.prev - (int32_t)bf[u] : age[u] + (int32_t)(s[u] & 0xffffu));
            tr[u] = since < C.tab_pre_len ? __ldg(C.tab_pre + since) : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            w1[u] = clamp_weight(w0[u] + (C.pre * tr[u] - C.post0) * C.lr, lo[u], hi[u]);
            // target below the source in caller order: its update of prev ran before the launch
            if (h[u] & NC_KEY_BEFORE) cap[u] = w1[u];
        }
    }
    uint32_t win = 0u;
    bool arrived = false;
    const unsigned nl0 = nl;
    float* xq = P.x + 4 * (int64_t)Q;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const bool fs = f[u] & 1u;
        // free: prev - arrival >= KC + [target above source]
        const bool launch = fs && age[u] >= C.kc + (int32_t)(h[u] & NC_KEY_AFTER);
        const bool now = age[u] == 0;
        win |= (uint32_t)age[u] < (uint32_t)C.kc ? 1u << u : 0u;
        // arrival branch
        const float v = clamp_weight(w1[u] + row.chg, lo[u], hi[u]);
        w2[u] = now ? v : w1[u];
        // AP_depolFac = 0.2f; *= 52.0; *= weight  (src/NeuCor.cpp:729-731)
        if (launch) xq[u] = C.dt * (C.c52 * cap[u]);
        const int32_t d = (int32_t)((h[u] & dmask) >> NC_KEY_DELAY_SHIFT);
        if (kWide) {
            bf[u] = launch ? s[u] : bf[u];
            s[u] = launch ? (uint32_t)(C.prev + d) : s[u];
        } else {
            // nc_state_word(prev, -d, d + age)
            const uint32_t ns = (uint32_t)d * 65537u + (((uint32_t)C.prev << 16) + (uint32_t)age[u]);
            s[u] = launch ? ns : s[u];
        }
        arrived |= now;
        nl += launch ? 1u : 0u;
        nf += fs ? 1u : 0u;
    }
    if (!kWide && C.refresh) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (nc_state_age(s[u], C.prev) >= NC_AGE_LIMIT) s[u] = nc_state_word(C.prev, NC_AGE_OLD, 0);
    }
    if ((row.tf & 1u) || arrived) *((float4*)P.w + Q) = make_float4(w2[0], w2[1], w2[2], w2[3]);
    if (nl != nl0 || (!kWide && C.refresh)) {
        *((uint4*)P.state + Q) = make_uint4(s[0], s[1], s[2], s[3]);
        if (kWide) *((uint4*)(P.state + C.wide) + Q) = make_uint4(bf[0], bf[1], bf[2], bf[3]);
    }
    return win;
}

// This stream thread's slots of the ring: components apart, so that a warp's 16-byte
// accesses are contiguous; then the word that holds the quad's row byte.  (.ca copies: a
// .cg copy of 16 bytes per lane fetched every 32-byte sector twice.)  Weights and states are
// about to be written, so half of their lines ask L2 to evict others first: 100k x 100
// 48.2 -> 46.1 us a step, 400k x 100 181 -> 175, 2M x 200 1,640 -> 1,591 (all of them: 46.5,
// 175, 1,589; captures too, or keys marked to go first: slower on 2M).  What runs next finds
// its own data in L2 as fast as before after some 20 passes either way.
struct Ring {
    uint32_t quad;     // shared address of slot 0's key
    uint32_t part;     // bytes between components
    uint32_t row;      // shared address of slot 0's row word
    __device__ __forceinline__ Ring(unsigned char* dyn, uint32_t threads)
    {
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(dyn);
        part = 16u * threads;
        quad = base + 16u * threadIdx.x;
        row = base + kRing * 3u * part + 4u * threadIdx.x;
    }
    __device__ __forceinline__ uint4 load(int slot, int c) const
    {
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(quad + (slot * 3 + c) * part));
        return v;
    }
    __device__ __forceinline__ uint32_t load_row(int slot) const
    {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(row + slot * (part >> 2)));
        return v;
    }
    // the part of a quad that no step writes, and the part that steps write
    __device__ __forceinline__ void fetch_key(const NcPools& P, int slot, uint32_t Q) const
    {
        async16(quad + slot * 3 * part, (const uint4*)P.key + Q);
        async4(row + slot * (part >> 2), (const uint32_t*)P.qrow + (Q >> 2));
    }
    __device__ __forceinline__ void fetch_state(const NcPools& P, int slot, uint32_t Q) const
    {
        const uint32_t to = quad + slot * 3 * part;
        const uint64_t keep = keep_half();
        async16_kept(to + part, (const uint4*)P.state + Q, keep);
        async16_kept(to + 2 * part, (const uint4*)P.w + Q, keep);
    }
    __device__ __forceinline__ void fetch(const NcPools& P, int slot, uint32_t Q) const
    {
        fetch_key(P, slot, Q);
        fetch_state(P, slot, Q);
    }
};

// The tiles of a block that are due in a launch, in order: blocks take the plan's shares
// blockIdx.x, blockIdx.x + gridDim.x, ...  Every other launch goes through a share backwards
// (`back`, the caller's): what a step touched last is what the L2 cache still holds when the
// next one begins (100k x 100, 160 MB of arrays against 129 MB of L2: 53.4 -> 48.5 us a step).
// The plan is known before the launch's wait for the step before it; what is due only after
// (settle_first).
template <bool kFlush>
struct Tiles {
    const NcPools& P;
    int share, ti, begin, end;  // begin <= ti < end
    bool back;
    int single;  // one net: 1 when it is due, 0 when not; -1: several nets
    __device__ __forceinline__ static bool due_net(const NcNetDesc& D)
    {
        const int32_t t = D.t;
        return D.active && (kFlush ? t >= 2 && D.stdp_done < t - 1 : t <= D.t_end);
    }
    __device__ __forceinline__ Tiles(const NcPools& p, bool back_) : P(p), share(blockIdx.x), back(back_) { enter(); }
    __device__ __forceinline__ bool planned() const { return ti >= begin && ti < end; }
    __device__ __forceinline__ void settle_first()
    {
        single = P.n_nets == 1 ? (due_net(P.nets[0]) ? 1 : 0) : -1;
        settle();
    }
    __device__ __forceinline__ void enter()
    {
        begin = end = ti = 0;
        if (share >= P.row_blocks) return;
        begin = P.rstart[share];
        end = P.rstart[share + 1];
        ti = back ? end - 1 : begin;
    }
    // to the first due tile from ti on; ti = -1 past the last
    __device__ __forceinline__ void settle()
    {
        while (true) {
            if (share >= P.row_blocks || single == 0) {
                ti = -1;
                return;
            }
            if (planned()) {
                if (single > 0 || due_net(P.nets[P.rtiles[ti].net])) return;
                ti += back ? -1 : 1;
                continue;
            }
            share += gridDim.x;
            enter();
        }
    }
    __device__ __forceinline__ void next()
    {
        ti += back ? -1 : 1;
        settle();
    }
};

// Adds a stream warp's counts to its net's.
__device__ __forceinline__ void count_events(const NcNetDesc& D, unsigned nl, unsigned nf, int lane)
{
    nl = __reduce_add_sync(kFull, nl);
    nf = __reduce_add_sync(kFull, nf);
    if (lane == 0 && nl) atomicAdd(D.stats + 1, (unsigned long long)nl);
    if (lane == 0 && nf != nl) atomicAdd(D.stats + 2, (unsigned long long)(nf - nl));
}

// Fired words of prev of a quad's four sources, and their bits.
template <bool kWide>
__device__ __forceinline__ void fired_words(const TileConst& C, const uint4& key, uint32_t (&f)[4])
{
    const uint32_t k[4] = {key.x, key.y, key.z, key.w};
#pragma unroll
    for (int u = 0; u < 4; ++u) f[u] = C.fprev[kWide ? k[u] >> 5 : k[u] >> (C.key_shift + 5)];
}
template <bool kWide>
__device__ __forceinline__ void fired_bits(const TileConst& C, const uint4& key, uint32_t (&f)[4])
{
    const uint32_t k[4] = {key.x, key.y, key.z, key.w};
#pragma unroll
    for (int u = 0; u < 4; ++u) f[u] = __funnelshift_r(f[u], 0u, kWide ? k[u] : k[u] >> C.key_shift);  // (slot mod 32)
}

// The quads of one tile.  The block's quads of one net are consecutive, [run0, run0 + run):
// this thread takes every threads-th of them, from Q on in steps of `step`, whichever tiles
// they fall into (Q is left at its first past the tile), and keeps its next ones under way.
template <bool kFlush, bool kStage, bool kWide, bool kInh>
__device__ __forceinline__ void tile_synapses(const NcPools& P, const TileConst& C, uint32_t q0, uint32_t nq,
                                              uint32_t run0, uint32_t run, bool due, const RowState* row,
                                              uint32_t row0, uint8_t* nib, uint32_t stage, const Ring& ring, uint32_t step,
                                              uint32_t& Q, int& slot, uint32_t (&f)[4], unsigned& nl, unsigned& nf)
{
    for (; Q - q0 < nq; Q += step) {
        async_wait();
        const int ahead = slot + 1 == kRing ? 0 : slot + 1;
        const uint4 st = ring.load(slot, 1);
        uint32_t win = 0u;
        uint32_t sums = 0u;  // (staged) bit 1: the row's sum counts
        if (due) {
            const uint4 key = ring.load(slot, 0);
            uint32_t fired[4] = {f[0], f[1], f[2], f[3]};
            fired_bits<kWide>(C, key, fired);
            // the next quad's fired words while this one is worked on
            if (Q + step - run0 < run) fired_words<kWide>(C, ring.load(ahead, 0), f);
            const uint4 w = ring.load(slot, 2);
            const uint32_t rb = ring.load_row(slot) >> (8 * (Q & 3u));
            const RowState rs = row[(rb - row0) & 31u];
            if (kStage) sums = rs.tf;
            win = quad_update<kWide, kInh>(P, C, Q, rs, key, st, w, fired, nl, nf);
        } else {
            if (kStage) sums = row[((ring.load_row(slot) >> (8 * (Q & 3u))) - row0) & 31u].tf;
            const uint32_t s[4] = {st.x, st.y, st.z, st.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int32_t age = kWide ? C.prev - (int32_t)s[u] : nc_state_age(s[u], C.prev);
                win |= (uint32_t)age < (uint32_t)C.kc ? 1u << u : 0u;
            }
        }
        if (!kFlush) nib[Q] = (uint8_t)win;
        if (kStage && win && (sums & 2u)) async16(stage + 16u * (Q - q0), (const float4*)P.x + Q);
        // the slot has been read: refill it
        const uint32_t next = Q + kRing * step;
        if (next - run0 < run) ring.fetch(P, slot, next);
        async_commit();
        slot = ahead;
    }
}

// The stream warps' part of a step (or of the flush of the last one).
template <bool kFlush, bool kAlone, Kind kKind>
__device__ __forceinline__ void stream_role(const NcPools& P, BlockShared& sh, unsigned char* dyn, bool back)
{
    constexpr bool kStage = kKind == kStaged;
    const int lane = threadIdx.x & 31;
    const uint32_t threads = blockDim.x - 32;
    const Ring ring(dyn, threads);
    const uint32_t stage = kStage ? (uint32_t)__cvta_generic_to_shared(dyn) + kRingBytes * threads : 0u;
    Tiles<kFlush> at(P, back);
    TileConst C;
    int net = -1, share = -1, slot = 0;
    const uint32_t step = at.back ? 0u - threads : threads;
    uint32_t Q = 0u, run0 = 0u, run = 0u;
    uint32_t f[4] = {0u, 0u, 0u, 0u};  // fired words of this thread's next quad
    const uint32_t* fired = nullptr;   // the net's fired words, of even steps
    bool due = false, inh = false;
    unsigned nl = 0u, nf = 0u;  // launches, and synapses whose source fired
    // the run of consecutive quads that `tile` begins, and this thread's first one of it
    auto begin_run = [&](const NcRowTile& tile) {
        int other = at.back ? at.begin : at.end - 1;  // the run's last tile in this order
        while (P.rtiles[other].net != tile.net) other += at.back ? 1 : -1;
        const NcRowTile& last = P.rtiles[other];
        run0 = at.back ? last.q0 : tile.q0;
        run = (at.back ? tile.q0 + (uint32_t)tile.nq : last.q0 + (uint32_t)last.nq) - run0;
        // chunks of `threads` quads from run0 on, the last one short
        Q = run0 + threadIdx.x + (at.back && run ? (run - 1u) / threads * threads : 0u);
        if (at.back && Q - run0 >= run) Q -= threads;
    };
    // what no step writes of a net's descriptor
    auto begin_net = [&](int n) {
        net = n;
        const NcNetDesc& D = P.nets[n];
        inh = !D.nonneg_terms;
        fired = P.fired + D.word_base;
        C.tab_pre = P.tables + D.table_base;
        C.tab_pre_len = D.tab_pre_len;
        C.kc = D.kc;
        C.key_shift = D.key_shift;
        C.dt = D.dt;
        C.c52 = D.c52;
        C.pre = D.pre_factor;
        C.lr = D.lr;
        C.post0 = D.post_factor * 0.0f;
        C.wide = D.wide;
    };
    auto begin_step = [&](int32_t t, int32_t done) {
        C.prev = t - 1;
        due = C.prev >= 1 && done < C.prev;  // launches and plasticity of prev
        C.fprev = fired + (int64_t)(C.prev & 1) * P.total_words;
        C.refresh = C.prev % NC_AGE_PERIOD == 0;
    };
    // Before the wait: the first tile, its net's constants and its first keys.  After it the
    // step counter, the first states and the first fired words (of both parities, the counter
    // tells which) come side by side: one round trip to L2 instead of five, while the step
    // before drains (the sphere of 750 7.5 -> 6.5 us a step, 1k x 50 7.05 -> 6.7, 30k x 73 15.3
    // -> 14.7, 20k x 100 with inhibitory synapses 21.5 -> 20.7, 100k x 100 46.1 -> 45.0).
    const int first = at.planned() ? at.ti : -1;
    if (kAlone && first >= 0) {
        const NcRowTile tile = P.rtiles[first];
        begin_run(tile);
#pragma unroll 1
        for (int k = 0; k < kRing; ++k)
            if (Q + k * step - run0 < run) ring.fetch_key(P, k, Q + k * step);
        async_commit();
        begin_net(tile.net);
    }
    if (kAlone) {
        wait_previous_step();
        release_next_step();
    }
    if (kAlone && first >= 0) {
        const NcNetDesc& D = P.nets[net];
        const int32_t t = D.t, done = D.stdp_done;
#pragma unroll 1
        for (int k = 0; k < kRing; ++k) {
            if (Q + k * step - run0 < run) ring.fetch_state(P, k, Q + k * step);
            async_commit();
        }
        async_wait_first();
        if (Q - run0 < run) {
            uint32_t odd[4];
            const uint4 key = ring.load(0, 0);
            C.fprev = fired;
            if (C.wide) fired_words<true>(C, key, f);
            else fired_words<false>(C, key, f);
            C.fprev = fired + P.total_words;
            if (C.wide) fired_words<true>(C, key, odd);
            else fired_words<false>(C, key, odd);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (!(t & 1)) f[u] = odd[u];
        }
        begin_step(t, done);
        share = at.share;
    }
    at.settle_first();
    if (kAlone && first >= 0 && (at.ti != first || at.share != share)) {  // it was not due
        async_wait_all();
        net = share = -1;
    }
    for (int n = 0; at.ti >= 0; at.next(), ++n) {
        const NcRowTile tile = P.rtiles[at.ti];
        const bool new_run = tile.net != net || at.share != share;
        if (new_run) {
            share = at.share;
            begin_run(tile);
#pragma unroll 1
            for (int k = 0; k < kRing; ++k) {
                const uint32_t q = Q + k * step;
                if (q - run0 < run) ring.fetch(P, slot + k < kRing ? slot + k : slot + k - kRing, q);
                async_commit();
            }
        }
        if (tile.net != net) {
            if (net >= 0) count_events(P.nets[net], nl, nf, lane);
            nl = nf = 0u;
            begin_net(tile.net);
            begin_step(P.nets[net].t, P.nets[net].stdp_done);
        }
        if (new_run && due) {  // the first quad's fired words
            async_wait();
            if (Q - run0 < run) {
                if (C.wide) fired_words<true>(C, ring.load(slot, 0), f);
                else fired_words<false>(C, ring.load(slot, 0), f);
            }
        }
        const int b = n & 1;
        // by pool index of the quad (a part's are read by whichever block ends last)
        uint8_t* nib = (tile.nq <= kNibCap && !(kKind == kSplit && tile.part) ? sh.nib[b] - tile.q0 : P.nib);
        bar_sync<kBarReady>(b);
        const uint32_t row0 = (uint32_t)tile.first, nq = (uint32_t)tile.nq;
        if (C.wide)
            tile_synapses<kFlush, kStage, true, true>(P, C, tile.q0, nq, run0, run, due, sh.row[b], row0, nib, stage, ring, step, Q,
                                              slot, f, nl, nf);
        else if (inh)
            tile_synapses<kFlush, kStage, false, true>(P, C, tile.q0, nq, run0, run, due, sh.row[b], row0, nib, stage, ring, step, Q,
                                               slot, f, nl, nf);
        else
            tile_synapses<kFlush, kStage, false, false>(P, C, tile.q0, nq, run0, run, due, sh.row[b], row0, nib, stage, ring, step, Q,
                                                slot, f, nl, nf);
        if (kStage) async_wait_all();
        bar_arrive<kBarFull>(b);
    }
    if (net >= 0) count_events(P.nets[net], nl, nf, lane);
    else bar_arrive<kBarFull>(0);  // nothing to do: the step counters have been read
}

// Row starts of a tile into L1, before the wait: nothing writes them.
__device__ __forceinline__ void prefetch_tile(const NcPools& P, const NcRowTile& tile, int lane)
{
    if (lane < tile.count) asm volatile("prefetch.global.L1 [%0];" ::"l"(P.in_ptr + tile.ptr + lane));
}

// Rows of tile `ti` into sh.row[b], and the buffer handed to the stream warps.
__device__ __forceinline__ void give_rows(const NcPools& P, BlockShared& sh, int ti, int b, int lane)
{
    if (lane < P.rtiles[ti].count) {
        const NcNetDesc& D = P.nets[P.rtiles[ti].net];
        const int32_t i = P.rtiles[ti].neuron + lane;
        // the target's trace at prev; the arriving synapse's own is 0
        const int32_t lf = P.lf[i];
        const float trT = P.pst[i];
        const uint32_t sums = lf == NC_NEVER || D.t - lf >= D.kc ? 2u : 0u;
        sh.row[b][lane] = RowState{(D.pre_factor * 0.0f - D.post_factor * trT) * D.lr, lf == D.t - 1 ? 1u | sums : sums};
    }
    bar_arrive<kBarReady>(b);
}

// The neuron warp's part of a step.
template <bool kFlush, bool kAlone, Kind kKind>
__device__ __forceinline__ void neuron_role(const NcPools& P, BlockShared& sh, unsigned char* dyn, bool back)
{
    constexpr bool kStage = kKind == kStaged;
    const int lane = threadIdx.x & 31;
    Tiles<kFlush> at(P, back);
    // (the first tile's rows, into the L1 or at least the L2)
    if (kAlone && at.planned()) prefetch_tile(P, P.rtiles[at.ti], lane);
    if (kAlone) {
        wait_previous_step();
        release_next_step();
    }
    at.settle_first();
    // the tile whose rows are given next: up to two ahead of the one being summed
    Tiles<kFlush> ahead = at;
    int given = 0;
    for (; given < 2 && ahead.ti >= 0; ++given, ahead.next()) give_rows(P, sh, ahead.ti, given & 1, lane);
    unsigned arrived = 0u;
    unsigned fires = 0u;
    int net = -1;
    bool counted = false;
    for (int n = 0; at.ti >= 0; ++n) {
        const int b = n & 1;
        const NcRowTile tile = P.rtiles[at.ti];
        at.next();
        if (kFlush) {
            bar_sync<kBarFull>(b);
            if (at.ti < 0) {
                counted = true;
                if (lane == 0) arrived = atomicAdd(P.done_ctr, 1u);
            }
            if (ahead.ti >= 0) {
                give_rows(P, sh, ahead.ti, b, lane);
                ahead.next();
            }
            continue;
        }
        const NcNetDesc& D = P.nets[tile.net];
        if (tile.net != net) {
            if (net >= 0 && lane == 0 && fires) atomicAdd(P.nets[net].stats + 0, (unsigned long long)fires);
            net = tile.net;
            fires = 0u;
        }
        const int32_t t = D.t;
        const int32_t kc = D.kc;
        const int32_t i = tile.first + lane, pj = tile.neuron + lane;
        auto streamed = [&] {
            bar_sync<kBarFull>(b);
            if (at.ti < 0) {  // the block's last tile: all its warps have read the step counters
                counted = true;
                if (lane == 0) arrived = atomicAdd(P.done_ctr, 1u);
            }
        };
        // the neurons of a split tile are the last block's
        bool mine = true;
        if (kKind == kSplit && tile.part) {
            streamed();
            mine = last_part(P, tile.part, lane);
        }
        const bool live = mine && lane < tile.count;
        const bool stop = D.nonneg_terms != 0;
        const float leak = D.leak;
        const float* tables = P.tables + D.table_base;
        uint8_t* fired_t = (uint8_t*)(P.fired + (int64_t)(t & 1) * P.total_words + D.word_base);
        uint8_t* forced_t = (uint8_t*)(P.forced + (int64_t)(t & 1) * P.total_words + D.word_base);
        uint8_t* ufire_t = (uint8_t*)(P.ufire + (int64_t)(t & 1) * P.total_words + D.word_base);
        uint32_t* forced_n = P.forced + (int64_t)((t + 1) & 1) * P.total_words + D.word_base;
        int32_t lf = NC_NEVER;
        float pot = 0.0f, ap = 0.0f, ap0 = 0.0f, trace = 0.0f;
        bool forced = false, input = false;
        int q0 = 0, nq = 0;
        if (live) {
            lf = P.lf[pj];
            pot = P.pot[pj];
            q0 = (int)((__ldg(P.in_ptr + tile.ptr + lane) >> 2) - (int64_t)tile.q0);
            nq = (int)((__ldg(P.in_ptr + tile.ptr + lane + 1) >> 2) - (int64_t)tile.q0) - q0;
            forced = (forced_t[i >> 3] >> (i & 7)) & 1u;
            input = (ufire_t[i >> 3] >> (i & 7)) & 1u;
            // the AP table's entries now and after a fire, the trace without one
            if (lf != NC_NEVER && t - lf < kc) ap = __ldg(P.tables + D.ap_base + (t - lf));
            ap0 = __ldg(P.tables + D.ap_base);
            trace = trace_at_u(tables + D.tab_pre_len, D.tab_post_len, t, lf);
            // input requests; background fires for step t+1 (src/NeuCor.cpp:604-607), drawn per
            // caller id
            const int32_t cid = D.permuted ? __ldg(P.orig_id + pj) : i;
            if (D.n_groups && input_request(P, D, cid, t)) forced = true;
            if (D.bg_period > 0) {
                uint32_t o[4];
                philox((uint32_t)cid, (uint32_t)t, NC_STREAM_BACKGROUND, 0u, D, o);
                if (o[0] % (uint32_t)D.bg_period == 0u) {
                    uint32_t bg = o[1] % (uint32_t)D.n;
                    if (D.permuted) bg = (uint32_t)P.slot_of[D.neuron_base + bg];
                    atomicOr(forced_n + (bg >> 5), 1u << (bg & 31));
                }
            }
        }
        // inside its AP (t - lastFire < KC) a neuron's potential comes from the AP table
        // whatever its sum is, and it cannot cross the threshold; with no negative term a
        // neuron already over the threshold fires whatever its sum
        const bool can = lf == NC_NEVER || t - lf >= kc;
        const TermFactor F = term_factor(D);
        const bool need = live && can && !(stop && fires_at(pot, leak));
        if (kKind != kSplit || !tile.part) {
            streamed();
            const uint8_t* nib = tile.nq <= kNibCap ? sh.nib[b] : P.nib + tile.q0;
            const float* x = kStage ? (const float*)(dyn + kRingBytes * (blockDim.x - 32)) : P.x + 4 * (int64_t)tile.q0;
            if (need) pot = fold_row<kStage>(nib, q0, nq, x, pot, leak, F, stop);
        } else {
            pot = fold_split_rows(P.nib, P.x, (int64_t)tile.q0 + q0, need ? nq : 0, pot, leak, F.hi, F.lo, F.e_term, stop,
                                  sh.nib[b]);
        }
        __syncwarp();
        if (ahead.ti >= 0) {
            give_rows(P, sh, ahead.ti, b, lane);
            ahead.next();
        }
        bool fired = false;
        if (live) {
            // charge_passive (src/NeuCor.cpp:677-680)
            pot = (pot - -70.0f) * leak + -70.0f;
            // charge_thresholdCheck (src/NeuCor.cpp:682-686); vesicles stay positive.  An input
            // firer's Neuron::fire has no threshold or refractory test
            fired = input || ((-55.0f < pot || forced) && can);
            // AP (src/NeuCor.cpp:706-714)
            if (fired) {
                P.lf[pj] = t;
                atomicAdd(P.firings + pj, 1u);  // (nothing waits for a value)
                pot = ap0;
            } else if (!can) {
                pot = ap;
            }
            P.pot[pj] = pot;
            // getTrace at t (src/NeuCor.cpp:671-675; 0 when it fired at t) for the next step
            P.pst[pj] = fired ? 0.0f : trace;
        }
        const uint32_t fmask = __ballot_sync(kFull, fired);
        // a tile may hold part of a word: bytes (8 neurons) are written on their own
        if (mine && lane < 4 && 8 * lane < tile.count) {
            const int32_t at_byte = tile.first / 8 + lane;
            const uint8_t v = (uint8_t)(fmask >> (8 * lane));
            fired_t[at_byte] = v;
            forced_t[at_byte] = 0;
            ufire_t[at_byte] = 0;
            if (D.raster_len > 0 && t >= D.raster_t0 && t - D.raster_t0 < D.raster_len)
                ((uint8_t*)(D.raster + (int64_t)(t - D.raster_t0) * D.n_words))[at_byte] = v;
        }
        fires += __popc(fmask);
    }
    if (net >= 0 && lane == 0 && fires) atomicAdd(P.nets[net].stats + 0, (unsigned long long)fires);
    if (!counted) {  // a block with nothing to do (its other warps have read the counters)
        bar_sync<kBarFull>(0);
        if (lane == 0) arrived = atomicAdd(P.done_ctr, 1u);
    }
    if (__shfl_sync(kFull, arrived, 0) == gridDim.x - 1u) advance_steps<kFlush ? kFlushed : kStep>(P, lane);
}

// One step (or the flush of the last one) of every tile of this block.
template <bool kFlush, bool kAlone, Kind kKind>
__device__ __forceinline__ void dense_pass(const NcPools& P, BlockShared& sh, unsigned char* dyn, bool back)
{
    if (threadIdx.x >= blockDim.x - 32) {
        neuron_role<kFlush, kAlone, kKind>(P, sh, dyn, back);
    } else {
        stream_role<kFlush, kAlone, kKind>(P, sh, dyn, back);
    }
}

#ifndef NC_DENSE_MIN_BLOCKS
#define NC_DENSE_MIN_BLOCKS 3
#endif
template <bool kFlush, Kind kKind>
__global__ void __launch_bounds__(kMaxThreads, NC_DENSE_MIN_BLOCKS) k_dense_step(NcPools P, bool back)
{
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ BlockShared sh;
    dense_pass<kFlush, true, kKind>(P, sh, dyn, back);
}

// ---------------------------------------------------------------- fused multi-step launch
// `ticks` whole steps of every net in one cooperative launch, a grid barrier after each.
// The grid is at most one wave (cudaLaunchCooperativeKernel refuses more), so every
// block reaches every barrier; each barrier wait is still bounded, and one that gives
// up sets NC_DEV_ERR_BARRIER and ends its block.  (No periodic input firers: they run as
// their own kernel before a step.)
constexpr uint32_t kBarrierPolls = 1u << 24;  // polls (64 ns sleeps) before a barrier gives up

// bar[0]: arrivals, bar[1]: generation.  gen: this block's view of the generation.
__device__ bool grid_barrier(unsigned* bar, unsigned& gen, uint32_t* dev_err, BlockShared& sh)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        __threadfence();
        const unsigned g = gen;
        if (atomicAdd(&bar[0], 1u) == gridDim.x - 1u) {
            atomicExch(&bar[0], 0u);
            __threadfence();
            atomicExch(&bar[1], g + 1u);
        } else {
            uint32_t it = 0;
            while (atomicAdd(&bar[1], 0u) == g) {
                if (++it > kBarrierPolls) {
                    atomicOr(dev_err, NC_DEV_ERR_BARRIER);
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        gen = g + 1u;
        sh.ok = ok;
    }
    __syncthreads();
    return sh.ok != 0;
}

template <Kind kKind>
__global__ void __launch_bounds__(kMaxThreads, NC_DENSE_MIN_BLOCKS) k_dense_fused(NcPools P, int32_t ticks,
                                                                                unsigned* bar)
{
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ BlockShared sh;
    unsigned gen = 0u;
    if (threadIdx.x == 0) gen = atomicAdd(&bar[1], 0u);
    for (int32_t k = 0; k < ticks; ++k) {
        dense_pass<false, false, kKind>(P, sh, dyn, k & 1);
        if (!grid_barrier(bar, gen, P.dev_err, sh)) return;
    }
}

// The kernels by kind, of one step and of several.
const void* step_kernel(Kind kind)
{
    return kind == kStaged ? (const void*)k_dense_step<false, kStaged>
           : kind == kSplit ? (const void*)k_dense_step<false, kSplit>
                            : (const void*)k_dense_step<false, kWhole>;
}
const void* fused_kernel(Kind kind)
{
    return kind == kSplit ? (const void*)k_dense_fused<kSplit> : (const void*)k_dense_fused<kWhole>;
}

// Blocks of one wave of a kind's kernel with `threads` threads on the current device (cached per
// device and block size).  Returns 0 when the device cannot run it (the launch then reports an
// error).
int resident_blocks(bool fused, Kind kind, int threads)
{
    static std::atomic<int> cache[2][3][64][kMaxThreads / 32 + 1];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::atomic<int>& c = cache[fused][kind][dev][threads / 32];
    int n = c.load(std::memory_order_relaxed);
    if (n == 0) {
        int sms = 0, per_sm = 0;
        const size_t dyn = dyn_bytes(threads - 32, kind == kStaged);
        const void* fn = fused ? fused_kernel(kind) : step_kernel(kind);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, dyn) != cudaSuccess || sms * per_sm <= 0)
            return 0;
        // no more shared memory than the blocks need: the rest is L1 for the gathers
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess) return 0;
        const size_t need = (size_t)per_sm * (fa.sharedSizeBytes + dyn + 1024);
        cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)std::min<size_t>(100, (need * 100 + 233471) / 233472));
        n = sms * per_sm;
        c.store(n, std::memory_order_relaxed);
    }
    return n;
}

// Threads per block: a neuron warp and at least one stream warp.
int block_threads(const nc::LaunchShape& L) { return std::max(L.neuron_block, 64); }

// A step's or flush's kernel as a programmatic dependent launch.
int launch_dependent(void (*fn)(NcPools, bool), int blocks, int threads, size_t dyn, const NcPools& P, bool back,
                     void* stream)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = dyn;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, fn, P, back) != cudaSuccess) return -1;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace

namespace nc {

// Whether a step of `threads`-thread blocks can keep its captured charges in shared memory: one
// tile to a block, it fits, and a wave holds every block.  (Blocks of several tiles would need
// two buffers, and large networks their L1.)
bool dense_stages(const std::vector<NcRowTile>& tiles, const std::vector<int32_t>& start, int threads)
{
    for (size_t b = 0; b + 1 < start.size(); ++b)
        if (start[b + 1] - start[b] > 1) return false;
    for (const NcRowTile& t : tiles)
        if (t.nq > kStageQuads || t.part) return false;
    return resident_blocks(false, kStaged, std::max(threads, 64)) >= (int)start.size() - 1;
}

int dense_resident_blocks(int threads)
{
    resident_blocks(false, kSplit, std::max(threads, 64));
    return resident_blocks(false, kWhole, std::max(threads, 64));
}

int launch_step_dense(const NcPools& P, const LaunchShape& L, bool back, void* stream)
{
    // a net with no neuron has no tile, but its step counter still advances
    const int threads = block_threads(L);
    const int blocks = L.dense_blocks > 0 ? std::min(L.dense_blocks, P.row_blocks) : P.row_blocks;
    // (another launch shape than the plan's may not hold every block in a wave)
    const bool stage = P.stage && L.dense_blocks == 0 && resident_blocks(false, kStaged, threads) >= blocks;
    return launch_dependent(stage     ? k_dense_step<false, kStaged>
                            : P.split ? k_dense_step<false, kSplit>
                                      : k_dense_step<false, kWhole>,
                            blocks, threads, dyn_bytes(threads - 32, stage), P, back, stream);
}

int launch_fused_dense(const NcPools& P, int32_t ticks, const LaunchShape& L, unsigned* bar, void* stream)
{
    if (ticks <= 0) return 0;
    const int threads = block_threads(L);
    const Kind kind = P.split ? kSplit : kWhole;
    const int resident = resident_blocks(true, kind, threads);
    if (resident <= 0) return -1;
    // at most one wave
    const int blocks = std::min(resident, P.row_blocks);
    const cudaStream_t s = (cudaStream_t)stream;
    // the arrival count starts at zero (a barrier that gave up may have left it set)
    if (cudaMemsetAsync(bar, 0, sizeof(unsigned), s) != cudaSuccess) return -1;
    NcPools p = P;
    void* args[] = {(void*)&p, (void*)&ticks, (void*)&bar};
    if (cudaLaunchCooperativeKernel(fused_kernel(kind), dim3((unsigned)blocks), dim3((unsigned)threads), args,
                                    dyn_bytes(threads - 32, false), s) != cudaSuccess)
        return -1;
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_flush_dense(const NcPools& P, const LaunchShape& L, void* stream)
{
    const int threads = block_threads(L);
    return launch_dependent(k_dense_step<true, kWhole>, P.row_blocks, threads, dyn_bytes(threads - 32, false), P, false,
                            stream);
}

}  // namespace nc
