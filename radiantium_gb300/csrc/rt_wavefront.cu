/*
 * rt_wavefront.cu - wavefront renderer for the `path` integrator.
 *
 * The megakernel runs PathTracer.Li (Integrators/PathTracer.cs) as one loop
 * per thread.  Here the loop is cut at its ray casts and the pieces run as
 * separate kernels over compacted queues:
 *
 *   k_wf_trace_closest / k_wf_trace_shadow   the queued rays: extension and
 *                area lights' MIS rays (closest hit), shadow rays and infinite
 *                lights' MIS rays (any hit), each kind in its own persistent
 *                kernel with dynamic ray fetch;
 *   k_wf_sort_count / k_wf_sort_scatter   regroup the active list by shade
 *                key (finished, missed, material type) so that a warp runs
 *                one material's code instead of the union of several;
 *   k_wf_shade   per path: first adds the direct-lighting term scheduled in
 *                the previous shade (its shadow / MIS rays are now resolved),
 *                then runs one bounce of the reference loop on the new
 *                extension hit and enqueues the next rays.
 *
 * All random numbers of a bounce are drawn in k_wf_shade in the reference's
 * order, and the radiance of a path is accumulated in the reference's order
 * (the deferred direct term of bounce b is added before the emission of
 * bounce b+1), so every sample is bit-identical to the megakernel and to the
 * CPU oracle.  Path slots whose path has finished are refilled with the next
 * camera sample, which keeps the queues full to the end of a render.
 *
 * A run renders a batch of jobs (rt_wavefront.h): a path slot records its
 * job, and the scene view and parameters of that job drive its traversal and
 * shading, so paths of every scene of a batch share one set of launches.
 * Every launch reads its work count from device memory and the active lists
 * alternate by iteration parity, so the launch sequence of one bounce never
 * changes and can be captured into a CUDA graph loop.
 */
#include <cuda_runtime.h>
#include <algorithm>
#include "rt_wavefront.cuh"

namespace {

__global__ void __launch_bounds__(256) k_wf_start(WfState W) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = slot < W.slots;
    const long long sid = claim_sample(W, 0xffffffffu, in);
    float4 o, d;
    const bool ok = in && init_path(W, slot, sid, &o, &d);
    int qs, qx, qm, qe, qa;
    queue_append<true>(W, 0, false, false, false, ok, false, &qs, &qx, &qm, &qe, &qa);
    if (ok) push_ray4(W, qe, slot, WF_RAY_EXT, o, d);
}

/* resident blocks of 128 threads per SM the trace kernels are compiled for
 * (the register budget: 65536 / (128 * blocks)) */
#ifndef RT_CLOSEST_BLOCKS
#define RT_CLOSEST_BLOCKS 6
#endif
#ifndef RT_SHADOW_BLOCKS
#define RT_SHADOW_BLOCKS 7
#endif
/* the fast traversal's wide nodes keep eight children's distances in registers:
 * trace ms of an 8-spp 640x360 pass over the 64 instances at closest / shadow 6 / 7: 11.9,
 * 5 / 6: 11.0, 5 / 5: 11.2, 4 / 5: 11.6 */
#ifndef RT_WIDE_CLOSEST_BLOCKS
#define RT_WIDE_CLOSEST_BLOCKS 5
#endif
#ifndef RT_WIDE_SHADOW_BLOCKS
#define RT_WIDE_SHADOW_BLOCKS 6
#endif
template <NodeMode kMode> constexpr int kClosestBlocks = kMode == kNodesWide ? RT_WIDE_CLOSEST_BLOCKS : RT_CLOSEST_BLOCKS;
template <NodeMode kMode> constexpr int kShadowBlocks = kMode == kNodesWide ? RT_WIDE_SHADOW_BLOCKS : RT_SHADOW_BLOCKS;
/* the same for the shade kernels of `path` (the host-driven render pass; the
 * graph-driven and adjoint-replay variants keep 5, where 6 spills far more), of
 * the light tracer and of vol_path.  Path shade at 6 / 7 / 8, ms: Cornell frame
 * 7.54 / 7.33 / 7.42, instances 69.6 / 68.8 / 68.3, batch 34.1 / 33.5 / 33.8. */
#ifndef RT_SHADE_BLOCKS
#define RT_SHADE_BLOCKS 7
#endif
#ifndef RT_PSHADE_BLOCKS
#define RT_PSHADE_BLOCKS 7       /* light tracer, ms: 13.4 at 5, 13.2 at 6, 13.1 at 7 */
#endif
#ifndef RT_VSHADE_BLOCKS
#define RT_VSHADE_BLOCKS 6       /* volume, ms: 20.7 at 4, 20.4 at 5, 20.3 at 6 */
#endif

/* closest-hit rays: extension and MIS rays (queue [0, n_closest)) */
template <bool kSh, NodeMode kMode>
__global__ void __launch_bounds__(RT_TRACE_BLOCK, kClosestBlocks<kMode>) k_wf_trace_closest(WfState W, uint32_t* status,
                                                                                            unsigned long long* stats, bool counting) {
    const int n = min(W.ctr->n_closest, 2 * W.slots);
    trace_queued<kClosestHit, kSh, kMode>(W, W.refill, [&](unsigned idle, bool* exhausted) {
        const int e = fetch_entry(&W.ctr->fetch[0], n, idle, exhausted);
        return e < n ? e : -1;
    }, status, stats, counting);
}

/* shadow rays and infinite lights' MIS rays: any-hit (queue [shadow_base, shadow_base + n_shadow)) */
template <bool kSh, NodeMode kMode>
__global__ void __launch_bounds__(RT_TRACE_BLOCK, kShadowBlocks<kMode>) k_wf_trace_shadow(WfState W, uint32_t* status,
                                                                                          unsigned long long* stats, bool counting) {
    const int n = min(W.ctr->n_shadow, 2 * W.slots);
    trace_queued<kAnyHit, kSh, kMode>(W, W.refill, [&](unsigned idle, bool* exhausted) {
        const int e = fetch_entry(&W.ctr->fetch[1], n, idle, exhausted);
        return e < n ? W.shadow_base + e : -1;
    }, status, stats, counting);
}

__global__ void __launch_bounds__(128, RT_VSHADE_BLOCKS) k_wf_shade_vol(WfState W, uint32_t* status, unsigned long long* stats,
                                                         bool counting, bool sorted) {
    const int cur = W.ctr->iter & 1;
    const int n = min(W.ctr->n_active[cur], W.slots);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int slot = -1;
    VolOut o;
    o.trw = o.itw = o.ext = o.keep = o.restart = false;
    if (i < n) { slot = sorted ? W.sorted[i] : W.active[cur][i]; shade_vol_path(&o, W, slot, status, stats, counting); }
    vol_queues(W, slot, cur ^ 1, o);
}

/* the active paths of this iteration, one thread each over the sorted list
 * (or, `sorted` false, the active list as built): either a grid sized to the
 * active count, or (kDynamic, inside a graph where the count is unknown at
 * launch) a resident grid whose warps take the next 32 entries from a
 * counter until the list is done.  The replay pass of the adjoint (kAdj)
 * sums its alpha gradients per block in shared memory. */
template <bool kAdj, bool kDynamic>
__global__ void __launch_bounds__(128, (kAdj || kDynamic) ? 5 : RT_SHADE_BLOCKS) k_wf_shade(WfState W, uint32_t* status, unsigned long long* stats, bool counting,
                                                       int pass, WfAdjoint A, bool sorted) {
    const int32_t* list;
    __shared__ float s_alpha[kAdj ? RT_ADJ_MAX_ALPHA : 1];
    if (kAdj) {
        for (int i = threadIdx.x; i < A.n_alpha; i += blockDim.x) s_alpha[i] = 0.0f;
        __syncthreads();
    }
    const int cur = W.ctr->iter & 1;
    const int n = min(W.ctr->n_active[cur], W.slots);
    list = sorted ? W.sorted : W.active[cur];
    if (!kDynamic) {
        const int i = blockIdx.x * blockDim.x + threadIdx.x;
        int slot = -1;
        PathOut o;
        o.shadow = o.mis_any = o.mis = o.ext = o.keep = o.restart = false;
        if (i < n) { slot = list[i]; shade_path<kAdj>(&o, W, slot, status, stats, counting, pass, A, s_alpha); }
        path_queues<true>(W, slot, cur ^ 1, o);
    } else {
        const int lane = threadIdx.x & 31;
        while (true) {
            int base = 0;
            if (lane == 0) base = atomicAdd(&W.ctr->shade_fetch, 32);
            base = __shfl_sync(kFullWarp, base, 0);
            if (base >= n) break;
            const int i = base + lane;
            int slot = -1;
            PathOut o;
            o.shadow = o.mis_any = o.mis = o.ext = o.keep = o.restart = false;
            if (i < n) { slot = list[i]; shade_path<kAdj>(&o, W, slot, status, stats, counting, pass, A, s_alpha); }
            __syncwarp();
            path_queues<false>(W, slot, cur ^ 1, o);
        }
    }
    if (kAdj) {
        __syncthreads();
        for (int i = threadIdx.x; i < A.n_alpha; i += blockDim.x)
            if (s_alpha[i] != 0.0f) atomicAdd(A.grad_alpha + i, s_alpha[i]);
    }
}

__global__ void __launch_bounds__(256) k_wf_start_particles(WfState W) {
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    PartOut o;
    o.splat = o.ext = o.keep = false;
    const bool in = slot < W.slots;
    const long long sid = claim_particle(W, in);
    if (in) start_particle(W, slot, sid, &o);
    /* the first active list is built from the slots' flags afterwards */
    int qs, qx, qm, qe, a;
    queue_append<true>(W, 0, false, false, false, o.ext, false, &qs, &qx, &qm, &qe, &a);
    if (o.ext) push_ray4(W, qe, slot, WF_RAY_EXT, o.eo, o.ed);
}

/* `sorted`: the list regrouped by shade key, else the active list as built
 * (scenes of one material type gain nothing from the regrouping) */
__global__ void __launch_bounds__(128, RT_PSHADE_BLOCKS) k_wf_shade_particle(WfState W, uint32_t* status, bool sorted) {
    const int cur = W.ctr->iter & 1;
    const int n = min(W.ctr->n_active[cur], W.slots);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int slot = -1;
    PartOut o;
    o.splat = o.ext = o.keep = false;
    bool restart = false;
    if (i < n) { slot = sorted ? W.sorted[i] : W.active[cur][i]; restart = shade_particle(W, slot, status, &o); }
    /* a finished particle's slot takes the next particle at once */
    const long long sid = claim_particle(W, restart);
    if (restart) start_particle(W, slot, sid, &o);
    particle_queues(W, slot, cur ^ 1, o);
}

__global__ void k_wf_active_init(WfState W) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= W.slots) return;
    bool alive = (W.flags[i] & F_ALIVE) != 0;
    int a = warp_append(&W.ctr->n_active[0], alive);
    if (alive) set_active(W, 0, a, i);
    else W.mark[i] = 0;
}

/* Code key of an active path: which code the shade kernel will run for it.
 * 0 finished (pending term, then a new sample), 1 missed the scene, 2 hit a
 * medium boundary without a surface, 3 + RT_MAT_* hit that material type,
 * 15 vol_path boundary walks.  The shade key puts the job (mod 64) above it,
 * so a batch shades - and then traces - one scene's paths together. */
DF int shade_key(const WfState& W, int slot) {
    const uint32_t fl = W.flags[slot];
    const int job = W.job[slot];
    const int jk = (job & 63) << 4;
    if (fl & (F_WTR | F_WIT)) return jk | 15;
    if (fl & F_DONE) return jk;
    const int hs = __float_as_int(W.ext_hit[slot].w);
    if (hs < 0) return jk | 1;
    const RtSceneView* S = W.jobs[job].view;
    const int prim = __float_as_int(__ldg(S->slots + 3 * (int64_t)hs).w);
    const int m = S->prims[prim].material;
    if (m < 0) return jk | 2;
    return jk | min(3 + S->materials[m].type, 14);
}

/* between trace and shade: the queues are consumed, reset their counters */
__global__ void k_wf_phase(WfState W) {
    if (threadIdx.x == 0) {
        WfCounters* c = W.ctr;
        c->n_closest = 0; c->n_shadow = 0; c->fetch[0] = 0; c->fetch[1] = 0; c->shade_fetch = 0;
        c->n_active[(c->iter & 1) ^ 1] = 0;
    }
    for (int k = threadIdx.x; k < 2 * WF_SHADE_KEYS; k += blockDim.x) W.key_count[k] = 0;
}

/* The sort's input order.  While at least one slot in WF_DENSE_SORT is active
 * (and the run allows it: W.dense_sort),
 * the sort walks the slots in index order (their marks say which are on this
 * iteration's list): a warp's entries of one key then land together in slot
 * order, so the shade's warps read path state of nearby slots - fewer sectors
 * per field than the appended list's scattered order.  Below that it walks the
 * active list itself.  Both kernels take the same decision from the same count. */
#ifndef WF_DENSE_SORT
#define WF_DENSE_SORT 8
#endif
DF bool sort_dense(const WfState& W, int n) { return W.dense_sort && n * WF_DENSE_SORT >= W.slots; }
DF int sort_span(const WfState& W, int n) { return sort_dense(W, n) ? W.slots : n; }
/* entry i of the sort's input: a slot, or -1 (a slot not on the list) */
DF int sort_input(const WfState& W, int cur, int n, int i) {
    if (!sort_dense(W, n)) return W.active[cur][i];
    return W.mark[i] == cur + 1 ? i : -1;
}

/* both sort kernels are grid-stride loops: one pass with a grid sized to the
 * active count, several with a resident grid inside a graph */
__global__ void __launch_bounds__(256) k_wf_sort_count(WfState W) {
    const int cur = W.ctr->iter & 1;
    const int n = min(W.ctr->n_active[cur], W.slots);
    const int span = sort_span(W, n);
    for (int i0 = blockIdx.x * blockDim.x; i0 < span; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + threadIdx.x;
        if (i >= span) break;
        const int slot = sort_input(W, cur, n, i);
        if (slot < 0) continue;
        const int key = shade_key(W, slot);
        W.sort_key[i] = (uint16_t)key;
        const unsigned peers = __match_any_sync(__activemask(), key);
        if ((threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1)) atomicAdd(W.key_count + key, __popc(peers));
    }
}

/* counting-sort scatter: entries of one key stay together, in any order
 * (every path's result is independent of the order paths are shaded in).
 * Each block turns the key counts into bases with a shared-memory scan. */
#define WF_KEYS_PER_THREAD (WF_SHADE_KEYS / 256)
static_assert(WF_SHADE_KEYS % 256 == 0, "the scatter's scan gives each of 256 threads the same number of keys");
__global__ void __launch_bounds__(256) k_wf_sort_scatter(WfState W) {
    __shared__ int base[WF_SHADE_KEYS];
    __shared__ int part[256];
    const int cur = W.ctr->iter & 1;
    const int n = min(W.ctr->n_active[cur], W.slots);
    const int span = sort_span(W, n);
    if ((int)(blockIdx.x * blockDim.x) >= span) return;
    const int t = threadIdx.x;
    /* exclusive scan of the key counts: each thread sums its run of keys,
     * the 256 sums are scanned (Hillis-Steele), then each run is filled in */
    int v[WF_KEYS_PER_THREAD], sum = 0;
#pragma unroll
    for (int j = 0; j < WF_KEYS_PER_THREAD; j++) { v[j] = W.key_count[t * WF_KEYS_PER_THREAD + j]; sum += v[j]; }
    part[t] = sum;
    __syncthreads();
    for (int off = 1; off < 256; off <<= 1) {
        const int add = t >= off ? part[t - off] : 0;
        __syncthreads();
        part[t] += add;
        __syncthreads();
    }
    int run = part[t] - sum;
#pragma unroll
    for (int j = 0; j < WF_KEYS_PER_THREAD; j++) { base[t * WF_KEYS_PER_THREAD + j] = run; run += v[j]; }
    __syncthreads();
    const unsigned lane = threadIdx.x & 31;
    for (int i0 = blockIdx.x * blockDim.x; i0 < span; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + threadIdx.x;
        if (i >= span) break;
        const int slot = sort_input(W, cur, n, i);
        if (slot < 0) continue;
        const int key = W.sort_key[i];
        const unsigned peers = __match_any_sync(__activemask(), key);
        const int leader = __ffs(peers) - 1;
        int first = 0;
        if ((int)lane == leader) first = atomicAdd(W.key_count + WF_SHADE_KEYS + key, __popc(peers));
        first = __shfl_sync(peers, first, leader);
        const int dst = base[key] + first + __popc(peers & ((1u << lane) - 1u));
        if (in_bounds(W, dst, W.slots)) W.sorted[dst] = slot;
    }
}

/* end of an iteration: the next active list becomes current */
__global__ void k_wf_tail(WfState W) {
    if (threadIdx.x == 0) W.ctr->iter++;
}
__global__ void k_wf_tail_loop(WfState W, cudaGraphConditionalHandle loop, uint32_t* status) {
    if (threadIdx.x == 0) {
        const int next = (W.ctr->iter & 1) ^ 1;
        W.ctr->iter++;
        /* the loop runs until the kernel that ends the round can take over; without it, queued
         * shadow rays keep it going: a finished light-tracer particle leaves its last splat in
         * the queue without an active slot */
        bool more = W.finish_max > 0 ? W.ctr->n_active[next] > W.finish_max
                                     : W.ctr->n_active[next] > 0 || W.ctr->n_shadow > 0;
        if (more && W.ctr->iter >= W.iter_cap) { atomicOr(status, RT_STATUS_WFITER); more = false; }
        cudaGraphSetConditional(loop, more ? 1u : 0u);
    }
}

}  // namespace

cudaError_t rt_wf_start(const WfState& W, cudaStream_t s, bool particle) {
    if (particle) k_wf_start_particles<<<grid_for(W.slots, 256), 256, 0, s>>>(W);
    else k_wf_start<<<grid_for(W.slots, 256), 256, 0, s>>>(W);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_wf_active_init<<<grid_for(W.slots, 256), 256, 0, s>>>(W);
    return cudaGetLastError();
}

namespace {

typedef void (*TraceKernel)(WfState, uint32_t*, unsigned long long*, bool);
/* the trace kernels by [node mode][shared-memory stack] */
const TraceKernel kClosest[4][2] = {
    {k_wf_trace_closest<false, kNodesGeneral>, k_wf_trace_closest<true, kNodesGeneral>},
    {k_wf_trace_closest<false, kNodesShort>, k_wf_trace_closest<true, kNodesShort>},
    {k_wf_trace_closest<false, kNodesWide>, k_wf_trace_closest<true, kNodesWide>},
    {k_wf_trace_closest<false, kNodesGrow>, k_wf_trace_closest<true, kNodesGrow>}};
const TraceKernel kShadow[4][2] = {
    {k_wf_trace_shadow<false, kNodesGeneral>, k_wf_trace_shadow<true, kNodesGeneral>},
    {k_wf_trace_shadow<false, kNodesShort>, k_wf_trace_shadow<true, kNodesShort>},
    {k_wf_trace_shadow<false, kNodesWide>, k_wf_trace_shadow<true, kNodesWide>},
    {k_wf_trace_shadow<false, kNodesShort>, k_wf_trace_shadow<true, kNodesShort>}};

/* resident blocks of every trace kernel */
struct TraceGrids {
    int closest[4][2], shadow[4][2];
    TraceGrids() {
        for (int m = 0; m < 4; m++)
            for (int d = 0; d < 2; d++) {
                closest[m][d] = resident_blocks(kClosest[m][d], RT_TRACE_BLOCK);
                shadow[m][d] = resident_blocks(kShadow[m][d], RT_TRACE_BLOCK);
            }
    }
};

}  // namespace

cudaError_t rt_wf_trace(const WfState& W, uint32_t* status, unsigned long long* stats, bool counting, cudaStream_t s,
                        bool deep, bool wide, bool general, bool grow, const WfFork* fork) {
    static const TraceGrids grids;
    const int m = wide ? kNodesWide : (general || counting ? kNodesGeneral : (grow ? kNodesGrow : kNodesShort)), d = deep ? 1 : 0;
    cudaError_t e = cudaSuccess;
    if (fork) {
        e = cudaEventRecord(fork->fork, s);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(fork->side, fork->fork, 0);
        if (e != cudaSuccess) return e;
    }
    kClosest[m][d]<<<grids.closest[m][d], RT_TRACE_BLOCK, 0, s>>>(W, status, stats, counting);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    kShadow[m][d]<<<grids.shadow[m][d], RT_TRACE_BLOCK, 0, fork ? fork->side : s>>>(W, status, stats, counting);
    e = cudaGetLastError();
    if (e != cudaSuccess || !fork) return e;
    e = cudaEventRecord(fork->join, fork->side);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, fork->join, 0);
    return e;
}

cudaError_t rt_wf_phase(const WfState& W, cudaStream_t s) {
    k_wf_phase<<<1, 256, 0, s>>>(W);
    return cudaGetLastError();
}

cudaError_t rt_wf_shade(const WfState& W, int n_hint, uint32_t* status, unsigned long long* stats, bool counting,
                        cudaGraphConditionalHandle loop, bool has_loop, cudaStream_t s, uint64_t* launches,
                        int pass, const WfAdjoint* adj, bool vol, bool particle, bool sort) {
    static const int sort_blocks = resident_blocks(k_wf_sort_scatter, 256);
    static const int shade_blocks = resident_blocks(k_wf_shade<false, true>, 128);
    const WfAdjoint A = adj ? *adj : WfAdjoint{-1, 0, nullptr, nullptr, nullptr, nullptr};
    const bool known = n_hint >= 0;
    const int n = known ? std::min(n_hint, W.slots) : W.slots;
    k_wf_phase<<<1, 256, 0, s>>>(W);
    if (n > 0) {
        const unsigned sb = known ? grid_for(n, 256) : (unsigned)sort_blocks;
        if (sort) {
            k_wf_sort_count<<<sb, 256, 0, s>>>(W);
            k_wf_sort_scatter<<<sb, 256, 0, s>>>(W);
        } else {
            *launches -= 2;
        }
        if (particle) k_wf_shade_particle<<<grid_for(n, 128), 128, 0, s>>>(W, status, sort);
        else if (vol) k_wf_shade_vol<<<grid_for(n, 128), 128, 0, s>>>(W, status, stats, counting, sort);
        else if (!known) k_wf_shade<false, true><<<shade_blocks, 128, 0, s>>>(W, status, stats, counting, pass, A, sort);
        else if (pass == WF_PASS_REPLAY) k_wf_shade<true, false><<<grid_for(n, 128), 128, 0, s>>>(W, status, stats, counting, pass, A, sort);
        else k_wf_shade<false, false><<<grid_for(n, 128), 128, 0, s>>>(W, status, stats, counting, pass, A, sort);
        *launches += 3;
    }
    if (has_loop) k_wf_tail_loop<<<1, 32, 0, s>>>(W, loop, status);
    else k_wf_tail<<<1, 32, 0, s>>>(W);
    *launches += 2;
    return cudaGetLastError();
}
