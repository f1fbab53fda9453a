/*
 * rt_trace.cuh - the traversal of many rays by persistent warps: the wavefront's
 * ray queues (rt_wavefront.cuh) and the ray batches of the C ABI
 * (rt_kernels.cu).
 */
#ifndef RT_TRACE_CUH
#define RT_TRACE_CUH
#include "rt_device.cuh"

using namespace rtd;

namespace {

DF void warp_add64(unsigned long long* dst, uint32_t v) {
    unsigned mask = __activemask();
    uint32_t s = __reduce_add_sync(mask, v);
    if ((threadIdx.x & 31) == (unsigned)(__ffs(mask) - 1) && s) atomicAdd(dst, (unsigned long long)s);
}

/* Persistent traversal with dynamic ray fetch (Aila & Laine 2009): each warp
 * keeps its lanes busy by handing a new queue entry to every lane whose ray
 * has finished, as soon as W.refill lanes are idle, instead of idling until
 * the warp's longest ray is done.  The traversal is the step machine of
 * Traversal, so a lane can take a new ray between any two steps
 * and the per-ray results are the same as a one-ray-per-thread launch. */
constexpr unsigned kFullWarp = 0xffffffffu;

/* One warp-wide fetch: returns this lane's queue entry (>= n: none) and sets
 * `exhausted` (warp-uniform) once the queue has been handed out. */
DF int fetch_entry(int32_t* counter, int n, unsigned idle, bool* exhausted) {
    const unsigned lane = threadIdx.x & 31;
    int first = 0;
    if (lane == 0) first = atomicAdd(counter, __popc(idle));
    first = __shfl_sync(kFullWarp, first, 0);
    *exhausted = first + __popc(idle) >= n;
    return first + __popc(idle & ((1u << lane) - 1u));
}

/* The traversal stack of a trace kernel: with kSh (scenes with tall trees)
 * its bottom RT_SH_STACK entries live in shared memory, which keeps the stack
 * of a deep traversal out of the L1 lines the node data needs; shallow trees
 * keep the whole stack in local memory, where it stays in a few hot lines. */
template <bool kSh> struct TraceStack;
template <> struct TraceStack<false> {
    int2 a[2 * RT_STACK_SIZE];
    DF int2* get() { return a; }
};
template <> struct TraceStack<true> {
    int2 a[2 * RT_STACK_SIZE];
    DF SplitStack get() {
        __shared__ int2 sh[RT_SH_STACK * RT_TRACE_BLOCK];
        return SplitStack{sh + threadIdx.x, a};
    }
};

/* When a warp stops descending: as soon as this many of 32 live lanes wait for
 * a LeafStep (a share of the live lanes when fewer are live).  A low count
 * runs the leaf, instance-entry and instance-exit code for few lanes at a
 * time, a high one lets the lanes that reached a leaf idle; deep trees reach
 * leaves less often, so they wait less.  Trace ms of a 64-spp Cornell frame
 * (5-level tree) at 12 / 16 / 20 / 24: 3.70 / 3.58 / 3.53 / 3.52, against 3.73
 * with up to three nodes and one leaf per step; of a 16-spp pass over the
 * 64 x 200 k-triangle instances at 4 / 8 / 12 / 14 / 16 / 20: 82.7 / 76.3 /
 * 73.1 / 72.8 / 72.7 / 75.3, against 79.6 with up to five nodes per step.
 * With the short node visit: Cornell frame at 12 / 18 / 20 / 22 / 24: 2.83 / 2.62 /
 * 2.57 / 2.52 / 2.50, the instances at 12 / 14 / 16: 48.7 / 48.1 / 47.8; whole calls
 * at 24 and 16 take 0.4 to 1.5 % less, with wide nodes 0.5 % more. */
#ifndef RT_LEAF_WAIT
#define RT_LEAF_WAIT 22          /* shallow trees */
#endif
#ifndef RT_LEAF_WAIT_DEEP
#define RT_LEAF_WAIT_DEEP 14     /* trees of RT_DEEP_TREE levels and more */
#endif
/* nodes a lane may visit in one run before the warp's fetch check (8 to 64 measured alike) */
#ifndef RT_DESCEND_RUN
#define RT_DESCEND_RUN 16
#endif

/* The traversal of a list of rays by one warp.  Lane by lane, `fetch` hands
 * out entries of the list (-1: none for this lane; called by the whole warp
 * when at least `refill` lanes are idle, until it sets its second argument);
 * for kEitherHit an entry's top bit marks an any-hit ray.  `load` gives an
 * entry's ray and scene, `report` takes its finished traversal.
 * Bound by lane utilisation and by the latency of dependent node loads (the
 * tree sits in L2): lanes at nodes, leaves and instance boundaries would
 * otherwise run one after another in every step, so the warp runs one kind at
 * a time for all lanes that wait for it. */
#define WF_ANY_BIT ((int)0x80000000)
template <HitForm kForm, bool kSh, NodeMode kMode, class Fetch, class Load, class Report>
DF void trace_rays(int refill, Fetch fetch, Load load, Report report, uint32_t* status, unsigned long long* stats,
                   bool counting) {
    constexpr bool kWide = kMode == kNodesWide;
    if (kMode == kNodesShort || kMode == kNodesGrow) counting = false;
    TraceStack<kSh> stk;
    const auto stack = stk.get();
    typedef decltype(stk.get()) Stk;
    TravStats st = {0, 0, 0};
    TravStats* pst = counting ? &st : nullptr;
    uint32_t done = 0;
    Traversal T;
    T.cur = RT_NO_NODE;
    T.first = kForm == kAnyHit;
    const RtSceneView* S = nullptr;
    bool on = false, exhausted = false;      /* on: the lane has a ray */
    auto finish = [&]() {
        report(S, T);
        done++;
        on = false;
        T.cur = RT_NO_NODE;
    };
    while (true) {
        const unsigned busy = __ballot_sync(kFullWarp, on);
        if (exhausted) {
            if (!busy) break;
        } else if (32 - __popc(busy) >= refill) {
            const int e = fetch(~busy, &exhausted);
            if (!on && e != -1) {
                const int q = kForm == kEitherHit ? e & ~WF_ANY_BIT : e;
                if (kForm == kEitherHit) T.first = e < 0;
                on = true;
                Ray ray;
                S = load(q, &ray);
                if (TraversalBegin<kWide>(S, ray, T, pst)) finish();
            }
        }
        bool over = false;
        if (on && ++T.guard > RT_TRAVERSAL_CAP) { atomicOr(status, RT_STATUS_TRAV); over = true; T.cur = RT_NO_NODE; }
        const int live = __popc(__ballot_sync(kFullWarp, on && !over));
        const int wait = (live * (kSh ? RT_LEAF_WAIT_DEEP : RT_LEAF_WAIT) + 31) >> 5;
#pragma unroll 1
        for (int k = 0; k < RT_DESCEND_RUN; k++) {
            if (T.cur >= 0 && DescendStep<Stk, kMode>(T, stack, status, pst)) over = true;
            if (live - __popc(__ballot_sync(kFullWarp, T.cur >= 0)) >= wait) break;
        }
        if (on && T.cur < 0 && (over || LeafStep<kForm, Stk, kWide>(S, T, stack, status, pst))) finish();
    }
    if (counting) {
        warp_add64(stats + (kForm == kAnyHit ? 2 : 1), done);
        warp_add64(stats + 3, st.nodes);
        warp_add64(stats + 4, st.prims);
        warp_add64(stats + 5, st.insts);
    }
}

/* resident blocks of a grid-stride kernel: every SM filled once */
template <typename K>
int resident_blocks(K kernel, int block) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0) != cudaSuccess || per_sm <= 0)
        per_sm = 1, sms = sms > 0 ? sms : 1;
    return sms * per_sm;
}

}  // namespace

#endif
