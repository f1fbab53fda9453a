/*
 * rt_finish.cu - the kernel that ends a wavefront round.
 *
 * Towards the end of a round (and for all of a small one) few paths are left,
 * and an iteration of the wavefront loop is bound by its launches and by its
 * longest ray, not by the work in it.  This kernel takes over at that point:
 * each warp takes a few of the remaining paths and runs them to their end - shade,
 * trace the rays that the shades left, shade again - as a wavefront of its own,
 * without a launch or a grid-wide wait between bounces.  The shades and the
 * traversal are the loop's own (rt_wavefront.cuh), so every sample has the same
 * bits; a finished path's slot takes the next camera sample here too.
 *
 * Measured against the loop running to its end (ms): volume 16 spp 26.4 -> 20.1
 * (its loop made about 90 iterations of under 64 Ki paths, each as long as its
 * longest ray), light tracer 15.5 -> 13.1, gradient step 5.2 -> 4.9, 256 x 256
 * preview 0.53 -> 0.36, batch of twelve scenes 34.3 -> 33.3.
 */
#include "rt_wavefront.cuh"

namespace {

enum FinishKind { kFinishPath, kFinishVol, kFinishParticle };

/* resident blocks per SM.  Path, whole rounds, ms at 3 / 4 / 5: Cornell box 16 Ki
 * samples 0.31 / 0.29 / 0.36, 64 Ki 0.48 / 0.36 / 0.42, 96 Ki 0.65 / 0.54 / 0.54; in
 * rough plastic 0.42 / 0.42 / 0.52, 0.65 / 0.48 / 0.57, 0.92 / 0.73 / 0.74; with a
 * displaced sphere 0.53 / 0.51 / 0.57, 0.85 / 0.66 / 0.73, 1.07 / 0.93 / 0.91.
 * vol_path and the light tracer, which take over long tails: 20.5 / 13.4 ms at 4,
 * 20.4 / 13.3 at 3, 20.6 / 13.3 at 2. */
#ifndef RT_FINISH_BLOCKS
#define RT_FINISH_BLOCKS 3
#endif
#ifndef RT_FINISH_PATH_BLOCKS
#define RT_FINISH_PATH_BLOCKS 4
#endif
#define RT_FINISH_MIN 4          /* fewest paths a warp takes at a time (1: the same) */
#define RT_FINISH_REFILL 4       /* idle lanes before a warp hands out more of its rays (1: the same) */
#define WF_FINISH_BLOCK 128

/* Entered with the rays of the current active list traced (rt_wf_trace) and
 * the counters reset (rt_wf_phase). */
template <FinishKind kKind, NodeMode kMode>
__global__ void __launch_bounds__(WF_FINISH_BLOCK, kKind == kFinishPath ? RT_FINISH_PATH_BLOCKS : RT_FINISH_BLOCKS) k_wf_finish(WfState W, uint32_t* status, unsigned long long* stats,
                                                                int pass) {
    __shared__ int s_rays[WF_FINISH_BLOCK / 32][3 * 32];
    int* const rays = s_rays[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int cur = W.ctr->iter & 1;
    const int n = min(W.ctr->n_active[cur], W.slots);
    const int warps = gridDim.x * (WF_FINISH_BLOCK / 32);
    const int per = min(32, max(RT_FINISH_MIN, (n + warps - 1) / warps));
    while (true) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&W.ctr->shade_fetch, per);
        base = __shfl_sync(kFullWarp, base, 0);
        if (base >= n) break;
        int slot = lane < per && base + lane < n ? W.active[cur][base + lane] : -1;
        for (int iter = W.ctr->iter;; iter++) {
            if (iter >= W.iter_cap) {
                if (lane == 0) atomicOr(status, RT_STATUS_WFITER);
                break;
            }
            /* the rays of every slot, side by side: region k of the ray arrays holds one ray per slot */
            int count = 0;
            auto put = [&](bool want, int region, int kind, bool any, float4 o, float4 d) {
                const unsigned m = __ballot_sync(kFullWarp, want);
                if (want) {
                    const int q = region * W.slots + slot;
                    push_ray4(W, q, slot, kind, o, d);
                    rays[count + __popc(m & ((1u << lane) - 1u))] = any ? q | WF_ANY_BIT : q;
                }
                count += __popc(m);
            };
            const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (kKind == kFinishPath) {
                PathOut o;
                o.shadow = o.mis_any = o.mis = o.ext = o.keep = o.restart = false;
                if (slot >= 0) shade_path<false>(&o, W, slot, status, stats, false, pass, WfAdjoint{}, nullptr);
                __syncwarp();
                const long long sid = claim_sample(W, kFullWarp, o.restart);
                float4 eo = none, ed = none;
                if (o.restart) {
                    o.keep = init_path(W, slot, sid, &eo, &ed);
                    o.ext = o.keep;
                } else if (o.ext) {
                    eo = W.ray_o[slot]; ed = W.ray_d[slot];
                }
                const bool mis = o.mis || o.mis_any;
                put(o.ext, 0, WF_RAY_EXT, false, eo, ed);
                put(mis, 1, o.mis ? WF_RAY_MIS : WF_RAY_MIS_ANY, o.mis_any, mis ? W.pd_ray_o[slot] : none,
                    mis ? W.pd_ray_d[slot] : none);
                put(o.shadow, 2, WF_RAY_SHADOW, true, o.shadow ? o.so : none, o.shadow ? o.sd : none);
                if (!o.keep) slot = -1;
            } else if (kKind == kFinishVol) {
                VolOut o;
                o.trw = o.itw = o.ext = o.keep = o.restart = false;
                if (slot >= 0) shade_vol_path(&o, W, slot, status, stats, false);
                __syncwarp();
                const long long sid = claim_sample(W, kFullWarp, o.restart);
                float4 eo = none, ed = none, to = none, td = none;
                if (o.restart) {
                    o.keep = init_path(W, slot, sid, &eo, &ed);
                    o.ext = o.keep;
                } else if (o.ext) {
                    eo = W.ray_o[slot]; ed = W.ray_d[slot];
                }
                if (o.itw) {
                    const float4 id = W.itw_d[slot];
                    eo = W.itw_o[slot];
                    ed = make_float4(id.x, id.y, id.z, kFMax);
                }
                if (o.trw) trw_ray(W, slot, &to, &td);
                put(o.ext || o.itw, 0, o.itw ? WF_RAY_MIS : WF_RAY_EXT, false, eo, ed);
                put(o.trw, 1, WF_RAY_TRW, false, to, td);
                if (!o.keep) slot = -1;
            } else {
                PartOut o;
                o.splat = o.ext = o.keep = false;
                bool restart = false;
                if (slot >= 0) restart = shade_particle(W, slot, status, &o);
                __syncwarp();
                const long long sid = claim_particle(W, restart);
                if (restart) start_particle(W, slot, sid, &o);
                __syncwarp();
                put(o.ext, 0, WF_RAY_EXT, false, o.ext ? o.eo : none, o.ext ? o.ed : none);
                put(o.splat, 2, WF_RAY_SPLAT, true, o.splat ? o.so : none, o.splat ? o.sd : none);
                if (!o.keep) slot = -1;
            }
            __syncwarp();
            int next = 0;
            if (count > 0)
                trace_queued<kEitherHit, false, kMode>(W, RT_FINISH_REFILL, [&](unsigned idle, bool* exhausted) {
                    const int e = next + __popc(idle & ((1u << lane) - 1u));
                    next += __popc(idle);
                    *exhausted = next >= count;
                    return (idle >> lane & 1u) && e < count ? rays[e] : -1;
                }, status, stats, false);
            __syncwarp();
            if (!__any_sync(kFullWarp, slot >= 0)) break;
        }
    }
}

typedef void (*FinishKernel)(WfState, uint32_t*, unsigned long long*, int);
/* by [kind][short, wide, grow]; the light tracer's closest-hit rays have no finite MaxT */
const FinishKernel kFinish[3][3] = {
    {k_wf_finish<kFinishPath, kNodesShort>, k_wf_finish<kFinishPath, kNodesWide>, k_wf_finish<kFinishPath, kNodesGrow>},
    {k_wf_finish<kFinishVol, kNodesShort>, k_wf_finish<kFinishVol, kNodesWide>, k_wf_finish<kFinishVol, kNodesGrow>},
    {k_wf_finish<kFinishParticle, kNodesShort>, k_wf_finish<kFinishParticle, kNodesWide>,
     k_wf_finish<kFinishParticle, kNodesShort>}};

struct FinishGrids {
    int blocks[3][3];
    FinishGrids() {
        for (int k = 0; k < 3; k++)
            for (int w = 0; w < 3; w++) blocks[k][w] = resident_blocks(kFinish[k][w], WF_FINISH_BLOCK);
    }
};

}  // namespace

static const FinishGrids& finish_grids() {
    static const FinishGrids grids;
    return grids;
}

int rt_wf_finish_lanes(bool wide, bool grow) {
    return finish_grids().blocks[kFinishPath][wide ? 1 : (grow ? 2 : 0)] * WF_FINISH_BLOCK;
}

cudaError_t rt_wf_finish(const WfState& W, uint32_t* status, unsigned long long* stats, cudaStream_t s, int pass, bool vol,
                         bool particle, bool wide, bool grow) {
    const FinishGrids& grids = finish_grids();
    cudaError_t e = rt_wf_phase(W, s);
    if (e != cudaSuccess) return e;
    const int k = particle ? kFinishParticle : (vol ? kFinishVol : kFinishPath), w = wide ? 1 : (grow ? 2 : 0);
    kFinish[k][w]<<<grids.blocks[k][w], WF_FINISH_BLOCK, 0, s>>>(W, status, stats, pass);
    return cudaGetLastError();
}
