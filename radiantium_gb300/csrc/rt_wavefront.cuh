/*
 * rt_wavefront.cuh - device functions of the wavefront renderer, shared by its
 * kernels (rt_wavefront.cu) and by the kernel that ends a round
 * (rt_finish.cu): queue appends, the traversal of a ray list, and one shade of
 * a path, vol_path or light-tracer slot.
 */
#ifndef RT_WAVEFRONT_CUH
#define RT_WAVEFRONT_CUH
#include <cuda_runtime.h>
#include "rt_integrators.cuh"
#include "rt_adjoint.cuh"
#include "rt_trace.cuh"
#include "rt_wavefront.h"

using namespace rtd;

namespace {

enum : uint32_t {
    F_ALIVE = 1u,        /* the slot holds a path */
    F_SPECULAR = 2u,     /* isSpecularPath */
    F_PENDING = 4u,      /* a direct-lighting term waits for its rays */
    F_L1 = 8u,           /* pending light-sample term (gated by the shadow ray) */
    F_L2 = 16u,          /* pending BSDF-sample term (resolved by the MIS ray) */
    F_DZERO = 32u,       /* pending direct term is exactly zero (no light / no estimate) */
    F_DONE = 64u,        /* the path ends once its pending term is added */
    F_EXT = 128u,        /* an extension ray was enqueued */
    F_WTR = 256u,        /* vol_path: a Transmittance-walk segment is being traced */
    F_WIT = 512u,        /* vol_path: an IntersectTr-walk segment is being traced */
    F_CONT = 1024u,      /* vol_path: the next extension ray waits for the pending term */
    F_ANY = 4096u,       /* the pending BSDF-sample term's ray is an any-hit ray (WF_RAY_MIS_ANY) */
    F_ALL = 2048u,       /* path, All light strategy: the vertex's lights are estimated one per iteration */
};

/* warp-aggregated append to a queue counter */
DF int warp_append(int* counter, bool want) {
    unsigned mask = __ballot_sync(__activemask(), want);
    if (!want) return -1;
    int leader = __ffs(mask) - 1;
    int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(mask));
    base = __shfl_sync(mask, base, leader);
    return base + __popc(mask & ((1u << lane) - 1u));
}

/* Appends a shade's rays and its slot for the next iteration in one pass:
 * the any-hit queue (the warp's shadow rays, then its WF_RAY_MIS_ANY rays),
 * the closest-hit queue (its MIS rays, then its extension rays) and the next active list `next`.  kBlock: one atomic per
 * counter per block, every thread of the block calls it (blockDim.x a
 * multiple of 32); else one per warp, every lane of the warp calls it.  The
 * three counters' atomics are in flight together.  Outputs are queue
 * positions (the shadow one including shadow_base), -1 where not wanted. */
template <bool kBlock>
DF void queue_append(const WfState& W, int next, bool shadow, bool any, bool mis, bool ext, bool keep,
                     int* qs, int* qx, int* qm, int* qe, int* qa) {
    const unsigned full = 0xffffffffu;
    const unsigned bs = __ballot_sync(full, shadow), bx = __ballot_sync(full, any), bm = __ballot_sync(full, mis),
                   be = __ballot_sync(full, ext), ba = __ballot_sync(full, keep);
    const int lane = threadIdx.x & 31;
    int b0, b1, b2;
    if (kBlock) {
        __shared__ int s_cnt[3][32];
        __shared__ int s_base[3];
        const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
        if (lane == 0) { s_cnt[0][w] = __popc(bs) + __popc(bx); s_cnt[1][w] = __popc(bm) + __popc(be); s_cnt[2][w] = __popc(ba); }
        __syncthreads();
        if (threadIdx.x < 3) {
            int* c = threadIdx.x == 0 ? &W.ctr->n_shadow : (threadIdx.x == 1 ? &W.ctr->n_closest : &W.ctr->n_active[next]);
            int t = 0;
            for (int k = 0; k < nw; k++) { const int v = s_cnt[threadIdx.x][k]; s_cnt[threadIdx.x][k] = t; t += v; }
            s_base[threadIdx.x] = t ? atomicAdd(c, t) : 0;
        }
        __syncthreads();
        b0 = s_base[0] + s_cnt[0][w]; b1 = s_base[1] + s_cnt[1][w]; b2 = s_base[2] + s_cnt[2][w];
        __syncthreads();
    } else {
        int v = 0;
        if (lane < 3) {
            const int t = lane == 0 ? __popc(bs) + __popc(bx) : (lane == 1 ? __popc(bm) + __popc(be) : __popc(ba));
            int* c = lane == 0 ? &W.ctr->n_shadow : (lane == 1 ? &W.ctr->n_closest : &W.ctr->n_active[next]);
            if (t) v = atomicAdd(c, t);
        }
        b0 = __shfl_sync(full, v, 0); b1 = __shfl_sync(full, v, 1); b2 = __shfl_sync(full, v, 2);
    }
    const unsigned lt = (1u << lane) - 1u;
    *qs = shadow ? W.shadow_base + b0 + __popc(bs & lt) : -1;
    *qx = any ? W.shadow_base + b0 + __popc(bs) + __popc(bx & lt) : -1;
    *qm = mis ? b1 + __popc(bm & lt) : -1;
    *qe = ext ? b1 + __popc(bm) + __popc(be & lt) : -1;
    *qa = keep ? b2 + __popc(ba & lt) : -1;
}

/* Debug-bounds builds (-DRT_DEBUG_BOUNDS) check every computed index into a
 * path-state buffer: one outside its buffer sets RT_STATUS_BOUNDS and the
 * access is skipped (no trap), so the host reports RT_ERR_BOUNDS. */
#ifdef RT_DEBUG_BOUNDS
DF bool in_bounds(const WfState& W, long long i, long long n) {
    if (i >= 0 && i < n) return true;
    atomicOr(W.status, RT_STATUS_BOUNDS);
    return false;
}
#else
DF bool in_bounds(const WfState&, long long, long long) { return true; }
#endif
DF void set_active(const WfState& W, int list, int a, int slot) {
    if (in_bounds(W, a, W.slots)) W.active[list][a] = slot;
    if (in_bounds(W, slot, W.slots)) W.mark[slot] = (uint8_t)(list + 1);
}
/* a shaded slot that leaves the active lists */
DF void clear_active(const WfState& W, int slot) {
    if (slot >= 0 && in_bounds(W, slot, W.slots)) W.mark[slot] = 0;
}

DF void push_ray4(const WfState& W, int q, int path, int kind, float4 o, float4 d) {
    if (!in_bounds(W, q, 4LL * W.slots)) return;
    W.q_o[q] = o;
    W.q_d[q] = d;
    W.q_meta[q] = (path << 10) | ((int)W.job[path] << 2) | kind;
}

DF void ray4(const Ray& r, float4* o, float4* d) {
    *o = make_float4(r.O.x, r.O.y, r.O.z, r.MinT);
    *d = make_float4(r.D.x, r.D.y, r.D.z, r.MaxT);
}

DF int meta_path(int meta) { return meta >> 10; }
DF int meta_job(int meta) { return (meta >> 2) & (WF_MAX_JOBS - 1); }
DF int meta_kind(int meta) { return meta & 3; }

/* job of a batch-wide sample id (jobs are ordered by their first id) */
DF int job_of(const WfState& W, long long sid) {
    int lo = 0, hi = W.ctr->n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (W.jobs[mid].first <= sid) lo = mid; else hi = mid - 1;
    }
    return lo;
}

/* Rng resumed at draw n of its stream */
DF void rng_resume(Rng& r, uint64_t seed, uint32_t x, uint32_t y, uint32_t s, uint32_t n) {
    rng_init(r, seed, x, y, s);
    r.n = n;
    if (n & 3u) philox(r.c0, r.c1, r.c2, n >> 2, r.k0, r.k1, r.buf);
}

/* sample id -> (crop pixel, sample index in chunk): ids are dense over the
 * crop; within a sample index the pixels run through bands of four rows,
 * column by column, so 32 consecutive ids cover an 8x4 pixel tile */
DF void sample_pixel(const RtParams& P, int64_t sid, int* lx, int* ly, int* k) {
    const int64_t npix = (int64_t)P.w * P.h;
    *k = (int)(sid / npix);
    const int r = (int)(sid - (int64_t)(*k) * npix);
    const int band = r / (4 * P.w);
    const int bh = min(4, P.h - band * 4);
    const int rr = r - band * 4 * P.w;
    *lx = rr / bh;
    *ly = band * 4 + rr % bh;
}

/* The lanes of `active` with `want` claim consecutive sample ids with one
 * atomic; -1 for the others and for ids past the round's end.  Every lane of
 * `active` calls it. */
DF long long claim_sample(const WfState& W, unsigned active, bool want) {
    const unsigned m = __ballot_sync(active, want);
    if (!want) return -1;
    const int leader = __ffs(m) - 1, lane = threadIdx.x & 31;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(&W.ctr->next_sample, (unsigned long long)__popc(m));
    base = __shfl_sync(m, base, leader);
    const long long id = (long long)base + __popc(m & ((1u << lane) - 1u));
    return id < W.ctr->total ? id : -1;
}

/* Initialises camera sample `sid` in `slot`; its first ray goes to W.ray_o /
 * ray_d and to (o, d).  sid < 0 empties the slot.  Returns whether a path
 * started. */
DF bool init_path(const WfState& W, int slot, long long sid, float4* o, float4* d) {
    if (sid < 0) { W.flags[slot] = 0; return false; }
    const int j = job_of(W, sid);
    const WfJob& J = W.jobs[j];
    const RtParams P = J.P;
    W.job[slot] = (uint8_t)j;
    int lx, ly, k;
    sample_pixel(P, sid - J.first, &lx, &ly, &k);
    int px = P.x0 + lx, py = P.y0 + ly, t = P.sample_begin + P.chunk_begin + k;
    Rng rand;
    rng_init(rand, P.seed, (uint32_t)px, (uint32_t)py, (uint32_t)t);
    V2 jit = NextVec2(rand);
    Ray ray = CameraRay(J.view->camera, v2((float)px + jit.x, (float)py + jit.y));
    W.pix[slot] = make_int4(lx, ly, k, t);
    W.rng_n[slot] = rand.n;
    W.coeff[slot] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    W.rad[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    W.bounce[slot] = make_int2(0, 0);
    W.flags[slot] = F_ALIVE | F_SPECULAR | F_EXT;
    W.vol_env[slot] = J.view->global_medium;
    ray4(ray, o, d);
    W.ray_o[slot] = *o;
    W.ray_d[slot] = *d;
    return true;
}

DF Ray queued_ray(const WfState& W, int q) {
    const float4 o = W.q_o[q], d = W.q_d[q];
    return mkray(v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), o.w, d.w);
}

DF void closest_done(const WfState& W, int meta, const Traversal& T) {
    const int path = meta_path(meta);
    const float4 h = make_float4(T.best.t, T.best.u, T.best.v, __int_as_float(T.any ? T.best.slot : -1));
    const int kind = meta_kind(meta);
    if (kind == WF_RAY_EXT) { W.ext_hit[path] = h; W.ext_sub[path] = T.best.sub; }
    else if (kind == WF_RAY_MIS) { W.mis_hit[path] = h; W.mis_sub[path] = T.best.sub; }
    else { W.trw_hit[path] = h; W.trw_sub[path] = T.best.sub; }
}

/* a shadow ray's answer: the path's occlusion flag, or for a light-tracer
 * camera connection its splat, added to the film sums when nothing is in the
 * way (the reference's `lock (renderTarget)` add, AdjointParticleIntegrator.cs:53-66) */
DF void shadow_done(const WfState& W, int meta, bool hit) {
    const int path = meta_path(meta);
    const int kind = meta_kind(meta);
    if (kind == WF_RAY_SHADOW) { W.occluded[path] = hit ? 1 : 0; return; }
    if (kind == WF_RAY_MIS_ANY) { W.mis_sub[path] = hit ? 1 : 0; return; }
    if (hit) return;
    const float4 sp = W.pd_l1[path];
    const int pix = __float_as_int(sp.w);
    const WfJob& J = W.jobs[meta_job(meta)];
    if (pix >= 0 && in_bounds(W, pix, (long long)J.P.w * J.P.h))
        atomicAdd(reinterpret_cast<float4*>(J.samples) + pix, make_float4(sp.x, sp.y, sp.z, 0.0f));
}


/* The rays of W's queue: `fetch` hands out its entries (for kEitherHit an entry's
 * top bit marks an any-hit ray), the results go to the paths' state. */
template <HitForm kForm, bool kSh, NodeMode kMode, class Fetch>
DF void trace_queued(const WfState& W, int refill, Fetch fetch, uint32_t* status, unsigned long long* stats, bool counting) {
    int meta = 0;
    trace_rays<kForm, kSh, kMode>(refill, fetch, [&](int q, Ray* ray) {
        meta = W.q_meta[q];
        *ray = queued_ray(W, q);
        return W.jobs[meta_job(meta)].view;
    }, [&](const RtSceneView*, const Traversal& T) {
        if (kForm == kAnyHit || (kForm == kEitherHit && T.first)) shadow_done(W, meta, T.any);
        else closest_done(W, meta, T);
    }, status, stats, counting);
}

DF bool load_hit(const RtSceneView* S, const Ray& ray, float4 h, int sub, Isect* it) {
    int slot = __float_as_int(h.w);
    if (slot < 0) return false;
    Best b;
    b.t = h.x; b.u = h.y; b.v = h.z; b.slot = slot; b.sub = sub; b.flags = 0;
    b.pw = v3s(0);
    /* instance hits: the world point is recomputed exactly as during traversal */
    float4 s1 = __ldg(S->slots + 3 * (int64_t)slot + 1);
    uint32_t kr = __float_as_uint(s1.w);
    if ((kr >> RT_KIND_SHIFT) == RT_KIND_INSTANCE) {
        const RtInstance& I = S->instances[kr & RT_REF_MASK];
        float w2m[12], m2w[12];
        for (int q = 0; q < 12; q++) { w2m[q] = I.w2m[q]; m2w[q] = I.m2w[q]; }
        float4 p1 = __ldg(S->slots + 3 * (int64_t)sub + 1);
        uint32_t pkr = __float_as_uint(p1.w);
        V3 pm;
        if ((pkr >> RT_KIND_SHIFT) == RT_KIND_TRI) {
            V3 bary = v3(1 - (b.u + b.v), b.u, b.v);
            RtTri t = S->tris[pkr & RT_REF_MASK];
            pm = bary.x * f4xyz(S->pos[t.v0]) + bary.y * f4xyz(S->pos[t.v1]) + bary.z * f4xyz(S->pos[t.v2]);
        } else {
            RtSphere sph = S->spheres[pkr & RT_REF_MASK];
            V3 c = v3(sph.center[0], sph.center[1], sph.center[2]);
            Ray mr = XfRay(ray, w2m);
            float tm = 0;
            SphereTest(c, sph.radius, mr, &tm);
            V3 n = Normalize(At(mr, tm) - c);
            pm = n * sph.radius + c;
        }
        b.pw = Xf12(pm, m2w);
    }
    Finish(S, ray, b, it);
    return true;
}

DF void finish_path(const WfJob& J, const WfState& W, int slot, C3 rad, unsigned long long* stats, int pass) {
    if (pass == WF_PASS_REPLAY) return;
    bool invalid = !IsValid(rad);
    if (invalid && pass == WF_PASS_RENDER) { rad = c3s(0.0f); atomicAdd(stats + 6, 1ull); }
    int4 px = W.pix[slot];
    const RtParams& P = J.P;
    const int64_t npix = (int64_t)P.w * P.h;
    const int64_t sample = (int64_t)px.z * npix + (int64_t)px.x * P.h + px.y;
    if (!in_bounds(W, sample, J.count)) return;
    float* o = J.samples + sample * 3;
    o[0] = rad.r; o[1] = rad.g; o[2] = rad.b;
}

/* What a path shade leaves for the queues: its shadow ray, whether it
 * queued a MIS ray (in pd_ray_o / pd_ray_d; mis_any: as an any-hit ray) or an
 * extension ray (in ray_o / ray_d), whether the slot stays active, and whether the path is over (the
 * caller starts the next camera sample in the slot). */
struct PathOut {
    float4 so, sd;
    bool shadow, mis_any, mis, ext, keep, restart;
};

/* The MIS ray towards an infinite light: EstimateDirect (PathTracer.cs:370-399)
 * takes the radiance of what the ray hits only where that is the sampled light
 * itself, which no primitive is, and the environment where it hits nothing.
 * So the ray stops at its first hit - the same answer as the closest hit's
 * existence - and the term it gates is complete when it is queued: the next
 * shade adds it as it adds a light-sample term, without an intersection or the
 * ray's direction and BSDF value.  A ray that could carry nothing is not traced. */
DF bool MisAny(const WfState& W, const RtSceneView* S, int light) {
    return W.mis_any && S->lights[light].kind == RT_LIGHT_INFINITE;
}

/* Schedules one light's direct term at vertex `it` (PathTracer.cs:309-399
 * for Mis, :95-190 for Nee): draws its light sample and, for Mis, its BSDF
 * sample, stores the term's parts and queues its shadow / MIS rays; the next
 * shade adds it once they are traced.  lightPdf: SampleLight's pdf (Uniform)
 * or 1 (All). */
template <bool kAdj>
DF void schedule_direct(PathOut* o, const WfState& W, const RtSceneView* S, int slot, const Isect& it, V3 wo, int mat,
                        const MatAt& at, int light, float lightPdf, C3 coeff, int method, Rng& rand, uint32_t& fl, float4& rho) {
    if (method == RT_METHOD_MIS) {
        fl |= F_PENDING;
        W.pd_coeff[slot] = make_float4(coeff.r, coeff.g, coeff.b, lightPdf);
        if (lightPdf > 0.0f) {
            V3 wod = it.Wr;
            LSample ls = LightSampleLi(S, light, it.P, rand);
            if (ls.Pdf > 0.0f && !IsBlack(ls.Li)) {
                const float4 ev = MatEval(S, mat, at, Lo(it, wod), Lo(it, ls.Wi));
                C3 fr = c3(ev.x, ev.y, ev.z);
                const float scatteringPdf = ev.w;
                if (!IsBlack(fr)) {
                    /* IsOccluded(it.P, ls.P) */
                    V3 vec = ls.P - it.P;
                    float dis = Length(vec);
                    if (!(dis < 0.001f)) {
                        fr = fr * AbsCosTheta(Lo(it, ls.Wi));
                        float weight = PowerHeuristic(ls.Pdf, scatteringPdf);
                        if (kAdj && __float_as_int(rho.w) >= 0)
                            rho.x = DirectDln(S, mat, Lo(it, wod), Lo(it, ls.Wi), weight, true, it.UV);
                        C3 l1 = fr * ls.Li * weight / ls.Pdf;
                        W.pd_l1[slot] = make_float4(l1.r, l1.g, l1.b, 0);
                        fl |= F_L1;
                        ray4(mkray(it.P, Normalize(vec), 0.0001f, dis - 0.0001f), &o->so, &o->sd);
                        o->shadow = true;
                    }
                }
            }
            BSample sample = MatSampleAt(S, mat, at, Lo(it, wod), rand);
            C3 fr = sample.Fr * AbsCosTheta(sample.Wi);
            float scatteringPdf = sample.Pdf;
            bool sampledSpecular = (sample.Type & BX_SPECULAR) != 0;
            if (!IsBlack(fr) && scatteringPdf > 0) {
                const V3 wiw = Wo(it, sample.Wi);
                const bool any = MisAny(W, S, light);
                C3 env = c3s(0.0f);          /* any: the radiance the ray carries if it hits nothing */
                float weight = 1;
                bool go = true;
                if (!sampledSpecular) {
                    float bxdfToLightPdf;
                    if (any) {
                        const float4 e = EnvPdfLe(S, light, wiw);
                        env = c3(e.x, e.y, e.z);
                        bxdfToLightPdf = e.w;
                    } else {
                        bxdfToLightPdf = LightPdfLi(S, light, it.P, wiw);
                    }
                    if (bxdfToLightPdf == 0.0f) go = false;
                    else weight = PowerHeuristic(scatteringPdf, bxdfToLightPdf);
                } else if (any) {
                    env = EvalAllInfinite(S, wiw);
                }
                if (go) {
                    if (kAdj && __float_as_int(rho.w) >= 0)
                        rho.y = DirectDln(S, mat, Lo(it, wod), sample.Wi, sampledSpecular ? 2.0f : weight, false,
                                          it.UV);
                    const Ray toLight = Spawn(it, wiw);
                    if (!any) {
                        V3 wle = Wo(it, -sample.Wi);
                        W.pd_fr[slot] = make_float4(fr.r, fr.g, fr.b, weight);
                        W.pd_mis[slot] = make_float4(scatteringPdf, __int_as_float(light), 0, 0);
                        W.pd_w[slot] = make_float4(wle.x, wle.y, wle.z, 0);
                        fl |= F_L2;
                        o->mis = true;
                    } else if (!IsBlack(env)) {
                        const C3 l2 = fr * env * weight / scatteringPdf;
                        W.pd_fr[slot] = make_float4(l2.r, l2.g, l2.b, 0);
                        fl |= F_L2 | F_ANY;
                        o->mis_any = true;
                    }
                    if (o->mis || o->mis_any) {
                        W.pd_ray_o[slot] = make_float4(toLight.O.x, toLight.O.y, toLight.O.z, toLight.MinT);
                        W.pd_ray_d[slot] = make_float4(toLight.D.x, toLight.D.y, toLight.D.z, toLight.MaxT);
                    }
                }
            }
        } else {
            fl |= F_DZERO;
        }
    } else { /* NEE: NeeEstimateLight */
        if (lightPdf > 0.0f) {
            fl |= F_PENDING;
            W.pd_coeff[slot] = make_float4(coeff.r, coeff.g, coeff.b, lightPdf);
            LSample r = LightSampleLi(S, light, it.P, rand);
            bool zero = true;
            if (r.Pdf > 0.0f) {
                V3 vec = r.P - it.P;
                float dis = Length(vec);
                if (!(dis < 0.001f)) {
                    C3 fr = MatFrAt(S, mat, at, Lo(it, wo), Lo(it, r.Wi));
                    C3 e = fr * r.Li * AbsCosTheta(Lo(it, r.Wi)) / r.Pdf;
                    W.pd_l1[slot] = make_float4(e.r, e.g, e.b, 0);
                    zero = false;
                    ray4(mkray(it.P, Normalize(vec), 0.0001f, dis - 0.0001f), &o->so, &o->sd);
                    o->shadow = true;
                }
            }
            if (zero) fl |= F_DZERO;
        }
    }
}

/* Adds the direct term that the slot's previous shade scheduled, then runs one
 * bounce of PathTracer.Mis / NextEventEstimation / OnlySampleBxdf after its
 * extension hit (PathTracer.cs:43-270); its rays and what becomes of the slot go
 * to `o`. */
template <bool kAdj>
DF void shade_path(PathOut* o, const WfState& W, int slot, uint32_t* status, unsigned long long* stats, bool counting,
                   int pass, const WfAdjoint& A, float* s_alpha) {
    const WfJob& J = W.jobs[W.job[slot]];
    const RtSceneView* S = J.view;
    const RtParams P = J.P;                  /* registers: the path-state stores below cannot alias it */
    uint32_t fl = W.flags[slot];
    float4 cf = W.coeff[slot], rd = W.rad[slot];
    C3 coeff = c3(cf.x, cf.y, cf.z), radiance = c3(rd.x, rd.y, rd.z);
    /* replay: the sample's radiance from the forward pass and its pixel's dL/dI */
    C3 Ltot = c3s(0.0f), dL = c3s(0.0f);
    bool grad = false;
    if (kAdj) {
        const int4 q = W.pix[slot];
        const int64_t pix = (int64_t)q.x * P.h + q.y;
        const float* ls = J.samples + ((int64_t)q.z * P.w * P.h + pix) * 3;
        Ltot = c3(ls[0], ls[1], ls[2]);
        dL = c3(A.dLdI[pix * 3], A.dLdI[pix * 3 + 1], A.dLdI[pix * 3 + 2]);
        grad = IsValid(Ltot) && (dL.r != 0.0f || dL.g != 0.0f || dL.b != 0.0f);
    }

    /* 1. the direct term scheduled by the previous bounce (or, All strategy,
     * the term of one light of this vertex) */
    bool resume = false;                     /* All: the vertex's last light is in, its continuation runs below */
    if (fl & F_PENDING) {
        float4 pc = W.pd_coeff[slot];
        C3 coeffb = c3(pc.x, pc.y, pc.z);
        float lightPdf = pc.w;
        const bool all = (fl & F_ALL) != 0;
        if (P.method == RT_METHOD_MIS) {
            C3 direct = c3s(0);
            C3 tl = c3s(0.0f), tb = c3s(0.0f);
            C3 le = c3s(0.0f);
            if (!(fl & F_DZERO)) {
                if ((fl & F_L1) && !W.occluded[slot]) {
                    float4 l1 = W.pd_l1[slot];
                    tl = c3(l1.x, l1.y, l1.z);
                    le = le + tl;
                }
                if ((fl & F_L2) && (fl & F_ANY)) {
                    if (!W.mis_sub[slot]) {
                        const float4 l2 = W.pd_fr[slot];
                        tb = c3(l2.x, l2.y, l2.z);
                        le = le + tb;
                    }
                } else if (fl & F_L2) {
                    float4 fr2 = W.pd_fr[slot];
                    float4 mi = W.pd_mis[slot];
                    float4 wl = W.pd_w[slot];
                    const int light = __float_as_int(mi.y);
                    C3 li = c3s(0);
                    Isect lit;
                    float4 mo = W.pd_ray_o[slot], md = W.pd_ray_d[slot];
                    Ray mr = mkray(v3(mo.x, mo.y, mo.z), v3(md.x, md.y, md.z), mo.w, md.w);
                    if (load_hit(S, mr, W.mis_hit[slot], W.mis_sub[slot], &lit)) {
                        if (LightOf(S, lit) >= 0 && LightOf(S, lit) == light) li = IsectLe(S, lit, v3(wl.x, wl.y, wl.z));
                    } else {
                        li = EvalAllInfinite(S, mr.D);
                    }
                    if (!IsBlack(li)) { tb = c3(fr2.x, fr2.y, fr2.z) * li * fr2.w / mi.x; le = le + tb; }
                }
                if (!all) direct = direct + le / lightPdf;
            }
            if (all) {
                /* PathTracer.cs:297-304: result += EstimateDirect(light) over Scene.Lights */
                const float4 ac = W.pd_acc[slot];
                const C3 acc = c3(ac.x, ac.y, ac.z) + le;
                W.pd_acc[slot] = make_float4(acc.r, acc.g, acc.b, ac.w);
            } else {
                radiance = radiance + coeffb * direct;
            }
            if (kAdj && grad && !all) {
                /* alpha terms of the pending vertex: its two direct terms, then its
                 * continuation, which carries everything after its direct light */
                const float4 ar = W.adj_rho[slot];
                const int aslot = __float_as_int(ar.w);
                if (aslot >= 0) {
                    float g = ar.z * Dot3(dL, Ltot - radiance);
                    if (!IsBlack(tl)) g += ar.x * Dot3(dL, coeffb * tl) / lightPdf;
                    if (!IsBlack(tb)) g += ar.y * Dot3(dL, coeffb * tb) / lightPdf;
                    if (g != 0.0f) atomicAdd(s_alpha + aslot, g);
                }
            }
        } else { /* NEE */
            C3 e = c3s(0);
            if (!(fl & F_DZERO) && !W.occluded[slot]) { float4 l1 = W.pd_l1[slot]; e = c3(l1.x, l1.y, l1.z); }
            radiance = all ? radiance + coeffb * e : radiance + coeffb * e / lightPdf;
        }
        fl &= ~(F_PENDING | F_L1 | F_L2 | F_DZERO | F_ANY);
        if (all) {
            const float4 ac = W.pd_acc[slot];
            const int next = __float_as_int(ac.w) + 1;
            if (next < S->light_count) {
                /* the next light at the same vertex: its draws follow the previous light's */
                const float4 ro = W.ray_o[slot], rdd = W.ray_d[slot];
                const Ray ray = mkray(v3(ro.x, ro.y, ro.z), v3(rdd.x, rdd.y, rdd.z), ro.w, rdd.w);
                Isect it;
                load_hit(S, ray, W.ext_hit[slot], W.ext_sub[slot], &it);
                const int4 px = W.pix[slot];
                Rng rand;
                rng_resume(rand, P.seed, (uint32_t)(P.x0 + px.x), (uint32_t)(P.y0 + px.y), (uint32_t)px.w, W.rng_n[slot]);
                float4 rho = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
                const int mat = PrimOf(S, it).material;
                schedule_direct<kAdj>(o, W, S, slot, it, -ray.D, mat, MatLookup(S, S->materials[mat], it.UV), next, 1.0f,
                                      coeffb, P.method, rand, fl, rho);
                W.pd_acc[slot] = make_float4(ac.x, ac.y, ac.z, __int_as_float(next));
                W.rng_n[slot] = rand.n;
                W.flags[slot] = fl;
                W.rad[slot] = make_float4(radiance.r, radiance.g, radiance.b, 0);
                o->keep = true;
                return;
            }
            if (P.method == RT_METHOD_MIS) radiance = radiance + coeffb * c3(ac.x, ac.y, ac.z);
            fl &= ~F_ALL;
            resume = true;
        }
    }

    bool done = (fl & F_DONE) != 0;
    if (!done) {
        /* 2. the bounce itself */
        int2 bc = W.bounce[slot];
        int bounces = bc.x, guard = bc.y;
        float4 ro = W.ray_o[slot], rdd = W.ray_d[slot];
        Ray ray = mkray(v3(ro.x, ro.y, ro.z), v3(rdd.x, rdd.y, rdd.z), ro.w, rdd.w);
        int4 px = W.pix[slot];
        Rng rand;
        rng_resume(rand, P.seed, (uint32_t)(P.x0 + px.x), (uint32_t)(P.y0 + px.y), (uint32_t)px.w, W.rng_n[slot]);
        bool isSpecularPath = (fl & F_SPECULAR) != 0;
        Ray nray = ray;
        bool ext = false;
        do {
            if (!resume && ++guard > RT_LOOP_CAP) { atomicOr(status, RT_STATUS_ITER); done = true; break; }
            Isect it;
            bool isHit = load_hit(S, ray, W.ext_hit[slot], W.ext_sub[slot], &it);
            V3 wo = -ray.D;
            if (resume) {
                /* All: emission and the lights of this vertex are in; its continuation follows */
            } else if (P.method == RT_METHOD_BXDF) {
                if (!isHit) { radiance = radiance + coeff * EvalAllInfinite(S, ray.D); done = true; break; }
                if (P.max_depth != -1 && bounces >= P.max_depth) { done = true; break; }
                if (!HasSurface(S, it)) { nray = mkray(it.P, ray.D, ray.MinT); ext = true; break; }
                if (LightOf(S, it) >= 0) radiance = radiance + coeff * IsectLe(S, it, wo);
            } else {
                if (bounces == 0 || isSpecularPath) {
                    if (isHit) radiance = radiance + coeff * IsectLe(S, it, wo);
                    else radiance = radiance + coeff * EvalAllInfinite(S, ray.D);
                }
                if (!isHit) { done = true; break; }
                if (P.max_depth != -1 && bounces >= P.max_depth) { done = true; break; }
                if (!HasSurface(S, it)) { nray = mkray(it.P, ray.D, ray.MinT); ext = true; break; }
            }
            /* the vertex's texture values, for its direct light and its continuation */
            const int mat = PrimOf(S, it).material;
            const MatAt at = MatLookup(S, S->materials[mat], it.UV);
            if (!resume && P.method != RT_METHOD_BXDF) {
                /* direct lighting: everything but the two ray casts */
                float4 rho = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
                if (kAdj && grad) {
                    if (UsesAlbedo(S, A.albedo_tex, mat)) {
                        const C3 R = TexSample(S, A.albedo_tex, it.UV);
                        const C3 rest = Ltot - radiance;
                        ScatterAlbedo(S, A.albedo_tex, A.grad_albedo, it.UV,
                                      c3(R.r > 0 ? dL.r * rest.r / R.r : 0.0f, R.g > 0 ? dL.g * rest.g / R.g : 0.0f,
                                         R.b > 0 ? dL.b * rest.b / R.b : 0.0f));
                    }
                    if (A.alpha_slot) rho.w = __int_as_float(A.alpha_slot[mat]);
                }
                if (P.strategy == RT_STRATEGY_ALL) {
                    if (S->light_count > 0) {
                        /* light 0 now, the others one per iteration; the continuation waits */
                        fl |= F_ALL;
                        W.pd_acc[slot] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(0));
                        schedule_direct<kAdj>(o, W, S, slot, it, wo, mat, at, 0, 1.0f, coeff, P.method, rand, fl, rho);
                        break;
                    }
                    if (P.method == RT_METHOD_MIS) radiance = radiance + coeff * c3s(0.0f);
                } else {
                    int light;
                    float lightPdf = SampleLight(S, rand, &light);
                    schedule_direct<kAdj>(o, W, S, slot, it, wo, mat, at, light, lightPdf, coeff, P.method, rand, fl, rho);
                }
                if (kAdj) W.adj_rho[slot] = rho;
            }
            /* continuation */
            BSample s = MatSampleAt(S, mat, at, Lo(it, wo), rand);
            if (kAdj && P.method == RT_METHOD_MIS && (fl & F_PENDING)) {
                float4 rho = W.adj_rho[slot];
                float rc = 0.0f, rcp;
                if (__float_as_int(rho.w) >= 0 && s.Pdf > 0.0f)
                    DlnAlpha(S, mat, Lo(it, wo), s.Wi, it.UV, &rc, &rcp);
                rho.z = rc;
                W.adj_rho[slot] = rho;
            }
            if (P.method != RT_METHOD_BXDF) isSpecularPath = (s.Type & BX_SPECULAR) != 0;
            if (s.Pdf > 0.0f) coeff = coeff * (s.Fr * AbsCosTheta(s.Wi) / s.Pdf);
            else { done = true; break; }
            nray = Spawn(it, Wo(it, s.Wi));
            if (bounces > P.min_depth) {
                float q = nmin(MaxElement(coeff), P.rr);
                if (NextFloat(rand) > q) { done = true; break; }
                coeff = coeff / q;
            }
            bounces++;
            ext = true;
        } while (false);
        if (ext) {
            W.ray_o[slot] = make_float4(nray.O.x, nray.O.y, nray.O.z, nray.MinT);
            W.ray_d[slot] = make_float4(nray.D.x, nray.D.y, nray.D.z, nray.MaxT);
            o->ext = true;
        }
        W.bounce[slot] = make_int2(bounces, guard);
        W.rng_n[slot] = rand.n;
        fl = (fl & ~F_SPECULAR) | (isSpecularPath ? F_SPECULAR : 0u);
        if (done) fl |= F_DONE;
    }
    W.coeff[slot] = make_float4(coeff.r, coeff.g, coeff.b, 0);
    W.rad[slot] = make_float4(radiance.r, radiance.g, radiance.b, 0);
    /* the slot stays active while it waits for rays */
    if ((fl & F_PENDING) || !(fl & F_DONE)) {
        W.flags[slot] = fl;
        o->keep = true;
        return;
    }
    finish_path(J, W, slot, radiance, stats, pass);
    if (counting) warp_add64(stats + 0, 1u);
    o->restart = true;
}

/* The shade's queue appends, for the block (kBlock) or the warp: a finished
 * path's slot takes the next camera sample at once. */
template <bool kBlock>
DF void path_queues(const WfState& W, int slot, int next, PathOut& o) {
    const long long sid = claim_sample(W, 0xffffffffu, o.restart);
    float4 ro, rd;
    if (o.restart && init_path(W, slot, sid, &ro, &rd)) { o.ext = true; o.keep = true; }
    int qs, qx, qm, qe, qa;
    queue_append<kBlock>(W, next, o.shadow, o.mis_any, o.mis, o.ext, o.keep, &qs, &qx, &qm, &qe, &qa);
    if (o.shadow) push_ray4(W, qs, slot, WF_RAY_SHADOW, o.so, o.sd);
    if (o.mis_any) push_ray4(W, qx, slot, WF_RAY_MIS_ANY, W.pd_ray_o[slot], W.pd_ray_d[slot]);
    if (o.mis) push_ray4(W, qm, slot, WF_RAY_MIS, W.pd_ray_o[slot], W.pd_ray_d[slot]);
    if (o.ext) {
        if (!o.restart) { ro = W.ray_o[slot]; rd = W.ray_d[slot]; }
        push_ray4(W, qe, slot, WF_RAY_EXT, ro, rd);
    }
    if (o.keep) set_active(W, next, qa, slot);
    else clear_active(W, slot);
}

/* ---- vol_path (VolumetricPathTracer.Li, Integrators/VolumetricPathTracer.cs) ----
 * A bounce draws all of its random numbers in one shade, in the reference's
 * order: medium distance, light choice and sample, phase / BSDF sample of
 * the direct term, continuation, Russian roulette.  The boundary walks of
 * the direct term (Scene.Transmittance towards the light sample,
 * Scene.IntersectTr along the phase / BSDF sample) draw none; each of their
 * segments is one closest-hit ray, traced in later iterations while the
 * path waits.  When both walks are done the direct term is added, then the
 * continuation ray (already sampled) is enqueued, so radiance accumulates
 * in the reference's order. */

DF int pack_env(int env, int count) { return (count << 16) | ((env + 1) & 0xFFFF); }
DF int env_of(int packed) { return (packed & 0xFFFF) - 1; }
DF int count_of(int packed) { return packed >> 16; }

/* the next Transmittance segment from the walk's current start (o, d); false: the walk is over */
DF bool trw_ray(const WfState& W, int slot, float4* o, float4* d) {
    const float4 st = W.trw_start[slot], en = W.trw_end[slot], dr = W.trw_dir[slot];
    const V3 start = v3(st.x, st.y, st.z), to = v3(en.x, en.y, en.z);
    const float dis = Length(to - start);
    if (dis < 0.0001f) return false;
    ray4(mkray(start, v3(dr.x, dr.y, dr.z), 0.0001f, dis - 0.0001f), o, d);
    return true;
}
DF bool trw_next(const WfState& W, int slot) {
    float4 o, d;
    return trw_ray(W, slot, &o, &d);
}
/* Scene.Transmittance (Scene.cs:72-103), one traced segment; true: continues */
DF bool trw_step(const RtSceneView* S, const WfState& W, int slot) {
    float4 st = W.trw_start[slot], en = W.trw_end[slot];
    const float4 dr = W.trw_dir[slot], trv = W.trw_tr[slot];
    V3 start = v3(st.x, st.y, st.z);
    const V3 to = v3(en.x, en.y, en.z), dir = v3(dr.x, dr.y, dr.z);
    int env = __float_as_int(st.w), count = __float_as_int(en.w);
    const float dis = Length(to - start);
    const Ray ray = mkray(start, dir, 0.0001f, dis - 0.0001f);
    Isect inct;
    const bool anyHit = load_hit(S, ray, W.trw_hit[slot], W.trw_sub[slot], &inct);
    C3 tr = c3(trv.x, trv.y, trv.z);
    bool more = true;
    if (anyHit && HasSurface(S, inct)) { tr = c3s(0.0f); more = false; }
    else {
        if (env >= 0) tr = tr * MedTr(S->media[env], ray);
        if (!anyHit) more = false;
        else {
            start = inct.P;
            env = GetMedium(S, inct, dir);
            if (++count >= RT_WALK_CAP) { more = false; atomicOr(W.status, RT_STATUS_WALK); }
        }
    }
    W.trw_tr[slot] = make_float4(tr.r, tr.g, tr.b, 0.0f);
    if (!more) return false;
    W.trw_start[slot] = make_float4(start.x, start.y, start.z, __int_as_float(env));
    W.trw_end[slot] = make_float4(to.x, to.y, to.z, __int_as_float(count));
    return trw_next(W, slot);
}
/* Scene.IntersectTr (Scene.cs:105-131), one traced segment; true: continues.
 * When over, itw_o holds the radiance found (light-identity check of
 * EstimateDirect, or the environment on a miss) and itw_tr the throughput. */
DF bool itw_step(const RtSceneView* S, const WfState& W, int slot, int light, V3 wle) {
    const float4 o = W.itw_o[slot], d = W.itw_d[slot], trv = W.itw_tr[slot];
    Ray ray = mkray(v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), o.w);
    const int packed = __float_as_int(trv.w);
    int env = env_of(packed), count = count_of(packed);
    C3 tr = c3(trv.x, trv.y, trv.z);
    Isect inct;
    const bool anyHit = load_hit(S, ray, W.mis_hit[slot], W.mis_sub[slot], &inct);
    C3 li = c3s(0.0f);
    bool more = false;
    if (!anyHit) {
        if (env >= 0) tr = tr * MedTr(S->media[env], ray);
        li = EvalAllInfinite(S, ray.D);
    } else {
        if (env >= 0) {
            const Ray realPath = mkray(ray.O, ray.D, ray.MinT, Length(At(ray, inct.T)));
            tr = tr * MedTr(S->media[env], realPath);
        }
        if (HasSurface(S, inct)) {
            if (LightOf(S, inct) >= 0 && LightOf(S, inct) == light) li = IsectLe(S, inct, wle);
        } else if (++count >= RT_WALK_CAP) {
            li = EvalAllInfinite(S, ray.D);             /* the walk gives up: a miss */
            atomicOr(W.status, RT_STATUS_WALK);
        } else {
            ray = mkray(inct.P, ray.D, 0.001f);
            env = GetMedium(S, inct, ray.D);
            more = true;
        }
    }
    if (more) {
        W.itw_o[slot] = make_float4(ray.O.x, ray.O.y, ray.O.z, ray.MinT);
        W.itw_tr[slot] = make_float4(tr.r, tr.g, tr.b, __int_as_float(pack_env(env, count)));
        return true;
    }
    W.itw_o[slot] = make_float4(li.r, li.g, li.b, 0.0f);
    W.itw_tr[slot] = make_float4(tr.r, tr.g, tr.b, 0.0f);
    return false;
}

/* What a vol_path shade leaves for the queues: a Transmittance segment
 * (its ray rebuilt from trw_*), an IntersectTr segment (from itw_*) or the
 * extension ray (ray_o / ray_d), whether the slot stays active, whether the
 * path is over.  A shade starts walk segments or an extension ray, never both. */
struct VolOut {
    bool trw, itw, ext, keep, restart;
};

/* one shade of a vol_path slot */
DF void shade_vol_path(VolOut* o, const WfState& W, int slot, uint32_t* status, unsigned long long* stats,
                       bool counting) {
    const WfJob& J = W.jobs[W.job[slot]];
    const RtSceneView* S = J.view;
    const RtParams P = J.P;
    uint32_t fl = W.flags[slot];
    /* 1. the boundary walks of a pending direct term */
    if (fl & (F_WTR | F_WIT)) {
        if ((fl & F_WTR) && !trw_step(S, W, slot)) fl &= ~F_WTR;
        if (fl & F_WIT) {
            const float4 mi = W.pd_mis[slot], wl = W.pd_w[slot];
            if (!itw_step(S, W, slot, __float_as_int(mi.y), v3(wl.x, wl.y, wl.z))) fl &= ~F_WIT;
        }
        if (fl & (F_WTR | F_WIT)) {
            W.flags[slot] = fl;
            o->trw = (fl & F_WTR) != 0;
            o->itw = (fl & F_WIT) != 0;
            o->keep = true;
            return;
        }
    }
    float4 cf = W.coeff[slot], rdv = W.rad[slot];
    C3 coeff = c3(cf.x, cf.y, cf.z), radiance = c3(rdv.x, rdv.y, rdv.z);
    bool ext = false;
    for (int pass = 0; pass < 2; pass++) {
        /* 2. the direct term, now that its walks are done (EstimateDirectSurface / Medium) */
        if (fl & F_PENDING) {
            const float4 pc = W.pd_coeff[slot];
            C3 direct = c3s(0.0f);
            if (!(fl & F_DZERO)) {
                C3 le = c3s(0.0f);
                if (fl & F_L1) {
                    const float4 l1 = W.pd_l1[slot], lr = W.vol_li[slot], t = W.trw_tr[slot];
                    const C3 lightLi = c3(lr.x, lr.y, lr.z) * c3(t.x, t.y, t.z);
                    if (!IsBlack(lightLi)) le = le + c3(l1.x, l1.y, l1.z) * lightLi * l1.w / W.pd_mis[slot].z;
                }
                if (fl & F_L2) {
                    const float4 fr2 = W.pd_fr[slot], mi = W.pd_mis[slot], li = W.itw_o[slot], t = W.itw_tr[slot];
                    const C3 L = c3(li.x, li.y, li.z);
                    if (!IsBlack(L)) le = le + c3(fr2.x, fr2.y, fr2.z) * L * c3(t.x, t.y, t.z) * fr2.w / mi.x;
                }
                direct = direct + le / pc.w;
            }
            radiance = radiance + c3(pc.x, pc.y, pc.z) * direct;
            fl &= ~(F_PENDING | F_L1 | F_L2 | F_DZERO);
        }
        if (fl & F_DONE) break;
        if (fl & F_CONT) {                       /* 3. the continuation sampled with the term */
            fl &= ~F_CONT;
            ext = true;
            break;
        }
        if (pass == 1) break;
        /* 4. one iteration of the Li loop on the extension hit */
        int2 bc = W.bounce[slot];
        int bounces = bc.x, guard = bc.y;
        float4 ro = W.ray_o[slot], rd = W.ray_d[slot];
        Ray ray = mkray(v3(ro.x, ro.y, ro.z), v3(rd.x, rd.y, rd.z), ro.w, rd.w);
        int env = W.vol_env[slot];
        const int4 px = W.pix[slot];
        Rng rand;
        rng_resume(rand, P.seed, (uint32_t)(P.x0 + px.x), (uint32_t)(P.y0 + px.y), (uint32_t)px.w, W.rng_n[slot]);
        bool isSpecularPath = (fl & F_SPECULAR) != 0;
        bool done = false, rr = true;
        do {
            if (++guard > RT_LOOP_CAP) { atomicOr(status, RT_STATUS_ITER); done = true; break; }
            const V3 wo = -ray.D;
            if (ray.MaxT <= ray.MinT) { done = true; break; }
            Isect it;
            const bool isHit = load_hit(S, ray, W.ext_hit[slot], W.ext_sub[slot], &it);
            MedSample msr; msr.sampled = false;
            if (env >= 0) {
                const Ray realRay = mkray(ray.O, ray.D, ray.MinT, isHit ? it.T : kFMax);
                msr = MedSampleDist(S->media[env], realRay, rand);
                coeff = coeff * msr.Tr;
            }
            if (IsBlack(coeff)) { done = true; break; }
            if (msr.sampled) {
                if (bounces >= P.max_depth) { done = true; break; }   /* VolumetricPathTracer.cs:55 */
                const RtMedium& M = S->media[env];
                int light;
                const float lightPdf = SampleLight(S, rand, &light);
                fl |= F_PENDING;
                W.pd_coeff[slot] = make_float4(coeff.r, coeff.g, coeff.b, lightPdf);
                if (lightPdf > 0.0f) {
                    const LSample ls = LightSampleLi(S, light, msr.P, rand);
                    if (ls.Pdf > 0.0f && !IsBlack(ls.Li)) {
                        const float p = MedP(M, msr.Wo, ls.Wi);
                        if (p != 0.0f) {
                            fl |= F_L1 | F_WTR;
                            const float weight = PowerHeuristic(ls.Pdf, p);
                            W.pd_l1[slot] = make_float4(p, p, p, weight);
                            W.vol_li[slot] = make_float4(ls.Li.r, ls.Li.g, ls.Li.b, 0.0f);
                            const V3 dir = Normalize(ls.P - msr.P);
                            W.trw_start[slot] = make_float4(msr.P.x, msr.P.y, msr.P.z, __int_as_float(env));
                            W.trw_end[slot] = make_float4(ls.P.x, ls.P.y, ls.P.z, __int_as_float(0));
                            W.trw_dir[slot] = make_float4(dir.x, dir.y, dir.z, 0.0f);
                            W.trw_tr[slot] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
                        }
                    }
                    V3 swi;
                    const float sp = MedSampleWi(M, msr.Wo, rand, &swi);
                    if (sp > 0) {
                        const float b2l = LightPdfLi(S, light, msr.P, swi);
                        if (b2l != 0.0f) {
                            fl |= F_L2 | F_WIT;
                            const float weight = PowerHeuristic(sp, b2l);
                            const Ray toLight = mkray(msr.P, swi);
                            W.pd_fr[slot] = make_float4(sp, sp, sp, weight);
                            W.pd_mis[slot] = make_float4(sp, __int_as_float(light), ls.Pdf, 0.0f);
                            W.pd_w[slot] = make_float4(-swi.x, -swi.y, -swi.z, 0.0f);
                            W.itw_o[slot] = make_float4(toLight.O.x, toLight.O.y, toLight.O.z, toLight.MinT);
                            W.itw_d[slot] = make_float4(toLight.D.x, toLight.D.y, toLight.D.z, 0.0f);
                            W.itw_tr[slot] = make_float4(1.0f, 1.0f, 1.0f, __int_as_float(pack_env(env, 0)));
                        } else {
                            W.pd_mis[slot] = make_float4(sp, __int_as_float(light), ls.Pdf, 0.0f);
                        }
                    } else {
                        W.pd_mis[slot] = make_float4(0.0f, __int_as_float(light), ls.Pdf, 0.0f);
                    }
                } else {
                    fl |= F_DZERO;
                }
                V3 swi;
                MedSampleWi(M, wo, rand, &swi);
                ray = mkray(msr.P, swi, ray.MinT);
                isSpecularPath = false;
            } else {
                if (bounces == 0 || isSpecularPath) {
                    if (isHit) radiance = radiance + coeff * IsectLe(S, it, wo);
                    else radiance = radiance + coeff * EvalAllInfinite(S, ray.D);
                }
                if (!isHit) { done = true; break; }
                if (P.max_depth != -1 && bounces >= P.max_depth) { done = true; break; }
                if (!HasSurface(S, it)) {
                    ray = mkray(it.P, ray.D, ray.MinT);
                    env = GetMedium(S, it, ray.D);
                    bounces--;
                    rr = false;                  /* `continue`: no Russian roulette this iteration */
                    break;
                }
                const int mat = PrimOf(S, it).material;
                const MatAt at = MatLookup(S, S->materials[mat], it.UV);
                int light;
                const float lightPdf = SampleLight(S, rand, &light);
                fl |= F_PENDING;
                W.pd_coeff[slot] = make_float4(coeff.r, coeff.g, coeff.b, lightPdf);
                if (lightPdf > 0.0f) {
                    const V3 wod = it.Wr;
                    const LSample ls = LightSampleLi(S, light, it.P, rand);
                    if (ls.Pdf > 0.0f && !IsBlack(ls.Li)) {
                        const float4 ev = MatEval(S, mat, at, Lo(it, wod), Lo(it, ls.Wi));
                        C3 fr = c3(ev.x, ev.y, ev.z);
                        const float scatteringPdf = ev.w;
                        if (!IsBlack(fr)) {
                            fl |= F_L1 | F_WTR;
                            fr = fr * AbsCosTheta(Lo(it, ls.Wi));
                            const float weight = PowerHeuristic(ls.Pdf, scatteringPdf);
                            W.pd_l1[slot] = make_float4(fr.r, fr.g, fr.b, weight);
                            W.vol_li[slot] = make_float4(ls.Li.r, ls.Li.g, ls.Li.b, 0.0f);
                            const V3 dir = Normalize(ls.P - it.P);
                            W.trw_start[slot] = make_float4(it.P.x, it.P.y, it.P.z, __int_as_float(env));
                            W.trw_end[slot] = make_float4(ls.P.x, ls.P.y, ls.P.z, __int_as_float(0));
                            W.trw_dir[slot] = make_float4(dir.x, dir.y, dir.z, 0.0f);
                            W.trw_tr[slot] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
                        }
                    }
                    const BSample sample = MatSampleAt(S, mat, at, Lo(it, wod), rand);
                    const C3 fr = sample.Fr * AbsCosTheta(sample.Wi);
                    const float scatteringPdf = sample.Pdf;
                    const bool sampledSpecular = (sample.Type & BX_SPECULAR) != 0;
                    float mis_pdf = 0.0f;
                    if (!IsBlack(fr) && scatteringPdf > 0) {
                        float weight = 1;
                        bool go = true;
                        if (!sampledSpecular) {
                            const float b2l = LightPdfLi(S, light, it.P, Wo(it, sample.Wi));
                            if (b2l == 0.0f) go = false;
                            else weight = PowerHeuristic(scatteringPdf, b2l);
                        }
                        if (go) {
                            fl |= F_L2 | F_WIT;
                            mis_pdf = scatteringPdf;
                            const Ray toLight = Spawn(it, Wo(it, sample.Wi));
                            const V3 wle = Wo(it, -sample.Wi);
                            W.pd_fr[slot] = make_float4(fr.r, fr.g, fr.b, weight);
                            W.pd_w[slot] = make_float4(wle.x, wle.y, wle.z, 0.0f);
                            W.itw_o[slot] = make_float4(toLight.O.x, toLight.O.y, toLight.O.z, toLight.MinT);
                            W.itw_d[slot] = make_float4(toLight.D.x, toLight.D.y, toLight.D.z, 0.0f);
                            W.itw_tr[slot] = make_float4(1.0f, 1.0f, 1.0f, __int_as_float(pack_env(env, 0)));
                        }
                    }
                    W.pd_mis[slot] = make_float4(mis_pdf, __int_as_float(light), ls.Pdf, 0.0f);
                } else {
                    fl |= F_DZERO;
                }
                const BSample sample = MatSampleAt(S, mat, at, Lo(it, wo), rand);
                isSpecularPath = (sample.Type & BX_SPECULAR) != 0;
                if (sample.Pdf > 0.0f) coeff = coeff * (sample.Fr * AbsCosTheta(sample.Wi) / sample.Pdf);
                else { done = true; break; }
                const V3 nextDir = Wo(it, sample.Wi);
                ray = mkray(it.P, nextDir, ray.MinT);
                env = GetMedium(S, it, nextDir);
            }
        } while (false);
        if (!done && rr && bounces > P.min_depth) {
            const float q = nmin(MaxElement(coeff), P.rr);
            if (NextFloat(rand) > q) done = true;
            else coeff = coeff / q;
        }
        if (!done) {
            bounces++;
            fl |= F_CONT;
            W.ray_o[slot] = make_float4(ray.O.x, ray.O.y, ray.O.z, ray.MinT);
            W.ray_d[slot] = make_float4(ray.D.x, ray.D.y, ray.D.z, ray.MaxT);
            W.vol_env[slot] = env;
        } else {
            fl |= F_DONE;
        }
        W.bounce[slot] = make_int2(bounces, guard);
        W.rng_n[slot] = rand.n;
        fl = (fl & ~F_SPECULAR) | (isSpecularPath ? F_SPECULAR : 0u);
        /* start the walks of the new direct term; if there are none, resolve it now */
        if (fl & F_WTR) {
            if (!trw_next(W, slot)) fl &= ~F_WTR;
        }
        if (fl & (F_WTR | F_WIT)) break;
    }
    W.coeff[slot] = make_float4(coeff.r, coeff.g, coeff.b, 0.0f);
    W.rad[slot] = make_float4(radiance.r, radiance.g, radiance.b, 0.0f);
    if (ext || (fl & (F_WTR | F_WIT))) {
        W.flags[slot] = fl;
        o->trw = (fl & F_WTR) != 0;
        o->itw = (fl & F_WIT) != 0;
        o->ext = ext;
        o->keep = true;
        return;
    }
    /* the path is over */
    finish_path(J, W, slot, radiance, stats, WF_PASS_RENDER);
    if (counting) warp_add64(stats + 0, 1u);
    o->restart = true;
}

/* The vol_path shade's queue appends for the block: a Transmittance segment
 * takes the first closest-hit position of the lane, an IntersectTr segment or
 * the extension ray the second; a finished path's slot takes the next camera
 * sample at once. */
DF void vol_queues(const WfState& W, int slot, int next, VolOut& o) {
    const long long sid = claim_sample(W, 0xffffffffu, o.restart);
    float4 ro, rd;
    if (o.restart && init_path(W, slot, sid, &ro, &rd)) { o.ext = true; o.keep = true; }
    int qs, qx, qt, qe, qa;
    queue_append<true>(W, next, false, false, o.trw, o.itw || o.ext, o.keep, &qs, &qx, &qt, &qe, &qa);
    if (o.trw) {
        float4 to, td;
        trw_ray(W, slot, &to, &td);
        push_ray4(W, qt, slot, WF_RAY_TRW, to, td);
    }
    if (o.itw) {
        const float4 io = W.itw_o[slot], id = W.itw_d[slot];
        push_ray4(W, qe, slot, WF_RAY_MIS, io, make_float4(id.x, id.y, id.z, kFMax));
    } else if (o.ext) {
        if (!o.restart) { ro = W.ray_o[slot]; rd = W.ray_d[slot]; }
        push_ray4(W, qe, slot, WF_RAY_EXT, ro, rd);
    }
    if (o.keep) set_active(W, next, qa, slot);
    else clear_active(W, slot);
}

/* ---- light tracing (AdjointParticleIntegrator.EmitParticle, AdjointParticleIntegrator.cs:24-79) ----
 * A slot holds one particle; the job's `samples` is the film sums (float4 per
 * pixel) and its `first` the index of the round's first particle.  The loop
 * is cut at its two ray casts: the extension ray (Scene.Intersect) and the
 * camera connection's shadow ray (Scene.IsOccluded), both traced in the next
 * trace phase.  A shade runs one vertex: camera connection (its splat waits
 * in pd_l1 and the shadow-ray kernel adds it when the way is clear),
 * importance-mode BSDF sample, and the top of the reference's loop (depth
 * limit, Russian roulette) before the next extension ray, so the random
 * numbers are drawn in the reference's order.  A finished particle's slot
 * takes the next particle at once: the new particle writes no splat before
 * the pending shadow ray has been traced. */

/* top of the bounce loop (AdjointParticleIntegrator.cs:34-42); false ends the particle */
DF bool particle_continue(const RtParams& P, int bounces, C3* coeff, Rng& rand) {
    if (P.max_depth != -1 && bounces >= P.max_depth) return false;
    if (bounces > P.min_depth) {
        if (NextFloat(rand) > P.rr) return false;
        *coeff = *coeff / P.rr;
    }
    return true;
}

/* What a light-tracer shade leaves for the queues: the camera connection's
 * splat ray, the next extension ray, and whether the slot holds a particle
 * for the next iteration.  The kernel appends them for the whole block. */
struct PartOut {
    float4 so, sd, eo, ed;
    bool splat, ext, keep;
};

/* Claims particles for `slot`, the first one `sid` (claimed by the caller),
 * until one has an extension ray to trace (a particle can end before its
 * first ray: no light, black emission, depth limit or roulette).  The ray
 * goes to `o`; o->keep is false once every particle of the round is claimed. */
DF void start_particle(const WfState& W, int slot, long long sid, PartOut* o) {
    const WfJob& J = W.jobs[0];
    const RtSceneView* S = J.view;
    const RtParams P = J.P;
    for (bool first = true;; first = false) {
        if (!first) sid = (long long)atomicAdd(&W.ctr->next_sample, 1ull);
        if (sid >= W.ctr->total) { W.flags[slot] = 0; o->keep = false; return; }
        const long long i = J.first + sid;
        Rng rand;
        rng_init(rand, P.seed, (uint32_t)(uint64_t)i, (uint32_t)((uint64_t)i >> 32), RT_PARTICLE_STREAM);
        int light;
        const float selectPdf = SampleLight(S, rand, &light);
        if (selectPdf == 0.0f) continue;
        const Emit e = LightSampleEmit(S, light, rand);
        if (IsBlack(e.le)) continue;
        C3 coeff = e.le * AbsDot(e.dir, e.n) / (selectPdf * e.pdf_pos * e.pdf_dir);
        const Ray ray = mkray(e.pos, e.dir, 0.0001f);
        if (!particle_continue(P, 1, &coeff, rand)) continue;
        W.job[slot] = 0;
        W.pix[slot] = make_int4((int)(uint32_t)(uint64_t)i, (int)(uint32_t)((uint64_t)i >> 32), 0, 0);
        W.rng_n[slot] = rand.n;
        W.coeff[slot] = make_float4(coeff.r, coeff.g, coeff.b, 0.0f);
        W.bounce[slot] = make_int2(1, 1);
        W.flags[slot] = F_ALIVE | F_EXT;
        ray4(ray, &o->eo, &o->ed);
        W.ray_o[slot] = o->eo;
        W.ray_d[slot] = o->ed;
        o->ext = true;
        o->keep = true;
        return;
    }
}

/* The warp's lanes with `want` claim consecutive particle ids with one atomic;
 * -1 for the others.  Every lane of the warp calls it. */
DF long long claim_particle(const WfState& W, bool want) {
    const unsigned m = __ballot_sync(0xffffffffu, want);
    if (!m) return -1;
    const int leader = __ffs(m) - 1, lane = threadIdx.x & 31;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(&W.ctr->next_sample, (unsigned long long)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    return want ? (long long)base + __popc(m & ((1u << lane) - 1u)) : -1;
}

/* queue the block's splat and extension rays and its next active slots */
DF void particle_queues(const WfState& W, int slot, int next, const PartOut& o) {
    int qs, qx, qm, qe, a;
    queue_append<true>(W, next, o.splat, false, false, o.ext, o.keep, &qs, &qx, &qm, &qe, &a);
    if (o.splat) push_ray4(W, qs, slot, WF_RAY_SPLAT, o.so, o.sd);
    if (o.ext) push_ray4(W, qe, slot, WF_RAY_EXT, o.eo, o.ed);
    if (o.keep) set_active(W, next, a, slot);
    else clear_active(W, slot);
}

/* One vertex of the slot's particle; its rays go to `o`.  Returns true when
 * the particle is over (the caller starts the next one in the slot). */
DF bool shade_particle(const WfState& W, int slot, uint32_t* status, PartOut* o) {
    const WfJob& J = W.jobs[0];
    const RtSceneView* S = J.view;
    const RtParams P = J.P;
    uint32_t fl = W.flags[slot];
    bool done = (fl & F_DONE) != 0;
    if (!done) {
        /* 1. the vertex at the extension hit */
        int2 bc = W.bounce[slot];
        int bounces = bc.x, guard = bc.y;
        const float4 cf = W.coeff[slot];
        C3 coeff = c3(cf.x, cf.y, cf.z);
        const float4 ro = W.ray_o[slot], rdd = W.ray_d[slot];
        const Ray ray = mkray(v3(ro.x, ro.y, ro.z), v3(rdd.x, rdd.y, rdd.z), ro.w, rdd.w);
        const int4 id = W.pix[slot];
        Rng rand;
        rng_resume(rand, P.seed, (uint32_t)id.x, (uint32_t)id.y, RT_PARTICLE_STREAM, W.rng_n[slot]);
        Ray nray = ray;
        bool ext = false;
        do {
            Isect it;
            if (!load_hit(S, ray, W.ext_hit[slot], W.ext_sub[slot], &it)) { done = true; break; }
            if (HasSurface(S, it)) {
                const int mat = PrimOf(S, it).material;
                const V3 wo = Lo(it, it.Wr);
                CamWi cw;
                if (CameraSampleWi(S->camera, it.P, &cw) && cw.we != 0.0f) {
                    /* Scene.IsOccluded(camera, it.P): closer than 0.001 counts as occluded, no ray */
                    const V3 vec = it.P - cw.pos;
                    const float dis = Length(vec);
                    if (!(dis < 0.001f)) {
                        const V3 wi = Lo(it, cw.dir);
                        const C3 f = MatFr<true>(S, mat, wo, wi, it.UV);
                        const C3 color = coeff * f * cw.we * AbsCosTheta(wi);
                        int pix = -1;   /* a NaN position (the reference throws) splats nothing */
                        if (cw.sx == cw.sx && cw.sy == cw.sy) {
                            const int x = (int)floorf(cw.sx), y = (int)floorf(cw.sy);
                            if (x >= 0 && x < S->camera.width && y >= 0 && y < S->camera.height)
                                pix = x * S->camera.height + y;
                        }
                        W.pd_l1[slot] = make_float4(color.r, color.g, color.b, __int_as_float(pix));
                        ray4(mkray(cw.pos, Normalize(vec), 0.0001f, dis - 0.0001f), &o->so, &o->sd);
                        o->splat = true;
                    }
                }
                const BSample bs = MatSample<true>(S, mat, wo, it.UV, rand);
                if (bs.Pdf > 0.0f) coeff = coeff * (bs.Fr * AbsCosTheta(bs.Wi) / bs.Pdf);
                else { done = true; break; }
                nray = Spawn(it, Wo(it, bs.Wi));
                bounces++;
            } else {
                nray = mkray(it.P, ray.D, ray.MinT);   /* bounces-- and continue: the same depth again */
            }
            /* 2. the top of the next loop iteration */
            if (++guard > RT_LOOP_CAP) { atomicOr(status, RT_STATUS_ITER); done = true; break; }
            if (!particle_continue(P, bounces, &coeff, rand)) { done = true; break; }
            ext = true;
        } while (false);
        if (ext) {
            ray4(nray, &o->eo, &o->ed);
            o->ext = true;
            W.ray_o[slot] = o->eo;
            W.ray_d[slot] = o->ed;
        }
        W.bounce[slot] = make_int2(bounces, guard);
        W.rng_n[slot] = rand.n;
        W.coeff[slot] = make_float4(coeff.r, coeff.g, coeff.b, 0.0f);
        if (done) fl |= F_DONE;
    }
    if (!(fl & F_DONE)) {
        W.flags[slot] = fl;
        o->keep = true;
        return false;
    }
    return true;
}

inline unsigned grid_for(int64_t n, int block) { return (unsigned)((n + block - 1) / block); }

}  // namespace

#endif
