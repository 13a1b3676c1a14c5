// Persistent, request-batched wavefront form of the bounce loop.
//
// A fixed pool of path slots (the wavefront) is advanced one vertex per
// iteration by small kernels instead of one large one:
//   regen   : resolve finished samples into their request's film and list the
//             free slots.
//   camera  : take the next (request, sample, pixel) work items, trace their
//             camera rays and start the paths that hit something in free slots.
//   extend  : closest hit of every other live path's current ray.
//   scatter : optionally, the live slots by material (a counting sort in chunks),
//             so that shade's warps hold one material.
//   shade   : one TraceRay vertex (medium, emission, NEE, BSDF sample, RR).
//             Shadow rays go to a queue instead of being traced inline.
//   plan    : the iteration's bookkeeping: whether the loop goes on, and the ray
//             sorts' key scans.
//   sscatter: optionally, the shadow records in key order.
//   occlude : any-hit (or the transparent walk) of the queued shadow rays;
//             visible contributions are added to their path's accumulator.
// The iteration is the body of a loop in a CUDA graph, which plan ends on the
// device when every request's samples are done.
//
// Many requests of uneven resolution, spp and depth share the pool: a work id
// maps to (request, sample, pixel) with a binary search over the requests'
// prefix offsets, samples outermost so a warp shares a sample index.
//
// The same loop runs the path-replay adjoint (rt_adjoint) in two passes over
// a range of samples: WF_RECORD renders them with the forward kernels and
// regen and camera store each finished sample's end state (lp, la, pre, att0) by
// work id instead of adding it to a film; WF_REPLAY traces the same samples
// again, regen starts each path itself with the adjoints of its recorded
// resolve, and
// k_wf_adjoint (wf_adjoint.cuh) replaces shade and occlude: it runs the vertex
// with the replay's gradient hooks and its shadow rays inline.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "adjoint.cuh"
#include "integrator.cuh"

namespace rt {

enum : int {
    PF_ALIVE = 1,       // a ray is in flight
    PF_DONE = 2,        // finished: the sample waits for resolve
    PF_PREV_DELTA = 4,
    PF_FIRST = 8,
    PF_CLAMP = 16,
    PF_DEAD = 32,       // 32, 64, 128: channels of la closed by the per-frame sanitize
    PF_INSIDE = 512,    // the slot's interior state (ab, ior) is set: absorption or a non-empty IOR stack
    PF_TRACED = 256,    // a camera path of this iteration: its hit is in place, extend skips it
};

struct WfRequest {
    RenderConst rc;
    int scene;
    int x0, y0, ww, wh;   // render window inside the W x H image
    int spp, spp0;
    long long begin;      // first global work id of this request
    long long count;      // ww * wh * spp
    double* accum;        // 3 * ww * wh: sums of clamped samples (planar, pixels in strip_pixel order).
                          // Double: a float sum of 65 536 samples of one pixel drifts by ~1e-3 of its
                          // value through the rounding of every addition.
};

// SoA path state. A vertex reads and writes o, d, beta, w (64 B) and reads id
// (16 B) and the hit (16 B); the radiance sums lp and la are touched where a
// term is added and at resolve, pre and att0 written at the first surface
// vertex and read at resolve.
struct WfPaths {
    float4* o;      // o.xyz, prev_pdf
    float4* d;      // d.xyz, flags
    float4* beta;   // beta.xyz, depth
    float4* w;      // w.xyz, rng dim
    int4* id;       // sample index, pixel (lx | ly << 16, window-local), request, pixel seed
    float4* lp;     // lp.xyz, -
    float4* la;     // la.xyz, -
    float4* pre;    // pre.xyz, -   (set once PF_CLAMP is)
    float4* att0;   // att0.xyz, -  (set once PF_CLAMP is)
    float4* ab;     // cur_abs.xyz, ior count   (dielectric scenes)
    float* ior;     // 8 per slot                (dielectric scenes)
    float4* hit;    // t, u, v, kind << 30 | slot
    int* free;      // free slots, for the iteration's camera paths
    int* order;     // slot order for shade (material-sorted or identity); for extend under the ray sort
    int* keys;      // material key per slot (sorting); after shade, the ray sort's key
    int* rrank;     // ray sort: the slot's rank among the rays of its key
};

// Shadow records. Thread t of shade writes its vertex's k-th record at
// k * nslots + t and the number it wrote to cnt[t]: no queue counter (a
// returning atomic per light sample in the middle of the vertex), and the
// records of a warp lie side by side.
struct WfShadow {
    float4* o;    // o.xyz, tmax
    float4* d;    // d.xyz, slot << 1 | to_la
    float4* c;    // contribution.xyz, scene
    int* cnt;     // per shade thread: its records
    int per;      // records a vertex can write (the most of any scene)
    int limit;    // test only, > 0: at most this many records per iteration, counted in ctl->nrec
    int* key;     // shadow sort: the record's ray_key
    int* rank;    // shadow sort: its rank among the records of its key
    int* order;   // shadow sort: records in key order, for occlude
};

struct WfCtl {
    unsigned long long next;    // next global work id
    unsigned long long total;   // total work ids
    unsigned long long iter_first;   // replay: the first work id of this iteration
    int live;                   // slots alive after the last regen and camera
    int nlive;                  // live slots in order[] (the material sort's total)
    int shaded;                 // nlive of the iteration's shade, for occlude
    int err;                    // a kernel's RT_ERR_* (traversal stack, index checks)
    int overflow;               // shadow queue overflow (its arrays hold every record: a test's limit)
    int iters, limit;           // iterations run, and the host's bound on them
    int done;                   // every work id resolved
    unsigned ext_next;          // persistent extend: next slot to fetch
    unsigned occ_next;          // persistent occlude: next shadow record to fetch
    int nbounce;                // ray sort: bounce rays shade continued (order[0 .. nbounce))
    int nshadow;                // shadow sort: records counted by key
    int nfree, free_next;       // slots in the free list, and the first one not yet reserved
    int nrec;                   // records written this iteration (counted under a test's limit alone)
};

// Buckets of the bounce-ray sort.
constexpr int kRayKeys = 1 << 15;

enum : int { WF_RENDER = 0, WF_RECORD = 1, WF_REPLAY = 2 };
// float4s of a replayed slot's adjoint state: 5 for the resolve adjoints, the
// interior material, the film gradient and the clamped value, then 5 for the
// throughput's log derivatives (dlb) while a medium slot is differentiated
constexpr int kAdjState = 10;

// The adjoint passes' buffers and parameters.
struct WfAdjoint {
    float4* rec;            // per work id, 4 float4: {lp, clamp flag}, la, pre, att0 of the finished sample
    long long nrec;         // work ids the record holds
    float4* st;             // per slot, kAdjState float4: the replay's resolve adjoints, interior material,
                            // film gradient and clamped value
    const float* dimg;      // dLoss/dfilm, 3 planes of W x H
    int W, H;
    float inv_spp;          // 1 / the request's spp: the film is the mean of its samples
    const float* params;    // raw parameter vector, 16 per material, then the medium's 6
    const unsigned* mmask;  // per material: bit k = slot k is differentiated
    const DMat* dmat;       // per material and BSDF slot: the dual material
    unsigned gmask;         // the medium's slots
    int nparams, medium_base;
    const int* act;         // the differentiated slots, nact of them
    int nact;
    int use_local;          // gradients gather in per-thread arrays (nparams <= kAdjLocal)
    int use_shared;         // ... otherwise in shared memory (nparams floats), else global atomics
    double* grad;           // nparams accumulators
};

struct WfArgs {
    const SceneView* views;
    int nviews;
    const WfRequest* reqs;
    int nreq;
    int nslots;
    int opaque;       // every scene of the batch is opaque: any-hit shadows
    int sort;
    int nkeys;        // material keys (sum over scenes) for sorting
    const int* key_base;   // per scene: first key
    int regroup;      // extend/occlude regroup their block's rays by kind (block_group)
    int replay;       // the replay pass: regen starts its camera paths, extend traces them
    int raysort;      // extend walks the bounce rays sorted by ray_key
    int rkey_bits;    // ray_key of bounce rays: origin cell bits per axis (0 .. 4)
    int rdir_bits;    // ray_key of bounce rays: direction bits (0, 3: octant, or an even count up to 8)
    int skey_bits;    // the same two for shadow records
    int sdir_bits;
    int* rhist;       // kRayKeys: bounce rays per key (filled by shade)
    int* roff;        // kRayKeys: the keys' first positions in order (the scanned histogram)
    int shadowsort;   // occlude walks the shadow records sorted by ray_key
    int* shist;       // kRayKeys: shadow records per key (filled by shade)
    int* soff;        // kRayKeys: the keys' first positions in S.order
    WfPaths P;
    WfShadow S;
    WfCtl* ctl;
    int* err;
    int any4;         // opaque shadow rays may walk the four-wide records (their stack bound fits)
    const WfAdjoint* J;   // the adjoint passes' buffers and parameters (null in WF_RENDER)
};

// The scene of a call with one scene, and the constants of one with one
// request, in constant memory: the kernels' ONE variants read them as
// instruction operands instead of through two dependent loads (request, then
// scene view) per thread. wf_render, which holds a process-wide lock until its
// kernels are done, writes them on the stream before the first iteration. Shade
// takes them for one request alone (with the view constant and the request's
// constants in global memory it lost 2% on a Cornell box); extend and occlude
// for one scene (extend 1.29 to 1.23 ms, occlude 0.78 to 0.73 ms on a Cornell
// box of 256x256x64 samples).
struct WfOne {
    SceneView view;
    RenderConst rc;
};
__constant__ WfOne c_wf_one;

RT_D int fbits(float f) { return __float_as_int(f); }
RT_D float ibits(int i) { return __int_as_float(i); }

// Stores a whole path state (the adjoint's replay).
RT_D void wf_store(const WfArgs& a, int i, const PathState& ps, int flags) {
    int dead = (ps.mask.x == 0.0f ? PF_DEAD : 0) | (ps.mask.y == 0.0f ? 2 * PF_DEAD : 0) |
               (ps.mask.z == 0.0f ? 4 * PF_DEAD : 0);
    a.P.o[i] = make_float4(ps.o.x, ps.o.y, ps.o.z, ps.prev_pdf);
    a.P.d[i] = make_float4(ps.d.x, ps.d.y, ps.d.z, ibits(flags | dead));
    a.P.beta[i] = make_float4(ps.beta.x, ps.beta.y, ps.beta.z, ibits(ps.depth));
    a.P.w[i] = make_float4(ps.w.x, ps.w.y, ps.w.z, ibits((int)ps.rng.dim));
    a.P.lp[i] = make_float4(ps.lp.x, ps.lp.y, ps.lp.z, 0.0f);
    a.P.la[i] = make_float4(ps.la.x, ps.la.y, ps.la.z, 0.0f);
    a.P.pre[i] = make_float4(ps.pre.x, ps.pre.y, ps.pre.z, 0.0f);
    a.P.att0[i] = make_float4(ps.att0.x, ps.att0.y, ps.att0.z, 0.0f);
}

template <class PS>
RT_D int wf_flags(const PS& ps, int alive) {
    return (alive ? PF_ALIVE : PF_DONE) | (ps.prev_delta ? PF_PREV_DELTA : 0) | (ps.first ? PF_FIRST : 0) |
           (ps.clamp_mode ? PF_CLAMP : 0);
}

// The window's pixels in 8-pixel-wide column strips, rows inside a strip:
// work ids run in this order, so the 32 camera rays of a warp of the camera kernel
// cover an 8x4 block rather than a 32x1 run, and the accumulation buffer is
// laid out the same way, so that the film atomics of consecutive slots stay
// contiguous. The last strip is narrower when ww % 8 != 0.
constexpr int kStripW = 8;   // 4 and 16 measured the same
RT_D void strip_pixel(int p, int ww, int wh, int& lx, int& ly) {
    int strip = p / (kStripW * wh);
    int in = p - strip * kStripW * wh;
    int sw = min(kStripW, ww - kStripW * strip);
    lx = kStripW * strip + in % sw;
    ly = in / sw;
}
// A request's local work id as (sample, pixel in strip order): samples outermost.
// 32-bit division where the request's ids fit.
RT_D void split_id(unsigned long long local, int npix, int& s, int& p) {
    if (local >> 32) {
        s = (int)(local / (unsigned)npix);
        p = (int)(local % (unsigned)npix);
    } else {
        unsigned q = (unsigned)local / (unsigned)npix;
        s = (int)q;
        p = (int)((unsigned)local - q * (unsigned)npix);
    }
}
RT_D int strip_index(int lx, int ly, int ww, int wh) {
    int strip = lx / kStripW;
    int sw = min(kStripW, ww - kStripW * strip);
    return strip * kStripW * wh + ly * sw + (lx - kStripW * strip);
}

RT_D uint32_t pixel_seed(int px, int py) { return ((uint32_t)px * 73856093u) ^ ((uint32_t)py * 19349663u); }

// Rebuilds the whole path state of slot i (the adjoint's replay).
RT_D void wf_load(const WfArgs& a, int i, const WfRequest& R, PathState& ps) {
    float4 o = a.P.o[i], d = a.P.d[i], b = a.P.beta[i], w = a.P.w[i], lp = a.P.lp[i], la = a.P.la[i],
           pre = a.P.pre[i], at = a.P.att0[i];
    int4 id = a.P.id[i];
    int flags = fbits(d.w);
    ps.o = v3(o.x, o.y, o.z);
    ps.prev_pdf = o.w;
    ps.d = v3(d.x, d.y, d.z);
    ps.beta = v3(b.x, b.y, b.z);
    ps.depth = fbits(b.w);
    ps.w = v3(w.x, w.y, w.z);
    ps.lp = v3(lp.x, lp.y, lp.z);
    ps.la = v3(la.x, la.y, la.z);
    ps.pre = v3(pre.x, pre.y, pre.z);
    ps.att0 = v3(at.x, at.y, at.z);
    ps.mask = v3((flags & PF_DEAD) ? 0.0f : 1.0f, (flags & (2 * PF_DEAD)) ? 0.0f : 1.0f,
                 (flags & (4 * PF_DEAD)) ? 0.0f : 1.0f);
    ps.prev_delta = (flags & PF_PREV_DELTA) != 0;
    ps.first = (flags & PF_FIRST) != 0;
    ps.clamp_mode = (flags & PF_CLAMP) != 0;
    ps.rng = Sampler{(uint32_t)id.w, (uint32_t)id.x, (uint32_t)fbits(w.w)};
    ps.cur_abs = v3(0.0f);
    ps.iors.n = 0;
    if (R.rc.dielectrics) {
        float4 ab = a.P.ab[i];
        ps.cur_abs = v3(ab.x, ab.y, ab.z);
        ps.iors.n = fbits(ab.w);
        for (int k = 0; k < 8; k++) ps.iors.slot[k] = a.P.ior[(size_t)i * 8 + k];
    }
}

RT_D void wf_store_media(const WfArgs& a, int i, const PathState& ps) {
    a.P.ab[i] = make_float4(ps.cur_abs.x, ps.cur_abs.y, ps.cur_abs.z, ibits(ps.iors.n));
    for (int k = 0; k < 8; k++) a.P.ior[(size_t)i * 8 + k] = ps.iors.slot[k];
}

// Adds a term to a slot's radiance sum (its own thread's, between extend and
// occlude). Out of line: a vertex does so at an emitter, the sky or a
// non-finite NEE term alone.
__device__ __noinline__ void wf_add(float4* dst, float x, float y, float z) {
    float4 v = *dst;
    v.x += x;
    v.y += y;
    v.z += z;
    *dst = v;
}

// The part of a path's state that a forward vertex works on. The radiance sums
// and the primary clamp's terms stay in their slot and are written where they
// change: a whole PathState held 15 more registers through the vertex and
// moved 128 B more per slot. With both gone and a lone request's view and
// constants in constant memory, shade went from 7.2 to 5.9 ms on a Cornell box
// of 256x256x64 samples and from 42.2 to 34.8 ms on a full-HD icosphere frame of
// 64 samples.

// A batch with transmissive materials: the interior absorption and the depth of
// the IOR stack. The stack's entries stay in the slot (a dielectric surface
// alone reads them), and outside every dielectric (PF_INSIDE clear) there is
// nothing to load or store.
struct LeanMedia {
    V3 cur_abs;
    int ior_n;
};
struct NoMedia {};
template <bool TRANSMIT>
struct LeanPath : std::conditional_t<TRANSMIT, LeanMedia, NoMedia> {
    V3 o, d, beta, w;
    float prev_pdf;
    int prev_delta, first, clamp_mode, depth;
    int dead;         // PF_DEAD bits
    Sampler rng;
    const WfArgs* a;
    int slot;

    // Volumetrics/IorStack.cs (capacity 8), as IorStackD
    RT_D float* ior_at(int k) const { return a->P.ior + (size_t)slot * 8 + k; }
    RT_D float ior_top() const { return this->ior_n == 0 ? 1.0f : *ior_at(this->ior_n - 1); }
    RT_D float ior_enclosing() const { return this->ior_n >= 2 ? *ior_at(this->ior_n - 2) : 1.0f; }
    RT_D void ior_push(float v) {
        if (this->ior_n >= 8) {
            for (int k = 0; k < 7; k++) *ior_at(k) = *ior_at(k + 1);
            *ior_at(7) = v;
            return;
        }
        *ior_at(this->ior_n++) = v;
    }
    RT_D void ior_pop() {
        if (this->ior_n > 0) this->ior_n--;
    }
    RT_D void add(V3 x, int to_la) {   // PathState::add
        if (!to_la) {
            wf_add(a->P.lp + slot, x.x, x.y, x.z);
            return;
        }
        if (!isfinite(x.x)) dead |= PF_DEAD;
        if (!isfinite(x.y)) dead |= 2 * PF_DEAD;
        if (!isfinite(x.z)) dead |= 4 * PF_DEAD;
        wf_add(a->P.la + slot, (dead & PF_DEAD) ? 0.0f : x.x, (dead & (2 * PF_DEAD)) ? 0.0f : x.y,
               (dead & (4 * PF_DEAD)) ? 0.0f : x.z);
    }
    RT_D void set_primary(V3 att) {
        a->P.pre[slot] = make_float4(w.x, w.y, w.z, 0.0f);
        a->P.att0[slot] = make_float4(att.x, att.y, att.z, 0.0f);
    }
};

RT_D int find_request(const WfRequest* reqs, int n, unsigned long long id) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if ((unsigned long long)reqs[mid].begin <= id) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Adds a sample's clamped radiance to its request's film sums.
RT_D void film_add(const WfRequest& R, int lx, int ly, V3 L) {
    size_t plane = (size_t)R.ww * R.wh, k = (size_t)RT_IX(strip_index(lx, ly, R.ww, R.wh), plane);
    atomicAdd(R.accum + k, (double)L.x);
    atomicAdd(R.accum + plane + k, (double)L.y);
    atomicAdd(R.accum + 2 * plane + k, (double)L.z);
}

// Regen resolves finished paths and lists the free slots: bound by memory (64 B
// read and three film atomics per finished path, 16 B of flags per slot).
// Threads of a block: one atomic per counter and block, on addresses that every
// block shares.
constexpr int kRegenBlock = 512;
template <int MODE>
__global__ void __launch_bounds__(kRegenBlock) k_wf_regen(const __grid_constant__ WfArgs a) {
    // The free slots go to the free list, or in the replay to the next work ids,
    // with one atomic per block (a ballot prefix over the block's free slots),
    // and the live count with one more: a per-warp atomic on one address
    // serialised in L2.
    __shared__ int s_warp[kRegenBlock / 32];   // per-warp free-slot offsets
    __shared__ unsigned long long s_base;
    __shared__ int s_live;
    const unsigned full = 0xffffffffu;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    bool in = i < a.nslots;
    int flags = in ? fbits(a.P.d[i].w) : 0;
    bool alive = in && (flags & PF_ALIVE);
    bool need = in && !alive;
    if (MODE != WF_REPLAY && need && (flags & PF_DONE)) {
        // a finished sample: resolve reads lp, la and, past a first surface vertex, pre and att0
        float4 lp = a.P.lp[i], la = a.P.la[i];
        float4 pre = make_float4(1.0f, 1.0f, 1.0f, 0.0f), at = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        int4 id = a.P.id[i];
        if (flags & PF_CLAMP) {
            pre = a.P.pre[i];
            at = a.P.att0[i];
        }
        const WfRequest& R = a.reqs[RT_IX(id.z, a.nreq)];
        int lx = id.y & 0xFFFF, ly = id.y >> 16;
        if (MODE == WF_RECORD) {   // keep its end state
            long long rid = R.begin + (long long)(id.x - R.spp0) * ((long long)R.ww * R.wh) +
                            strip_index(lx, ly, R.ww, R.wh);
            if (rid >= 0 && rid < a.J->nrec) {
                float4* r = a.J->rec + 4 * rid;
                r[0] = make_float4(lp.x, lp.y, lp.z, ibits(flags & PF_CLAMP));
                r[1] = la;
                r[2] = pre;
                r[3] = at;
            } else {
                atomicExch(a.err, RT_ERR_BOUNDS);
            }
        } else {   // its clamped radiance into the film
            PathState ps;
            ps.lp = v3(lp.x, lp.y, lp.z);
            ps.la = v3(la.x, la.y, la.z);
            ps.pre = v3(pre.x, pre.y, pre.z);
            ps.att0 = v3(at.x, at.y, at.z);
            ps.clamp_mode = (flags & PF_CLAMP) != 0;
            V3 L = path_resolve(ps, R.rc);
            if (!is_zero(L)) film_add(R, lx, ly, L);
        }
    }
    unsigned m = __ballot_sync(full, need);
    if (lane == 0) s_warp[wid] = __popc(m);
    if (threadIdx.x == 0) s_live = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
        int tot = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            int c = s_warp[w];
            s_warp[w] = tot;
            tot += c;
        }
        s_base = 0ull;
        if (tot && MODE == WF_REPLAY) s_base = atomicAdd(&a.ctl->next, (unsigned long long)tot);
        else if (tot) s_base = (unsigned long long)atomicAdd(&a.ctl->nfree, tot);
    }
    __syncthreads();
    bool live = alive;
    if (alive && a.raysort) {
        // a bounce ray shade continued: its key's first position plus the rank
        // shade's count gave it
        int pos = a.roff[RT_IX(a.P.keys[i], kRayKeys)] + a.P.rrank[i];
        if (pos < a.ctl->nbounce) a.P.order[pos] = i;
        else atomicExch(a.err, RT_ERR_BOUNDS);
    }
    if (MODE != WF_REPLAY && need) {
        a.P.d[i].w = ibits(0);
        a.P.free[RT_IX((int)s_base + s_warp[wid] + __popc(m & ((1u << lane) - 1u)), a.nslots)] = i;
    } else if (need) {
        unsigned long long id = s_base + (unsigned long long)(s_warp[wid] + __popc(m & ((1u << lane) - 1u)));
        if (id >= a.ctl->total) {
            a.P.d[i].w = ibits(0);
        } else {
            int req = RT_IX(find_request(a.reqs, a.nreq, id), a.nreq);
            const WfRequest& R = a.reqs[req];
            int lx, ly, s, p;
            split_id(id - (unsigned long long)R.begin, R.ww * R.wh, s, p);
            strip_pixel(p, R.ww, R.wh, lx, ly);
            PathState ps;
            path_init(ps, R.rc, R.x0 + lx, R.y0 + ly, (uint32_t)(R.spp0 + s));
            int al = path_alive(ps);
            // the adjoints of the recorded resolve; no gradient, no replay
            const WfAdjoint& J = *a.J;
            size_t plane = (size_t)J.W * J.H, fi = (size_t)(R.y0 + ly) * J.W + (R.x0 + lx);
            V3 delta = v3(J.dimg[fi], J.dimg[plane + fi], J.dimg[2 * plane + fi]) * J.inv_spp;
            AdjResolve ar{};
            if (id < (unsigned long long)J.nrec && !is_zero(delta)) {
                const float4* r = J.rec + 4 * id;
                float4 r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3];
                ar = adjoint_resolve(R.rc, v3(r0.x, r0.y, r0.z), v3(r1.x, r1.y, r1.z), v3(r2.x, r2.y, r2.z),
                                     v3(r3.x, r3.y, r3.z), fbits(r0.w) != 0, delta);
            }
            al = al && !is_zero(ar.g_a);
            float4* q = J.st + kAdjState * (size_t)i;
            q[0] = make_float4(ar.tot_a.x, ar.tot_a.y, ar.tot_a.z, ar.tot_la.x);
            q[1] = make_float4(ar.tot_la.y, ar.tot_la.z, ar.g_a.x, ar.g_a.y);
            q[2] = make_float4(ar.g_a.z, ar.g_la.x, ar.g_la.y, ar.g_la.z);
            q[3] = make_float4(ar.g_att0.x, ar.g_att0.y, ar.g_att0.z, ibits(-1));
            q[4] = make_float4(ar.delta.x, ar.delta.y, ar.delta.z, ar.val);
            if (J.gmask & 0x3Fu)
                for (int k = 5; k < kAdjState; k++) q[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            a.P.o[i] = make_float4(ps.o.x, ps.o.y, ps.o.z, ps.prev_pdf);
            a.P.d[i] = make_float4(ps.d.x, ps.d.y, ps.d.z, ibits(wf_flags(ps, al)));
            a.P.beta[i] = make_float4(1.0f, 1.0f, 1.0f, ibits(ps.depth));
            a.P.w[i] = make_float4(1.0f, 1.0f, 1.0f, ibits((int)ps.rng.dim));
            a.P.id[i] = make_int4((int)ps.rng.index, lx | (ly << 16), req, (int)ps.rng.seed);
            a.P.lp[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            a.P.la[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            a.P.pre[i] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
            a.P.att0[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (R.rc.dielectrics) a.P.ab[i] = make_float4(0.0f, 0.0f, 0.0f, ibits(0));
            live = true;
            if (a.raysort) {   // camera rays after the bounce rays, in work-id (pixel) order
                long long pos = (long long)a.ctl->nbounce + (long long)(id - a.ctl->iter_first);
                if (pos < a.nslots) a.P.order[pos] = al ? i : -1;
                else atomicExch(a.err, RT_ERR_BOUNDS);
            }
        }
    }
    int wl = __popc(__ballot_sync(full, live));
    if (lane == 0 && wl) atomicAdd(&s_live, wl);
    __syncthreads();
    if (threadIdx.x == 0 && s_live) atomicAdd(&a.ctl->live, s_live);
}

// Block-local counting partition; blockDim.x is a multiple of 32, at most 256,
// and every thread of the block calls it. Each thread offers one item of class
// cls (cls < 0: none). On return s_idx[0 .. n) holds the block's items ordered
// by class, in thread order within a class, and n is returned.
template <int NC>
RT_D int block_group(int item, int cls, int* s_idx, int (*s_cnt)[8], int* s_tot) {
    static_assert(NC <= 32, "one class per lane of the scanning warp");
    const unsigned full = 0xffffffffu;
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned mine = 0;
#pragma unroll
    for (int c = 0; c < NC; c++) {
        unsigned m = __ballot_sync(full, cls == c);
        if (cls == c) mine = m;
        if (lane == 0) s_cnt[c][wid] = __popc(m);
    }
    __syncthreads();
    if (wid == 0) {
        // lane c: the class's count, an exclusive scan over the classes, then
        // the running offsets of its warps (class-major order)
        int sum = 0;
        if (lane < NC)
            for (int w = 0; w < nw; w++) sum += s_cnt[lane][w];
        int incl = sum;
        for (int off = 1; off < 32; off <<= 1) {
            int v = __shfl_up_sync(full, incl, off);
            if (lane >= off) incl += v;
        }
        int run = incl - sum;
        if (lane < NC)
            for (int w = 0; w < nw; w++) {
                int c = s_cnt[lane][w];
                s_cnt[lane][w] = run;
                run += c;
            }
        if (lane == 31) *s_tot = incl;   // lanes past NC add nothing: lane 31 holds the total
    }
    __syncthreads();
    if (cls >= 0) s_idx[s_cnt[cls][wid] + __popc(mine & ((1u << lane) - 1u))] = item;
    __syncthreads();
    return *s_tot;
}

RT_D int octant(float x, float y, float z) { return (x < 0.0f) | ((y < 0.0f) << 1) | ((z < 0.0f) << 2); }

// Spreads the low 4 bits of v to bits 0, 3, 6, 9 (a Morton code's axis).
RT_D unsigned spread3(unsigned v) { return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4) | ((v & 8u) << 6); }

// Sort key of a bounce ray (0 .. kRayKeys): the origin's cell in the scene's
// sort box, cb bits per axis in Morton order, above a direction bin of db
// bits: none, the octant for 3, else a square grid over the octahedral map of
// the direction. Rays that share a key start close together in similar
// directions, so they walk much the same BVH nodes.
RT_D int ray_key(const SceneView& s, V3 o, V3 d, int cb, int db) {
    unsigned cell = 0;
    if (cb > 0) {
        float n = (float)(1 << cb);
        V3 u = (o - s.sort_lo) * s.sort_scale;
        unsigned cx = (unsigned)fminf(fmaxf(u.x * n, 0.0f), n - 1.0f);
        unsigned cy = (unsigned)fminf(fmaxf(u.y * n, 0.0f), n - 1.0f);
        unsigned cz = (unsigned)fminf(fmaxf(u.z * n, 0.0f), n - 1.0f);
        cell = spread3(cx) | (spread3(cy) << 1) | (spread3(cz) << 2);
    }
    unsigned dir = 0;
    if (db == 3) {
        dir = (unsigned)octant(d.x, d.y, d.z);
    } else if (db > 0) {
        // octahedral map of the direction onto [-1, 1]^2
        float l1 = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
        float px = l1 > 0.0f ? d.x / l1 : 0.0f, py = l1 > 0.0f ? d.y / l1 : 0.0f;
        if (d.z < 0.0f) {
            float qx = (1.0f - fabsf(py)) * (px < 0.0f ? -1.0f : 1.0f);
            float qy = (1.0f - fabsf(px)) * (py < 0.0f ? -1.0f : 1.0f);
            px = qx;
            py = qy;
        }
        float g = (float)(1 << (db / 2));
        unsigned gx = (unsigned)fminf(fmaxf((px * 0.5f + 0.5f) * g, 0.0f), g - 1.0f);
        unsigned gy = (unsigned)fminf(fmaxf((py * 0.5f + 0.5f) * g, 0.0f), g - 1.0f);
        dir = gx | (gy << (db / 2));
    }
    return (int)((cell << db) | dir) & (kRayKeys - 1);
}

// Stores slot i's closest hit and, when sorting, its material key: misses and
// emitters sort after the materials, and a path whose free flight ends in the
// medium before the hit after those. The flight's two draws are the vertex's
// first (rng as shade will have it), so its outcome is known here; a warp of
// shade that held both kinds of vertex ran the medium's and the surface's code,
// which in a foggy box, where 19 of 20 vertices are in mid-air, most warps did.
RT_D void hit_store(const WfArgs& a, int i, int req, const SceneView& s, const Hit& h, const Sampler& rng) {
    int packed = h.kind == HIT_NONE ? 0 : ((h.kind << 30) | h.slot);
    a.P.hit[i] = make_float4(h.t, h.u, h.v, ibits(packed));
    if (a.sort) {
        int key = a.nkeys;
        if (h.kind != HIT_NONE) {
            int ent = h.kind == HIT_TRI ? s.tri_entity[RT_IX(h.slot, s.n_tris)] : h.slot;
            key = RT_IX(a.key_base[a.reqs[req].scene] + s.entities[RT_IX(ent, s.n_entities)].material, a.nkeys);
        }
        if (s.has_medium) {
            Sampler r = rng;
            float t;
            V3 beta;
            if (medium_sample(s, h.kind != HIT_NONE ? h.t : 1e30f, r, t, beta)) key = a.nkeys + 1;
        }
        a.P.keys[i] = key;
    }
}

// A bounce ray's closest hit. One that leaves a scene with neither medium nor
// sky ends its path here: shade would add nothing.
RT_D void extend_store(const WfArgs& a, int i, int req, const SceneView& s, const Hit& h) {
    if (h.kind == HIT_NONE && !s.has_medium && !s.sky_on) {
        a.P.d[i].w = ibits((fbits(a.P.d[i].w) & ~PF_ALIVE) | PF_DONE);
        return;
    }
    Sampler rng{0u, 0u, 0u};
    if (a.sort && s.has_medium) {
        int4 id = a.P.id[i];
        rng = Sampler{(uint32_t)id.w, (uint32_t)id.x, (uint32_t)fbits(a.P.w[i].w)};
    }
    hit_store(a, i, req, s, h, rng);
}

// One thread per slot. With regroup, the block first reorders its live slots:
// camera rays, then bounce rays by direction octant. Regen hands a block's free
// slots consecutive pixels, so its camera rays are coherent, but they sit
// between the bounce rays of paths still in flight; regrouped, a warp holds
// one kind of ray and no longer waits on its slowest bounce ray.
// The register budget of 5 blocks of 256 (48 registers) lets 10 blocks of the
// autotuned 128 threads share an SM instead of 9: extend -2.5% per 64-spp
// icosphere frame, for an 8-byte spill (6 blocks spill 100 bytes: -0.5% there,
// +10% on a Cornell box; 4 blocks: +1%). For the same budget the flags are read
// again where a miss changes them (mixed batch 20.0 to 19.7 ms).
template <int STACK, bool L4, bool ONE>
__global__ void __launch_bounds__(256, 5) k_wf_extend(const __grid_constant__ WfArgs a) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (a.raysort) {
        // order[0 .. nbounce): bounce rays by key; then, in the replay, this iteration's camera rays
        long long n = a.ctl->nbounce;
        if (a.replay) {
            unsigned long long nx = a.ctl->next < a.ctl->total ? a.ctl->next : a.ctl->total;
            long long ncam = (long long)nx - (long long)a.ctl->iter_first;
            if (ncam > 0) n += ncam;
        }
        if ((long long)i >= n || i >= a.nslots) return;
        i = a.P.order[i];
        if (i < 0) return;
        i = RT_IX(i, a.nslots);
    } else if (a.regroup) {
        __shared__ int s_idx[256], s_cnt[9][8], s_tot;
        int cls = -1;
        if (i < a.nslots) {
            float4 d = a.P.d[i];
            int fl = fbits(d.w);
            if ((fl & PF_ALIVE) && !(fl & PF_TRACED)) cls = (fl & PF_FIRST) ? 0 : 1 + octant(d.x, d.y, d.z);
        }
        int n = block_group<9>(i, cls, s_idx, s_cnt, &s_tot);
        if ((int)threadIdx.x >= n) return;
        i = s_idx[threadIdx.x];
    } else if (i >= a.nslots) {
        return;
    }
    float4 d = a.P.d[i];
    int flags = fbits(d.w);
    if (!(flags & PF_ALIVE) || (flags & PF_TRACED)) return;
    float4 o = a.P.o[i];
    int req = ONE && a.nreq == 1 ? 0 : RT_IX(a.P.id[i].z, a.nreq);
    const SceneView& s = ONE ? c_wf_one.view : a.views[RT_IX(a.reqs[req].scene, a.nviews)];
    Hit h;
    trace<false, STACK, L4>(s, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), kEps, kInf, h, nullptr, a.err);
    extend_store(a, i, req, s, h);
}

// Persistent form with dynamic ray fetch (Aila and Laine 2009): a grid sized
// to fill the GPU once walks rays in rounds (Walker::step). Between rounds,
// once kRefill lanes of a warp have finished (or all of them), the finished
// lanes take the next slots from a global counter, so a few long rays no
// longer keep a warp whose other lanes are done. The rays, their walks and
// their results are those of the one-thread-per-slot kernel.
constexpr int kRefill = 8;

template <int STACK>
__global__ void __launch_bounds__(256) k_wf_extend_pt(const __grid_constant__ WfArgs a) {
    const unsigned full = 0xffffffffu;
    int lane = threadIdx.x & 31;
    Walker<false, STACK> w;
    int slot = -1, req = 0, flags = 0;
    bool exhausted = false;
    for (;;) {
        bool idle = slot < 0 && !exhausted;
        unsigned need = __ballot_sync(full, idle);
        unsigned busy = __ballot_sync(full, slot >= 0);
        if (!need && !busy) break;
        if (need && (__popc(need) >= kRefill || !busy)) {
            int leader = __ffs(need) - 1;
            unsigned base = 0;
            if (lane == leader) base = atomicAdd(&a.ctl->ext_next, (unsigned)__popc(need));
            base = __shfl_sync(full, base, leader);
            if (idle) {
                unsigned i = base + (unsigned)__popc(need & ((1u << lane) - 1u));
                if (i >= (unsigned)a.nslots) {
                    exhausted = true;
                } else {
                    float4 d = a.P.d[i];
                    flags = fbits(d.w);
                    if ((flags & PF_ALIVE) && !(flags & PF_TRACED)) {
                        float4 o = a.P.o[i];
                        req = a.nreq == 1 ? 0 : RT_IX(a.P.id[i].z, a.nreq);
                        slot = (int)i;
                        w.start(a.views[RT_IX(a.reqs[req].scene, a.nviews)], v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), kEps, kInf,
                                nullptr, false, 0);
                    }
                }
            }
            continue;
        }
        if (slot >= 0) {
            const SceneView& s = a.views[RT_IX(a.reqs[req].scene, a.nviews)];
            if (w.step(s, nullptr, a.err)) {
                extend_store(a, slot, req, s, w.best);
                slot = -1;
            }
        }
    }
}

// Resident blocks of 128 per SM the camera kernel is compiled for; a build knob.
#ifndef RT_CAMERA_MIN_BLOCKS
#define RT_CAMERA_MIN_BLOCKS 8
#endif
// Camera paths: generation and first hit in one kernel, on persistent warps.
// A warp takes 32 consecutive work ids (an 8x4 block of pixels), traces their
// camera rays and gives a slot only to the paths that go on: a ray that
// leaves a scene without a medium is a finished sample (the sky's radiance or
// nothing) and never touches the path state. In an open scene those are most
// camera rays: with a slot each, they cost the state's writes and reads in
// regen, extend and shade, and left few bounce rays per iteration to sort. A
// full-HD icosphere frame of 64 samples took 152.9 ms with a slot for each and
// takes 141.5 (regen and the camera rays 13.7 to 22.7 ms, extend 51.3 to 37.8,
// shade 34.8 to 29.3). The rays' walk bounds it: the warp's 8x4 block of pixels
// is as coherent as the scene allows.
// The paths that go on store only what their first vertex does not know: shade
// sets the rest of a PF_FIRST path itself.
//
// Slots are reserved from the free list 32 at a time before the rays are
// traced, so that every hit has one; what a warp does not use stays free until
// the next iteration. Once the list is dry a warp goes on with what it has
// left, down to half a warp of rays (but at least one round). Every round
// consumes work ids, so the loop ends.
template <int STACK, int MODE, bool ONE>
__global__ void __launch_bounds__(128, RT_CAMERA_MIN_BLOCKS) k_wf_camera(const __grid_constant__ WfArgs a) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned long long total = a.ctl->total;
    const int nfree = a.ctl->nfree;   // complete: regen has run
    int b0 = 0, n0 = 0, b1 = 0, n1 = 0;   // the warp's reserved ranges of the free list
    int kept = 0;
    bool dry = false, first = true;
    for (;;) {
        if (!dry && n0 + n1 < 32) {
            int b = 0;
            if (lane == 0) b = atomicAdd(&a.ctl->free_next, 32);
            b = __shfl_sync(full, b, 0);
            b1 = b;
            n1 = min(32, max(0, nfree - b));   // n1 was 0: n0 + n1 < 32 with n1 in {0, 32}
            dry = n1 < 32;
            if (n0 == 0) {
                b0 = b1;
                n0 = n1;
                n1 = 0;
            }
        }
        int n = min(32, n0 + n1);
        if (n == 0 || (dry && n < 16 && !first)) break;
        first = false;
        unsigned long long id0 = 0;
        if (lane == 0) id0 = atomicAdd(&a.ctl->next, (unsigned long long)n);
        id0 = __shfl_sync(full, id0, 0);
        if (id0 >= total) break;
        unsigned long long id = id0 + (unsigned long long)lane;
        bool keep = false;
        int req = 0, pix = 0, seed = 0, sample = 0;
        V3 dir = v3(0.0f);
        Hit h;
        h.kind = HIT_NONE;
        if (lane < n && id < total) {
            req = RT_IX(find_request(a.reqs, a.nreq, id), a.nreq);
            const WfRequest& R = a.reqs[req];
            const RenderConst& rc = R.rc;
            const SceneView& s = ONE ? c_wf_one.view : a.views[RT_IX(R.scene, a.nviews)];
            int lx, ly, si, p;
            split_id(id - (unsigned long long)R.begin, R.ww * R.wh, si, p);
            strip_pixel(p, R.ww, R.wh, lx, ly);
            PathState ps;
            path_init(ps, rc, R.x0 + lx, R.y0 + ly, (uint32_t)(R.spp0 + si));
            pix = lx | (ly << 16);
            seed = (int)ps.rng.seed;
            sample = (int)ps.rng.index;
            dir = ps.d;
            V3 L = v3(0.0f);
            if (path_alive(ps)) {
                traverse<false, STACK>(s, ps.o, ps.d, kEps, kInf, h, nullptr, a.err);
                keep = h.kind != HIT_NONE || s.has_medium;
                if (!keep && s.sky_on) L = L + weight_sky(s, rc, 0.0f, 1);   // shade_vertex's sky term, w = 1
            }
            if (!keep && MODE == WF_RECORD) {
                if ((long long)id < a.J->nrec) {
                    float4* r = a.J->rec + 4 * id;
                    r[0] = make_float4(L.x, L.y, L.z, ibits(0));
                    r[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    r[2] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
                    r[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                } else {
                    atomicExch(a.err, RT_ERR_BOUNDS);
                }
            } else if (!keep && !is_zero(L)) {
                film_add(R, lx, ly, clamp_lum(L, rc.max_rad));
            }
        }
        unsigned m = __ballot_sync(full, keep);
        int c = __popc(m), rank = __popc(m & ((1u << lane) - 1u));
        if (keep) {
            int i = RT_IX(a.P.free[rank < n0 ? b0 + rank : b1 + (rank - n0)], a.nslots);
            a.P.d[i] = make_float4(dir.x, dir.y, dir.z,
                                   ibits(PF_ALIVE | PF_PREV_DELTA | PF_FIRST | PF_TRACED));
            a.P.id[i] = make_int4(sample, pix, req, seed);
            a.P.lp[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            a.P.la[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const SceneView& s = ONE ? c_wf_one.view : a.views[RT_IX(a.reqs[req].scene, a.nviews)];
            hit_store(a, i, req, s, h, Sampler{(uint32_t)seed, (uint32_t)sample, 2u});
        }
        kept += c;
        if (c >= n0) {
            b0 = b1 + (c - n0);
            n0 = n1 - (c - n0);
            n1 = 0;
        } else {
            b0 += c;
            n0 -= c;
        }
    }
    if (lane == 0 && kept) atomicAdd(&a.ctl->live, kept);
}

// Exclusive scan over the block of one value per thread (blockDim.x a multiple
// of 32, at most 1024); *total receives the sum. s_w holds 32 ints.
RT_D int block_scan(int v, int* s_w, int* total) {
    const unsigned full = 0xffffffffu;
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        int x = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) s_w[w] = incl;
    __syncthreads();
    if (w == 0) {
        int x = lane < nw ? s_w[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(full, x, o);
            if (lane >= o) x += y;
        }
        s_w[lane] = x;
    }
    __syncthreads();
    *total = s_w[nw - 1];
    return (w ? s_w[w - 1] : 0) + incl - v;
}

// Sorts the live slots by material, chunk by chunk: a cluster of blocks orders
// its run of kSortChunk slots through shared memory and appends it to order[]
// with one atomic. Shade wants warps of one material, not one global order: a
// material's run in a chunk is long enough for that, and there is no global
// histogram, whose few hot counters took an atomic per warp and material in
// extend, in camera and twice here. (Chunks of 8192 slots, one block's: shade
// 27.1 to 30.4 ms on the full-HD icosphere frame with its 65 materials.)
constexpr int kSortThreads = 1024, kSortPer = 8, kSortCluster = 8;
constexpr int kSortChunk = kSortThreads * kSortPer * kSortCluster;
constexpr int kSortKeys = 256;   // keys of a chunk's counts
__global__ void __cluster_dims__(kSortCluster, 1, 1) __launch_bounds__(kSortThreads)
    k_wf_scatter(const __grid_constant__ WfArgs a) {
    __shared__ int s_w[32], s_cnt[kSortKeys], s_all[kSortCluster][kSortKeys], s_base;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned rank = cluster.block_rank();
    const int tid = threadIdx.x, first = blockIdx.x * (kSortThreads * kSortPer) + tid;
    // A block's shared memory may be written by another once that block runs:
    // all arrive here, and wait before the first remote store, behind the loads.
    cluster.barrier_arrive();
    if (tid < kSortKeys) s_cnt[tid] = 0;
    __syncthreads();
    int key[kSortPer], pos[kSortPer];
#pragma unroll
    for (int k = 0; k < kSortPer; k++) {
        int i = first + k * kSortThreads;
        key[k] = i < a.nslots && (fbits(a.P.d[i].w) & PF_ALIVE) ? RT_IX(a.P.keys[i], a.nkeys + 2) : -1;
    }
#pragma unroll
    for (int k = 0; k < kSortPer; k++) {
        // one shared-memory atomic per distinct key of the warp
        unsigned grp = __match_any_sync(0xffffffffu, key[k]);
        int lane = tid & 31, leader = __ffs(grp) - 1, base = 0;
        if (key[k] >= 0 && lane == leader) base = atomicAdd(&s_cnt[key[k]], __popc(grp));
        pos[k] = __shfl_sync(0xffffffffu, base, leader) + __popc(grp & ((1u << lane) - 1u));
    }
    __syncthreads();
    cluster.barrier_wait();
    // every block gets every block's counts: a key's slots of the earlier blocks go first
    if (tid < kSortKeys)
        for (int q = 0; q < kSortCluster; q++) cluster.map_shared_rank(&s_all[0][0], q)[rank * kSortKeys + tid] = s_cnt[tid];
    cluster.sync();
    int sum = 0, before = 0, live;
    if (tid < kSortKeys)
        for (int q = 0; q < kSortCluster; q++) {
            int c = s_all[q][tid];
            if (q < (int)rank) before += c;
            sum += c;
        }
    int off = block_scan(sum, s_w, &live);
    if (tid < kSortKeys) s_cnt[tid] = off + before;
    if (rank == 0 && tid == 0) {
        int b = live ? atomicAdd(&a.ctl->nlive, live) : 0;
        for (int q = 0; q < kSortCluster; q++) *cluster.map_shared_rank(&s_base, q) = b;
    }
    cluster.sync();
#pragma unroll
    for (int k = 0; k < kSortPer; k++)
        if (key[k] >= 0) a.P.order[RT_IX(s_base + s_cnt[key[k]] + pos[k], a.nslots)] = first + k * kSortThreads;
}

// Shadow sink of the wavefront: queue the ray with its contribution.
struct QueueShadows : NoAdjoint {
    const WfArgs* a;
    int t, slot, scene;   // shade's thread, its slot and scene
    int n;                // records written
    template <class PS>
    RT_D void shadow(PS& ps, int li, V3 o, V3 d, float tmax, V3 c, int to_la) {
        if (!isfinite(c.x) || !isfinite(c.y) || !isfinite(c.z)) {
            ps.add(c, to_la);   // records the per-frame sanitize in the mask
            return;
        }
        if (n >= a->S.per || (a->S.limit > 0 && atomicAdd(&a->ctl->nrec, 1) >= a->S.limit)) {
            atomicExch(&a->ctl->overflow, 1);
            return;
        }
        int j = n * a->nslots + t;
        n++;
        a->S.o[j] = make_float4(o.x, o.y, o.z, tmax);
        a->S.d[j] = make_float4(d.x, d.y, d.z, ibits((slot << 1) | to_la));
        a->S.c[j] = make_float4(c.x, c.y, c.z, ibits(scene));
        if (a->shadowsort) {   // the record's sort key and its rank in the key's count
            // above the origin's cell: the light, among up to eight, else the direction's octant
            const SceneView& s = a->views[scene];
            int key = ray_key(s, o, d, a->skey_bits, a->sdir_bits);
            if (s.num_lights > 1 && s.num_lights <= 8) key = (key & ~7) | li;
            unsigned grp = __match_any_sync(__activemask(), key);
            int lane = threadIdx.x & 31, leader = __ffs(grp) - 1;
            int base = 0;
            if (lane == leader) base = atomicAdd(&a->shist[key], __popc(grp));
            base = __shfl_sync(grp, base, leader);
            a->S.key[j] = key;
            a->S.rank[j] = base + __popc(grp & ((1u << lane) - 1u));
        }
    }
    RT_D void skipped(V3, V3, float) {}
};

// Under the ray sort: the continued ray's sort key and its rank in the key's
// count (one returning atomic per distinct key in the warp).
RT_D void wf_rank_ray(const WfArgs& a, const SceneView& s, V3 o, V3 d, int i) {
    int key = ray_key(s, o, d, a.rkey_bits, a.rdir_bits);
    unsigned grp = __match_any_sync(__activemask(), key);
    int lane = threadIdx.x & 31, leader = __ffs(grp) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&a.rhist[key], __popc(grp));
    base = __shfl_sync(grp, base, leader);
    a.P.keys[i] = key;
    a.P.rrank[i] = base + __popc(grp & ((1u << lane) - 1u));
}

// Starts the loads of what a vertex reads of slot i first on their way into L2.
// Shade does this for the slot that a thread of the block
// kAheadBlocks later will work on, when the material order has scattered the
// slots: their one block an SM runs in lockstep, so nothing else of the SM covers
// the first loads, and the slots, over a gigabyte, come from DRAM. The distance
// is the number of blocks in flight, one an SM. (Shade, with the first loads
// issued together: four foggy views of 256x256x64 samples 17.6 to 15.9 ms, a
// mixed batch 43.4 to 42.2, a full-HD icosphere frame of 64 samples 26.4 to 26.2.
// The adjoint's vertex gained nothing from it.)
constexpr int kAheadBlocks = 148;
RT_D void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
RT_D void wf_prefetch(const WfArgs& a, int i) {
    prefetch_l2(a.P.d + i);
    prefetch_l2(a.P.id + i);
    prefetch_l2(a.P.hit + i);
    prefetch_l2(a.P.o + i);
    prefetch_l2(a.P.beta + i);
    prefetch_l2(a.P.w + i);
}

// Hit record of slot i as extend wrote it.
RT_D Hit wf_hit(const WfArgs& a, int i) {
    float4 hh = a.P.hit[i];
    int packed = fbits(hh.w);
    Hit h;
    h.t = hh.x;
    h.u = hh.y;
    h.v = hh.z;
    h.kind = packed == 0 ? HIT_NONE : ((unsigned)packed >> 30);
    h.slot = packed & 0x3FFFFFFF;
    return h;
}

// Threads of a shade block: 512 at 128 registers fill an SM. Shade waits for
// instructions, and the warps of one block start together and share what they
// fetch: with two blocks of 256 instead, shade took 29.4 against 26.7 ms on a
// full-HD icosphere frame of 64 samples and 44.0 against 39.2 ms on four foggy
// views; blocks of 768 and 1024 threads (80 and 64 registers) spill and took
// 26.8 and 27.6, 42.5 and 45.5 ms.
constexpr int kShadeBlock = 512;
template <bool MEDIUM, bool TRANSMIT, bool ONE>
__global__ void __launch_bounds__(kShadeBlock, 1) k_wf_shade(const __grid_constant__ WfArgs a) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    int i, next = -1;
    if (a.sort) {
        // the scatter left the live slots in material order in order[0 .. live)
        if (t >= a.ctl->nlive) return;
        i = RT_IX(a.P.order[RT_IX(t, a.nslots)], a.nslots);
        next = t + kAheadBlocks * blockDim.x;
        next = next < a.ctl->nlive ? RT_IX(a.P.order[next], a.nslots) : -1;
    } else {
        if (t >= a.nslots) return;
        i = t;
    }
    float4 d = a.P.d[i];
    int4 id = a.P.id[i];
    Hit h = wf_hit(a, i);
    if (next >= 0) wf_prefetch(a, next);
    int flags = fbits(d.w);
    if (!(flags & PF_ALIVE)) {
        a.S.cnt[t] = 0;
        return;
    }
    int req = ONE ? 0 : RT_IX(id.z, a.nreq);
    const RenderConst& rc = ONE ? c_wf_one.rc : a.reqs[req].rc;
    int scene = ONE ? 0 : RT_IX(a.reqs[req].scene, a.nviews);
    const SceneView& s = ONE ? c_wf_one.view : a.views[scene];
    LeanPath<TRANSMIT> ps;
    ps.a = &a;
    ps.slot = i;
    ps.d = v3(d.x, d.y, d.z);
    ps.prev_delta = (flags & PF_PREV_DELTA) != 0;
    ps.first = (flags & PF_FIRST) != 0;
    ps.clamp_mode = (flags & PF_CLAMP) != 0;
    ps.dead = flags & (7 * PF_DEAD);
    // a camera path as path_init leaves it (it stored no more), else the slot's state
    float4 o = make_float4(rc.cam.origin.x, rc.cam.origin.y, rc.cam.origin.z, 0.0f);
    float4 b = make_float4(1.0f, 1.0f, 1.0f, ibits(rc.max_depth)), w = make_float4(1.0f, 1.0f, 1.0f, ibits(2));
    if (!ps.first) {
        o = a.P.o[i];
        b = a.P.beta[i];
        w = a.P.w[i];
    }
    ps.o = v3(o.x, o.y, o.z);
    ps.prev_pdf = o.w;
    ps.beta = v3(b.x, b.y, b.z);
    ps.depth = fbits(b.w);
    ps.w = v3(w.x, w.y, w.z);
    ps.rng = Sampler{(uint32_t)id.w, (uint32_t)id.x, (uint32_t)fbits(w.w)};
    if constexpr (TRANSMIT) {
        ps.cur_abs = v3(0.0f);
        ps.ior_n = 0;
        if (flags & PF_INSIDE) {
            float4 ab = a.P.ab[i];
            ps.cur_abs = v3(ab.x, ab.y, ab.z);
            ps.ior_n = fbits(ab.w);
        }
    }
    QueueShadows sink{{}, &a, t, i, scene, 0};
    bool alive = shade_vertex<MEDIUM, TRANSMIT>(s, rc, ps, h, sink);
    a.S.cnt[t] = sink.n;
    int keep = wf_flags(ps, alive) | ps.dead;
    if constexpr (TRANSMIT) {
        if (alive && rc.dielectrics && (ps.ior_n > 0 || !is_zero(ps.cur_abs))) {
            keep |= PF_INSIDE;
            a.P.ab[i] = make_float4(ps.cur_abs.x, ps.cur_abs.y, ps.cur_abs.z, ibits(ps.ior_n));
        }
    }
    a.P.d[i] = make_float4(ps.d.x, ps.d.y, ps.d.z, ibits(keep));
    if (!alive) return;   // resolve reads the flags and the radiance sums alone
    a.P.o[i] = make_float4(ps.o.x, ps.o.y, ps.o.z, ps.prev_pdf);
    a.P.beta[i] = make_float4(ps.beta.x, ps.beta.y, ps.beta.z, ibits(ps.depth));
    a.P.w[i] = make_float4(ps.w.x, ps.w.y, ps.w.z, ibits((int)ps.rng.dim));
    if (a.raysort) wf_rank_ray(a, s, ps.o, ps.d, i);
}

// Exclusive scan of a ray-sort key histogram (kRayKeys counts) into off by one
// cluster of kPlanCluster blocks of 1024 threads, four neighbouring keys a
// thread, clearing the histogram for the next shade; *total receives the sum.
// Blocks exchange their sums through distributed shared memory. (One block
// whose threads each read a run of 32 keys took about 10 us longer.)
constexpr int kPlanCluster = 8;
RT_D void key_scan(int* hist, int* off, int* total) {
    static_assert(kRayKeys == kPlanCluster * 1024 * 4, "four keys a thread");
    __shared__ int s_w[32], s_sum[kPlanCluster];
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned rank = cluster.block_rank();
    const int at = (int)rank * 1024 + threadIdx.x;
    cluster.barrier_arrive();   // every block of the cluster runs: see k_wf_scatter
    int4 v = reinterpret_cast<int4*>(hist)[at];
    reinterpret_cast<int4*>(hist)[at] = make_int4(0, 0, 0, 0);
    int sum;
    int base = block_scan(v.x + v.y + v.z + v.w, s_w, &sum);
    cluster.barrier_wait();
    if (threadIdx.x < kPlanCluster) *cluster.map_shared_rank(&s_sum[rank], threadIdx.x) = sum;
    cluster.sync();
    int all = 0;
#pragma unroll
    for (unsigned k = 0; k < kPlanCluster; k++) {
        if (k < rank) base += s_sum[k];
        all += s_sum[k];
    }
    int4 r;
    r.x = base;
    r.y = r.x + v.x;
    r.z = r.y + v.y;
    r.w = r.z + v.z;
    reinterpret_cast<int4*>(off)[at] = r;
    if (rank == 0 && threadIdx.x == 0) *total = all;
}

// Between shade and occlude, one launch: block 0 ends the iteration's
// bookkeeping (whether the loop goes on: a host that read the progress back
// every few iterations cost a thumbnail of 12 K samples 0.83 against 0.44 ms and a
// Cornell box of 4 M 11.4 against 10.0 ms; and the counters that the next
// iteration accumulates, none of which occlude reads), the first cluster scans
// the bounce rays' keys and the second the shadow records'. loop: the graph's
// loop condition, in_loop: whether there is one (a handle has no value that means
// none, and a loop that nobody ends does not end).
__global__ void __cluster_dims__(kPlanCluster, 1, 1) __launch_bounds__(1024)
    k_wf_plan(const __grid_constant__ WfArgs a, cudaGraphConditionalHandle loop, bool in_loop) {
    WfCtl* c = a.ctl;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        c->iters++;
        c->done = c->next >= c->total && c->live == 0;
        if (in_loop && (c->done || c->overflow || c->err || c->iters >= c->limit)) cudaGraphSetConditional(loop, 0);
        c->iter_first = c->next;
        c->live = 0;
        c->ext_next = 0;
        c->occ_next = 0;
        c->nfree = 0;
        c->free_next = 0;
        c->nrec = 0;
        c->shaded = c->nlive;
        c->nlive = 0;
    }
    if (blockIdx.x >= kPlanCluster) key_scan(a.shist, a.soff, &c->nshadow);
    else if (a.raysort) key_scan(a.rhist, a.roff, &c->nbounce);
}

// The record that thread t of shade wrote k-th, or -1. Under the material sort
// shade ran the threads below the live count alone.
RT_D int shadow_record(const WfArgs& a, int t, int k) {
    int live = a.sort ? a.ctl->shaded : a.nslots;
    if (t >= live || k >= a.S.cnt[RT_IX(t, a.nslots)]) return -1;
    return k * a.nslots + t;
}

// Occlude and the shadow scatter run a row of blocks per record that a vertex may
// write (shade's threads along x). Rows lie along y and, past that axis's 65 535
// (a light of 256 x 256 samples), along z.
constexpr int kMaxRows = 65535;
RT_D int shadow_row() { return (int)(blockIdx.z * gridDim.y + blockIdx.y); }

// Shadow sort: each queued record goes to its key's offset plus its rank. Few
// threads that take many turns: with a thread per possible record most blocks
// had nothing to do, and starting them took longer than the records (8 M slots
// of two records: 40 us an iteration; all sorting of a full-HD icosphere frame of
// 64 samples 4.10 to 3.51 ms, smooth mesh 0.76 to 0.67, mixed batch 4.49 to 3.99).
// Occlude is not launched so: the long rays of its blocks want the hardware's
// own scheduling (0.75 M threads: 29.2 to 31.2 ms; a thread a slot: 29.5).
constexpr int kScatterBlocks = 148 * 10;
__global__ void k_wf_sscatter(const __grid_constant__ WfArgs a) {
    const int n = a.sort ? a.ctl->shaded : a.nslots;
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < (unsigned)n; t += gridDim.x * blockDim.x) {
        int j = shadow_record(a, (int)t, shadow_row());
        if (j < 0) continue;
        int pos = a.soff[RT_IX(a.S.key[j], kRayKeys)] + a.S.rank[j];
        if (pos < a.ctl->nshadow) a.S.order[pos] = j;
        else atomicExch(a.err, RT_ERR_BOUNDS);
    }
}

// Persistent any-hit for opaque batches (the walk is one any-hit traversal):
// the dynamic-fetch scheme of k_wf_extend_pt over the shadow queue.
template <int STACK>
__global__ void __launch_bounds__(256) k_wf_occlude_pt(const __grid_constant__ WfArgs a) {
    const unsigned full = 0xffffffffu;
    int lane = threadIdx.x & 31;
    unsigned n = (unsigned)a.nslots * (unsigned)a.S.per;
    Walker<true, STACK> w;
    int rec = -1;
    bool exhausted = false;
    for (;;) {
        bool idle = rec < 0 && !exhausted;
        unsigned need = __ballot_sync(full, idle);
        unsigned busy = __ballot_sync(full, rec >= 0);
        if (!need && !busy) break;
        if (need && (__popc(need) >= kRefill || !busy)) {
            int leader = __ffs(need) - 1;
            unsigned base = 0;
            if (lane == leader) base = atomicAdd(&a.ctl->occ_next, (unsigned)__popc(need));
            base = __shfl_sync(full, base, leader);
            if (idle) {
                unsigned j = base + (unsigned)__popc(need & ((1u << lane) - 1u));
                if (j >= n) {
                    exhausted = true;
                } else if ((rec = shadow_record(a, (int)(j % (unsigned)a.nslots), (int)(j / (unsigned)a.nslots))) >= 0) {
                    float4 o = a.S.o[rec], d = a.S.d[rec], c = a.S.c[rec];
                    w.start(a.views[RT_IX(fbits(c.w), a.nviews)], v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), kEps, o.w, nullptr, false, 0);
                }
            }
            continue;
        }
        if (rec >= 0) {
            float4 c = a.S.c[rec];
            if (w.step(a.views[RT_IX(fbits(c.w), a.nviews)], nullptr, a.err)) {
                if (w.best.kind == HIT_NONE) {   // visible: transmittance 1
                    int packed = fbits(a.S.d[rec].w);
                    int slot = RT_IX(packed >> 1, a.nslots);
                    float4* dst = (packed & 1) ? (a.P.la + slot) : (a.P.lp + slot);
                    float* f = reinterpret_cast<float*>(dst);
                    atomicAdd(f, c.x);
                    atomicAdd(f + 1, c.y);
                    atomicAdd(f + 2, c.z);
                }
                rec = -1;
            }
        }
    }
}

// OPAQUE: a batch with no transmissive material, whose shadow rays are any-hit
// walks. That variant has a register budget of 5 blocks of 256 (48 registers):
// 10 blocks of the autotuned 128 threads per SM instead of 8, occlude -7.8%
// per 64-spp icosphere frame. The transparent variant keeps the full budget
// its longer walk needs.
template <int STACK, bool L4, bool OPAQUE, bool ONE>
__global__ void __launch_bounds__(256, OPAQUE ? 5 : 1) k_wf_occlude(const __grid_constant__ WfArgs a) {
    int j;
    if (a.shadowsort) {   // a flat grid over the sorted order
        long long p = (long long)shadow_row() * gridDim.x * blockDim.x + (long long)blockIdx.x * blockDim.x + threadIdx.x;
        int n = a.ctl->nshadow;
        if (p >= n) return;
        j = RT_IX(a.S.order[p], a.nslots * a.S.per);
    } else {
        j = shadow_record(a, blockIdx.x * blockDim.x + threadIdx.x, shadow_row());
        if (a.regroup) {   // shadow rays by direction octant
            __shared__ int s_idx[256], s_cnt[8][8], s_tot;
            int cls = -1;
            if (j >= 0) {
                float4 d = a.S.d[j];
                cls = octant(d.x, d.y, d.z);
            }
            int m = block_group<8>(j, cls, s_idx, s_cnt, &s_tot);
            if ((int)threadIdx.x >= m) return;
            j = s_idx[threadIdx.x];
        } else if (j < 0) {
            return;
        }
    }
    // The any-hit walk has no register to spare for what a visible ray adds: it
    // is read after it, and added in one vector operation (full-HD icosphere frame
    // of 64 samples 29.8 to 29.2 ms, smooth mesh 1.40 to 1.35, Cornell box 0.74 to
    // 0.70). The transparent walk has, and takes it along: read late it lost 2%.
    constexpr bool LATE = OPAQUE && ONE;
    float4 o = a.S.o[j], d = a.S.d[j], c;
    if (!LATE) c = a.S.c[j];
    const SceneView& s = ONE ? c_wf_one.view : a.views[RT_IX(fbits(c.w), a.nviews)];
    V3 tr = shadow_transmittance<STACK, L4>(s, OPAQUE ? 1 : a.opaque, v3(o.x, o.y, o.z), v3(d.x, d.y, d.z), kEps,
                                            o.w, nullptr, a.err);
    if (near_zero(tr)) return;
    if (LATE) c = a.S.c[j];
    int packed = fbits(LATE ? a.S.d[j].w : d.w);
    int slot = RT_IX(packed >> 1, a.nslots);
    V3 v = v3(c.x, c.y, c.z) * tr;
    atomicAdd((packed & 1) ? (a.P.la + slot) : (a.P.lp + slot), make_float4(v.x, v.y, v.z, 0.0f));
}

// Mean of the accumulated sums into the films (Renderer.cs:711).
__global__ void k_wf_finalize(const WfRequest* reqs, int nreq, float* const* films, const int* film_w,
                              const int* film_h) {
    int r = blockIdx.y;
    if (r >= nreq) return;
    const WfRequest& R = reqs[r];
    long long plane = (long long)R.ww * R.wh;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < plane; i += (long long)gridDim.x * blockDim.x) {
        int lx, ly;
        strip_pixel((int)i, R.ww, R.wh, lx, ly);   // the accumulation buffer is in strip order
        size_t fp = (size_t)film_w[r] * film_h[r];
        size_t fi = (size_t)(R.y0 + ly) * film_w[r] + (R.x0 + lx);
        for (int c = 0; c < 3; c++) films[r][c * fp + fi] = (float)(R.accum[c * plane + i] / (double)R.spp);
    }
}

}  // namespace rt
