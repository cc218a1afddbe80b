// Wavefront path tracer: a pool of path slots advanced one bounce per iteration by a
// fixed sequence of kernels, replayed from a CUDA graph until every work item is done.
// Works on any number of views (one view = one camera over one scene), which is how a
// batch of scenes renders in one launch.
//
// One iteration is six launches: trace (traversal only), resolve of continuation rays
// (emission, shading queues) and of MIS and shadow rays (their contributions), shade for
// Disney surfaces, shade for the other materials, logic (finish samples, start new ones);
// independent ones run side by side (see run_wavefront).  Adjoint renders add the two shading kernels of replayed vertices and a kernel that
// scatters finished vertices' parameter gradients onto texels and material constants.
// Ray queues (filled by the shade and logic kernels, consumed by the next trace):
//   cont    slot ids whose continuation ray is in the slot's ray registers
//   mis     MIS-BSDF rays (origin|slot, direction|pdf, weight|view)
//   shadow  NEE shadow rays (origin|t_max, direction|slot, contribution|view)
// Shading queues (filled by k_wf_resolve_cont, consumed by the shade kernels):
//   disney / simple   slot ids whose continuation ray hit a surface of that class
// Entries are appended with warp-aggregated atomics (one atomic per warp and queue:
// ballot, popcount, prefix), so each queue is dense and its float4 records are read
// coalesced.  The resolve kernels add MIS and shadow contributions, and the emission a
// continuation ray sees at the first bounce, to the slot's accumulator; the logic
// kernel folds it into the path.
//
// Work items are (view, pixel, chunk of `chunk` consecutive samples).  A slot runs its
// item's samples one after another with Kahan-compensated sums and writes the item's
// partial sums once; a final kernel sums the chunks of each pixel in chunk order.  When
// a path ends, its slot immediately starts the next sample (path regeneration).
//
// The buffers, pinned staging, events and the instantiated graph live in a per-context
// workspace (WfCache) that later renders reuse; the graph is launched again as long as
// the launch state (WfState, tuning, iteration bound) is byte-identical.
#include <cmath>
#include <cstring>
#include <utility>
#include <vector>

#include "fm_bsdf_grad.cuh"
#include "fm_path.cuh"
#include "fm_render.h"
#include "fm_trace.cuh"

namespace fm {

namespace {

// slot flags (depth in bits 8..): a continuation ray was queued / shadow or MIS rays of
// this slot are queued, both set by the shading kernels and read by the logic kernel
constexpr int kNextCont = 1;
constexpr int kPending = 2;
// adjoint renders: the slot is replaying its sample's path (second pass)
constexpr int kReplay = 4;
// the slot has no work item yet / will get none any more
constexpr int kNeedItem = 8;
constexpr int kDone = 16;
// queue counters: two sets of the three ray queues (the one being filled for the next trace
// and the one being traced; they change places every iteration, see WfState::qw), slots
// still holding work, the shading queues (two classes, and in adjoint renders two more
// for replayed vertices) and the trace kernel's next unclaimed ray.  Each counter has a
// 128-byte line of its own: atomics from every warp of the GPU on counters that share a
// line queue behind one another at the L2 (one line for all of them cost 9 % of the
// batched step).
constexpr int kQcLine = 32;
constexpr int kQcCont = 0 * kQcLine, kQcMis = 1 * kQcLine, kQcShadow = 2 * kQcLine;   // within a set
constexpr int kQcSet = 3 * kQcLine;
constexpr int kQcActive = 6 * kQcLine, kQcDisney = 7 * kQcLine, kQcSimple = 8 * kQcLine;
constexpr int kQcTraceNext = 9 * kQcLine, kQcDisneyR = 10 * kQcLine, kQcSimpleR = 11 * kQcLine;
constexpr int kQcGrad = 12 * kQcLine, kQcBodies = 13 * kQcLine, kQcLimit = 14 * kQcLine;
constexpr int kQcCount = 16 * kQcLine;

// Records of queued MIS and shadow rays.
struct RayQueue {
    float4 *mis_o, *mis_d, *mis_a;
    float4 *sh_o, *sh_d, *sh_c;
};

struct WfState {
    int64_t pool;
    const WfView* views;
    int32_t nviews;
    int64_t total_items;
    unsigned long long* next_item;
    // per slot
    int64_t* item;        // global work item (unless kNeedItem or kDone)
    int32_t* k;           // sample within the item
    int32_t* view;
    int32_t* flags;       // kNextCont | kPending | kReplay | kNeedItem | kDone | depth << 8
    uint64_t* rng;
    float4* beta;
    float4* col;
    float4* ro;
    float4* rd;
    float4* hit;
    float4* acc;          // adjoint renders: the iteration's MIS, shadow and emission contributions
                          // (atomic adds from the resolve kernels; forward renders add them to col
                          // and have none)
    float4* isum;
    float4* icomp;
    float4* asum;         // where aov is set (null otherwise)
    float4* nsum;
    // queues
    int32_t* cont_q;
    int32_t* disney_q;    // slots whose continuation ray hit a Disney surface
    int32_t* simple_q;    // ... a Lambert, conductor or dielectric surface
    int32_t* disney_r;    // adjoint renders: the same for slots replaying their path
    int32_t* simple_r;
    RayQueue rq;          // MIS and shadow rays being traced
    RayQueue wq;          // ... being queued for the next iteration (the same buffers when resolution
                          // of the traced rays ends before shading begins)
    float4* cont_h;       // trace results in continuation-queue order: hit (t, prim, b1, b2)
    int32_t* cont_v;      // ... and the ray's view, so that hit resolution starts from
                          // coalesced loads instead of the slot indirection
    float4* mis_h;        // trace results: MIS ray hits (t, prim, b1, b2)
    uint32_t* sh_h;       // ... shadow ray occluded (1) or not (0)
    int64_t cap_cont, cap_mis, cap_sh;
    unsigned* qc;         // kQc* counters
    unsigned* qr;         // the counter set of the rays being traced (appends beyond a queue's
                          // capacity count too: readers clamp with traced_rays)
    unsigned* qw;         // the counter set being filled for the next iteration
    int32_t aov;          // some view wants albedo or normal images: asum / nsum are kept
    int64_t trace_tail;   // rays from the end of the trace queues below which warps claim exactly what they need
    // trace kernel span of the current iteration (earliest block start, latest block
    // end, device global timer in ns) and the sum of the spans so far
    unsigned long long* tspan;
    Counters* cnt;
    uint32_t* status;
    // adjoint renders only (null otherwise)
    float4* lp;           // primal radiance of the slot's current sample
    float4* dfr;          // [5 per slot] the slot's current vertex: dlw[15] (c*5+i), material, u, v
    float4* vg;           // [2 per slot] gradient collected for that vertex (g[5]; NEE / MIS, resolve kernels)
    float4* gq;           // [3 per entry] finished vertices' gradients: g[5], u, v, material, view
    int64_t cap_grad;
    float4* sh_g;         // [3 per shadow ray] g[5], u, v, material, env weight e[3], env score s
    float4* mis_g;        // [8 per MIS ray] B[15] (c*5+i), material, u, v, e[3], a[5], b[5]
    float* const* tex_acc;     // per scene texture: NULL or tex_copies[t] x w*h*3 FP32 accumulators
    const int32_t* tex_copies;
    float* mat_acc;            // num_materials * 5 FP32 accumulators, or NULL
    double* env_row;           // env importance: per-row and global score sums (see scatter_env_score)
    double* env_total;
};

FM_D unsigned lanemask_lt() { return (1u << (threadIdx.x & 31)) - 1u; }

// Warp-aggregated append: returns this lane's index (or -1 when !want).
FM_D int64_t wagg_append(unsigned* counter, bool want)
{
    const unsigned mask = __activemask();
    const unsigned b = __ballot_sync(mask, want);
    if (!want) return -1;
    const int leader = __ffs(b) - 1;
    unsigned base = 0;
    if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(counter, (unsigned)__popc(b));
    base = __shfl_sync(b, base, leader);
    return (int64_t)base + __popc(b & lanemask_lt());
}

// Block-aggregated append to one of NQ queues (which = -1: none), the queue k counted
// by qc[ci[k]].  Every thread of the block calls it at the same point of block-uniform
// control flow; `sh` is 2 * NQ words of shared memory.  One shared-memory atomic per warp
// and queue and one global atomic per block and queue: appends from every warp of the
// GPU to one counter wait on one another at the L2, so a hot queue is cheaper to fill a
// block at a time.
template <int NQ>
FM_D int64_t block_append(unsigned* qc, const int* ci, int which, unsigned* sh)
{
    if (threadIdx.x < NQ) sh[threadIdx.x] = 0u;
    __syncthreads();
    unsigned local = 0;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
        const unsigned b = __ballot_sync(0xffffffffu, which == k);
        if (b == 0u) continue;
        const int leader = __ffs(b) - 1;
        unsigned base = 0;
        if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(&sh[k], (unsigned)__popc(b));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (which == k) local = base + __popc(b & lanemask_lt());
    }
    __syncthreads();
    if (threadIdx.x < NQ && sh[threadIdx.x]) {
        int c = ci[0];
#pragma unroll
        for (int k = 1; k < NQ; ++k)
            if ((int)threadIdx.x == k) c = ci[k];
        sh[NQ + threadIdx.x] = atomicAdd(&qc[c], sh[threadIdx.x]);
    }
    __syncthreads();
    return which < 0 ? -1 : (int64_t)sh[NQ + which] + local;
}

// wagg_append for call sites where lanes of one warp may reach the append with
// different counters at once (divergent jobs whose appends the compiler may merge):
// lanes are grouped by counter before the ballot.
FM_D int64_t wagg_append_grouped(unsigned* counter, bool want)
{
    const unsigned mask = __activemask();
    const unsigned peers = __match_any_sync(mask, (unsigned long long)counter);
    const unsigned b = __ballot_sync(mask, want) & peers;
    if (!want) return -1;
    const int leader = __ffs(b) - 1;
    unsigned base = 0;
    if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(counter, (unsigned)__popc(b));
    base = __shfl_sync(b, base, leader);
    return (int64_t)base + __popc(b & lanemask_lt());
}

// One vector atomic (each component added atomically) instead of three scalar ones.
FM_D void acc_add(float4* a, f3 c) { atomicAdd(a, make_float4(c.x, c.y, c.z, 0.0f)); }

// Where hit resolution adds a slot's radiance contributions: the sample's radiance col
// itself in forward renders; in adjoint renders the iteration's accumulator acc, which
// the logic kernel adds to col (the replay reads the radiance before this iteration's
// contributions).
template <bool ADJ>
FM_D float4* rad_acc(const WfState& st, int slot) { return ADJ ? &st.acc[slot] : &st.col[slot]; }

FM_D int find_view(const WfState& st, int64_t item)
{
    int lo = 0, hi = st.nviews - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (st.views[mid].item_base <= item)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// ---- adjoint helpers -------------------------------------------------------------
//
// The adjoint renders each sample twice in the same slot: a primal pass that records
// the path's radiance L, then a replay with the same random numbers.  Each term V of a
// sample's radiance is a product of factors along the path, and the derivative of the
// expected image is E[dV/dp + V d log q/dp] summed over the sampled directions, q the
// density they were drawn with (sampled directions held fixed).  At a replayed vertex
// k with throughput beta_k and BSDF f_k (parameters p = basecolor, metallic,
// roughness of that vertex):
//   NEE term c (if unshadowed): dc/dp = beta Le cos w_l / pdf_l df/dp
//                                       + c (-2 (1 - w_l) dlog pdf_b/dp)     (MIS weight)
//   MIS term c (if it hits an emitter): beta Le cos w_b / pdf_b df/dp
//                                       + c (dlog q/dp - dlog pdf_b/dp + 2 (1 - w_b) dlog pdf_b/dp)
//   continuation: (L - C_<=k) (df/dp / f + dlog q/dp - dlog pdf_b/dp)
// pdf_b is the BSDF density the reference reports and q the sampler's true density
// (they differ for the Disney reflection lobes; see fm_bsdf_grad.cuh); C_<=k is the
// radiance collected up to and including vertex k.  The first two are collected by the
// resolve kernel once visibility and the emitter are known; the third is deferred to the
// next shaded vertex, where L - C_<=k is known.  Environment texels enter through Le
// (bilinear taps) and through the light's sampling and reported densities (importance
// tables normalised per row and over the whole map), handled by scatter_env and
// scatter_env_score.  Every part is contracted with the pixel's dLoss/dI / spp before it
// is scattered, so a payload holds one float per parameter (or per parameter and
// channel while Le is still unknown).

// dLoss/dI of the slot's pixel divided by spp (the image is a mean over samples).
FM_D f3 pixel_delta(const WfState& st, int slot, const WfView& V)
{
    const int64_t local = st.item[slot] - V.item_base;
    const int npix = V.cfg.width * V.cfg.height;
    const int p = (int)(local % npix);
    const float inv = 1.0f / (float)V.cfg.spp;
    const float* d = V.drgb + 3 * (size_t)p;
    return f3{__ldg(d) * inv, __ldg(d + 1) * inv, __ldg(d + 2) * inv};
}

// Texel gradients are accumulated in FP32 (reductions with no return value) in several
// copies per texture (more for small textures, whose texels are hit more often), a
// block writing to copy blockIdx % copies, which spreads the updates that concurrent
// blocks make to the same texel; the copies are summed in FP64 after the render
// (fm_adjoint.cu).
FM_D float* grad_copy(const WfState& st, int tex, const DevTexture& t)
{
    const int copies = st.tex_copies[tex];
    return st.tex_acc[tex] + (size_t)(blockIdx.x % copies) * ((size_t)t.w * t.h * 3);
}

// Sum of v over the lanes in `peers` (which must all be active and call this together).
FM_D float peer_sum(unsigned peers, float v)
{
    float sum = 0.0f;
    for (unsigned m = peers; m; m &= m - 1u) sum += __shfl_sync(peers, v, __ffs(m) - 1);
    return sum;
}

// Adds g[c] * (weight of each tap) to channel c0 + c of the taps tex_sample reads.
// Neighbouring pixels often read the same taps; lanes of the warp whose taps coincide
// (same accumulator, texture and first tap, hence the same four taps) add their values
// together first, and one lane issues the reductions.
FM_D void tex_scatter(const WfState& st, int tex, const DevTexture& t, float u, float v, int c0, int nc,
                      const float* g)
{
    const TexTaps tp = tex_taps(t, u, v);
    float* base = grad_copy(st, tex, t);
    float* first = base + 3 * ((size_t)tp.y[0] * t.w + tp.x[0]) + c0;
    const unsigned peers = __match_any_sync(__activemask(), (unsigned long long)(uintptr_t)first);
    const bool leader = (int)(threadIdx.x & 31) == __ffs(peers) - 1;
    for (int k = 0; k < tp.n; ++k) {
        float* at = base + 3 * ((size_t)tp.y[k] * t.w + tp.x[k]) + c0;
        for (int c = 0; c < nc; ++c) {
            const float sum = peer_sum(peers, tp.w[k] * g[c]);
            if (leader && sum != 0.0f) atomicAdd(at + c, sum);
        }
    }
}

// Lanes of the warp that pass the same key sum their n values; one lane per key adds
// the sums to base[0..n).
FM_D void warp_add_by_key(int key, const float* v, int n, float* base)
{
    const unsigned peers = __match_any_sync(__activemask(), key);
    const int leader = __ffs(peers) - 1;
    for (int i = 0; i < n; ++i) {
        float sum = 0.0f;
        for (unsigned m = peers; m; m &= m - 1u) sum += __shfl_sync(peers, v[i], __ffs(m) - 1);
        if ((int)(threadIdx.x & 31) == leader && sum != 0.0f) atomicAdd(base + i, sum);
    }
}

// Material whose parameters a vertex's gradient goes to, or -1 (no differentiable
// parameters: conductor, dielectric, per-vertex attributes).
FM_D int grad_target(const DevScene& S, const HitInfo& h)
{
    const DevMaterial& M = S.materials[h.mat];
    if (M.vattr_offset >= 0) return -1;
    return (M.type == 0 || M.type == 3) ? h.mat : -1;
}

// Scatters d/d{basecolor rgb, metallic, roughness} at (u, v) of material `mat` to the
// textures those parameters read (basecolor: rgb; metallic: the third channel;
// roughness: the second), or to the material's constants.
FM_D void scatter_params(const WfState& st, const DevScene& S, int mat, float u, float v, const float* g)
{
    if (mat < 0) return;
    const DevMaterial& M = S.materials[mat];
    const int which[3] = {MP_BASECOLOR, MP_METALLIC, MP_ROUGHNESS};
    const int first[3] = {0, 3, 4}, count[3] = {3, 1, 1}, chan[3] = {0, 2, 1};
    float cst[kGradParams] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    bool any_cst = false;
    for (int k = 0; k < 3; ++k) {
        const float* gg = g + first[k];
        const TexRef& r = M.p[which[k]];
        if (r.tex < 0) {
            for (int c = 0; c < count[k]; ++c) cst[first[k] + c] = gg[c];
            any_cst = true;
            continue;
        }
        bool any = false;
        for (int c = 0; c < count[k]; ++c) any = any || gg[c] != 0.0f;
        if (any && st.tex_acc && st.tex_acc[r.tex]) tex_scatter(st, r.tex, S.textures[r.tex], u, v, chan[k], count[k], gg);
    }
    if (any_cst && st.mat_acc) warp_add_by_key(mat, cst, kGradParams, st.mat_acc + (size_t)mat * kGradParams);
}

// Scatters e (per channel, before the env factor) to the env texels seen along `dir`.
FM_D void scatter_env(const WfState& st, const DevScene& S, f3 dir, f3 e)
{
    if (!st.tex_acc || S.env_light < 0) return;
    const DevEnv& E = S.env;
    if (!st.tex_acc[E.tex]) return;
    float u, v, th;
    spherical_uv(xf_vec(E.w2l, dir), u, v, th);
    const float g[3] = {e.x * E.factor, e.y * E.factor, e.z * E.factor};
    tex_scatter(st, E.tex, S.textures[E.tex], u, v, 0, 3, g);
}

// Texel (i, j) of the env map that holds direction `dir` and its luminance (the cell
// EnvLight::Pdf reads).
FM_D bool env_texel(const DevScene& S, f3 dir, int& i, int& j, float& lumt)
{
    const DevEnv& E = S.env;
    float u, v, th;
    spherical_uv(xf_vec(E.w2l, dir), u, v, th);
    i = (int)(u * (float)E.w);
    j = (int)(v * (float)E.h);
    i = i < 0 ? 0 : (i > E.w - 1 ? E.w - 1 : i);
    j = j < 0 ? 0 : (j > E.h - 1 ? E.h - 1 : j);
    const float4 t = __ldg(S.textures[E.tex].texels + (size_t)j * E.w + i);
    lumt = luminance(f3{t.x, t.y, t.z});
    return lumt > 0.0f;
}

// s * d log(density)/d texels for the env light's densities at `dir`: the sampled
// texel's own term (d log lum = L_c / lum) here; the normalisation terms are summed
// into env_row[j] (reported density: divided by the row sum) or env_total (sampling
// density: divided by the map's sum) and spread over the texels after the render.
FM_D void scatter_env_score(const WfState& st, const DevScene& S, f3 dir, float s, bool per_row)
{
    if (s == 0.0f || !st.tex_acc || S.env_light < 0) return;
    if (!st.tex_acc[S.env.tex]) return;
    int i, j;
    float lumt;
    if (!env_texel(S, dir, i, j, lumt)) return;
    float* at = grad_copy(st, S.env.tex, S.textures[S.env.tex]) + 3 * ((size_t)j * S.env.w + i);
    const unsigned tpeers = __match_any_sync(__activemask(), (unsigned long long)(uintptr_t)at);
    const float k = peer_sum(tpeers, s / lumt);
    if ((int)(threadIdx.x & 31) == __ffs(tpeers) - 1) {
        atomicAdd(at, 0.2126f * k);
        atomicAdd(at + 1, 0.7152f * k);
        atomicAdd(at + 2, 0.0722f * k);
    }
    // one FP64 add per warp and target
    const int key = per_row ? j : -1;
    const unsigned peers = __match_any_sync(__activemask(), key);
    double sum = 0.0;
    for (unsigned m = peers; m; m &= m - 1u) sum += (double)__shfl_sync(peers, s, __ffs(m) - 1);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(per_row ? st.env_row + j : st.env_total, sum);
}

// Completes the vertex gradient record of `slot` (NEE / MIS parts collected in vg, plus
// the continuation part dLoss/dI * R . dlw with R the radiance still to come after that
// vertex), queues it for k_wf_grad_scatter and clears the record.  The scatter runs in
// its own small kernel: done here, its tap arithmetic and atomics ran at the low
// occupancy of the replay shading kernels.
FM_D void flush_vertex(const WfState& st, int vid, int slot, f3 wr)
{
    float4* D = st.dfr + 5 * (size_t)slot;
    const float4 d3 = D[3];
    const int mat = __float_as_int(d3.w);
    if (mat < 0) return;
    const float4 d0 = D[0], d1 = D[1], d2 = D[2], d4 = D[4];
    const float4 v0 = st.vg[2 * (size_t)slot], v1 = st.vg[2 * (size_t)slot + 1];
    const float dl[15] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w, d2.x, d2.y, d2.z, d2.w, d3.x, d3.y, d3.z};
    const float vg[kGradParams] = {v0.x, v0.y, v0.z, v0.w, v1.x};
    float g[kGradParams];
    bool any = false;
    for (int i = 0; i < kGradParams; ++i) {
        g[i] = vg[i] + wr.x * dl[i] + wr.y * dl[5 + i] + wr.z * dl[10 + i];
        any = any || g[i] != 0.0f;
    }
    D[3] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
    const int64_t q = wagg_append(&st.qc[kQcGrad], any);
    if (!any) return;
    if (q < st.cap_grad) {
        float4* E = st.gq + 3 * q;
        E[0] = make_float4(g[0], g[1], g[2], g[3]);
        E[1] = make_float4(g[4], d4.x, d4.y, __int_as_float(mat));
        E[2] = make_float4(__int_as_float(vid), 0.0f, 0.0f, 0.0f);
    } else {
        atomicOr(st.status, 2u);
    }
}

// NEE / MIS gradient of the slot's current vertex, once the ray's outcome is known.
FM_D void add_vertex_grad(const WfState& st, int slot, const float* g)
{
    float* v = reinterpret_cast<float*>(st.vg + 2 * (size_t)slot);
    for (int i = 0; i < kGradParams; ++i)
        if (g[i] != 0.0f) atomicAdd(v + i, g[i]);
}

// Last kernel of a conditional graph body (iters_per_graph iterations): run the body
// again while any slot holds work, no queue overflowed (status bit 2: work was dropped,
// so the render has failed) and the iteration bound is not reached (status bit 4
// reports that the bound stopped the loop).
__global__ void k_wf_continue(WfState st, cudaGraphConditionalHandle handle, unsigned max_bodies)
{
    const unsigned active = st.qc[kQcActive];
    const unsigned bodies = ++st.qc[kQcBodies];
    const bool overflow = (*(volatile uint32_t*)st.status & 2u) != 0u;
    if (active != 0u && !overflow && bodies >= max_bodies) atomicOr(st.status, 4u);
    cudaGraphSetConditional(handle, (active != 0u && !overflow && bodies < max_bodies) ? 1u : 0u);
}

// After the iteration at which a caller's limit falls inside a graph body: the body's nth run
// reports the limit if a slot still holds work there.
__global__ void k_wf_limit(WfState st, unsigned nth)
{
    if (++st.qc[kQcLimit] != nth || st.qc[kQcActive] == 0u) return;
    if ((*(volatile uint32_t*)st.status & 2u) == 0u) atomicOr(st.status, 4u);
}

// Rays of the current iteration, [cont | MIS | shadow].  A queue that overflowed counted
// appends beyond its capacity (only the first cap entries were written, and status bit 2
// is set): counts are clamped to the capacity so that no kernel reads an entry that was
// never written.
struct TracedRays {
    uint32_t cont, mis, shadow;
};
FM_D TracedRays traced_rays(const WfState& st)
{
    return TracedRays{(uint32_t)min((int64_t)st.qr[kQcCont], st.cap_cont), (uint32_t)min((int64_t)st.qr[kQcMis], st.cap_mis),
                      (uint32_t)min((int64_t)st.qr[kQcShadow], st.cap_sh)};
}

// Called once by the trace kernel: clears the counters that the rest of the iteration
// fills.  Their last readers ran before this kernel.
FM_D void clear_counters(const WfState& st)
{
    st.qw[kQcCont] = 0;
    st.qw[kQcMis] = 0;
    st.qw[kQcShadow] = 0;
    st.qc[kQcActive] = 0;
    st.qc[kQcDisney] = 0;
    st.qc[kQcSimple] = 0;
    st.qc[kQcDisneyR] = 0;
    st.qc[kQcSimpleR] = 0;
    st.qc[kQcGrad] = 0;
}

FM_D unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The rays of the combined index space as a stream (trace_stream): continuation rays by
// slot, MIS and shadow rays from their queues.
struct WfRays {
    const WfState& st;
    uint32_t nc, ncm;   // continuation rays, continuation + MIS rays
    FM_D StreamRay load(uint32_t idx) const
    {
        StreamRay q;
        q.tmin = 0.0f;
        q.tmax = kRealMax;
        q.any = false;
        float4 o4, d4;
        int vid;
        if (idx < nc) {
            const int slot = st.cont_q[idx];
            vid = st.view[slot];
            o4 = st.ro[slot];
            d4 = st.rd[slot];
            st.cont_v[idx] = vid;
        } else if (idx < ncm) {
            o4 = st.rq.mis_o[idx - nc];
            d4 = st.rq.mis_d[idx - nc];
            vid = __float_as_int(st.rq.mis_a[idx - nc].w);
        } else {
            o4 = st.rq.sh_o[idx - ncm];
            d4 = st.rq.sh_d[idx - ncm];
            vid = __float_as_int(st.rq.sh_c[idx - ncm].w);
            q.tmin = kEps;
            q.tmax = o4.w;
            q.any = true;
        }
        q.scene = st.views[vid].scene;
        q.o = f3{o4.x, o4.y, o4.z};
        q.d = f3{d4.x, d4.y, d4.z};
        return q;
    }
    FM_D float tmin(uint32_t, bool any) const { return any ? kEps : 0.0f; }
    FM_D void finish(uint32_t idx, const Hit& h) const
    {
        if (idx < ncm) {
            float4* out = idx < nc ? st.cont_h + idx : st.mis_h + (idx - nc);
            *out = make_float4(h.t, __int_as_float(h.prim), h.b1, h.b2);
        } else {
            st.sh_h[idx - ncm] = h.prim >= 0 ? 1u : 0u;
        }
    }
};

// A continuation ray's result: the shading queue the slot goes to by the hit's material
// class (0 Disney, 1 other materials; 2 and 3 the same for vertices of adjoint renders
// being replayed), or -1 when a miss or a first-bounce emitter hit ends the path here.
template <bool ADJ>
FM_D int finish_cont(const WfState& st, int64_t idx, const DevScene& S, const Hit& h)
{
    const int cslot = st.cont_q[idx];
    const int cflags = st.flags[cslot];
    const int depth = cflags >> 8;
    int cls = -1;
    // the ray itself is needed only for a first-bounce miss or emitter hit
    auto ray_dir = [&]() {
        const float4 d4 = st.rd[cslot];
        return f3{d4.x, d4.y, d4.z};
    };
    if (h.prim < 0) {
        // the camera ray's beta is 1
        if (depth == 1 && S.env_light >= 0) {
            const f3 d = ray_dir();
            acc_add(rad_acc<ADJ>(st, cslot), env_radiance(S, d));
            if (ADJ && (cflags & kReplay)) scatter_env(st, S, d, pixel_delta(st, cslot, st.views[st.view[cslot]]));
        }
    } else {
        const int info = __ldg(S.prim_info + h.prim);
        const int li = depth == 1 ? (info >> 2) - 1 : -1;
        if (li >= 0) {
            const float4 o4 = st.ro[cslot];
            const HitInfo lh = make_hit(S, f3{o4.x, o4.y, o4.z}, ray_dir(), h);
            if (dot(lh.ng, lh.wo) > 0) acc_add(rad_acc<ADJ>(st, cslot), ld3(S.lights[li].radiance));
        } else {
            cls = (info & 3) - 1;
        }
    }
    // replayed vertices of an adjoint render go to their own queues, so that primal
    // vertices run in the forward shading kernels
    if (cls < 0) return -1;
    return ADJ && (cflags & kReplay) ? cls + 2 : cls;
}

// An MIS-BSDF ray's result: the emitter (or environment) it reaches, MIS-weighted.
template <bool ADJ>
FM_D void finish_mis(const WfState& st, int64_t q, const DevScene& S, const Hit& h)
{
    const float4 o4 = st.rq.mis_o[q], d4 = st.rq.mis_d[q], a4 = st.rq.mis_a[q];
    const int slot = __float_as_int(o4.w);
    const f3 o = f3{o4.x, o4.y, o4.z}, d = f3{d4.x, d4.y, d4.z}, A = f3{a4.x, a4.y, a4.z};
    const float pdf = d4.w;   // < 0: delta BSDF sample (no MIS weight)
    f3 c = mk(0.0f), Le = mk(0.0f);
    float w = 1.0f;
    bool env_hit = false;
    if (h.prim < 0) {
        if (S.env_light >= 0) {
            Le = env_radiance(S, d);
            c = A * Le;
            if (pdf >= 0.0f) {
                w = power_heuristic(pdf, env_pdf(S, d));
                c *= w;
            }
            env_hit = true;
        }
    } else {
        const int li = (__ldg(S.prim_info + h.prim) >> 2) - 1;
        if (li >= 0) {
            const HitInfo lh = make_hit(S, o, d, h);
            const f3 l2s = normalize(o - lh.pos);
            const DevLight& L = S.lights[li];
            const f3 rad = dot(lh.ng, l2s) > 0 ? ld3(L.radiance) : mk(0.0f);
            if (length(rad) >= kEpsPdf) {
                Le = rad;
                c = A * rad;
                if (pdf >= 0.0f) {
                    w = power_heuristic(pdf, area_light_pdf(S, L, o, lh.pos, lh.ng, l2s));
                    c *= w;
                }
            }
        }
    }
    if (c.x == 0.0f && c.y == 0.0f && c.z == 0.0f) return;
    acc_add(rad_acc<ADJ>(st, slot), c);
    // only rays of replayed vertices carry a gradient payload
    if (ADJ && (st.flags[slot] & kReplay)) {
        const float4* P = st.mis_g + 8 * q;
        const float4 p3 = P[3], p4 = P[4], p5 = P[5];
        const int mat = __float_as_int(p3.w);
        const f3 e = f3{p4.z, p4.w, p5.x};
        // sum_c dLoss/dc_c * c_c (e = dLoss/dI * A, c = A Le w)
        const float ec = e.x * Le.x * w + e.y * Le.y * w + e.z * Le.z * w;
        if (mat >= 0) {
            const float4 p0 = P[0], p1 = P[1], p2 = P[2], p6 = P[6], p7 = P[7];
            const float B[15] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w,
                                 p2.x, p2.y, p2.z, p2.w, p3.x, p3.y, p3.z};
            const float a[kGradParams] = {p5.y, p5.z, p5.w, p6.x, p6.y};
            const float b[kGradParams] = {p6.z, p6.w, p7.x, p7.y, p7.z};
            const f3 u3 = Le * w;
            const float wl = pdf >= 0.0f ? 1.0f - w : 0.0f;
            float g[kGradParams];
            for (int i = 0; i < kGradParams; ++i)
                g[i] = u3.x * B[i] + u3.y * B[5 + i] + u3.z * B[10 + i] + ec * (a[i] + wl * b[i]);
            add_vertex_grad(st, slot, g);
        }
        if (env_hit && (e.x != 0.0f || e.y != 0.0f || e.z != 0.0f)) {
            scatter_env(st, S, d, e * w);
            // MIS weight w_b = pdf_b^2 / (pdf_b^2 + pdf_env^2), pdf_env the reported
            // (per-row normalised) density
            if (pdf >= 0.0f) scatter_env_score(st, S, d, -2.0f * (1.0f - w) * ec, true);
        }
    }
}

// A shadow ray's result: the NEE contribution when unoccluded.
template <bool ADJ>
FM_D void finish_shadow(const WfState& st, int64_t q, const DevScene& S, const Hit& h)
{
    if (h.prim >= 0) return;
    const float4 d4 = st.rq.sh_d[q], c4 = st.rq.sh_c[q];
    const int slot = __float_as_int(d4.w);
    acc_add(rad_acc<ADJ>(st, slot), f3{c4.x, c4.y, c4.z});
    if (ADJ && (st.flags[slot] & kReplay)) {
        const float4* P = st.sh_g + 3 * q;
        const float4 p1 = P[1], p2 = P[2];
        const int mat = __float_as_int(p1.w);
        if (mat >= 0) {
            const float4 p0 = P[0];
            const float g[kGradParams] = {p0.x, p0.y, p0.z, p0.w, p1.x};
            add_vertex_grad(st, slot, g);
        }
        if (p2.x != 0.0f || p2.y != 0.0f || p2.z != 0.0f) {
            const f3 dir = f3{d4.x, d4.y, d4.z};
            scatter_env(st, S, dir, f3{p2.x, p2.y, p2.z});
            // env NEE: 1 / pdf_sample, its MIS weight and the score of the sampling
            // density leave 2 (1 - w_l) d log pdf_sample
            scatter_env_score(st, S, dir, p2.w, false);
        }
    }
}

// Traces every queued ray of the combined index space [cont | MIS | shadow]: continuation
// and MIS-BSDF rays (closest hit) and shadow rays (occlusion), and stores the results;
// the resolve kernels turn them into radiance and shading work.  64 registers: three and five
// blocks of 256 threads per SM traced the 16-scene batch in 32.0 and 35.4 ms against 29.1.
__global__ void __launch_bounds__(256, 4) k_wf_trace(WfState st)
{
    const TracedRays n = traced_rays(st);
    const uint32_t nc = n.cont, ncm = nc + n.mis;
    extern __shared__ float4 s_trace[];
    if (threadIdx.x == 0) atomicMin(&st.tspan[0], global_ns());
    if (blockIdx.x == 0 && threadIdx.x == 0) clear_counters(st);
    trace_stream(WfRays{st, nc, ncm}, ncm + n.shadow, &st.qc[kQcTraceNext], (uint32_t)st.trace_tail, s_trace,
                 st.status);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(&st.tspan[1], global_ns());
}

// Turns the continuation rays' results into radiance (emission at the first bounce, added to
// the slots' accumulators) and fills the shading queues.
template <bool ADJ>
__global__ void __launch_bounds__(256) k_wf_resolve_cont(WfState st)
{
    const int64_t nc = traced_rays(st).cont;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // the trace kernel's span, and its counters for the next iteration
        if (st.tspan[1] > st.tspan[0]) st.tspan[2] += st.tspan[1] - st.tspan[0];
        st.tspan[0] = ~0ull;
        st.tspan[1] = 0ull;
        st.qc[kQcTraceNext] = 0;
        if (nc) atomicAdd(&st.cnt->closest, (unsigned long long)nc);
    }
    constexpr int NQ = ADJ ? 4 : 2;
    __shared__ unsigned s_app[2 * NQ];
    const int shade_qc[4] = {kQcDisney, kQcSimple, kQcDisneyR, kQcSimpleR};
    for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x; i0 < nc; i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        int which = -1, slot = 0;
        if (i < nc) {
            slot = st.cont_q[i];
            const float4 h4 = st.cont_h[i];
            const int vid = st.cont_v[i];
            st.hit[slot] = h4;   // the shading kernels read it by slot
            which = finish_cont<ADJ>(st, i, *st.views[vid].scene, Hit{h4.x, __float_as_int(h4.y), h4.z, h4.w});
        }
        const int64_t q = block_append<NQ>(st.qc, shade_qc, which, s_app);
        if (which >= 0) {
            int32_t* const queue = which == 0 ? st.disney_q : which == 1 ? st.simple_q : which == 2 ? st.disney_r : st.simple_r;
            queue[q] = slot;
        }
    }
}

// Turns the MIS and shadow rays' results into radiance (and, in adjoint renders, their
// gradients), added to the slots' accumulators.
template <bool ADJ>
__global__ void __launch_bounds__(256) k_wf_resolve_rays(WfState st)
{
    const TracedRays n = traced_rays(st);
    const int64_t nm = n.mis, total = nm + n.shadow;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (n.mis) atomicAdd(&st.cnt->closest, (unsigned long long)n.mis);
        if (n.shadow) atomicAdd(&st.cnt->shadow, (unsigned long long)n.shadow);
    }
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        if (i < nm) {
            const float4 h4 = st.mis_h[i];
            finish_mis<ADJ>(st, i, *st.views[__float_as_int(st.rq.mis_a[i].w)].scene,
                            Hit{h4.x, __float_as_int(h4.y), h4.z, h4.w});
        } else {
            const int64_t q = i - nm;
            if (st.sh_h[q] == 0u)
                finish_shadow<ADJ>(st, q, *st.views[__float_as_int(st.rq.sh_c[q].w)].scene, Hit{0.0f, -1, 0.0f, 0.0f});
        }
    }
}

FM_D void kahan_add4(float4& sum, float4& c, f3 x)
{
    const float yx = x.x - c.x, yy = x.y - c.y, yz = x.z - c.z;
    const float tx = sum.x + yx, ty = sum.y + yy, tz = sum.z + yz;
    c.x = (tx - sum.x) - yx;
    c.y = (ty - sum.y) - yy;
    c.z = (tz - sum.z) - yz;
    sum.x = tx;
    sum.y = ty;
    sum.z = tz;
}

// The Kahan sums of the slot's item over its first `done` samples (nothing is stored before
// the first).
FM_D void item_sums(const WfState& st, int slot, int done, float4& sum, float4& cmp)
{
    sum = cmp = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (done > 0) {
        sum = st.isum[slot];
        cmp = st.icomp[slot];
    }
}

FM_D int item_samples(const WfView& V, int chunk_index)
{
    const int first = chunk_index * V.chunk;
    return min(V.chunk, V.cfg.spp - first);
}

// Start sample `k` of the slot's item: camera ray into the slot registers, enqueue it.
FM_D void start_sample(const WfState& st, int slot, const WfView& V, int64_t item_local, int k, int extra_flags = 0)
{
    const int npix = V.cfg.width * V.cfg.height;
    const int c = (int)(item_local / npix);
    const PixelRef pr = pixel_ref(V.cfg, (int)(item_local % npix));
    const int sample = c * V.chunk + k;
    Rng rng = rng_for(V.cfg.seed, pr.key, (uint64_t)(V.cfg.sample_offset + sample));
    const float fx = rng_1d(rng), fy = rng_1d(rng);
    const float lx = rng_1d(rng), ly = rng_1d(rng);
    const float px = ((float)pr.i + fx) / (float)V.cfg.img_w;
    const float py = ((float)pr.j + fy) / (float)V.cfg.img_h;
    f3 o, d;
    camera_ray(V.cam, px, py, lx, ly, o, d);
    st.ro[slot] = make_float4(o.x, o.y, o.z, 0.0f);
    st.rd[slot] = make_float4(d.x, d.y, d.z, 0.0f);
    st.rng[slot] = rng.state;
    st.beta[slot] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    st.col[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    st.flags[slot] = (1 << 8) | extra_flags;
    // a replay starts with no deferred continuation gradient
    if (extra_flags & kReplay) st.dfr[5 * (size_t)slot + 3] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
}

// One sampling step of a vertex in k_wf_shade, and what the step's gradient needs.
struct ShadeJob {
    int kind = 0;   // 1: shadow ray queued, 2: MIS ray queued, 3: continuation queued
    int64_t q = -1;
    f3 wi, gw, ge, f, base;
    float mis = 1.0f, dc = 0.0f;
    bool sdelta = false, env = false;
};

// Shading of the slots whose continuation ray hit a surface of material class CLS
// (k_wf_resolve_cont queued them): AOVs at the first bounce, next-event estimation (shadow
// rays), the MIS BSDF samples (MIS rays) and the continuation sample with Russian
// roulette.  Sets kNextCont / kPending so that the logic kernel keeps the slot's
// sample open.  Each class runs its own kernel, so a warp holds one kind of BSDF and
// the kernel's code holds only that kind's lobes.
template <int CLS, bool ADJ>
FM_D void shade_vertices(const WfState& st)
{
    // ADJ: the replayed vertices of an adjoint render; otherwise forward (or primal) ones
    const int64_t n = st.qc[CLS == kClsDisney ? (ADJ ? kQcDisneyR : kQcDisney) : (ADJ ? kQcSimpleR : kQcSimple)];
    const int32_t* queue = CLS == kClsDisney ? (ADJ ? st.disney_r : st.disney_q) : (ADJ ? st.simple_r : st.simple_q);
    unsigned long long n_bounces = 0;
    __shared__ unsigned s_app[2];
    const int cont_qc = kQcCont;
    for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x; i0 < n; i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        const bool valid = i < n;
        const int slot = valid ? queue[i] : 0;
        bool enqueue_cont = false;
        if (valid) {
            ++n_bounces;
            const int vid = st.view[slot];
            const WfView& V = st.views[vid];
            const DevScene& S = *V.scene;
            const int flags0 = st.flags[slot];
            const int depth = flags0 >> 8;
            const bool replay = ADJ;
            int flags = (depth << 8) | (flags0 & kReplay);
            const float4 h4 = st.hit[slot];
            const float4 o4 = st.ro[slot], d4 = st.rd[slot];
            const f3 o = f3{o4.x, o4.y, o4.z}, d = f3{d4.x, d4.y, d4.z};
            const float4 b4 = st.beta[slot];
            f3 beta = f3{b4.x, b4.y, b4.z};
            Hit hit;
            hit.t = h4.x;
            hit.prim = __float_as_int(h4.y);
            hit.b1 = h4.z;
            hit.b2 = h4.w;
            const HitInfo h = make_hit(S, o, d, hit);
            Rng rng;
            rng.state = st.rng[slot];
            const Bsdf b = make_bsdf<CLS>(S, h);
            f3 delta = mk(0.0f);
            int tgt = -1;
            if (ADJ && replay) {
                delta = pixel_delta(st, slot, V);
                tgt = grad_target(S, h);
                // the previous vertex's record: its NEE / MIS rays are resolved and the
                // radiance after it, L - C_<=k-1, is known now
                const float4 a4 = st.acc[slot], c4 = st.col[slot], l4 = st.lp[slot];
                const f3 R = f3{l4.x - (c4.x + a4.x), l4.y - (c4.y + a4.y), l4.z - (c4.z + a4.z)};
                flush_vertex(st, vid, slot, delta * R);
                // this vertex's record: target now, continuation part below
                float4* D = st.dfr + 5 * (size_t)slot;
                D[0] = D[1] = D[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                D[3] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(tgt));
                D[4] = make_float4(h.u, h.v, 0.0f, 0.0f);
                st.vg[2 * (size_t)slot] = st.vg[2 * (size_t)slot + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            if (depth == 1 && !replay && st.aov) {
                const f3 al = bsdf_albedo(b);
                float4 as = st.asum[slot], ns = st.nsum[slot];
                as.x += al.x; as.y += al.y; as.z += al.z;
                ns.x += h.ng.x; ns.y += h.ng.y; ns.z += h.ng.z;
                st.asum[slot] = as;
                st.nsum[slot] = ns;
            }
            // The vertex's sampling steps, in the forward render's random-number order: for
            // each of direct_loop rounds, NEE of every light and one MIS-BSDF sample; then
            // the continuation.  Replayed vertices of adjoint renders run the steps as one
            // flat loop of jobs and evaluate the BSDF's derivatives for each job's direction
            // at the end of the loop body: one call site keeps the dual-number code in the
            // instruction caches once instead of three times.
            const float inv_dl = 1.0f / (float)V.cfg.direct_loop;
            const int nl = S.num_lights;
            auto nee_job = [&](int r, ShadeJob& J) {
                const DevLight& L = S.lights[r];
                LightSample ls;
                bool ok = light_sample(S, L, h.pos, rng_3d(rng), ls);
                ok = ok && ls.pdf >= kEpsPdf && length(ls.radiance) >= kEpsPdf;
                float pb = 0.0f;
                f3 f = mk(0.0f);
                if (ok) {
                    f = bsdf_f<CLS>(b, h.wo, ls.wi);
                    ok = length(f) >= kEpsPdf;
                }
                if (ok) {
                    pb = bsdf_pdf<CLS>(b, h.wo, ls.wi);
                    ok = pb >= kEpsPdf;
                }
                const int64_t q = ADJ ? wagg_append_grouped(&st.qw[kQcShadow], ok) : wagg_append(&st.qw[kQcShadow], ok);
                if (!ok) return;
                f3 c = beta * (f * ls.radiance * absdot(ls.wi, h.ng)) / ls.pdf;
                if (!ls.delta) c *= power_heuristic(ls.pdf, pb);
                c *= inv_dl;
                if (q >= st.cap_sh) {
                    atomicOr(st.status, 2u);
                    return;
                }
                st.wq.sh_o[q] = make_float4(h.pos.x, h.pos.y, h.pos.z, ls.dist - kEps);
                st.wq.sh_d[q] = make_float4(ls.wi.x, ls.wi.y, ls.wi.z, __int_as_float(slot));
                st.wq.sh_c[q] = make_float4(c.x, c.y, c.z, __int_as_float(vid));
                flags |= kPending;
                if (ADJ) {
                    J.kind = 1;
                    J.q = q;
                    J.wi = ls.wi;
                    J.f = f;
                    J.mis = ls.delta ? 1.0f : power_heuristic(ls.pdf, pb);
                    J.base = beta * (absdot(ls.wi, h.ng) / ls.pdf * J.mis * inv_dl);
                    J.dc = dot(delta, c);   // sum_c dLoss/dc_c * c_c
                    J.gw = delta * J.base * ls.radiance;
                    J.sdelta = ls.delta;
                    J.env = L.kind == LK_ENV;
                }
            };
            auto mis_job = [&](ShadeJob& J) {
                const BsdfSample ms = bsdf_sample<CLS>(b, h.wo, rng_3d(rng));
                const bool ok = length(ms.f) >= kEpsPdf && ms.pdf >= kEpsPdf;
                const int64_t q = ADJ ? wagg_append_grouped(&st.qw[kQcMis], ok) : wagg_append(&st.qw[kQcMis], ok);
                if (!ok) return;
                const f3 wn = normalize(ms.wi);
                const f3 ro = spawn_origin(h, wn);
                const f3 A = beta * ms.f * absdot(h.ng, wn) / ms.pdf * inv_dl;
                if (q >= st.cap_mis) {
                    atomicOr(st.status, 2u);
                    return;
                }
                st.wq.mis_o[q] = make_float4(ro.x, ro.y, ro.z, __int_as_float(slot));
                st.wq.mis_d[q] = make_float4(wn.x, wn.y, wn.z, ms.delta ? -1.0f : ms.pdf);
                st.wq.mis_a[q] = make_float4(A.x, A.y, A.z, __int_as_float(vid));
                flags |= kPending;
                if (ADJ) {
                    J.kind = 2;
                    J.q = q;
                    J.wi = ms.wi;
                    J.gw = delta * beta * (absdot(h.ng, wn) / ms.pdf * inv_dl);
                    J.ge = delta * A;
                    J.sdelta = ms.delta;
                }
            };
            auto cont_job = [&](ShadeJob& J) {
                const BsdfSample sc = bsdf_sample<CLS>(b, h.wo, rng_3d(rng));
                if (!(length(sc.f) >= kEpsPdf && sc.pdf >= kEpsPdf)) return;
                beta *= sc.f * absdot(h.ng, sc.wi) / sc.pdf;
                if (depth >= V.cfg.depth) return;
                if (V.cfg.rr_enabled) {
                    if (rng_1d(rng) > V.cfg.rr_coef) return;
                    beta /= V.cfg.rr_coef;
                }
                const f3 no = spawn_origin(h, sc.wi);
                st.ro[slot] = make_float4(no.x, no.y, no.z, 0.0f);
                st.rd[slot] = make_float4(sc.wi.x, sc.wi.y, sc.wi.z, 0.0f);
                st.beta[slot] = make_float4(beta.x, beta.y, beta.z, 0.0f);
                flags = kNextCont | (flags & (kPending | kReplay)) | ((depth + 1) << 8);
                enqueue_cont = true;
                if (ADJ) {
                    J.kind = 3;
                    J.wi = sc.wi;
                }
            };
            if constexpr (ADJ) {
                const int njobs = V.cfg.direct_loop * (nl + 1) + 1;
                for (int j = 0; j < njobs; ++j) {
                    const int r = j == njobs - 1 ? -1 : j % (nl + 1);
                    ShadeJob J;
                    if (r < 0)
                        cont_job(J);
                    else if (r == nl)
                        mis_job(J);
                    else
                        nee_job(r, J);
                    if (J.kind == 0) continue;
                    BsdfGrads bg;
                    const bool grads = tgt >= 0 && !(J.kind == 2 && J.sdelta && CLS == kClsSimple);
                    if (grads) bsdf_grads<CLS>(b, h.wo, J.wi, bg);
                    if (J.kind == 1) {
                        // NEE: df/dp weighted by dLoss/dI beta Le cos w_l / pdf_l, and the MIS
                        // weight's dependence on pdf_b
                        float g[kGradParams] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
                        if (grads) {
                            contract(bg.f, J.gw, g);
                            if (!J.sdelta)
                                for (int i = 0; i < kGradParams; ++i) g[i] -= 2.0f * (1.0f - J.mis) * J.dc * bg.dlogp[i];
                        }
                        const f3 e = J.env ? delta * J.base * J.f : mk(0.0f);
                        const float senv = J.env ? 2.0f * (1.0f - J.mis) * J.dc : 0.0f;
                        float4* P = st.sh_g + 3 * J.q;
                        P[0] = make_float4(g[0], g[1], g[2], g[3]);
                        P[1] = make_float4(g[4], h.u, h.v, __int_as_float(tgt));
                        P[2] = make_float4(e.x, e.y, e.z, senv);
                    } else if (J.kind == 2) {
                        // MIS: df/dp per channel (Le and the MIS weight are known only
                        // after the trace), the density terms, and the env weight
                        float B[15], a[kGradParams], bb[kGradParams];
                        for (int k = 0; k < 15; ++k) B[k] = 0.0f;
                        for (int k = 0; k < kGradParams; ++k) a[k] = bb[k] = 0.0f;
                        if (grads) {
                            for (int i = 0; i < kGradParams; ++i) {
                                B[i] = J.gw.x * bg.f.x.d[i];
                                B[5 + i] = J.gw.y * bg.f.y.d[i];
                                B[10 + i] = J.gw.z * bg.f.z.d[i];
                            }
                            if (!J.sdelta)
                                for (int i = 0; i < kGradParams; ++i) {
                                    a[i] = bg.dscore[i];
                                    bb[i] = 2.0f * bg.dlogp[i];
                                }
                        }
                        float4* P = st.mis_g + 8 * J.q;
                        P[0] = make_float4(B[0], B[1], B[2], B[3]);
                        P[1] = make_float4(B[4], B[5], B[6], B[7]);
                        P[2] = make_float4(B[8], B[9], B[10], B[11]);
                        P[3] = make_float4(B[12], B[13], B[14], __int_as_float(tgt));
                        P[4] = make_float4(h.u, h.v, J.ge.x, J.ge.y);
                        P[5] = make_float4(J.ge.z, a[0], a[1], a[2]);
                        P[6] = make_float4(a[3], a[4], bb[0], bb[1]);
                        P[7] = make_float4(bb[2], bb[3], bb[4], 0.0f);
                    } else if (grads) {
                        // continuation: d log (f / pdf_b) / dp and the score of the
                        // sampler's density, used when the vertex's record is flushed
                        float dl[15];
                        for (int i = 0; i < kGradParams; ++i) {
                            dl[i] = bg.f.x.v > 0.0f ? bg.f.x.d[i] / bg.f.x.v + bg.dscore[i] : 0.0f;
                            dl[5 + i] = bg.f.y.v > 0.0f ? bg.f.y.d[i] / bg.f.y.v + bg.dscore[i] : 0.0f;
                            dl[10 + i] = bg.f.z.v > 0.0f ? bg.f.z.d[i] / bg.f.z.v + bg.dscore[i] : 0.0f;
                        }
                        float4* D = st.dfr + 5 * (size_t)slot;
                        D[0] = make_float4(dl[0], dl[1], dl[2], dl[3]);
                        D[1] = make_float4(dl[4], dl[5], dl[6], dl[7]);
                        D[2] = make_float4(dl[8], dl[9], dl[10], dl[11]);
                        D[3] = make_float4(dl[12], dl[13], dl[14], __int_as_float(tgt));
                    }
                }
            } else {
                ShadeJob J;
                for (int kk = 0; kk < V.cfg.direct_loop; ++kk) {
                    for (int r = 0; r < nl; ++r) nee_job(r, J);
                    mis_job(J);
                }
                cont_job(J);
            }
            st.rng[slot] = rng.state;
            st.flags[slot] = flags;
        }
        const int64_t q = block_append<1>(st.qw, &cont_qc, enqueue_cont ? 0 : -1, s_app);
        if (enqueue_cont) {
            if (q < st.cap_cont)
                st.cont_q[q] = slot;
            else
                atomicOr(st.status, 2u);
        }
    }
    for (int off = 16; off > 0; off >>= 1) n_bounces += __shfl_xor_sync(0xffffffffu, n_bounces, off);
    if ((threadIdx.x & 31) == 0 && n_bounces) atomicAdd(&st.cnt->bounces, n_bounces);
}

// The shading kernels.  The forward Disney kernel is capped at 64 registers (four 256-thread
// blocks per SM): it waits on dependent loads and instruction fetch, and the extra warps
// outweigh its spills (16-scene batch, all kernels but trace: 31.5 / 30.5 / 29.9 ms with two /
// three / four blocks).  The other materials' kernel keeps 80 (two / three / four / five
// blocks: 32.4 / 30.5 / 30.6 / 31.0 ms).  The replay kernels of adjoint renders keep the
// compiler's allocation (their dual-number code spills heavily under a cap).
template <int CLS>
__global__ void __launch_bounds__(256, CLS == kClsDisney ? 4 : 3) k_wf_shade(WfState st)
{
    shade_vertices<CLS, false>(st);
}

template <int CLS>
__global__ void __launch_bounds__(256) k_wf_shade_replay(WfState st)
{
    shade_vertices<CLS, true>(st);
}

// Per slot, after the shading kernels: a sample with neither a continuation ray nor
// rays in flight is finished: its colour (with the shadow, MIS and emission
// contributions the resolve kernels added; adjoint renders fold this iteration's in from
// acc first) goes into the item's Kahan sum and the slot starts its next sample, or
// takes a new work item.
// Most slots of most iterations have rays in flight or no work left, so a block first
// looks at the flags of PER slots per thread (16 bytes at once for four) and lists the slots
// that need more; the long part then runs with full warps over the list.  Deciding slot
// by slot ran it at 18-20 lanes of 32 and had every slot pass the block-wide queue append:
// all kernels but the trace kernel took 30.5 -> 28.9 ms of the 16-scene batch and 0.93 ->
// 0.74 ms of the Cornell box; in an adjoint render of 4 views 10.55 -> 10.47 ms.
// Five blocks per SM (48 registers): the long part waits on dependent loads; four and six
// are within 1 %.
template <bool ADJ, int PER>
__global__ void __launch_bounds__(256, 5) k_wf_logic(WfState st)
{
    unsigned long long n_paths = 0, n_nans = 0;
    unsigned n_active = 0;
    __shared__ unsigned s_app[2];
    __shared__ unsigned s_n;
    __shared__ uint16_t s_list[256 * PER];
    const int cont_qc = kQcCont;
    const int lane = threadIdx.x & 31;
    for (int64_t base = blockIdx.x * (int64_t)(256 * PER); base < st.pool; base += (int64_t)gridDim.x * (256 * PER)) {
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        {
            const int64_t first = base + PER * (int)threadIdx.x;
            const bool whole = first + PER <= st.pool;
            int f[PER];
            if (PER == 4 && whole) {
                const int4 f4 = *reinterpret_cast<const int4*>(st.flags + first);
                f[0] = f4.x;
                f[PER > 1 ? 1 : 0] = f4.y;
                f[PER > 2 ? 2 : 0] = f4.z;
                f[PER > 3 ? 3 : 0] = f4.w;
            } else {
                for (int k = 0; k < PER; ++k) f[k] = first + k < st.pool ? st.flags[first + k] : kDone;
            }
            unsigned todo = 0;
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                if (f[k] & kDone) continue;
                if (!(f[k] & kNeedItem) && (f[k] & (kNextCont | kPending))) {
                    ++n_active;
                    f[k] &= ~(kNextCont | kPending);
                    st.flags[first + k] = f[k];
                    if (ADJ) {
                        const float4 a4 = st.acc[first + k];
                        if (a4.x != 0.0f || a4.y != 0.0f || a4.z != 0.0f) {
                            const float4 c4 = st.col[first + k];
                            st.col[first + k] = make_float4(c4.x + a4.x, c4.y + a4.y, c4.z + a4.z, 0.0f);
                            st.acc[first + k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        }
                    }
                } else {
                    todo |= 1u << k;
                }
            }
            const int mine = __popc(todo);
            int upto = mine;
            for (int off = 1; off < 32; off <<= 1) {
                const int o = __shfl_up_sync(0xffffffffu, upto, off);
                if (lane >= off) upto += o;
            }
            unsigned at = 0;
            if (lane == 31 && upto) at = atomicAdd(&s_n, (unsigned)upto);
            at = __shfl_sync(0xffffffffu, at, 31) + (unsigned)(upto - mine);
#pragma unroll
            for (int k = 0; k < PER; ++k)
                if ((todo >> k) & 1u) s_list[at++] = (uint16_t)(PER * threadIdx.x + k);
        }
        __syncthreads();
        const int n = (int)s_n;
        for (int j0 = 0; j0 < n; j0 += 256) {
            const int j = j0 + (int)threadIdx.x;
            const bool listed = j < n;
            const int slot = listed ? (int)(base + s_list[j]) : 0;
            const int flags = listed ? st.flags[slot] : kDone;
            bool need_new = (flags & kNeedItem) != 0;
            bool enqueue_cont = false;
            // the sample to start (one start_sample call for every case below, so that the
            // lanes of a warp generate their camera rays together)
            int s_vid = 0, s_k = 0, s_flags = 0;
            int64_t s_local = 0;
            if (listed && !need_new) {
                const int64_t item = st.item[slot];
                // the sample's radiance: forward renders add contributions to col directly,
                // adjoint renders collect this iteration's in acc (the replay needs the radiance
                // before them)
                const float4 c4 = st.col[slot];
                f3 col = f3{c4.x, c4.y, c4.z};
                if (ADJ) {
                    const float4 a4 = st.acc[slot];
                    col = f3{c4.x + a4.x, c4.y + a4.y, c4.z + a4.z};
                    if (a4.x != 0.0f || a4.y != 0.0f || a4.z != 0.0f) st.acc[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
                if (ADJ && !(flags & kReplay)) {
                    // primal pass of this sample done: keep L, add it to the image, replay
                    const int vid = st.view[slot];
                    const WfView& V = st.views[vid];
                    st.lp[slot] = make_float4(col.x, col.y, col.z, 0.0f);
                    s_k = st.k[slot];
                    float4 sum, cmp;
                    item_sums(st, slot, s_k, sum, cmp);
                    kahan_add4(sum, cmp, col);
                    st.isum[slot] = sum;
                    st.icomp[slot] = cmp;
                    s_vid = vid;
                    s_local = item - V.item_base;
                    s_flags = kReplay;
                    enqueue_cont = true;
                } else {
                    const int vid = st.view[slot];
                    const WfView& V = st.views[vid];
                    if (ADJ) {
                        // the last vertex's record (its NEE / MIS rays are resolved)
                        const float4 l4 = st.lp[slot];
                        const f3 R = f3{l4.x - col.x, l4.y - col.y, l4.z - col.z};
                        flush_vertex(st, vid, slot, pixel_delta(st, slot, V) * R);
                    }
                    ++n_paths;
                    if (!isfinite(col.x) || !isfinite(col.y) || !isfinite(col.z)) ++n_nans;
                    const int k = st.k[slot];
                    float4 sum, cmp;
                    // the primal pass has added an adjoint render's sample already
                    item_sums(st, slot, ADJ ? k + 1 : k, sum, cmp);
                    if (!ADJ) kahan_add4(sum, cmp, clamp_sample(V.cfg, col));
                    const int kdone = k + 1;
                    const int64_t local = item - V.item_base;
                    const int npix = V.cfg.width * V.cfg.height;
                    const int chunk_index = (int)(local / npix);
                    if (kdone >= item_samples(V, chunk_index)) {
                        float4* P = V.partial + V.partial_f4 * (size_t)local;
                        P[0] = sum;
                        if (st.aov) {
                            P[1] = st.asum[slot];
                            P[2] = st.nsum[slot];
                        }
                        need_new = true;
                    } else {
                        st.isum[slot] = sum;
                        st.icomp[slot] = cmp;
                        st.k[slot] = kdone;
                        s_vid = vid;
                        s_local = local;
                        s_k = kdone;
                        enqueue_cont = true;
                    }
                }
            }
            // new work items for slots that finished theirs (one atomic per warp)
            {
                const unsigned mask = __activemask();
                const unsigned b = __ballot_sync(mask, need_new);
                if (need_new) {
                    const int leader = __ffs(b) - 1;
                    unsigned long long base = 0;
                    if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(st.next_item, (unsigned long long)__popc(b));
                    base = __shfl_sync(b, base, leader);
                    const int64_t it = (int64_t)(base + __popc(b & lanemask_lt()));
                    if (it >= st.total_items) {
                        st.flags[slot] = kDone;
                    } else {
                        const int vid = find_view(st, it);
                        const WfView& V = st.views[vid];
                        st.item[slot] = it;
                        st.view[slot] = vid;
                        st.k[slot] = 0;
                        if (st.aov) st.asum[slot] = st.nsum[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        s_vid = vid;
                        s_local = it - V.item_base;
                        s_k = 0;
                        enqueue_cont = true;
                    }
                }
            }
            if (enqueue_cont) start_sample(st, slot, st.views[s_vid], s_local, s_k, s_flags);
            const int64_t q = block_append<1>(st.qw, &cont_qc, enqueue_cont ? 0 : -1, s_app);
            if (enqueue_cont) {
                if (q < st.cap_cont)
                    st.cont_q[q] = slot;
                else
                    atomicOr(st.status, 2u);
            }
            if (enqueue_cont) ++n_active;
        }
        __syncthreads();   // the list is free again
    }
    for (int off = 16; off > 0; off >>= 1) {
        n_paths += __shfl_xor_sync(0xffffffffu, n_paths, off);
        n_nans += __shfl_xor_sync(0xffffffffu, n_nans, off);
        n_active += __shfl_xor_sync(0xffffffffu, n_active, off);
    }
    if ((threadIdx.x & 31) == 0) {
        if (n_paths | n_nans) {
            atomicAdd(&st.cnt->paths, n_paths);
            atomicAdd(&st.cnt->nans, n_nans);
        }
        if (n_active) atomicAdd(&st.qc[kQcActive], n_active);
    }
}

// Scatters the gradients of the vertices finished this iteration (queued by the replay
// shading and logic kernels) to the textures and constants of their materials.
__global__ void __launch_bounds__(256) k_wf_grad_scatter(WfState st)
{
    const int64_t n = min((int64_t)st.qc[kQcGrad], st.cap_grad);
    for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x; i0 < n; i0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        if (i >= n) continue;
        const float4 e0 = st.gq[3 * i], e1 = st.gq[3 * i + 1], e2 = st.gq[3 * i + 2];
        const float g[kGradParams] = {e0.x, e0.y, e0.z, e0.w, e1.x};
        scatter_params(st, *st.views[__float_as_int(e2.x)].scene, __float_as_int(e1.w), e1.y, e1.z, g);
    }
}

__global__ void k_wf_init(WfState st)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) st.tspan[0] = ~0ull;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < st.pool; s += (int64_t)gridDim.x * blockDim.x) {
        st.flags[s] = kNeedItem;
        if (st.acc) st.acc[s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        st.col[s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// Per pixel: sum the chunks in order (Kahan) and divide by spp.
__global__ void k_wf_reduce(WfView V)
{
    const int npix = V.cfg.width * V.cfg.height;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
        float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f), c = s;
        f3 a = mk(0.0f), n = mk(0.0f);
        for (int ch = 0; ch < V.nchunks; ++ch) {
            const float4* P = V.partial + V.partial_f4 * ((size_t)ch * npix + p);
            const float4 x = P[0];
            kahan_add4(s, c, f3{x.x, x.y, x.z});
            if (V.alb || V.nrm) {
                const float4 y = P[1], z = P[2];
                a += f3{y.x, y.y, y.z};
                n += f3{z.x, z.y, z.z};
            }
        }
        const float inv = 1.0f / (float)V.cfg.spp;
        st3(V.rgb + 3 * (size_t)p, f3{s.x, s.y, s.z} * inv);
        if (V.alb) st3(V.alb + 3 * (size_t)p, a * inv);
        if (V.nrm) st3(V.nrm + 3 * (size_t)p, n * inv);
    }
}

// Adds the counters of one render (workspace-owned, so that the cached graph's launch
// state does not depend on the caller's buffer) to the caller's.
__global__ void k_counters_add(Counters* dst, const Counters* src)
{
    dst->paths += src->paths;
    dst->closest += src->closest;
    dst->shadow += src->shadow;
    dst->bounces += src->bounces;
    dst->nans += src->nans;
}

}  // namespace

// The wavefront workspace of a context: the path-state and queue buffers (sized by the
// largest pool and queue capacities seen so far), the per-view partial sums, pinned
// host staging, events, and the instantiated graph with the launch state it was built
// for.  Renders of one batch shape class reuse all of it, so a render costs the host
// a views upload, a few memsets and one graph launch.
struct WfCache {
    bool adj = false;
    int64_t pool = 0, cap_mis = 0, cap_sh = 0, partial_f4 = 0;
    int64_t aov_pool = 0;        // capacity of asum and nsum, which only some renders need
    float4 *asum = nullptr, *nsum = nullptr;
    int32_t nviews = 0;
    size_t held = 0;             // device bytes of everything below
    int64_t builds = 0;          // times the state buffers were allocated
    std::vector<std::pair<void*, size_t>> allocs;   // state buffers and their bytes
    WfState bufs;                                   // their pointers
    RayQueue alt;                // forward renders: a second set of ray records (null: none)
    cudaStream_t side[2] = {nullptr, nullptr};   // the branches of an iteration's kernels
    cudaEvent_t fork = nullptr, join[2] = {nullptr, nullptr}, fork2 = nullptr;
    float4* partial = nullptr;
    WfView* d_views = nullptr;
    Counters* cnt = nullptr;
    WfView* h_views = nullptr;   // pinned
    void* h_block = nullptr;     // pinned: queue counters, status word, trace spans
    unsigned* h_qc = nullptr;
    uint32_t* h_status = nullptr;
    unsigned long long* h_span = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    std::vector<cudaEvent_t> pev;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    WfState g_st;
    int64_t g_pool = 0, g_max_bodies = 0, g_limit = 0;
    int g_trace_block = 0, g_shade_block = 0, g_iters = 0;
    bool g_profile = false;
    WfCache()
    {
        std::memset(&bufs, 0, sizeof(bufs));
        std::memset(&alt, 0, sizeof(alt));
        std::memset(&g_st, 0, sizeof(g_st));
    }
};

namespace {

void wf_cache_drop_graph(WfCache& c)
{
    if (c.exec) cudaGraphExecDestroy(c.exec);
    if (c.graph) cudaGraphDestroy(c.graph);
    c.exec = nullptr;
    c.graph = nullptr;
}

// Device memory of the workspace; refused beyond the context's limit as the driver refuses
// it when the device has no more.
cudaError_t wf_malloc(fm_ctx* ctx, WfCache& c, void** p, size_t bytes)
{
    if (ctx->wf_limit > 0 && c.held + bytes > ctx->wf_limit) return cudaErrorMemoryAllocation;
    const cudaError_t e = cudaMallocAsync(p, bytes, ctx->stream);
    if (e == cudaSuccess) c.held += bytes;
    return e;
}
void wf_free(WfCache& c, cudaStream_t s, void* p, size_t bytes)
{
    if (!p) return;
    cudaFreeAsync(p, s);
    c.held -= bytes;
}

// Frees state buffers until `keep` are left.
void wf_cache_free_allocs(WfCache& c, cudaStream_t s, size_t keep)
{
    while (c.allocs.size() > keep) {
        wf_free(c, s, c.allocs.back().first, c.allocs.back().second);
        c.allocs.pop_back();
    }
}

void wf_cache_free_state(WfCache& c, cudaStream_t s)
{
    wf_cache_free_allocs(c, s, 0);
    std::memset(&c.bufs, 0, sizeof(c.bufs));
    std::memset(&c.alt, 0, sizeof(c.alt));
    c.pool = c.cap_mis = c.cap_sh = 0;
}

void wf_cache_free_aov(WfCache& c, cudaStream_t s)
{
    wf_free(c, s, c.asum, sizeof(float4) * (size_t)c.aov_pool);
    wf_free(c, s, c.nsum, sizeof(float4) * (size_t)c.aov_pool);
    c.asum = c.nsum = nullptr;
    c.aov_pool = 0;
}

// Calls f(pointer, count) for every buffer of a set of ray records ...
template <class F>
void each_ray_buffer(RayQueue& r, int64_t cap_mis, int64_t cap_sh, F&& f)
{
    f(r.mis_o, cap_mis);
    f(r.mis_d, cap_mis);
    f(r.mis_a, cap_mis);
    f(r.sh_o, cap_sh);
    f(r.sh_d, cap_sh);
    f(r.sh_c, cap_sh);
}
// ... and of the state of `pool` path slots (one set of ray records included).
template <class F>
void each_state_buffer(WfState& b, bool adj, int64_t pool, int64_t cap_mis, int64_t cap_sh, F&& f)
{
    f(b.next_item, 1);
    f(b.item, pool);
    f(b.k, pool);
    f(b.view, pool);
    f(b.flags, pool);
    f(b.rng, pool);
    f(b.beta, pool);
    f(b.col, pool);
    f(b.ro, pool);
    f(b.rd, pool);
    f(b.hit, pool);
    f(b.isum, pool);
    f(b.icomp, pool);
    f(b.cont_q, pool);
    f(b.cont_h, pool);
    f(b.cont_v, pool);
    f(b.disney_q, pool);
    f(b.simple_q, pool);
    each_ray_buffer(b.rq, cap_mis, cap_sh, f);
    f(b.mis_h, cap_mis);
    f(b.sh_h, cap_sh);
    f(b.qc, kQcCount);
    f(b.tspan, 4);
    if (adj) {
        f(b.acc, pool);
        f(b.disney_r, pool);
        f(b.simple_r, pool);
        f(b.lp, pool);
        f(b.dfr, 5 * pool);
        f(b.vg, 2 * pool);
        f(b.gq, 6 * pool);
        f(b.sh_g, 3 * cap_sh);
        f(b.mis_g, 8 * cap_mis);
    }
}

// What a render of some views needs of the workspace at a tuning's pool.
struct WfSizes {
    int64_t pool = 0, cap_mis = 0, cap_sh = 0;
    int64_t items = 0, partial_f4 = 0;
    double samples = 0.0;
    int64_t aov_pool = 0;   // slots with albedo and normal sums: `pool`, or 0 when no view wants those images
};

// Sizes a render and splits the views' samples into work items: about four per path slot
// over the whole job.  Albedo and normal sums are kept, and their partial sums written, only
// when asked for (they are a third of a path's state traffic).
WfSizes size_views(std::vector<WfView>& views, int64_t tune_pool)
{
    WfSizes z;
    int64_t max_lights = 1, max_dl = 1;
    bool aov = false;
    for (const auto& v : views) {
        aov = aov || v.alb || v.nrm;
        z.samples += (double)v.cfg.width * v.cfg.height * v.cfg.spp;
        max_dl = std::max<int64_t>(max_dl, v.cfg.direct_loop);
        max_lights = std::max<int64_t>(max_lights, v.num_lights);
    }
    z.pool = std::max<int64_t>(1024, std::min<int64_t>(tune_pool, (int64_t)z.samples));
    z.aov_pool = aov ? z.pool : 0;
    z.cap_mis = z.pool * max_dl;
    z.cap_sh = z.pool * max_dl * max_lights;
    const double per_item = z.samples / (4.0 * (double)z.pool);
    for (auto& v : views) {
        const int chunk = (int)std::floor(per_item);
        v.chunk = std::max(1, std::min(chunk, v.cfg.spp));
        v.nchunks = (v.cfg.spp + v.chunk - 1) / v.chunk;
        v.item_base = z.items;
        const int64_t items = (int64_t)v.cfg.width * v.cfg.height * v.nchunks;
        z.items += items;
        v.partial_f4 = aov ? 3 : 1;
        z.partial_f4 += v.partial_f4 * items;
    }
    return z;
}

// Device bytes of the forward workspace for such a render, both sets of ray records included.
size_t forward_bytes(const WfSizes& z)
{
    size_t total = sizeof(float4) * (size_t)z.partial_f4;
    auto add = [&](auto*& p, size_t count) { total += sizeof(*p) * count; };
    WfState b;
    each_state_buffer(b, false, z.pool, z.cap_mis, z.cap_sh, add);
    each_ray_buffer(b.rq, z.cap_mis, z.cap_sh, add);
    return total + 2 * sizeof(float4) * (size_t)z.aov_pool;
}

bool wf_state_holds(const WfCache& c, const WfSizes& z)
{
    return z.pool <= c.pool && z.cap_mis <= c.cap_mis && z.cap_sh <= c.cap_sh;
}

// Releases a workspace, complete or not.
void wf_cache_destroy(WfCache*& c, cudaStream_t s)
{
    wf_cache_drop_graph(*c);
    wf_cache_free_state(*c, s);
    wf_cache_free_aov(*c, s);
    wf_free(*c, s, c->partial, sizeof(float4) * (size_t)c->partial_f4);
    wf_free(*c, s, c->d_views, sizeof(WfView) * (size_t)c->nviews);
    wf_free(*c, s, c->cnt, sizeof(Counters));
    cudaStreamSynchronize(s);
    if (c->h_views) cudaFreeHost(c->h_views);
    if (c->h_block) cudaFreeHost(c->h_block);
    for (cudaStream_t x : c->side)
        if (x) cudaStreamDestroy(x);
    for (cudaEvent_t ev : {c->fork, c->fork2, c->join[0], c->join[1], c->e0, c->e1})
        if (ev) cudaEventDestroy(ev);
    for (cudaEvent_t ev : c->pev) cudaEventDestroy(ev);
    delete c;
    c = nullptr;
}

// Makes the workspace of `ctx` (forward or adjoint) hold at least what a render needs.
fm_status wf_cache_reserve(fm_ctx* ctx, bool adj, const WfSizes& need, int32_t nviews, WfCache*& out)
{
    cudaStream_t s = ctx->stream;
    WfCache*& c = ctx->wf_cache[adj ? 1 : 0];
    if (!c) {
        c = new WfCache();
        c->adj = adj;
        const size_t hb = sizeof(unsigned) * kQcCount + sizeof(uint32_t) * 4 + sizeof(unsigned long long) * 4;
        const unsigned nt = cudaEventDisableTiming;
        if (cudaStreamCreateWithFlags(&c->side[0], cudaStreamNonBlocking) != cudaSuccess ||
            cudaStreamCreateWithFlags(&c->side[1], cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&c->fork, nt) != cudaSuccess || cudaEventCreateWithFlags(&c->fork2, nt) != cudaSuccess ||
            cudaEventCreateWithFlags(&c->join[0], nt) != cudaSuccess ||
            cudaEventCreateWithFlags(&c->join[1], nt) != cudaSuccess || cudaEventCreate(&c->e0) != cudaSuccess || cudaEventCreate(&c->e1) != cudaSuccess ||
            cudaMallocHost(&c->h_block, hb) != cudaSuccess || wf_malloc(ctx, *c, (void**)&c->cnt, sizeof(Counters)) != cudaSuccess) {
            cudaGetLastError();
            wf_cache_destroy(c, s);
            return set_error(ctx, FM_ERR_OOM, "wavefront: workspace allocation failed");
        }
        char* hp = static_cast<char*>(c->h_block);
        c->h_span = reinterpret_cast<unsigned long long*>(hp);
        c->h_qc = reinterpret_cast<unsigned*>(hp + sizeof(unsigned long long) * 4);
        c->h_status = reinterpret_cast<uint32_t*>(hp + sizeof(unsigned long long) * 4 + sizeof(unsigned) * kQcCount);
    }
    if (nviews > c->nviews) {
        wf_cache_drop_graph(*c);
        wf_free(*c, s, c->d_views, sizeof(WfView) * (size_t)c->nviews);
        if (c->h_views) {
            cudaStreamSynchronize(s);
            cudaFreeHost(c->h_views);
        }
        c->d_views = nullptr;
        c->h_views = nullptr;
        c->nviews = 0;
        WfView* d = nullptr;
        if (wf_malloc(ctx, *c, (void**)&d, sizeof(WfView) * (size_t)nviews) != cudaSuccess ||
            cudaMallocHost((void**)&c->h_views, sizeof(WfView) * (size_t)nviews) != cudaSuccess) {
            cudaGetLastError();
            wf_free(*c, s, d, sizeof(WfView) * (size_t)nviews);
            return set_error(ctx, FM_ERR_OOM, "wavefront: view table allocation failed");
        }
        c->d_views = d;
        c->nviews = nviews;
    }
    if (need.partial_f4 > c->partial_f4) {
        wf_free(*c, s, c->partial, sizeof(float4) * (size_t)c->partial_f4);
        c->partial = nullptr;
        c->partial_f4 = 0;
        if (wf_malloc(ctx, *c, (void**)&c->partial, sizeof(float4) * (size_t)need.partial_f4) != cudaSuccess) {
            cudaGetLastError();
            return set_error(ctx, FM_ERR_OOM, "wavefront: partial buffer allocation failed");
        }
        c->partial_f4 = need.partial_f4;
    }
    if (need.aov_pool > c->aov_pool) {
        wf_cache_drop_graph(*c);
        wf_cache_free_aov(*c, s);
        const size_t bytes = sizeof(float4) * (size_t)need.aov_pool;
        float4 *as = nullptr, *ns = nullptr;
        if (wf_malloc(ctx, *c, (void**)&as, bytes) != cudaSuccess || wf_malloc(ctx, *c, (void**)&ns, bytes) != cudaSuccess) {
            cudaGetLastError();
            wf_free(*c, s, as, bytes);
            return set_error(ctx, FM_ERR_OOM, "wavefront: albedo and normal sums' allocation failed");
        }
        c->asum = as;
        c->nsum = ns;
        c->aov_pool = need.aov_pool;
    }
    if (!wf_state_holds(*c, need)) {
        wf_cache_drop_graph(*c);
        const int64_t pool = std::max(need.pool, c->pool), cap_mis = std::max(need.cap_mis, c->cap_mis);
        const int64_t cap_sh = std::max(need.cap_sh, c->cap_sh);
        wf_cache_free_state(*c, s);
        bool ok = true;
        auto A = [&](auto*& p, size_t count) {
            void* q = nullptr;
            const size_t bytes = sizeof(*p) * count;
            if (ok && wf_malloc(ctx, *c, &q, bytes) == cudaSuccess) {
                c->allocs.emplace_back(q, bytes);
                p = static_cast<std::remove_reference_t<decltype(p)>>(q);
            } else {
                ok = false;
            }
        };
        each_state_buffer(c->bufs, adj, pool, cap_mis, cap_sh, A);
        if (!ok) {
            cudaGetLastError();
            wf_cache_free_state(*c, s);
            return set_error(ctx, FM_ERR_OOM, "wavefront: state allocation failed");
        }
        if (!adj) {
            // the second set of ray records; without room for it renders run with one
            const size_t kept = c->allocs.size();
            each_ray_buffer(c->alt, cap_mis, cap_sh, A);
            if (!ok) {
                cudaGetLastError();
                wf_cache_free_allocs(*c, s, kept);
                std::memset(&c->alt, 0, sizeof(c->alt));
            }
        }
        c->pool = pool;
        c->cap_mis = cap_mis;
        c->cap_sh = cap_sh;
        ++c->builds;
    }
    out = c;
    return FM_OK;
}

template <bool ADJ>
fm_status run_wavefront(fm_ctx* ctx, const std::vector<WfView>& views_in, const WfTuning& tune, const WfAdjoint* adj,
                        Counters* cnt, WfTimes* times)
{
    cudaStream_t s = ctx->stream;
    std::vector<WfView> views = views_in;
    const WfSizes z = size_views(views, tune.pool);
    const int64_t pool = z.pool;
    WfCache* c = nullptr;
    fm_status result = wf_cache_reserve(ctx, ADJ, z, (int32_t)views.size(), c);
    if (result != FM_OK) return result;
    {
        float4* p = c->partial;
        for (auto& v : views) {
            v.partial = p;
            p += v.partial_f4 * (int64_t)v.cfg.width * v.cfg.height * v.nchunks;
        }
    }
    // the launch state: the workspace's buffers, this call's sizes
    WfState st;
    std::memcpy(&st, &c->bufs, sizeof(st));
    st.pool = pool;
    st.nviews = (int32_t)views.size();
    st.aov = z.aov_pool > 0 ? 1 : 0;
    st.asum = st.aov ? c->asum : nullptr;
    st.nsum = st.aov ? c->nsum : nullptr;
    st.total_items = z.items;
    st.cap_cont = pool;
    st.cap_mis = z.cap_mis;
    st.cap_sh = z.cap_sh;
    if (tune.queue_limit > 0) {
        // below the allocated capacities: appends beyond them are counted and dropped
        st.cap_cont = std::min<int64_t>(st.cap_cont, tune.queue_limit);
        st.cap_mis = std::min<int64_t>(st.cap_mis, tune.queue_limit);
        st.cap_sh = std::min<int64_t>(st.cap_sh, tune.queue_limit);
    }
    st.views = c->d_views;
    st.wq = st.rq;
    st.qr = st.qc;
    st.qw = st.qc + kQcSet;
    st.trace_tail = (int64_t)ctx->num_sms * 64 * 32;   // a warp of rays for each of 64 resident warps per SM
    st.cnt = c->cnt;
    st.status = ctx->d_status;
    if (ADJ) {
        st.cap_grad = 2 * pool;   // a slot can finish two vertices in one iteration
        st.tex_acc = adj->tex_acc;
        st.tex_copies = adj->tex_copies;
        st.mat_acc = adj->mat_acc;
        st.env_row = adj->env_row;
        st.env_total = adj->env_total;
    }
    // the previous call ended with a stream synchronisation, so the pinned staging is free
    std::memcpy(c->h_views, views.data(), sizeof(WfView) * views.size());
    FM_CUDA_TRY(ctx, cudaMemcpyAsync(c->d_views, c->h_views, sizeof(WfView) * views.size(), cudaMemcpyHostToDevice, s),
                "wavefront views");
    FM_CUDA_TRY(ctx, cudaMemsetAsync(st.next_item, 0, sizeof(unsigned long long), s), "wavefront");
    FM_CUDA_TRY(ctx, cudaMemsetAsync(st.qc, 0, sizeof(unsigned) * kQcCount, s), "wavefront");
    FM_CUDA_TRY(ctx, cudaMemsetAsync(st.tspan, 0, sizeof(unsigned long long) * 4, s), "wavefront");
    FM_CUDA_TRY(ctx, cudaMemsetAsync(c->cnt, 0, sizeof(Counters), s), "wavefront");
    const int sms = ctx->num_sms;
    k_wf_init<<<sms * 8, 256, 0, s>>>(st);
    cudaEventRecord(c->e0, s);
    // One graph body = `iters_per_graph` iterations (an even number, as the counter sets and
    // ray records change places with every iteration) of
    //   trace -> resolve (continuation rays) -> shade (Disney) | shade (other materials)
    //         |  resolve (MIS and shadow rays)                                   -> logic
    // The branches run side by side: hit resolution waits on dependent loads while shading
    // issues, and in small renders each kernel is one latency.  Against one kernel after
    // another, with a launch between iterations that swapped the counters: 64^2 preview
    // 0.70 -> 0.58 ms, Cornell box 256^2 x 16 samples 1.69 -> 1.32, 1.3 M triangles at 1080p
    // 6.46 -> 6.03, 16-scene batch 61.2 -> 59.8, adjoint of 4 views 11.85 -> 11.34.  Shading queues its rays into
    // the second set of records meanwhile.  Adjoint renders resolve all rays first, since
    // replayed vertices read what their MIS and shadow rays collected, then shade all four
    // queues side by side, and scatter gradients after the logic kernel.
    const int body_iters = tune.iters_per_graph + (tune.iters_per_graph & 1);
    const bool overlap = !ADJ && c->alt.mis_o != nullptr;
    // what is resident at 64 registers per thread; more blocks would only find no rays left
    const int trace_grid = sms * (1024 / tune.trace_block);
    const size_t trace_smem = kTraceSmemPerThread * (size_t)tune.trace_block;
    const int shade_grid = (int)std::min<int64_t>((pool + tune.shade_block - 1) / tune.shade_block, (int64_t)sms * 32);
    // slots per thread of the logic kernel: four where that still leaves several blocks per SM
    const bool logic4 = pool >= (int64_t)sms * 4096;
    const int logic_grid = (int)std::min<int64_t>((pool + 255) / (logic4 ? 1024 : 256), (int64_t)sms * 32);
    const int resolve_grid = sms * 16;
    // Bound on iterations: every sample takes at most depth + 1 iterations and a slot
    // runs its samples one after another.
    int max_depth = 1, max_chunk = 1;
    for (const auto& v : views) {
        max_depth = std::max(max_depth, v.cfg.depth);
        max_chunk = std::max(max_chunk, v.chunk);
    }
    const double iter_bound =
        (z.samples / (double)pool + 4.0 * max_chunk + 8.0) * (max_depth + 2) * 4.0 * (ADJ ? 2.0 : 1.0) + 1000.0;
    // (the host's loop of timed renders sees the end of a body one launch later)
    int64_t max_bodies = (int64_t)(iter_bound / body_iters) + 16 + (tune.profile ? 1 : 0);
    // A caller's limit counts whole runs of iters_per_graph iterations, so with an odd number
    // it can fall inside a body: limit_at is the iteration of the last body that it follows.
    int64_t limit = 0;
    int limit_at = 0;
    if (tune.max_iterations > 0) {
        const int64_t runs = ((int64_t)tune.max_iterations + tune.iters_per_graph - 1) / tune.iters_per_graph;
        limit = (runs + (tune.profile ? 1 : 0)) * tune.iters_per_graph;
        const int64_t bodies = (limit + body_iters - 1) / body_iters;
        if (bodies <= max_bodies) {
            max_bodies = bodies;
            limit_at = (int)(limit % body_iters);
        }
    }
    // optional per-kernel timing: event-record nodes around every trace and shade launch
    std::vector<cudaEvent_t>& pev = c->pev;
    if (tune.profile) {
        while (pev.size() < 3 * (size_t)body_iters) {
            cudaEvent_t ev = nullptr;
            cudaEventCreate(&ev);
            pev.push_back(ev);
        }
    }
    double trace_ms = 0.0, shade_ms = 0.0;
    auto capture_iterations = [&]() {
        // work on `to` follows what `from` holds
        auto after = [](cudaEvent_t ev, cudaStream_t from, cudaStream_t to) {
            cudaEventRecord(ev, from);
            cudaStreamWaitEvent(to, ev, 0);
        };
        cudaStream_t s1 = c->side[0], s2 = c->side[1];
        for (int it = 0; it < body_iters; ++it) {
            WfState x = st;
            if (it & 1) std::swap(x.qr, x.qw);
            if (overlap) {
                x.rq = it & 1 ? c->alt : st.rq;
                x.wq = it & 1 ? st.rq : c->alt;
            }
            if (tune.profile) cudaEventRecordWithFlags(pev[3 * it], s, cudaEventRecordExternal);
            k_wf_trace<<<trace_grid, tune.trace_block, trace_smem, s>>>(x);
            if (tune.profile) cudaEventRecordWithFlags(pev[3 * it + 1], s, cudaEventRecordExternal);
            after(c->fork, s, s1);
            k_wf_resolve_rays<ADJ><<<resolve_grid, 256, 0, s1>>>(x);
            k_wf_resolve_cont<ADJ><<<resolve_grid, 256, 0, s>>>(x);
            if (!overlap) after(c->join[0], s1, s);
            after(c->fork2, s, s2);
            k_wf_shade<kClsDisney><<<shade_grid, tune.shade_block, 0, s>>>(x);
            k_wf_shade<kClsSimple><<<shade_grid, tune.shade_block, 0, s2>>>(x);
            if (ADJ) {
                k_wf_shade_replay<kClsDisney><<<shade_grid, tune.shade_block, 0, s>>>(x);
                k_wf_shade_replay<kClsSimple><<<shade_grid, tune.shade_block, 0, s2>>>(x);
            }
            after(c->join[1], s2, s);
            after(c->join[0], s1, s);
            if (logic4)
                k_wf_logic<ADJ, 4><<<logic_grid, 256, 0, s>>>(x);
            else
                k_wf_logic<ADJ, 1><<<logic_grid, 256, 0, s>>>(x);
            if (ADJ) k_wf_grad_scatter<<<sms * 8, 256, 0, s>>>(x);
            if (tune.profile) cudaEventRecordWithFlags(pev[3 * it + 2], s, cudaEventRecordExternal);
            if (it + 1 == limit_at) k_wf_limit<<<1, 1, 0, s>>>(x, (unsigned)std::min<int64_t>(max_bodies, 0x7fffffff));
        }
    };
    cudaError_t e = cudaSuccess;
    // The instantiated graph is kept in the workspace and launched again while the
    // launch state (buffers, sizes, tuning, iteration bound) is the same; a batch of the
    // same shape class re-uploads only its views.
    const bool reuse = c->exec && std::memcmp(&c->g_st, &st, sizeof(st)) == 0 && c->g_pool == tune.pool &&
                       c->g_trace_block == tune.trace_block && c->g_shade_block == tune.shade_block &&
                       c->g_iters == body_iters && c->g_profile == tune.profile &&
                       c->g_max_bodies == max_bodies && c->g_limit == limit;
    if (!reuse) {
        wf_cache_drop_graph(*c);
        cudaGraph_t graph = nullptr;
        if (!tune.profile) {
            // The whole render is one launch: a conditional WHILE node repeats the body
            // (iters_per_graph iterations and k_wf_continue) on the device until no slot
            // holds work, so the host never waits between iterations.
            e = cudaGraphCreate(&graph, 0);
            cudaGraphConditionalHandle handle{};
            if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&handle, graph, 1u, cudaGraphCondAssignDefault);
            cudaGraphNodeParams cp{};
            cp.type = cudaGraphNodeTypeConditional;
            cp.conditional.handle = handle;
            cp.conditional.type = cudaGraphCondTypeWhile;
            cp.conditional.size = 1;
            cudaGraphNode_t cnode = nullptr;
            if (e == cudaSuccess) e = cudaGraphAddNode(&cnode, graph, nullptr, 0, &cp);
            cudaGraph_t body = e == cudaSuccess ? cp.conditional.phGraph_out[0] : nullptr;
            if (e == cudaSuccess)
                e = cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
            if (e == cudaSuccess) {
                capture_iterations();
                k_wf_continue<<<1, 1, 0, s>>>(st, handle, (unsigned)std::min<int64_t>(max_bodies, 0x7fffffff));
                e = cudaStreamEndCapture(s, &body);
            }
        } else {
            e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
            if (e == cudaSuccess) {
                capture_iterations();
                e = cudaStreamEndCapture(s, &graph);
            }
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&c->exec, graph, 0);
        c->graph = graph;
        if (e != cudaSuccess) {
            wf_cache_drop_graph(*c);
            cudaStreamSynchronize(s);
            return cuda_error(ctx, e, "wavefront graph");
        }
        std::memcpy(&c->g_st, &st, sizeof(st));
        c->g_pool = tune.pool;
        c->g_trace_block = tune.trace_block;
        c->g_shade_block = tune.shade_block;
        c->g_iters = body_iters;
        c->g_profile = tune.profile;
        c->g_max_bodies = max_bodies;
        c->g_limit = limit;
    }
    unsigned* h_qc = c->h_qc;
    int64_t graph_launches = 0;
    if (!tune.profile) {
        uint32_t* hs = c->h_status;
        unsigned long long* span = c->h_span;
        e = cudaGraphLaunch(c->exec, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(h_qc, st.qc, sizeof(unsigned) * kQcCount, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(hs, st.status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(span, st.tspan, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess) {
            graph_launches = h_qc[kQcBodies];
            // the resolve launch after each trace launch adds that launch's span
            trace_ms = 1e-6 * (double)span[2];
            if (*hs & 4u) result = set_error(ctx, FM_ERR_TIMEOUT, "wavefront: iteration limit reached");
        }
    } else {
        int64_t guard = 0;
        for (;;) {
            e = cudaGraphLaunch(c->exec, s);
            if (e != cudaSuccess) break;
            ++graph_launches;
            e = cudaMemcpyAsync(h_qc, st.qc, sizeof(unsigned) * kQcCount, cudaMemcpyDeviceToHost, s);
            if (e != cudaSuccess) break;
            e = cudaMemcpyAsync(c->h_status, st.status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
            if (e != cudaSuccess) break;
            e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) break;
            for (int it = 0; it < body_iters; ++it) {
                float a = 0.0f, b = 0.0f;
                cudaEventElapsedTime(&a, pev[3 * it], pev[3 * it + 1]);
                cudaEventElapsedTime(&b, pev[3 * it + 1], pev[3 * it + 2]);
                trace_ms += a;
                shade_ms += b;
            }
            // done when no slot holds work after the last shade
            const bool limited = (*c->h_status & 4u) != 0u;
            if (h_qc[kQcActive] == 0u && !limited) break;
            if (limited || ++guard >= max_bodies) {
                result = set_error(ctx, FM_ERR_TIMEOUT, "wavefront: iteration limit reached");
                break;
            }
        }
    }
    if (e != cudaSuccess) result = cuda_error(ctx, e, "wavefront loop");
    if (result == FM_OK) {
        for (const auto& v : views) {
            const int npix = v.cfg.width * v.cfg.height;
            k_wf_reduce<<<std::min((npix + 255) / 256, sms * 16), 256, 0, s>>>(v);
        }
        k_counters_add<<<1, 1, 0, s>>>(cnt, c->cnt);
        e = cudaGetLastError();
        if (e != cudaSuccess) result = cuda_error(ctx, e, "wavefront reduce");
    }
    cudaEventRecord(c->e1, s);
    cudaStreamSynchronize(s);
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, c->e0, c->e1);
    if (times) {
        times->launches = 2 + graph_launches * ((ADJ ? 9 : 6) * body_iters + (tune.profile ? 0 : 1) + (limit_at > 0 ? 1 : 0)) +
                          (int64_t)views.size();
        times->total_ms = ms;
        times->trace_ms = trace_ms;
        // without event timing, everything but the trace kernel counts as shading
        times->shade_ms = tune.profile ? shade_ms : std::max(0.0, (double)ms - trace_ms);
    }
    // a failed render leaves the graph in an unknown state: build it again next time
    if (result != FM_OK) wf_cache_drop_graph(*c);
    return result;
}

}  // namespace

fm_status reduce_views(fm_ctx* ctx, const std::vector<WfView>& views)
{
    for (const auto& v : views) {
        const int npix = v.cfg.width * v.cfg.height;
        k_wf_reduce<<<std::min((npix + 255) / 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(v);
    }
    FM_CUDA_TRY(ctx, cudaGetLastError(), "reduce views");
    return FM_OK;
}

fm_status wavefront_views(fm_ctx* ctx, const std::vector<WfView>& views, const WfTuning& tune, Counters* cnt,
                          WfTimes* times)
{
    return run_wavefront<false>(ctx, views, tune, nullptr, cnt, times);
}

fm_status wavefront_adjoint(fm_ctx* ctx, const std::vector<WfView>& views, const WfTuning& tune, const WfAdjoint& adj,
                            Counters* cnt, WfTimes* times)
{
    return run_wavefront<true>(ctx, views, tune, &adj, cnt, times);
}

void wf_cache_release(fm_ctx* ctx)
{
    for (WfCache*& c : ctx->wf_cache)
        if (c) wf_cache_destroy(c, ctx->stream);
}

size_t wavefront_bytes(std::vector<WfView> views, int64_t pool) { return forward_bytes(size_views(views, pool)); }

namespace {

// The most device memory that fm_render's workspace takes for more than the default slots.
constexpr size_t kWideBytes = size_t(8000) * 1000 * 1000;

// Whether a render of more than the default slots has its workspace already or may let it
// grow: within kWideBytes, and within half of the memory that is free or that the workspace
// and the device's memory pool hold and would use again.  Asked before the present workspace
// is given up, so a pool that does not fit costs nothing, not even the kept graph.  A size
// that was refused all the same (another process took the memory) is not tried again.
bool wide_pool_fits(fm_ctx* ctx, const WfSizes& z)
{
    if (ctx->wf_refused > 0 && z.pool >= ctx->wf_refused) return false;
    const WfCache* c = ctx->wf_cache[0];
    WfSizes need = z;
    size_t held = 0;
    if (c) {
        if (wf_state_holds(*c, z) && z.partial_f4 <= c->partial_f4 && z.aov_pool <= c->aov_pool) return true;
        need.pool = std::max(z.pool, c->pool);
        need.cap_mis = std::max(z.cap_mis, c->cap_mis);
        need.cap_sh = std::max(z.cap_sh, c->cap_sh);
        need.partial_f4 = std::max(z.partial_f4, c->partial_f4);
        need.aov_pool = std::max(z.aov_pool, c->aov_pool);
        held = c->held;
    }
    const size_t bytes = forward_bytes(need);
    if (bytes > kWideBytes) return false;
    size_t free_b = 0, total_b = 0;
    uint64_t reserved = 0, used = 0;
    cudaMemPool_t mem;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || cudaDeviceGetDefaultMemPool(&mem, ctx->device) != cudaSuccess ||
        cudaMemPoolGetAttribute(mem, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(mem, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return bytes <= (free_b + (size_t)(reserved - std::min(reserved, used)) + held) / 2;
}

}  // namespace

fm_status launch_wavefront(fm_ctx* ctx, const fm_scene* scene, const DevCamera& cam, const RenderCfg& cfg, float* rgb,
                           float* alb, float* nrm, Counters* cnt)
{
    WfView v{};
    v.scene = scene->d_dev;
    v.num_lights = scene->dev.num_lights;
    v.cam = cam;
    v.cfg = cfg;
    v.rgb = rgb;
    v.alb = alb;
    v.nrm = nrm;
    // Path slots: the default 2^21, or more up to 2^23 where there are 1.5 samples or more per
    // slot -- more slots mean fewer iterations, so fewer launches and kernel tails
    // (1920x1080 through 1.3 M triangles with 2^21 / 2^22 / 2^23 / 2^24 slots: 5.76 / 5.49 /
    // 5.49 / 5.51 ms at 4 samples per pixel, 18.8 / 17.3 / 16.8 / 17.3 ms at 16) -- as long as
    // the device has room for their workspace.
    WfTuning t;
    const double samples = (double)cfg.width * cfg.height * cfg.spp;
    for (int64_t pool = (int64_t)1 << 23; pool > t.pool; pool /= 2) {
        if (samples < 1.5 * (double)pool) continue;
        std::vector<WfView> views{v};
        if (!wide_pool_fits(ctx, size_views(views, pool))) continue;
        WfTuning wide;
        wide.pool = pool;
        const std::string before = ctx->error;
        const fm_status st = wavefront_views(ctx, {v}, wide, cnt, nullptr);
        if (st != FM_ERR_OOM) return st;
        ctx->error = before;
        ctx->wf_refused = pool;
    }
    return wavefront_views(ctx, {v}, t, cnt, nullptr);
}

}  // namespace fm

// Used by tests: bounds the device memory of each of the context's workspaces and of the
// denoiser's records (0: by the device only), and reports the forward one's device bytes, how often its state was
// allocated and whether it has the second set of ray records.
extern "C" void fm_internal_limit_workspace(fm_ctx* ctx, int64_t bytes)
{
    if (!ctx) return;
    ctx->wf_limit = bytes > 0 ? (size_t)bytes : 0;
    ctx->wf_refused = 0;
}
extern "C" void fm_internal_workspace(const fm_ctx* ctx, int64_t* out)
{
    const fm::WfCache* c = ctx ? ctx->wf_cache[0] : nullptr;
    out[0] = c ? (int64_t)c->held : 0;
    out[1] = c ? c->builds : 0;
    out[2] = c && c->alt.mis_o ? 1 : 0;
}
