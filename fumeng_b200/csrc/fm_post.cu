// Post-processing of a finished frame on the device: the reference's PostProcess chain
// (core/renderer.h:131-135) and the 8-bit conversion its RenderTarget::save_to_file does
// before the PNG write (render_target.h:26-31, image/image.cpp:98-109).
//
// Per-pixel steps (tone mapping, linear <-> sRGB) run as one kernel per run of
// consecutive per-pixel steps; the denoise step is an image-level filter between them.
// The arithmetic of the per-pixel steps is the reference's float build's: every
// operation explicitly rounded in the reference's order (no multiply-add is contracted),
// pow from the device's powf.  So the 8-bit outputs equal the reference's bytes for the
// same float input, up to the last bit of powf on the sRGB steps (a value whose
// 255 x lands within one float ulp of a rounding boundary can then differ by one code).
//
// Denoise: the reference calls Intel Open Image Denoise's "RT" filter with the albedo and
// normal images as guides (post/oidn_denoise.cpp:36-78).  That filter is a trained
// network that is not available here; this file runs a different, non-learned filter on
// the same inputs instead: the edge-avoiding a-trous wavelet filter (Dammertz, Sewtz,
// Hanika and Lensch, "Edge-Avoiding A-Trous Wavelet Transform for fast Global
// Illumination Filtering", HPG 2010), five passes of a 5x5 B3-spline kernel with taps
// 1, 2, 4, 8, 16 pixels apart, each tap weighted by its colour, normal and albedo
// distance to the centre.  Its output is not the reference's.
#include <algorithm>
#include <cmath>
#include <vector>

#include "fm_common.cuh"
#include "fm_internal.h"
#include "fm_staging.h"

namespace fm {

namespace {

constexpr int kMaxPostSteps = 16;

struct PostChain {
    int n;
    int type[kMaxPostSteps];
    float lum[kMaxPostSteps];
};

// ToneMapping::FilmicCore (post/tonemapping.cpp:10-19), float, in the source's order.
FM_D float filmic_core(float x)
{
    const float A = 0.22f, B = 0.30f, C = 0.10f, D = 0.20f, E = 0.01f, F = 0.30f;
    const float num = __fadd_rn(__fmul_rn(x, __fadd_rn(__fmul_rn(A, x), __fmul_rn(C, B))), __fmul_rn(D, E));
    const float den = __fadd_rn(__fmul_rn(x, __fadd_rn(__fmul_rn(A, x), B)), __fmul_rn(D, F));
    return __fsub_rn(__fdiv_rn(num, den), __fdiv_rn(E, F));
}

// ToneMapping::Filmic (:21-25): FilmicCore(1.6 * value * lum) / FilmicCore(11.2).
FM_D float filmic(float v, float lum, float white)
{
    return __fdiv_rn(filmic_core(__fmul_rn(__fmul_rn(1.6f, v), lum)), white);
}

// LinearToSrgb / SrgbToLinear (core/utils.h:120-132), float.
FM_D float linear_to_srgb(float c)
{
    if (c <= 0.0031308f) return __fmul_rn(12.92f, c);
    return __fsub_rn(__fmul_rn(1.055f, powf(c, __fdiv_rn(1.0f, 2.4f))), 0.055f);
}

FM_D float srgb_to_linear(float c)
{
    if (c <= 0.04045f) return __fdiv_rn(__fmul_rn(c, 1.0f), 12.92f);
    return powf(__fdiv_rn(__fmul_rn(__fadd_rn(c, 0.055f), 1.0f), 1.055f), 2.4f);
}

__global__ void k_post_pointwise(float* __restrict__ rgb, int64_t n, PostChain chain, int first, int last)
{
    const float white = filmic_core(11.2f);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float v = rgb[i];
        for (int s = first; s < last; ++s) {
            if (chain.type[s] == FM_POST_TONEMAP)
                v = filmic(v, chain.lum[s], white);
            else if (chain.type[s] == FM_POST_LINEAR_TO_SRGB)
                v = linear_to_srgb(v);
            else if (chain.type[s] == FM_POST_SRGB_TO_LINEAR)
                v = srgb_to_linear(v);
        }
        rgb[i] = v;
    }
}

// RealToUInt8 (core/utils.h:134-137): Clamp(c, 0, 1) (utils.h:68-71), then
// round(255 c).  A NaN channel (left unchanged by the reference's Clamp, and undefined
// in its integer conversion) becomes 0.
__global__ void k_to_u8(const float* __restrict__ src, uint8_t* __restrict__ dst, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float c = src[i];
        c = c > 1.0f ? 1.0f : (c < 0.0f ? 0.0f : c);
        dst[i] = c == c ? (uint8_t)roundf(__fmul_rn(255.0f, c)) : (uint8_t)0;
    }
}

// What a tap of the a-trous filter reads, per pixel: the compressed colour t(c) = c / (1 + c)
// per channel with the colour's red, its green and blue, the unit normal and the albedo.
// 56 B in four loads.  Computed in every tap from the images as they are, the same values
// cost six divisions, a square root and nine 4-byte loads 12 bytes apart per tap.
struct DenoiseIn {
    const float4* t;   // t(c).xyz | c.x
    const float2* c;   // c.y, c.z
    const float4* n;   // unit normal (zero stays zero)
    const float4* a;   // albedo
};

// |v|^2 and a . b with their multiply-adds written out, so that the 8-bit images do not
// depend on how the compiler contracts the sums.
FM_D float square(f3 v) { return fmaf(v.z, v.z, fmaf(v.x, v.x, __fmul_rn(v.y, v.y))); }
FM_D float dot_fma(f3 a, f3 b) { return fmaf(a.z, b.z, fmaf(a.y, b.y, __fmul_rn(a.x, b.x))); }

FM_D f3 compress(f3 c)
{
    return f3{c.x / (1.0f + fmaxf(c.x, 0.0f)), c.y / (1.0f + fmaxf(c.y, 0.0f)), c.z / (1.0f + fmaxf(c.z, 0.0f))};
}

// A colour's records.  A colour that is not finite is never averaged into another pixel: its
// t.x is NaN, which makes every weight computed from it fail the test of a tap.
FM_D void put_colour(float4* t, float2* c, int64_t p, f3 v)
{
    const f3 u = compress(v);
    t[p] = make_float4(isfinite(v.x + v.y + v.z) ? u.x : __int_as_float(0x7fffffff), u.y, u.z, v.x);
    c[p] = make_float2(v.y, v.z);
}

// A rectangle of the image.
struct Rect {
    int x0, y0, w, h;
};

// The records of rectangle r's pixels, row by row (the whole image unless TILED).
template <bool TILED>
__global__ void k_denoise_pack(const float* __restrict__ rgb, const float* __restrict__ alb, const float* __restrict__ nrm,
                               int width, Rect r, float4* t, float2* c, float4* n, float4* a)
{
    const int64_t npix = (int64_t)r.w * r.h;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npix; p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t q = TILED ? (r.y0 + p / r.w) * (int64_t)width + r.x0 + p % r.w : p;
        put_colour(t, c, p, f3{rgb[3 * q], rgb[3 * q + 1], rgb[3 * q + 2]});
        f3 np = f3{nrm[3 * q], nrm[3 * q + 1], nrm[3 * q + 2]};
        const float nl = sqrtf(square(np));
        np = nl > 0.0f ? np / nl : np;
        n[p] = make_float4(np.x, np.y, np.z, 0.0f);
        a[p] = make_float4(alb[3 * q], alb[3 * q + 1], alb[3 * q + 2], 0.0f);
    }
}

// One pass of the edge-avoiding a-trous filter at tap distance `step` (pixels).
// Weights: B3-spline h(dx) h(dy) with h = (1, 4, 6, 4, 1) / 16, times
//   exp(-|t(c_q) - t(c_p)|^2 / sc^2)          colour; inv_sc2 = 1 / sc^2, a power of two
//   exp(-max(0, 1 - n_p . n_q) / sn^2)         normal (unit-normalised AOV means)
//   exp(-|a_q - a_p|^2 / sa^2)                 albedo
// with the colour scale halved at every pass (the finer detail has been removed).  The
// records are those of w x h pixels, which are all filtered, the results going to the next
// pass's records or, in the last pass, to the plain image (rgb set).  TILED: the rectangle
// `out` of them is filtered, to an image with rows `width` pixels apart.  Blocks
// are 32 x 8 pixels, so that the taps of the first passes are in the L1 cache.
// Bound by issue slots (about 70 instructions per tap, two of them IEEE divisions that
// the results depend on); 1920x1080: 418 -> 188 us per pass.
template <bool TILED>
__global__ void __launch_bounds__(256) k_atrous(DenoiseIn in, int w, int h, Rect out, int step, float inv_sc2, float sn,
                                                float sa, float4* __restrict__ t_out, float2* __restrict__ c_out,
                                                float* __restrict__ rgb, int width)
{
    const float hk[5] = {1.0f / 16.0f, 4.0f / 16.0f, 6.0f / 16.0f, 4.0f / 16.0f, 1.0f / 16.0f};
    const int tiles_x = ((TILED ? out.w : w) + 31) / 32;
    int x = (int)(blockIdx.x % tiles_x) * 32 + (threadIdx.x & 31), y = (int)(blockIdx.x / tiles_x) * 8 + (threadIdx.x >> 5);
    if (TILED) {
        if (x >= out.w || y >= out.h) return;
        x += out.x0;
        y += out.y0;
    } else if (x >= w || y >= h) {
        return;
    }
    const int64_t p = (int64_t)y * w + x;
    const float4 t4 = __ldg(in.t + p), n4 = __ldg(in.n + p), a4 = __ldg(in.a + p);
    const float2 c2 = __ldg(in.c + p);
    const f3 cp = f3{t4.w, c2.x, c2.y}, np = f3{n4.x, n4.y, n4.z}, ap = f3{a4.x, a4.y, a4.z};
    const f3 tp = t4.x == t4.x ? f3{t4.x, t4.y, t4.z} : compress(cp);
    f3 sum = mk(0.0f);
    float wsum = 0.0f;
#pragma unroll 1
    for (int dy = -2; dy <= 2; ++dy) {
        const int yy = y + dy * step;
        if (yy < 0 || yy >= h) continue;
#pragma unroll
        for (int dx = -2; dx <= 2; ++dx) {
            const int xx = x + dx * step;
            if (xx < 0 || xx >= w) continue;
            const int64_t q = (int64_t)yy * w + xx;
            const float4 tq4 = __ldg(in.t + q), nq4 = __ldg(in.n + q), aq4 = __ldg(in.a + q);
            const float2 cq2 = __ldg(in.c + q);
            const f3 tq = f3{tq4.x, tq4.y, tq4.z}, nq = f3{nq4.x, nq4.y, nq4.z}, aq = f3{aq4.x, aq4.y, aq4.z};
            const f3 dc = tq - tp, da = aq - ap;
            const float wc = __expf(-square(dc) * inv_sc2);
            const float wn = __expf(-fmaxf(0.0f, __fsub_rn(1.0f, dot_fma(np, nq))) / (sn * sn));
            const float wa = __expf(-square(da) / (sa * sa));
            const float wt = hk[dx + 2] * hk[dy + 2] * wc * wn * wa;
            if (!(wt > 0.0f)) continue;
            sum += f3{tq4.w, cq2.x, cq2.y} * wt;
            wsum += wt;
        }
    }
    const f3 r = wsum > 0.0f ? sum / wsum : cp;
    if (TILED)
        st3(rgb + 3 * ((int64_t)y * width + x), r);
    else if (rgb)
        st3(rgb + 3 * p, r);
    else
        put_colour(t_out, c_out, p, r);
}

// The filter's colour scale at pass k.
inline float inv_sc2(int k)
{
    const float sc = 0.5f / (float)(1 << k);
    return 1.0f / (sc * sc);
}

// What the denoiser works in: two sets of colour records and the guides', 80 B per pixel of
// the whole image -- or, where the device has no room for them, of one tile and its
// surroundings at a time, with a second image that the passes alternate with.
struct DenoiseBufs {
    float4* t[2];
    float2* c[2];
    float4 *n, *a;
    float* pong;   // tiled
};
constexpr int kPasses = 5, kReach = 2 << (kPasses - 1);   // the widest pass's taps, in pixels
constexpr int kTileW = 512, kTileH = 128;

template <bool TILED>
void launch_pack(cudaStream_t s, int num_sms, const DenoiseBufs& b, const float* rgb, const float* alb, const float* nrm,
                 int width, Rect r)
{
    const int64_t npix = (int64_t)r.w * r.h;
    const int grid = (int)std::min<int64_t>((npix + 255) / 256, (int64_t)num_sms * 16);
    k_denoise_pack<TILED><<<grid, 256, 0, s>>>(rgb, alb, nrm, width, r, b.t[0], b.c[0], b.n, b.a);
}

// Pass k over `out`, within the records of r, from record set `from` to the other one or to
// the image.
template <bool TILED>
void launch_atrous(cudaStream_t s, const DenoiseBufs& b, int k, int from, Rect r, Rect out, float* rgb, int width)
{
    const int tiles = ((out.w + 31) / 32) * ((out.h + 7) / 8);
    if (TILED) rgb += 3 * ((int64_t)r.y0 * width + r.x0);
    const Rect inside{out.x0 - r.x0, out.y0 - r.y0, out.w, out.h};
    k_atrous<TILED><<<tiles, 256, 0, s>>>(DenoiseIn{b.t[from], b.c[from], b.n, b.a}, r.w, r.h, inside, 1 << k, inv_sc2(k),
                                          0.35f, 0.1f, b.t[from ^ 1], b.c[from ^ 1], rgb, width);
}

// Five passes between two sets of colour records; the last one writes the image.
cudaError_t denoise(cudaStream_t s, int num_sms, const DenoiseBufs& b, float* rgb, const float* alb, const float* nrm, int w,
                    int h)
{
    const Rect all{0, 0, w, h};
    launch_pack<false>(s, num_sms, b, rgb, alb, nrm, w, all);
    for (int k = 0; k < kPasses; ++k) launch_atrous<false>(s, b, k, k & 1, all, all, k == kPasses - 1 ? rgb : nullptr, w);
    return cudaGetLastError();
}

// The same tile by tile: each pass reads one image and writes the other, the records of a
// tile and the taps around it made again for every pass (1920x1080: 3.55 ms against 0.94).
cudaError_t denoise_tiled(cudaStream_t s, int num_sms, const DenoiseBufs& b, float* rgb, const float* alb, const float* nrm,
                          int w, int h)
{
    float *src = rgb, *dst = b.pong;
    for (int k = 0; k < kPasses; ++k) {
        const int reach = 2 << k;
        for (int y = 0; y < h; y += kTileH)
            for (int x = 0; x < w; x += kTileW) {
                const Rect out{x, y, std::min(kTileW, w - x), std::min(kTileH, h - y)};
                const int x0 = std::max(0, x - reach), y0 = std::max(0, y - reach);
                const Rect r{x0, y0, std::min(w, out.x0 + out.w + reach) - x0, std::min(h, out.y0 + out.h + reach) - y0};
                launch_pack<true>(s, num_sms, b, src, alb, nrm, w, r);
                launch_atrous<true>(s, b, k, 0, r, out, dst, w);
            }
        std::swap(src, dst);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || src == rgb) return e;
    return cudaMemcpyAsync(rgb, src, 3 * sizeof(float) * (size_t)w * h, cudaMemcpyDeviceToDevice, s);
}

}  // namespace

}  // namespace fm

using namespace fm;

extern "C" fm_status fm_postprocess(fm_ctx* ctx, int32_t width, int32_t height, const fm_post_step* steps,
                                    int32_t num_steps, float* rgb, const float* albedo, const float* normal,
                                    uint8_t* rgb8, uint8_t* albedo8, uint8_t* normal8, int32_t flags)
{
    if (!ctx) return FM_ERR_INVALID;
    if (width <= 0 || height <= 0 || (int64_t)width * height > ((int64_t)1 << 30) || num_steps < 0 ||
        num_steps > kMaxPostSteps || (num_steps > 0 && !steps) || !rgb)
        return set_error(ctx, FM_ERR_INVALID, "postprocess: bad arguments");
    PostChain chain{};
    chain.n = num_steps;
    bool denoise_step = false;
    for (int i = 0; i < num_steps; ++i) {
        const int t = steps[i].type;
        if (t != FM_POST_TONEMAP && t != FM_POST_LINEAR_TO_SRGB && t != FM_POST_SRGB_TO_LINEAR && t != FM_POST_DENOISE)
            return set_error(ctx, FM_ERR_INVALID, "postprocess: unknown step type");
        chain.type[i] = t;
        chain.lum[i] = steps[i].lum;
        denoise_step = denoise_step || t == FM_POST_DENOISE;
    }
    if (denoise_step && (!albedo || !normal))
        return set_error(ctx, FM_ERR_INVALID, "postprocess: the denoise step needs the albedo and normal images");
    FM_CUDA_TRY(ctx, cudaSetDevice(ctx->device), "cudaSetDevice");
    cudaStream_t s = ctx->stream;
    const bool dev = (flags & FM_FLAG_DEVICE_PTRS) != 0;
    const int64_t n = (int64_t)width * height * 3;
    const size_t fbytes = (size_t)n * sizeof(float);
    // device copies when the caller's buffers are host memory, the 8-bit outputs, and the
    // denoiser's records
    const size_t npix = (size_t)width * height;
    const size_t base = (dev ? 0 : 3 * fbytes) + (dev ? 0 : 3 * (size_t)n) + 4096;
    char* tmp = nullptr;
    size_t recs = denoise_step ? npix : 0;   // pixels with records
    bool tiled = false;
    cudaError_t e = ctx->wf_limit > 0 && 80 * recs > ctx->wf_limit ? cudaErrorMemoryAllocation
                                                                  : cudaMallocAsync((void**)&tmp, base + 80 * recs, s);
    if (e == cudaErrorMemoryAllocation && denoise_step) {
        cudaGetLastError();
        tiled = true;
        recs = (size_t)std::min(width, kTileW + 2 * kReach) * std::min(height, kTileH + 2 * kReach);
        e = cudaMallocAsync((void**)&tmp, base + 80 * recs + fbytes, s);
    }
    FM_CUDA_TRY(ctx, e, "postprocess alloc");
    char* q = tmp;
    auto take = [&](size_t b) {
        char* r = q;
        q += (b + 255) / 256 * 256;
        return r;
    };
    float* d_rgb = rgb;
    const float* d_alb = albedo;
    const float* d_nrm = normal;
    uint8_t *d_rgb8 = rgb8, *d_alb8 = albedo8, *d_nrm8 = normal8;
    if (!dev) {
        d_rgb = reinterpret_cast<float*>(take(fbytes));
        float* a = albedo ? reinterpret_cast<float*>(take(fbytes)) : nullptr;
        float* nn = normal ? reinterpret_cast<float*>(take(fbytes)) : nullptr;
        std::vector<InCopy> in{InCopy{d_rgb, rgb, fbytes}};
        if (a) in.push_back(InCopy{a, albedo, fbytes});
        if (nn) in.push_back(InCopy{nn, normal, fbytes});
        e = copy_in(ctx, s, in);
        d_alb = a;
        d_nrm = nn;
        d_rgb8 = rgb8 ? reinterpret_cast<uint8_t*>(take((size_t)n)) : nullptr;
        d_alb8 = albedo8 && albedo ? reinterpret_cast<uint8_t*>(take((size_t)n)) : nullptr;
        d_nrm8 = normal8 && normal ? reinterpret_cast<uint8_t*>(take((size_t)n)) : nullptr;
    }
    DenoiseBufs den{};
    if (denoise_step) {
        for (int k = 0; k < 2; ++k) {
            den.t[k] = reinterpret_cast<float4*>(take(16 * recs));
            den.c[k] = reinterpret_cast<float2*>(take(8 * recs));
        }
        den.n = reinterpret_cast<float4*>(take(16 * recs));
        den.a = reinterpret_cast<float4*>(take(16 * recs));
        if (tiled) den.pong = reinterpret_cast<float*>(take(fbytes));
    }
    const int block = 256;
    const int grid = (int)std::min<int64_t>((n + block - 1) / block, (int64_t)ctx->num_sms * 16);
    int first = 0;
    for (int i = 0; i <= num_steps && e == cudaSuccess; ++i) {
        if (i < num_steps && chain.type[i] != FM_POST_DENOISE) continue;
        if (i > first) {
            k_post_pointwise<<<grid, block, 0, s>>>(d_rgb, n, chain, first, i);
            e = cudaGetLastError();
        }
        if (i < num_steps && e == cudaSuccess) {
            e = (tiled ? denoise_tiled : denoise)(s, ctx->num_sms, den, d_rgb, d_alb, d_nrm, width, height);
        }
        first = i + 1;
    }
    if (e == cudaSuccess && d_rgb8) {
        k_to_u8<<<grid, block, 0, s>>>(d_rgb, d_rgb8, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && d_alb8 && d_alb) {
        k_to_u8<<<grid, block, 0, s>>>(d_alb, d_alb8, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && d_nrm8 && d_nrm) {
        k_to_u8<<<grid, block, 0, s>>>(d_nrm, d_nrm8, n);
        e = cudaGetLastError();
    }
    if (!dev && e == cudaSuccess) {
        std::vector<OutCopy> out{OutCopy{rgb, d_rgb, fbytes}};
        if (d_rgb8) out.push_back(OutCopy{rgb8, d_rgb8, (size_t)n});
        if (d_alb8) out.push_back(OutCopy{albedo8, d_alb8, (size_t)n});
        if (d_nrm8) out.push_back(OutCopy{normal8, d_nrm8, (size_t)n});
        e = copy_results(ctx, s, out);
    }
    cudaFreeAsync(tmp, s);
    const cudaError_t e2 = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(ctx, e, "postprocess");
    if (e2 != cudaSuccess) return cuda_error(ctx, e2, "postprocess");
    return FM_OK;
}
