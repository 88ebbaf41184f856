// pf_kernels.cu -- sm_103a kernels of the PixelForge triangle pipeline.
//
//   k_vertex   one thread per vertex: transform, Gouraud lighting
//              (src/internal/primitives/triangles.c:72-104, lighting.c:24-134)
//   k_items    one thread per triangle-face item, in submission order:
//              2D/3D decision, projection, polygon clipping of the rare items
//              that cross a plane (triangles.c:157-280), setup, cull and
//              order-keyed binning into 8x8 tiles (triangles.c:287-339)
//   k_binsort  long bins back into submission order
//   k_raster   one warp per tile: restores submission order of a short
//              bin, then per batch of sub-triangles computes coverage with
//              the reference's integer edge functions, shades fragments
//              densely and resolves each pixel's fragments in order (depth
//              test, blend) (triangles.c:398-557); optionally starts from
//              a fused clear
//   k_rows     BGRA / unsigned-byte targets, one CTA per framebuffer row
//   k_clear, k_fill, k_hook  framebuffer-wide passes (pfClear,
//              pfClearFramebuffer, device post-process hooks)
//
// Framebuffers of other formats than RGBA / unsigned byte keep their raw
// pixels in HBM; the kernels read and write them through the format's
// getters and setters (pf_pixfmt.h).
//
// Arithmetic parity.  The file is compiled with -fmad=false so that no
// multiply-add is contracted (the reference is built for AVX2 without FMA);
// every floating-point expression keeps the reference's operation order.
// x86 conversion and min/max rules are restated explicitly (see x86_* below).
// Depth and Phong use exact 1/x and 1/sqrt(x) where the reference uses the
// approximate rcp/rsqrt instructions.

#include <cuda_runtime.h>
#include <stdint.h>
#include "pf_layout.h"
#include "pf_device.h"
#include "pf_limits.h"
#include "pf_pixfmt.h"

namespace {

#include "pf_common.cuh"

static_assert((unsigned)PFP_DEPTH_TEST == (unsigned)PFS_DEPTH_TEST && (unsigned)PFP_BLEND == (unsigned)PFS_BLEND &&
              (unsigned)PFP_DEPTH_WRITE == (unsigned)PFS_DEPTH_MASK, "host-set records carry draw-state bits");


// ---------------------------------------------------------------------------
// Gouraud lighting, ubyte arithmetic (lighting.c:24-134), Blinn-Phong
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t min255(int32_t n) { return (uint32_t)(n | ((255 - n) >> 31)) & 255u; }

// powf(x, y) for the Gouraud specular term (lighting.c:114), correctly
// rounded through double precision.  Whole exponents up to 256 (shininess is
// usually one) use binary powering in double -- at most 16 roundings of 2^-53
// each, far below the float rounding step -- instead of the FP64 pow routine,
// which is slow on this part.
__device__ __forceinline__ float pow_gouraud(float x, float y)
{
    if (y >= 1.0f && y <= 256.0f && y == truncf(y)) {
        uint32_t n = (uint32_t)y;
        double b = (double)x, r = 1.0;
        while (n) { if (n & 1u) r *= b; b *= b; n >>= 1; }
        return (float)r;
    }
    return (float)pow((double)x, (double)y);
}

__device__ uint32_t light_gouraud(const PFDrawState &S, const PFDevMaterial &m, uint32_t diffuse,
                                  const float *P, const float *N)
{
    uint32_t R = chn(m.emis, 0), G = chn(m.emis, 1), B = chn(m.emis, 2);
    const uint32_t dR = chn(diffuse, 0), dG = chn(diffuse, 1), dB = chn(diffuse, 2);
    const uint32_t aR = (chn(m.amb, 0) * dR) / 255, aG = (chn(m.amb, 1) * dG) / 255, aB = (chn(m.amb, 2) * dB) / 255;
    float V[3];
    {
        float lsq = 0.0f;
        for (int i = 0; i < 3; i++) { V[i] = S.viewPos[i] - P[i]; lsq += V[i]*V[i]; }
        float inv = __frcp_rn(sqrtf(lsq));
        for (int i = 0; i < 3; i++) V[i] = V[i] * inv;
    }
    const float shin = m.shininess;
    for (int li = 0; li < S.nLights; li++) {
        const PFDevLight &l = S.lights[li];
        uint32_t lR = 0, lG = 0, lB = 0;
        float L[3] = { l.pos[0] - P[0], l.pos[1] - P[1], l.pos[2] - P[2] };
        float dsq = L[0]*L[0] + L[1]*L[1] + L[2]*L[2];
        float dist = 0.0f;
        if (dsq != 0.0f) {
            dist = sqrtf(dsq);
            float inv = __frcp_rn(dist);
            L[0] = L[0] * inv; L[1] = L[1] * inv; L[2] = L[2] * inv;
        }
        uint32_t intensity = 255;
        bool skip = false;
        if ((double)l.inner < 3.14159265358979323846) {
            float nd[3] = { -l.dir[0], -l.dir[1], -l.dir[2] };
            float theta = v3_dot(L, nd);
            float eps = l.inner - l.outer;
            int32_t iv = x86_cvt_trunc(255.0f*(theta - l.outer)/eps);
            intensity = (uint32_t)(iv < 0 ? 0 : (iv > 255 ? 255 : iv));
            if (intensity == 0) skip = true;
        }
        if (!skip) {
            uint32_t att = 255;
            if (l.attL != 0.0f || l.attQ != 0.0f) {
                att = x86_ftoub(255.0f / (l.attC + l.attL*dist + l.attQ*dsq));
                if (att == 0) skip = true;
            }
            if (!skip) {
                uint32_t factor = (intensity * att) / 255;
                int32_t dI = x86_cvt_trunc(255.0f * v3_dot(N, L));
                uint32_t diff = (uint32_t)(dI > 0 ? dI : 0) & 255u;
                lR = min255((int32_t)(lR + (dR * chn(l.diff, 0) * diff) / (255 * 255)));
                lG = min255((int32_t)(lG + (dG * chn(l.diff, 1) * diff) / (255 * 255)));
                lB = min255((int32_t)(lB + (dB * chn(l.diff, 2) * diff) / (255 * 255)));
                float H[3] = { L[0] + V[0], L[1] + V[1], L[2] + V[2] };
                v3_normalize(H);
                float nh = fmaxf(v3_dot(N, H), 0.0f);
                float pw = pow_gouraud(nh, shin);
                uint32_t spec = x86_ftoub(255.0f * pw);
                lR = min255((int32_t)(lR + (chn(m.spec, 0) * chn(l.spec, 0) * spec) / (255 * 255)));
                lG = min255((int32_t)(lG + (chn(m.spec, 1) * chn(l.spec, 1) * spec) / (255 * 255)));
                lB = min255((int32_t)(lB + (chn(m.spec, 2) * chn(l.spec, 2) * spec) / (255 * 255)));
                lR = (lR * factor) / 255; lG = (lG * factor) / 255; lB = (lB * factor) / 255;
            }
        }
        R = min255((int32_t)(R + lR + (aR * chn(l.amb, 0)) / 255));
        G = min255((int32_t)(G + lG + (aG * chn(l.amb, 1)) / 255));
        B = min255((int32_t)(B + lB + (aB * chn(l.amb, 2)) / 255));
    }
    return R | (G << 8) | (B << 16) | (diffuse & 0xff000000u);
}

// scalar pfiBlendMultiplicative (blend.h:77-86)
__device__ __forceinline__ uint32_t blend_mul_scalar(uint32_t s, uint32_t d)
{
    uint32_t r = 0;
    for (int i = 0; i < 4; i++) r |= ((chn(s, i) * chn(d, i)) / 255) << (8 * i);
    return r;
}

// ---------------------------------------------------------------------------
// per-fragment operations, SIMD semantics
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack4(const int32_t *v)
{
    return (uint32_t)v[0] | ((uint32_t)v[1] << 8) | ((uint32_t)v[2] << 16) | ((uint32_t)v[3] << 24);
}

// blend.h:140-277 (SUB adds; channels are ORed without masks when packed)
__device__ uint32_t blend_simd(int mode, uint32_t src, uint32_t dst)
{
    if (mode == 1) {
        // alpha: (s a + d (256 - a)) >> 8 a channel, the source's alpha taken
        // as 255, two channels a multiply (a sum stays below 2^16)
        const uint32_t a = (src >> 24) + 1u, ia = 256u - a;
        const uint32_t rb = (src & 0x00ff00ffu) * a + (dst & 0x00ff00ffu) * ia;
        const uint32_t ga = (((src >> 8) & 0x000000ffu) | 0x00ff0000u) * a + ((dst >> 8) & 0x00ff00ffu) * ia;
        return ((rb >> 8) & 0x00ff00ffu) | (ga & 0xff00ff00u);
    }
    int32_t s[4], d[4], o[4];
    for (int i = 0; i < 4; i++) { s[i] = (int32_t)chn(src, i); d[i] = (int32_t)chn(dst, i); }
    switch (mode) {
    case 0: for (int i = 0; i < 4; i++) o[i] = (s[i] + d[i]) >> 1; break;
    case 2: for (int i = 0; i < 4; i++) { int32_t t = s[i] + d[i]; o[i] = t < 255 ? t : 255; } break;
    case 3: for (int i = 0; i < 4; i++) { int32_t t = s[i] + d[i]; o[i] = t > 0 ? t : 0; } break;
    case 4: for (int i = 0; i < 4; i++) o[i] = (s[i]*d[i]) >> 8; break;
    case 5: for (int i = 0; i < 4; i++) { int32_t t = ((d[i]*(255 - s[i])) >> 8) + s[i]; o[i] = t < 255 ? t : 255; } break;
    case 6: for (int i = 0; i < 4; i++) o[i] = s[i] > d[i] ? s[i] : d[i]; break;
    case 7: for (int i = 0; i < 4; i++) o[i] = s[i] < d[i] ? s[i] : d[i]; break;
    default: return src;
    }
    return pack4(o);
}

// depth.h:80-124 (NOTEQUAL compares equal there)
__device__ __forceinline__ bool depth_simd(int f, float src, float dst)
{
    switch (f) {
    case 0: case 1: return src == dst;
    case 2: return src < dst;
    case 3: return src <= dst;
    case 4: return src > dst;
    default: return src >= dst;
    }
}


// A texture as the rasterizer samples it.
struct TexDesc {
    const uint32_t *tex;
    uint32_t w, h;
    int32_t wrap, filter;
    float tx, ty;
};

// From the set-up record (texture parameters copied there by setup_prim),
// or from the draw state when they did not fit.
__device__ __forceinline__ TexDesc tex_desc(const PFPrim &P, const PFDrawState *states)
{
    TexDesc d;
    if (!(P.rstate & PFR_TEX_FROM_STATE)) {
        d.tex = reinterpret_cast<const uint32_t *>(P.src);
        d.w = P.nSrc & 0xffffu; d.h = P.nSrc >> 16;
        d.wrap = (int32_t)((P.rstate >> PFR_WRAP_SHIFT) & 3u); d.filter = (P.rstate & PFR_FILTER) ? 1 : 0;
        d.tx = P.texTx; d.ty = P.texTy;
    } else {
        const PFDrawState &S = states[P.flags >> 8];
        d.tex = S.tex; d.w = S.texW; d.h = S.texH; d.wrap = S.texWrap; d.filter = S.texFilter;
        d.tx = S.texTx; d.ty = S.texTy;
    }
    return d;
}

// Texel at linear offset y*w + x; offsets outside the texture read as 0
// (the reference reads past its buffer there).
__device__ __forceinline__ uint32_t tex_fetch(const TexDesc &T, int32_t x, int32_t y)
{
    int32_t off = (int32_t)((uint32_t)y * T.w + (uint32_t)x);
    if (off < 0 || (uint32_t)off >= T.w * T.h) return 0u;
    return __ldg(T.tex + off);
}

__device__ __forceinline__ uint32_t lerp_color(uint32_t a, uint32_t b, float t)
{
    const float inv255 = 1.0f / 255.0f;
    int32_t o[4];
    for (int i = 0; i < 4; i++) {
        float af = (float)chn(a, i) * inv255;
        float bf = (float)chn(b, i) * inv255;
        float r = af + t * (bf - af);
        o[i] = __float2int_rn(x86_min(x86_max(r, 0.0f), 1.0f) * 255.0f);   // clamped: in range
    }
    return pack4(o);
}

__device__ uint32_t tex_sample(const TexDesc &T, float u, float v)
{
    int32_t x0, y0;
    tex_map_wh(T.w, T.h, T.wrap, u, v, x0, y0);
    if (T.filter == 0) return tex_fetch(T, x0, y0);
    int32_t x1, y1;
    tex_map_wh(T.w, T.h, T.wrap, u + T.tx, v + T.ty, x1, y1);
    float fx = u * (float)T.w - (float)x0;
    float fy = v * (float)T.h - (float)y0;
    fx = x86_min(x86_max(fx, 0.0f), 1.0f);
    fy = x86_min(x86_max(fy, 0.0f), 1.0f);
    uint32_t c00 = tex_fetch(T, x0, y0), c10 = tex_fetch(T, x1, y0);
    uint32_t c01 = tex_fetch(T, x0, y1), c11 = tex_fetch(T, x1, y1);
    return lerp_color(lerp_color(c00, c10, fx), lerp_color(c01, c11, fx), fy);
}

// Cephes log/exp as adapted for SSE/AVX by J. Pommier and G. Garberoglio
// (zlib licence), the reference's per-fragment power (simd.h:183-300, 1158-1170).
__device__ float cephes_log(float x)
{
    const bool invalid = (x <= 0.0f);
    x = x86_max(x, __uint_as_float(0x00800000u));
    int32_t e_i = (int32_t)(__float_as_uint(x) >> 23);
    x = __uint_as_float((__float_as_uint(x) & ~0x7f800000u) | __float_as_uint(0.5f));
    e_i -= 0x7f;
    float e = (float)e_i;
    e = e + 1.0f;
    const bool lt = (x < 0.707106781186547524f);
    float tmp = lt ? x : 0.0f;
    x = x - 1.0f;
    e = e - (lt ? 1.0f : 0.0f);
    x = x + tmp;
    float z = x * x;
    float y = 7.0376836292E-2f;
    y = y * x; y = y + -1.1514610310E-1f;
    y = y * x; y = y + 1.1676998740E-1f;
    y = y * x; y = y + -1.2420140846E-1f;
    y = y * x; y = y + 1.4249322787E-1f;
    y = y * x; y = y + -1.6668057665E-1f;
    y = y * x; y = y + 2.0000714765E-1f;
    y = y * x; y = y + -2.4999993993E-1f;
    y = y * x; y = y + 3.3333331174E-1f;
    y = y * x;
    y = y * z;
    tmp = e * -2.12194440e-4f;
    y = y + tmp;
    tmp = z * 0.5f;
    y = y - tmp;
    tmp = e * 0.693359375f;
    x = x + y;
    x = x + tmp;
    return invalid ? __uint_as_float(0xffffffffu) : x;
}

__device__ float cephes_exp(float x)
{
    x = x86_min(x, 88.3762626647949f);
    x = x86_max(x, -88.3762626647949f);
    float fx = x * 1.44269504088896341f;
    fx = fx + 0.5f;
    float tmp = floorf(fx);
    fx = tmp - ((tmp > fx) ? 1.0f : 0.0f);
    tmp = fx * 0.693359375f;
    float z = fx * -2.12194440e-4f;
    x = x - tmp;
    x = x - z;
    z = x * x;
    float y = 1.9875691500E-4f;
    y = y * x; y = y + 1.3981999507E-3f;
    y = y * x; y = y + 8.3334519073E-3f;
    y = y * x; y = y + 4.1665795894E-2f;
    y = y * x; y = y + 1.6666665459E-1f;
    y = y * x; y = y + 5.0000001201E-1f;
    y = y * z;
    y = y + x;
    y = y + 1.0f;
    int32_t n = x86_cvt_trunc(fx) + 0x7f;
    return y * __uint_as_float((uint32_t)n << 23);
}

__device__ __forceinline__ void dir_simd(float *d, const float *a, const float *b)   // simd.h:2469-2490
{
    d[0] = a[0] - b[0]; d[1] = a[1] - b[1]; d[2] = a[2] - b[2];
    float lsq = d[0]*d[0] + d[1]*d[1];
    lsq = lsq + d[2]*d[2];
    lsq = x86_max(lsq, 1e-5f);
    float inv = __frcp_rn(sqrtf(lsq));
    d[0] = d[0] * inv; d[1] = d[1] * inv; d[2] = d[2] * inv;
}
__device__ __forceinline__ float dot_simd(const float *a, const float *b)
{
    float d = a[0]*b[0] + a[1]*b[1];
    return d + a[2]*b[2];
}

// pfiSimdLightingProcess (lighting.c:149-258), one lane
__device__ uint32_t light_phong(const PFDrawState &S, uint32_t frag, const PFDevMaterial &m,
                                const float *P, const float *N)
{
    const float inv255 = 1.0f / 255.0f;
    float cd[3], ca[3], cs[3];
    for (int i = 0; i < 3; i++) {
        cd[i] = (float)chn(frag, i) * inv255;
        ca[i] = (float)chn(m.amb, i) * inv255;
        cs[i] = (float)chn(m.spec, i) * inv255;
    }
    for (int i = 0; i < 3; i++) ca[i] = ca[i] * cd[i];
    float V[3]; dir_simd(V, S.viewPos, P);
    float acc[3] = { 0.0f, 0.0f, 0.0f };
    for (int li = 0; li < S.nLights; li++) {
        const PFDevLight &l = S.lights[li];
        float la[3], ld[3], ls[3];
        for (int i = 0; i < 3; i++) {
            la[i] = (float)chn(l.amb, i) * inv255;
            ld[i] = (float)chn(l.diff, i) * inv255;
            ls[i] = (float)chn(l.spec, i) * inv255;
        }
        float L[3]; dir_simd(L, l.pos, P);
        float amb[3], dif[3], spe[3];
        for (int i = 0; i < 3; i++) amb[i] = la[i] * ca[i];
        float diff = x86_max(dot_simd(N, L), 0.0f);
        for (int i = 0; i < 3; i++) { dif[i] = ld[i] * diff; dif[i] = dif[i] * cd[i]; }
        float H[3] = { L[0] + V[0], L[1] + V[1], L[2] + V[2] };
        float hs = H[0]*H[0] + H[1]*H[1];
        hs = hs + H[2]*H[2];
        float hinv = __frcp_rn(sqrtf(hs));
        for (int i = 0; i < 3; i++) H[i] = H[i] * hinv;
        float spec = x86_max(dot_simd(N, H), 0.0f);
        spec = cephes_exp(cephes_log(spec) * m.shininess);
        for (int i = 0; i < 3; i++) { spe[i] = ls[i] * spec; spe[i] = spe[i] * cs[i]; }
        if ((double)l.inner < 3.14159265358979323846) {
            float nd[3] = { -l.dir[0], -l.dir[1], -l.dir[2] };
            float theta = dot_simd(L, nd);
            float eps = l.inner - l.outer;
            float it = (theta - l.outer) / eps;
            it = x86_min(x86_max(it, 0.0f), 1.0f);
            for (int i = 0; i < 3; i++) { dif[i] = dif[i] * it; spe[i] = spe[i] * it; }
        }
        if (l.attL != 0.0f || l.attQ != 0.0f) {
            // pfiVec3DistanceSq_simd reads y for z (simd.h:2423-2442)
            float d0 = l.pos[0] - P[0], d1 = l.pos[1] - P[1], d2 = l.pos[1] - P[1];
            float dsq = d0*d0 + (d1*d1 + d2*d2);
            float dist = sqrtf(dsq);
            float att = __frcp_rn(l.attC + (l.attL*dist + l.attQ*dsq));
            for (int i = 0; i < 3; i++) { amb[i] = amb[i] * att; dif[i] = dif[i] * att; spe[i] = spe[i] * att; }
        }
        for (int i = 0; i < 3; i++) { acc[i] = acc[i] + amb[i]; acc[i] = acc[i] + dif[i]; acc[i] = acc[i] + spe[i]; }
    }
    int32_t o[4] = { 0, 0, 0, 0 };
    for (int i = 0; i < 3; i++) o[i] = __float2int_rn(x86_min(x86_max(acc[i], 0.0f), 1.0f) * 255.0f);
    return pack4(o);
}

// ---------------------------------------------------------------------------
// k_vertex
// ---------------------------------------------------------------------------
__device__ __forceinline__ int seg_of_vertex(const PFSegment *segs, int nSegs, uint32_t g)
{
    int lo = 0, hi = nSegs - 1;
    while (lo < hi) { int mid = (lo + hi + 1) >> 1; if (segs[mid].vtxBase <= g) lo = mid; else hi = mid - 1; }
    return lo;
}
__device__ __forceinline__ int seg_of_item(const PFSegment *segs, int nSegs, uint32_t g)
{
    int lo = 0, hi = nSegs - 1;
    while (lo < hi) { int mid = (lo + hi + 1) >> 1; if (segs[mid].itemBase <= g) lo = mid; else hi = mid - 1; }
    return lo;
}

// One thread per vertex of the batch.  The grid also clears the tile bin
// counters and the per-batch counters for k_items (so no memset launches),
// and puts the pixels that a fused clear keeps in place (a copy of their own
// costs a small launch more than it moves).
__global__ void k_vertex(const PFSegment *__restrict__ segs, int nSegs, const PFDrawState *__restrict__ states,
                         PFVertexOut *__restrict__ out, uint32_t nVerts, PFDevCounters *cnt,
                         uint32_t *__restrict__ binCount, uint32_t nTiles, const PFTarget *__restrict__ targets, int nTargets)
{
    __shared__ int sUniform, sAborted;
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // (no-op unless launched programmatically serialized)
    // thread 0 takes the block's decisions, behind one barrier: the abort
    // (one decision per block) and the segment of the block's vertices when
    // they share one (the usual case; the others search)
    const uint32_t g0 = blockIdx.x * blockDim.x;
    if (threadIdx.x == 0) {
        sAborted = cnt->abortCommand != 0xffffffffu;
        int su = -1;
        if (g0 < nVerts) {
            const int a = seg_of_vertex(segs, nSegs, g0), b = seg_of_vertex(segs, nSegs, min(g0 + blockDim.x, nVerts) - 1);
            su = (a == b) ? a : -1;
        }
        sUniform = su;
    }
    __syncthreads();
    if (sAborted) return;
    for (uint32_t t = g; t < nTiles; t += gridDim.x * blockDim.x) binCount[t] = 0;
    if (g == 0) {
        cnt->clipCount = 0; cnt->batchRasterized = 0; cnt->batchFragments = 0; cnt->tileQueue = 0; cnt->sortQueue = 0;
        cnt->tileListCount = 0;
        for (int l = 0; l < PF_HEAVY_LEVELS; l++) cnt->heavyCount[l] = 0;
    }
    if (g < (uint32_t)nTargets) {
        // the pixels a fused pfClear keeps, which came with the draw states
        const PFTarget &T = targets[g];
        if (T.headColor)
            for (int i = 0; i < 2 * pff_bytes(T.fmt); i++) static_cast<uint32_t *>(T.color)[i] = T.headColor[i];
        if (T.headDepth)
            for (int i = 0; i < 8; i++) T.depth[i] = T.headDepth[i];
    }
    if (g >= nVerts) return;
    // the segment and its draw state are read in place (one address for the
    // block: L1 serves it after the first access)
    const int su = sUniform;
    const PFSegment &sg = segs[su >= 0 ? su : seg_of_vertex(segs, nSegs, g)];
    const PFDrawState &S = states[sg.state];
    const uint32_t j = g - sg.vtxBase;
    float pos[4], nrm[3], uv[2];
    uint32_t col;
    if (sg.srcKind == PF_SRC_RECORDS) {
        const PFVertexIn &r = sg.records[j];
        for (int i = 0; i < 4; i++) pos[i] = r.pos[i];
        for (int i = 0; i < 3; i++) nrm[i] = r.normal[i];
        uv[0] = r.uv[0]; uv[1] = r.uv[1];
        col = r.color;
    } else {
        pos[0] = pos[1] = pos[2] = 0.0f; pos[3] = 1.0f;
        for (int k = 0; k < sg.posSize; k++) pos[k] = sg.pos[(size_t)j * sg.posSize + k];
        if (sg.nrm) { for (int k = 0; k < 3; k++) nrm[k] = sg.nrm[(size_t)j * 3 + k]; }
        else { nrm[0] = sg.constNormal[0]; nrm[1] = sg.constNormal[1]; nrm[2] = sg.constNormal[2]; }
        if (sg.uv) { uv[0] = sg.uv[(size_t)j * 2]; uv[1] = sg.uv[(size_t)j * 2 + 1]; }
        else { uv[0] = sg.constUv[0]; uv[1] = sg.constUv[1]; }
        if (sg.col) {
            col = 0xffffffffu;
            for (int k = 0; k < sg.colSize; k++) {
                uint32_t b = sg.col[(size_t)j * sg.colSize + k];
                col = (col & ~(255u << (8 * k))) | (b << (8 * k));
            }
        } else col = sg.constColor;
    }
    PFVertexOut o;
    uint32_t c0 = col, c1 = col;
    float n[3] = { nrm[0], nrm[1], nrm[2] };
    if (S.flags & PFS_LIGHTING) {
        v3_transform(n, nrm, S.normal);
        v3_normalize(n);
        uint32_t base[2] = { blend_mul_scalar(col, S.mat[0].diff), blend_mul_scalar(col, S.mat[1].diff) };
        if (!(S.flags & PFS_PHONG)) {
            float NdotV = v3_dot(n, S.view8);
            const PFDevMaterial &lm = S.mat[(NdotV < 0.0f) ? 0 : 1];
            base[0] = light_gouraud(S, lm, base[0], pos, n);
            base[1] = (S.mat[0].diff == S.mat[1].diff) ? base[0] : light_gouraud(S, lm, base[1], pos, n);
        }
        c0 = base[0]; c1 = base[1];
    }
    v4_transform(o.h, pos, S.mvp);
    o.uv[0] = uv[0]; o.uv[1] = uv[1];
    o.col[0] = c0; o.col[1] = c1;
    o.n[0] = n[0]; o.n[1] = n[1]; o.n[2] = n[2];
    o.p[0] = pos[0]; o.p[1] = pos[1]; o.p[2] = pos[2];
    o.pad[0] = o.pad[1] = 0;
    out[g] = o;
}

// ---------------------------------------------------------------------------
// setup + binning
// ---------------------------------------------------------------------------

struct BinArgs {
    uint32_t *binCount;
    uint32_t *tileList;        // the raster work lists
    uint32_t listStride;
    uint32_t *bins;
    uint32_t cap;
    const PFTarget *targets;
    PFDevCounters *cnt;
    uint32_t command;
    float4 *planes;            // depth_plane of each item's sub-triangle 0
    bool countSmall;           // triangles within 32x32 pixels are counted by k_items too
};

// Framebuffer geometry a sub-triangle is binned against.
struct TileSpace {
    uint32_t W, H, tilesX, tileBase;
    bool rows;                 // rasterized by k_rows, which counts its fragments
};

__device__ __forceinline__ TileSpace tile_space(const BinArgs &B, int target)
{
    const PFTarget &t = B.targets[target];
    return TileSpace{ t.W, t.H, t.tilesX, t.tileBase, t.fmt == PFF_BGRA8 };
}


// Tile range of a set-up sub-triangle: pixels x in [xMin, xMax) and y in
// [yMin, yMax], compared as unsigned (the reference's PFsizei loop bounds),
// clipped to the framebuffer.  Returns false when no pixel remains.
__device__ __forceinline__ bool tile_range(const TileSpace &T, const PFPrim &P, uint32_t &tx0, uint32_t &ty0,
                                           uint32_t &ntx, uint32_t &nty)
{
    uint32_t x0 = (uint32_t)P.xMin, x1 = (uint32_t)P.xMax, y0 = (uint32_t)P.yMin, y1 = (uint32_t)P.yMax;
    if (x1 > T.W) x1 = T.W;
    if (y1 >= T.H) y1 = T.H - 1;
    if (x0 >= x1 || y0 > y1) return false;
    tx0 = x0 / PF_TILE; ty0 = y0 / PF_TILE;
    ntx = (x1 - 1) / PF_TILE - tx0 + 1; nty = y1 / PF_TILE - ty0 + 1;
    return true;
}

// A triangle record's edge functions as the binning tests tiles with them:
// w_e(x, y) = x ex_e + y ey_e + c_e (triangles.c:336-349, 398-420), set
// only when every vertex coordinate and the box lie within (-2^13, 2^13)
// and the framebuffer is at most 2^13 pixels a side -- there the edge
// functions of every pixel of the box stay far inside 32 bits, where the
// reference's wrapping arithmetic is exact (on = false otherwise, and for
// points, lines and rectangles, which keep every tile of their box).
struct EdgeTest {
    int32_t ex[3], ey[3], c[3];
    int32_t xMin, xMax, yMin, yMax;
    bool on;
};
__device__ __forceinline__ bool edge_on(const PFPrim &P, uint32_t W, uint32_t H)
{
    const int32_t L = 1 << 13;
    const int32_t v[6] = { P.x1, P.y1, P.x2, P.y2, P.x3, P.y3 };
    bool ok = !(P.flags & PFP_KIND) && W <= (uint32_t)L && H <= (uint32_t)L &&
              P.xMin > -L && P.xMin < L && P.xMax > -L && P.xMax < L && P.yMin > -L && P.yMin < L && P.yMax > -L && P.yMax < L;
    for (int k = 0; k < 6; k++) ok = ok && v[k] > -L && v[k] < L;
    return ok;
}
__device__ __forceinline__ EdgeTest edge_test(const PFPrim &P, bool ok)
{
    EdgeTest E;
    const int32_t vx[3] = { P.x2, P.x3, P.x1 }, vy[3] = { P.y2, P.y3, P.y1 };
    const int32_t sgn = (P.flags & 1u) ? -1 : 1;
    const int32_t sx[3] = { P.y3 - P.y2, P.y1 - P.y3, P.y2 - P.y1 }, sy[3] = { P.x2 - P.x3, P.x3 - P.x1, P.x1 - P.x2 };
    for (int e = 0; e < 3; e++) {
        E.ex[e] = ok ? sgn * sx[e] : 0;
        E.ey[e] = ok ? sgn * sy[e] : 0;
        E.c[e] = ok ? -(vx[e] * E.ex[e] + vy[e] * E.ey[e]) : 0;
    }
    E.xMin = P.xMin; E.xMax = P.xMax; E.yMin = P.yMin; E.yMax = P.yMax;
    E.on = ok;
    return E;
}

// Whether the record may cover a pixel of tile (tx, ty): no, when one of
// its edge functions is negative on the whole rectangle where the tile and
// the box meet -- a pixel is covered only when no edge function is negative
// (triangles.c:415-420), and a linear function is largest at a corner.
__device__ __forceinline__ bool tile_touched(const EdgeTest &E, uint32_t tx, uint32_t ty, uint32_t W, uint32_t H)
{
    if (!E.on) return true;
    // the tile's pixels inside the box and the framebuffer (the box was
    // found inside it by tile_range)
    const int32_t x0 = max(E.xMin, (int32_t)(tx * PF_TILE));
    const int32_t x1 = min(min(E.xMax, (int32_t)(tx * PF_TILE + PF_TILE)), (int32_t)W) - 1;
    const int32_t y0 = max(E.yMin, (int32_t)(ty * PF_TILE));
    const int32_t y1 = min(min(E.yMax, (int32_t)(ty * PF_TILE + PF_TILE - 1)), (int32_t)H - 1);
    bool keep = true;
    for (int e = 0; e < 3; e++) {
        const int32_t w00 = x0 * E.ex[e] + y0 * E.ey[e] + E.c[e];
        const int32_t hi = w00 + max((x1 - x0) * E.ex[e], 0) + max((y1 - y0) * E.ey[e], 0);
        keep = keep && hi >= 0;
    }
    return keep;
}

__device__ __forceinline__ void bin_slot(const BinArgs &B, uint32_t t, uint32_t slot, uint32_t key)
{
    if (slot < B.cap) B.bins[(size_t)t * B.cap + slot] = key;
    else {
        atomicMax(&B.cnt->maxBin, slot + 1);
        if (slot == B.cap) {
            atomicOr(&B.cnt->status, (unsigned)PFD_BIN_OVERFLOW);
            atomicMin(&B.cnt->abortCommand, B.command);
        }
    }
}

// Raster work lists: a tile's bin growing from `before` to `before + added`
// entries puts the tile on the list of non-empty tiles (first entry) and on
// the list of each heavy level it reaches (32, 128, 512, 2048 entries),
// which the rasterizer takes first, heaviest level first, so that the
// longest tiles do not start last.
__device__ __forceinline__ uint32_t heavy_level(uint32_t count)
{
    uint32_t l = 0;                                    // 0: below the first level
#pragma unroll
    for (int k = 0; k < PF_HEAVY_LEVELS; k++) l += count >= ((uint32_t)PF_HEAVY_BASE << (2 * k)) ? 1u : 0u;
    return l;
}

__device__ __forceinline__ void list_tile(const BinArgs &B, uint32_t t, uint32_t before, uint32_t added)
{
    if (before == 0) B.tileList[atomicAdd(&B.cnt->tileListCount, 1u)] = t;
    for (uint32_t l = heavy_level(before) + 1; l <= heavy_level(before + added); l++)
        B.tileList[l * B.listStride + atomicAdd(&B.cnt->heavyCount[l - 1], 1u)] = t;
}

// The same for the tiles of a whole warp (every lane calls it; lanes that
// put nothing on a list pass added = 0): one atomic a list and warp.  The
// five counters share a cache line, so an atomic per tile and level queues
// there: the batch of 64 soups, 83,000 tiles past most levels, 777 -> 645 us
// of k_items in the first state of the binning below (312-326 now).
__device__ __forceinline__ void list_tiles_warp(const BinArgs &B, uint32_t t, uint32_t before, uint32_t added)
{
    const uint32_t from = heavy_level(before), to = heavy_level(before + added);
    if (!__any_sync(0xffffffffu, added && (before == 0 || to > from))) return;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t l = 0; l <= PF_HEAVY_LEVELS; l++) {
        const bool put = added && (l == 0 ? before == 0 : (from < l && l <= to));
        const uint32_t m = __ballot_sync(0xffffffffu, put);
        if (!m) continue;
        const uint32_t first = (uint32_t)(__ffs(m) - 1);
        uint32_t at = 0;
        if (lane == first) at = atomicAdd(l == 0 ? &B.cnt->tileListCount : &B.cnt->heavyCount[l - 1], (unsigned)__popc(m));
        at = __shfl_sync(0xffffffffu, at, first);
        if (put) B.tileList[l * B.listStride + at + __popc(m & ((1u << lane) - 1u))] = t;
    }
}

// Whether the record may raise a pixel's depth (a batch without such
// records only lowers depths).
__device__ __forceinline__ bool raises_depth(uint32_t rstate)
{
    const uint32_t func = (rstate >> 16) & 255u;
    return (rstate & PFS_DEPTH_MASK) && !((rstate & PFS_DEPTH_TEST) && (func == 2u || func == 3u || func == 0u));
}

// What k_raster needs to know of a record to drop it before loading it: a
// bound on its interpolated term 1 / depth over the image, the plane
// x + y px + z py, and a bound w over the whole triangle.  The plane only
// for triangles of more than a tile, whose corners' depths say little about
// their depth in one tile; m bounds the sum of its absolute terms over the
// tiles of the box, and 4e-6 m the rounding of this
// evaluation, k_raster's and a covered fragment's own (some twenty
// operations of 2^-24 each).  Infinite where there is no bound, w NaN when
// the record may raise a depth.
__device__ __forceinline__ float depth_bound(const PFPrim &P)
{
    const float inf = __int_as_float(0x7f800000);
    if (raises_depth(P.rstate)) return __int_as_float(0x7fffffff);
    if (!(P.zReject == P.zReject)) return inf;         // (none unless lo > 0 or hi < 0)
    const float lo = fminf(P.z1, fminf(P.z2, P.z3)), hi = fmaxf(P.z1, fmaxf(P.z2, P.z3));
    return hi * (lo > 0.0f ? 1.00001f : 0.99999f);
}

// Append `key` to the bin of every tile the sub-triangle touches (one
// thread; used by the clipping path).
__device__ void bin_prim(const BinArgs &B, const TileSpace &T, const PFPrim &P, uint32_t key)
{
    uint32_t tx0, ty0, ntx, nty;
    if (!tile_range(T, P, tx0, ty0, ntx, nty)) return;
    const EdgeTest ET = edge_test(P, edge_on(P, T.W, T.H));
    for (uint32_t ty = ty0; ty < ty0 + nty; ty++)
        for (uint32_t tx = tx0; tx < tx0 + ntx; tx++) {
            if (!tile_touched(ET, tx, ty, T.W, T.H)) continue;
            const uint32_t t = T.tileBase + ty * T.tilesX + tx;
            const uint32_t slot = atomicAdd(&B.binCount[t], 1u);
            list_tile(B, t, slot, 1u);
            bin_slot(B, t, slot, key);
        }
}

// Whether the record's box is that of its vertices, inside the framebuffer.
__device__ __forceinline__ bool whole_box(const PFPrim &P, const TileSpace &T)
{
    return P.xMin == min(P.x1, min(P.x2, P.x3)) && P.xMax == max(P.x1, max(P.x2, P.x3)) &&
           P.yMin == min(P.y1, min(P.y2, P.y3)) && P.yMax == max(P.y1, max(P.y2, P.y3)) &&
           P.xMin >= 0 && P.yMin >= 0 && (uint32_t)P.xMax <= T.W && (uint32_t)P.yMax < T.H;
}

// A lane's sub-triangle as its warp bins it, in shared memory: seven 16-byte
// words (a stride of 28 banks: 16-byte reads of eight different records
// touch every bank once).
struct __align__(16) BinRec {
    int32_t ex[3], ey[3], c[3];        // edge functions x ex + y ey + c (on), as EdgeTest
    float rex[3];                      // 1 / ex
    int32_t x0, x1, y0, y1;            // its pixels, inside the framebuffer (inclusive)
    uint32_t on;
    uint32_t first;                    // number of its first tile row
    uint32_t tileBase, tilesX;
    uint32_t key;
    uint32_t count;                    // its covered pixels: 0 not counted, 1 lattice_pixels, 2 row_pixels
    uint32_t right;                    // lattice_pixels: those of column xMax
    float z[3], wInvSum, bound;        // depth_plane
};
static_assert(sizeof(BinRec) == 112 && offsetof(BinRec, x0) == 48 && offsetof(BinRec, on) == 64 && offsetof(BinRec, key) == 80,
              "seven 16-byte words, written word by word");

// A tile row of a sub-triangle: a run of tiles.
struct __align__(16) BinRow {
    uint32_t tile, first, key, pad;    // first tile, number of its first (row, tile) pair
};

// Binning scratch of a warp.
struct BinWarp {
    BinRec rec[32];
    BinRow row[32];
};

// The pixel columns [lo, hi] of tile row ty that may hold covered pixels:
// those where no edge function is negative on the whole of the row's part
// of the column (the largest value is at one end of it), bounded by the
// root of that value, which is linear in x.  The root is found in single
// precision and widened by 1/32 of a pixel: |x| is below 2^13 and the
// value's integer terms below 2^30, so its error stays below 2^-7; a column
// too many costs nothing but a bin entry that covers no pixel.
__device__ __forceinline__ void row_columns(const BinRec &r, uint32_t ty, int32_t &lo, int32_t &hi)
{
    lo = r.x0; hi = r.x1;
    if (!r.on) return;
    const int32_t y0 = max(r.y0, (int32_t)(ty * PF_TILE)), y1 = min(r.y1, (int32_t)(ty * PF_TILE + PF_TILE - 1));
#pragma unroll
    for (int e = 0; e < 3; e++) {
        const int32_t v = r.c[e] + r.ey[e] * (r.ey[e] > 0 ? y1 : y0);      // its largest over the row at x = 0
        const float root = -(float)v * r.rex[e];
        if (r.ex[e] > 0) lo = max(lo, __float2int_ru(root - 0.03125f));
        else if (r.ex[e] < 0) hi = min(hi, __float2int_rd(root + 0.03125f));
        else if (v < 0) hi = lo - 1;
    }
}

// The covered pixels of tile row ty, columns [lo, hi] (none is covered
// outside them): per pixel row and edge the exact last column the edge
// function leaves non-negative -- floor division of its value at x = 0 by
// |ex|, found once in single precision and corrected by its remainder, then
// stepped row by row with quotient and remainder.  Only for records whose
// edge functions stay inside 32 bits (on).  A quotient beyond 2^21, which a
// single correction may leave off, stays far outside the columns whatever
// the rows add to it.
__device__ __forceinline__ uint32_t row_pixels(const BinRec &r, uint32_t ty, int32_t lo, int32_t hi)
{
    const int32_t y0 = max(r.y0, (int32_t)(ty * PF_TILE)), y1 = min(r.y1, (int32_t)(ty * PF_TILE + PF_TILE - 1));
    auto divide = [](int32_t v, int32_t d, float inv, int32_t &rem) {
        int32_t q = __float2int_rd((float)v * inv);
        rem = (int32_t)((uint32_t)v - (uint32_t)q * (uint32_t)d);
        if (rem < 0) { q--; rem += d; }
        if (rem >= d) { q++; rem -= d; }
        return q;
    };
    int32_t q[3], rem[3], qs[3], rs[3], d[3];
#pragma unroll
    for (int e = 0; e < 3; e++) {
        d[e] = abs(r.ex[e]);
        if (d[e] == 0) {
            // a horizontal edge's rows are wholly inside or outside: the
            // rows from the edge times 2^14, and 2^13 (columns stay below it)
            const int32_t v = r.c[e] + r.ey[e] * y0;
            q[e] = __float2int_rn((float)v * __frcp_rn(fabsf((float)r.ey[e]))) * (1 << 14) + (1 << 13);
            qs[e] = r.ey[e] > 0 ? 1 << 14 : -(1 << 14);
            rem[e] = rs[e] = 0; d[e] = 0x7fffffff;
            continue;
        }
        const float inv = fabsf(r.rex[e]);
        q[e] = divide(r.c[e] + r.ey[e] * y0, d[e], inv, rem[e]);
        qs[e] = divide(r.ey[e], d[e], inv, rs[e]);
    }
    uint32_t n = 0;
    for (int32_t y = y0; y <= y1; y++) {
        int32_t a = lo, b = hi;
#pragma unroll
        for (int e = 0; e < 3; e++) {
            if (r.ex[e] > 0) a = max(a, -q[e]); else b = min(b, q[e]);
            q[e] += qs[e]; rem[e] += rs[e];
            if (rem[e] >= d[e]) { rem[e] -= d[e]; q[e]++; }
        }
        n += (uint32_t)max(b - a + 1, 0);
    }
    return n;
}

// The depth plane of a record.
__device__ __forceinline__ float4 depth_plane(const BinRec &R)
{
    const float inf = __int_as_float(0x7f800000);
    float4 p = make_float4(inf, 0.0f, 0.0f, R.bound);
    if (!(fabsf(R.bound) < inf) || (R.x1 - R.x0 < PF_TILE && R.y1 - R.y0 < PF_TILE)) return p;
    float m = 0.0f;
    p.x = 0.0f;
#pragma unroll
    for (int e = 0; e < 3; e++) {
        const float zw = R.z[e] * R.wInvSum, fc = (float)R.c[e], fx = (float)R.ex[e], fy = (float)R.ey[e];
        p.x += fc * zw; p.y += fx * zw; p.z += fy * zw;
        m += (fabsf(fc) + fabsf(fx) * (float)(R.x1 + PF_TILE) + fabsf(fy) * (float)(R.y1 + PF_TILE)) * fabsf(zw);
    }
    p.x += 4e-6f * m;
    return p;
}

// The covered pixels of a record whose box is that of its vertices and whose
// edge functions stay inside 32 bits: the vertices are pixels, and the
// pixels where no edge function is negative are those of the closed
// triangle -- by Pick's theorem half its doubled area and of its boundary's
// pixels, and one -- less those of the column xMax, which the box leaves
// out.  A boundary's pixels are the greatest common divisors of its edges'
// components (Euclid's algorithm on the three at once; values below 2^14,
// so a quotient in single precision is at most one off).
__device__ __forceinline__ uint32_t lattice_pixels(const BinRec &R)
{
    int32_t a[3], b[3];
#pragma unroll
    for (int e = 0; e < 3; e++) { a[e] = abs(R.ex[e]); b[e] = abs(R.ey[e]); }
    while ((b[0] | b[1] | b[2]) != 0) {
#pragma unroll
        for (int e = 0; e < 3; e++) {
            const int32_t q = (int32_t)__fdividef((float)a[e], (float)b[e]);
            int32_t r = a[e] - q * b[e];
            if (r < 0) r += b[e]; else if (r >= b[e]) r -= b[e];
            if (b[e] != 0) { a[e] = b[e]; b[e] = r; }
        }
    }
    return (uint32_t)((R.c[0] + R.c[1] + R.c[2] + a[0] + a[1] + a[2]) / 2 + 1) - R.right;
}

// The covered pixels of the warp's records whose box was cut (count 2; few
// are), one after the other, a lane a tile row; returns the lane's share.
__device__ __noinline__ uint32_t clipped_pixels(const BinWarp &S, uint32_t records)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t pixels = 0;
    for (uint32_t k = 0; k < records; k++) {
        const BinRec &r = S.rec[k];
        if (r.count != 2u) continue;
        for (uint32_t ty = (uint32_t)r.y0 / PF_TILE + lane; ty <= (uint32_t)r.y1 / PF_TILE; ty += 32u) {
            int32_t lo, hi;
            row_columns(r, ty, lo, hi);
            if (lo <= hi) pixels += row_pixels(r, ty, lo, hi);
        }
    }
    return pixels;
}

// Warp-cooperative binning of the lanes' sub-triangles: the tile rows of all
// of them are numbered through and each lane takes one, finding the run of
// tiles the sub-triangle may cover there; then the (row, tile) pairs of 32
// rows are numbered through and each lane takes one pair at a time.  So the
// work is even whatever the sub-triangles' sizes, and only tiles that get
// an entry are visited.  Bound by instruction issue and, in small launches,
// by the round trips of the counter atomics.  Testing every tile of the box
// instead, one sub-triangle after the other, a batch of 64 soups (207,000
// items covering hundreds of tiles each, 4.5 tiles tested per entry) took
// 614 us of k_items, now 312-326; phong1080, whose triangles cover one or two
// tiles, 286 -> 229 us; the 2,000-triangle soup at 256x256 136 -> 17 us
// together with the items a warp (pfd_launch_items).  Depth planes and
// fragment counts are in the new figures: they cost 5 us of the batch and 40
// of phong1080, and save k_raster 300 and 59 (queue_refill).  Pairs of one
// window of 32 that touch the same tile share one atomic on its counter
// (neighbouring triangles of a mesh usually do), slots within a group follow
// lane order; the pairs of a single sub-triangle are distinct tiles and skip
// the grouping.  The counters of BIN_BURST windows are claimed before any of
// their slots is written, so that the atomics' round trips overlap.
// Every lane of the warp must call it (lanes with nothing to bin pass
// has = false).
#define BIN_BURST 4
__device__ void bin_prim_warp(const BinArgs &B, const TileSpace &T, bool has, const PFPrim &P, bool on, uint32_t key, BinWarp &S)
{
    const uint32_t all = 0xffffffffu;
    uint32_t tx0 = 0, ty0 = 0, ntx = 1, nty = 0;
    if (has && !tile_range(T, P, tx0, ty0, ntx, nty)) nty = 0;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1, le = lt | (1u << lane);
    uint32_t rows;
    const uint32_t firstRow = warp_offsets(nty, rows);
    const uint32_t owners = __ballot_sync(all, nty > 0);
    bool counts = false;
    if (nty > 0) {
        // (16 bytes at a time as they are known: the record in registers
        // beside P would spill)
        int4 *q = reinterpret_cast<int4 *>(&S.rec[__popc(owners & lt)]);
        q[3] = make_int4(P.xMin, (int32_t)min((uint32_t)P.xMax, T.W) - 1, P.yMin, (int32_t)min((uint32_t)P.yMax, T.H - 1u));
        q[4] = make_int4(on, (int32_t)firstRow, (int32_t)T.tileBase, (int32_t)T.tilesX);
        if (P.flags & (PFP_KIND | PFP_COUNT)) {
            // no bound, nothing to count here
            const float inf = __int_as_float(0x7f800000);
            q[5] = make_int4((int32_t)key, 0, 0, 0);
            B.planes[key >> PF_SUB_BITS] = make_float4(inf, 0.0f, 0.0f, raises_depth(P.rstate) ? __int_as_float(0x7fffffff) : inf);
        } else {
            const bool r1 = P.x1 == P.xMax, r2 = P.x2 == P.xMax, r3 = P.x3 == P.xMax;
            const int32_t right = 1 + (r1 && r2 ? abs(P.y1 - P.y2) : r2 && r3 ? abs(P.y2 - P.y3) : r1 && r3 ? abs(P.y3 - P.y1) : 0);
            counts = true;
            q[5] = make_int4((int32_t)key, whole_box(P, T) ? 1 : 2, right, __float_as_int(P.z1));
            q[6] = make_int4(__float_as_int(P.z2), __float_as_int(P.z3), __float_as_int(P.wInvSum), __float_as_int(depth_bound(P)));
        }
        const EdgeTest E = edge_test(P, on);
        q[0] = make_int4(E.ex[0], E.ex[1], E.ex[2], E.ey[0]);
        q[1] = make_int4(E.ey[1], E.ey[2], E.c[0], E.c[1]);
        q[2] = make_int4(E.c[2], __float_as_int(__frcp_rn((float)E.ex[0])), __float_as_int(__frcp_rn((float)E.ex[1])),
                         __float_as_int(__frcp_rn((float)E.ex[2])));
    }
    __syncwarp();
    for (uint32_t r0 = 0; r0 < rows; r0 += 32u) {
        // my row: of the last sub-triangle whose first row is not past it
        BinRow w{ 0, 0, 0, 0 };
        uint32_t n = 0;
        {
            const uint32_t before = __popc(__ballot_sync(all, nty > 0 && firstRow < r0));
            const uint32_t heads = __reduce_or_sync(all, (nty > 0 && firstRow - r0 < 32u) ? 1u << (firstRow - r0) : 0u);
            if (r0 + lane < rows) {
                const BinRec &r = S.rec[before + __popc(heads & le) - 1u];
                const uint32_t ty = (uint32_t)r.y0 / PF_TILE + (r0 + lane - r.first);
                int32_t lo, hi;
                row_columns(r, ty, lo, hi);
                if (lo <= hi) {
                    n = (uint32_t)hi / PF_TILE - (uint32_t)lo / PF_TILE + 1u;
                    w.tile = r.tileBase + ty * r.tilesX + (uint32_t)lo / PF_TILE;
                }
                w.key = r.key;
            }
        }
        uint32_t total;
        w.first = warp_offsets(n, total);
        const uint32_t filled = __ballot_sync(all, n > 0);
        if (n > 0) S.row[__popc(filled & lt)] = w;
        __syncwarp();
        for (uint32_t p0 = 0; p0 < total; p0 += 32u * BIN_BURST) {
            uint32_t tt[BIN_BURST], gg[BIN_BURST], bb[BIN_BURST], kk[BIN_BURST];
#pragma unroll
            for (int u = 0; u < BIN_BURST; u++) {
                const uint32_t w0 = p0 + 32u * (uint32_t)u, p = w0 + lane;
                tt[u] = 0xffffffffu; gg[u] = 0; bb[u] = 0; kk[u] = 0;
                if (w0 >= total) continue;                     // uniform over the warp
                const uint32_t before = __popc(__ballot_sync(all, n > 0 && w.first < w0));
                const uint32_t heads = __reduce_or_sync(all, (n > 0 && w.first - w0 < 32u) ? 1u << (w.first - w0) : 0u);
                const BinRow q = S.row[before + __popc(heads & le) - 1u];    // (past the last pair: the last row)
                const bool act = p < total;
                const uint32_t t = act ? q.tile + (p - q.first) : 0xffffffffu;
                const uint32_t key0 = __shfl_sync(all, q.key, 0);
                const uint32_t grp = __all_sync(all, q.key == key0) ? 1u << lane : __match_any_sync(all, t);
                tt[u] = t; gg[u] = grp; kk[u] = q.key;
                if (act && lane == (uint32_t)(__ffs(grp) - 1)) bb[u] = atomicAdd(&B.binCount[t], (unsigned)__popc(grp));
            }
#pragma unroll
            for (int u = 0; u < BIN_BURST; u++) {
                if (p0 + 32u * (uint32_t)u >= total) continue;
                const uint32_t grp = gg[u], leader = (uint32_t)(__ffs(grp) - 1);
                const uint32_t base = __shfl_sync(all, bb[u], leader);
                const bool act = tt[u] != 0xffffffffu;
                list_tiles_warp(B, tt[u], base, act && lane == leader ? (uint32_t)__popc(grp) : 0u);
                if (act) bin_slot(B, tt[u], base + __popc(grp & lt), kk[u]);
            }
        }
        __syncwarp();                                          // the rows are free
    }
    // the depth planes and the fragments, once the entries are on their way
    // (read back from shared memory: held through the loops above they
    // would spill)
    if (!__any_sync(all, counts)) return;
    const uint32_t records = __popc(__ballot_sync(all, nty > 0));
    uint32_t count = 0, pixels = 0;
    if (lane < records) {
        const BinRec &r = S.rec[lane];
        count = r.count;
        if (count) B.planes[r.key >> PF_SUB_BITS] = depth_plane(r);
        if (count == 1u) pixels = lattice_pixels(r);
    }
    if (__any_sync(all, count == 2u)) pixels += clipped_pixels(S, records);
    pixels = __reduce_add_sync(all, pixels);
    if (lane == 0 && pixels) atomicAdd(&B.cnt->batchFragments, (unsigned long long)pixels);
}

__device__ __forceinline__ void store_phong(PFPrimPhong *dst, const SVert &a, const SVert &b, const SVert &c)
{
    PFPrimPhong q;
    for (int i = 0; i < 3; i++) {
        q.n1[i] = a.n[i]; q.n2[i] = b.n[i]; q.n3[i] = c.n[i];
        q.p1[i] = a.p[i]; q.p2[i] = b.p[i]; q.p3[i] = c.p[i];
    }
    q.pad[0] = q.pad[1] = 0.0f;
    *dst = q;
}

__device__ __forceinline__ void item_vertices(const PFSegment &sg, uint32_t k, uint32_t v[3], int &face, unsigned *status)
{
    uint32_t s[3];
    if (sg.itemKind == PF_ITEMS_TRIS) {
        uint32_t tri = (sg.nFaces == 2) ? (k >> 1) : k;
        face = (sg.nFaces == 2) ? (int)(k & 1) : sg.face0;
        s[0] = 3 * tri; s[1] = 3 * tri + 1; s[2] = 3 * tri + 2;
    } else {
        const int4 e = reinterpret_cast<const int4 *>(sg.explicitItems)[k];
        s[0] = (uint32_t)e.x; s[1] = (uint32_t)e.y; s[2] = (uint32_t)e.z; face = e.w;
    }
    for (int m = 0; m < 3; m++) {
        uint32_t j = sg.idx ? __ldg(sg.idx + s[m]) : s[m];
        if (j >= sg.nVerts) {                          // the host sizes nVerts from the indices, except for
            j = sg.nVerts - 1;                         // device indices (pfDrawElementsDevice): clamped, flagged
            atomicOr(status, (unsigned)PFD_BOUNDS);
        }
        v[m] = sg.vtxRead + j;
    }
}

// ---------------------------------------------------------------------------
// polygon clipping (triangles.c:157-280), for the rare items that cross a
// clip plane; called out of line from k_items
// ---------------------------------------------------------------------------
struct CVert { float h[4]; float pos[4]; float n[3]; float uv[2]; uint32_t c; };

// pfiLerpVertex (internal/context/context.c:67-90)
__device__ void lerp_vert(CVert &r, const CVert &s, const CVert &e, float t)
{
    uint32_t uT = x86_ftoub(255.0f * t);
    r.c = 0;
    for (int i = 0; i < 4; i++) {
        r.h[i] = s.h[i] + t*(e.h[i] - s.h[i]);
        r.pos[i] = s.pos[i] + t*(e.pos[i] - s.pos[i]);
        int32_t sc = (int32_t)chn(s.c, i), ec = (int32_t)chn(e.c, i);
        r.c |= ((uint32_t)(sc + ((int32_t)uT * (ec - sc)) / 255) & 255u) << (8 * i);
    }
    r.uv[0] = s.uv[0] + t*(e.uv[0] - s.uv[0]);
    r.uv[1] = s.uv[1] + t*(e.uv[1] - s.uv[1]);
    for (int i = 0; i < 3; i++) r.n[i] = s.n[i] + t*(e.n[i] - s.n[i]);
}

__device__ int clip_plane(CVert *poly, int n, CVert *tmp, int ax, int sign)
{
    // sign 0: w clip (w < eps is outside); sign +1: h[ax] <= w; sign -1: -h[ax] <= w
    for (int i = 0; i < n; i++) tmp[i] = poly[i];
    int m = 0;
    int prev = n - 1;
    auto inside = [&](const CVert &v) -> int {
        if (sign == 0) return (v.h[3] < 1e-5f) ? -1 : 1;
        if (sign > 0) return (v.h[ax] <= v.h[3]) ? 1 : -1;
        return (-v.h[ax] <= v.h[3]) ? 1 : -1;
    };
    int pd = inside(tmp[prev]);
    for (int i = 0; i < n; i++) {
        int cd = inside(tmp[i]);
        if (pd * cd < 0 && m < PF_CLIP_MAXV) {
            const CVert &p = tmp[prev], &c = tmp[i];
            float t;
            if (sign == 0) t = (1e-5f - p.h[3]) / (c.h[3] - p.h[3]);
            else if (sign > 0) t = (p.h[3] - p.h[ax]) / ((p.h[3] - p.h[ax]) - (c.h[3] - c.h[ax]));
            else t = (p.h[3] + p.h[ax]) / ((p.h[3] + p.h[ax]) - (c.h[3] + c.h[ax]));
            lerp_vert(poly[m++], p, c, t);
        }
        if (cd > 0 && m < PF_CLIP_MAXV) poly[m++] = tmp[i];
        pd = cd; prev = i;
    }
    return m;
}

struct ItemOut {
    PFPrim *prims;
    PFPrimPhong *primsPh;
    PFPrim *pool;
    PFPrimPhong *poolPh;
    uint32_t poolCap;
    uint64_t *rowInfo;          // launches with a row-rasterized target: per item, row_info (null otherwise)
    uint64_t *rowGroup;         // and per 32 items (a k_items warp), the rows their records span
};
static_assert(PF_MAX_SUBTRIS <= 16, "an item's sub-triangles are the bits of a 16-bit mask");

// What k_rows needs to know of an item without reading its records: bit s
// (s < 16) set when sub-triangle s has a record that draws something, and
// the first and last framebuffer row of those records (24 bits each, at
// bits 16 and 40; rows are unsigned, as tile_edge reads a box).
__device__ __forceinline__ void row_info_add(uint64_t &info, uint32_t sub, const PFPrim &P)
{
    const uint32_t xMin = (uint32_t)P.xMin, xMax = (uint32_t)P.xMax, lo = (uint32_t)P.yMin, hi = (uint32_t)P.yMax;
    if (xMin >= xMax || lo > hi || hi == 0xffffffffu) return;           // an empty box: nothing drawn
    uint64_t l = min(lo, 0xffffffu), h = min(hi, 0xffffffu);
    if (info & 0xffffu) { l = min(l, (info >> 16) & 0xffffffu); h = max(h, info >> 40); }
    info = (info & 0xffffu) | (1ull << sub) | (l << 16) | (h << 40);
}
// The rows spanned by the records of a warp's 32 items (row_info words w of
// its lanes, 0 past the end): bit 0 set when there is any, the first and
// last row at bits 16 and 40.
__device__ __forceinline__ uint64_t row_group(uint64_t w)
{
    const bool any = (w & 0xffffu) != 0;
    uint32_t lo = any ? (uint32_t)((w >> 16) & 0xffffffu) : 0xffffffu, hi = any ? (uint32_t)(w >> 40) : 0u;
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    return __any_sync(0xffffffffu, any) ? (1ull | (uint64_t)lo << 16 | (uint64_t)hi << 40) : 0ull;
}

// rowInfo[g] of an item whose only record is P (kept) or that has none.
// (In line: taking the record's address would keep it in local memory.)
__device__ __forceinline__ void store_row_info(uint64_t *rowInfo, uint32_t g, const PFPrim &P, bool kept)
{
    uint64_t rows = 0;
    if (kept) row_info_add(rows, 0, P);
    rowInfo[g] = rows;
}

__device__ __noinline__ void clip_item(const PFDrawState &S, int stateIdx, const PFVertexOut *const *V, int face,
                                       uint32_t g, const ItemOut &O, const BinArgs &B, const TileSpace &T)
{
    CVert poly[PF_CLIP_MAXV], tmp[PF_CLIP_MAXV];
    if (O.rowInfo) O.rowInfo[g] = 0;
    for (int m = 0; m < 3; m++) {
        const PFVertexOut &o = *V[m];
        for (int i = 0; i < 4; i++) poly[m].h[i] = o.h[i];
        poly[m].pos[0] = o.p[0]; poly[m].pos[1] = o.p[1]; poly[m].pos[2] = o.p[2];
        poly[m].pos[3] = 1.0f;     // object-space w is not read after clipping
        for (int i = 0; i < 3; i++) poly[m].n[i] = o.n[i];
        poly[m].uv[0] = o.uv[0]; poly[m].uv[1] = o.uv[1];
        poly[m].c = o.col[face];
    }
    int n = clip_plane(poly, 3, tmp, 3, 0);
    for (int ax = 0; ax < 3 && n > 0; ax++) {
        n = clip_plane(poly, n, tmp, ax, +1);
        if (n == 0) break;
        n = clip_plane(poly, n, tmp, ax, -1);
    }
    if (n < 3) return;
    SVert s[PF_CLIP_MAXV];
    for (int i = 0; i < n; i++) {
        float hz = __frcp_rn(poly[i].h[2]);
        s[i].u = poly[i].uv[0] * hz; s[i].v = poly[i].uv[1] * hz;
        float invW = __frcp_rn(poly[i].h[3]);
        to_screen(S, poly[i].h[0] * invW, poly[i].h[1] * invW, s[i].sx, s[i].sy);
        s[i].z = hz;
        s[i].c = poly[i].c;
        for (int k = 0; k < 3; k++) { s[i].n[k] = poly[i].n[k]; s[i].p[k] = poly[i].pos[k]; }
    }
    const int nsub = n - 2;
    uint32_t base = 0;
    if (nsub > 1) {
        base = atomicAdd(&B.cnt->clipCount, (unsigned)(nsub - 1));
        if (base + (uint32_t)(nsub - 1) > O.poolCap) {
            atomicOr(&B.cnt->status, (unsigned)PFD_CLIP_OVERFLOW);
            atomicMin(&B.cnt->abortCommand, B.command);
            return;
        }
    }
    PFPrim first;
    bool firstSet = false;
    uint64_t rows = 0;
    for (int i = 0; i < nsub; i++) {
        PFPrim P;
        if (!setup_prim(S, face, true, s[0], s[i + 1], s[i + 2], stateIdx, P)) continue;
        P.flags |= PFP_COUNT;
        row_info_add(rows, (uint32_t)i, P);
        atomicAdd(&B.cnt->batchRasterized, 1ull);
        if (i == 0) { first = P; firstSet = true; }
        else {
            O.pool[base + i - 1] = P;
            if (S.flags & PFS_PHONG) store_phong(&O.poolPh[base + i - 1], s[0], s[i + 1], s[i + 2]);
        }
        bin_prim(B, T, P, (g << PF_SUB_BITS) | (uint32_t)i);
    }
    // prims[g] carries the pool base of sub-triangles >= 1 even when
    // sub-triangle 0 was culled.
    if (!firstSet) { first.flags = 0; first.xMin = 1; first.xMax = 0; }
    first.poolBase = (int32_t)base;
    O.prims[g] = first;
    {
        const float inf = __int_as_float(0x7f800000);      // (its pieces have no bound)
        B.planes[g] = make_float4(inf, 0.0f, 0.0f, raises_depth(raster_state(S)) ? __int_as_float(0x7fffffff) : inf);
    }
    if (O.rowInfo) O.rowInfo[g] = rows;
    if (firstSet && (S.flags & PFS_PHONG)) store_phong(&O.primsPh[g], s[0], s[1], s[2]);
}

// ---------------------------------------------------------------------------
// k_items: one thread per triangle-face item, in submission order
// ---------------------------------------------------------------------------
// Project, clip if needed and set up item g.  Returns true when its
// unclipped sub-triangle survived culling and must be binned by the caller
// (clipped items bin their sub-triangles themselves).
__device__ __forceinline__ bool item_setup(const PFSegment &sg, const PFDrawState *sState,
                                           const PFDrawState *__restrict__ states,
                                           const PFVertexOut *__restrict__ vout, uint32_t g, const ItemOut &O,
                                           const BinArgs &B, const TileSpace &T, PFPrim &P, bool &on)
{
    const PFDrawState &S = sState ? *sState : states[sg.state];
    const uint32_t k = g - sg.itemBase + sg.itemSkip;
    if (sg.itemKind == PF_ITEMS_EXPLICIT && reinterpret_cast<const int4 *>(sg.explicitItems)[k].w < 0) {
        // a point or a line set up on the host: its record, under this draw state
        const uint32_t r = (uint32_t)reinterpret_cast<const int4 *>(sg.explicitItems)[k].x;
        P = static_cast<const PFPrim *>(sg.prebuilt)[r];
        P.flags = (P.flags & 0xffu) | ((uint32_t)sg.state << 8);
        // its own depth test, blending and depth write stand in for the
        // state's (a thick line's centre is always tested; pfRectf does none)
        P.rstate = (raster_state(S) & ~(uint32_t)PFP_OPS) | (P.flags & PFP_OPS);
        P.zReject = __int_as_float(0x7fffffff);
        O.prims[g] = P;
        if (O.rowInfo) store_row_info(O.rowInfo, g, P, true);
        return true;
    }
    uint32_t vi[3]; int face;
    item_vertices(sg, k, vi, face, &B.cnt->status);
    const PFVertexOut *V[3] = { &vout[vi[0]], &vout[vi[1]], &vout[vi[2]] };
    float4 hv[3];
    for (int m = 0; m < 3; m++) hv[m] = *reinterpret_cast<const float4 *>(V[m]->h);
    float ws = 0.0f;
    for (int m = 0; m < 3; m++) ws += hv[m].w;
    const bool is2D = fabsf(ws - 3.0f) < 1e-5f;
    if (!is2D) {
        bool inside = true;
        for (int m = 0; m < 3; m++) {
            const float4 h = hv[m];
            inside = inside && !(h.w < 1e-5f) && (h.x <= h.w) && (-h.x <= h.w) && (h.y <= h.w) && (-h.y <= h.w) &&
                     (h.z <= h.w) && (-h.z <= h.w);
        }
        if (!inside) { clip_item(S, sg.state, V, face, g, O, B, T); return false; }
    }
    SVert s[3];
    for (int m = 0; m < 3; m++) {
        // (the vertex's other three 16-byte words: uv and colours, normal and
        // position)
        const float4 *vw = reinterpret_cast<const float4 *>(V[m]);
        const float4 h = hv[m], uv = vw[1];
        if (is2D) {
            to_screen(S, h.x, h.y, s[m].sx, s[m].sy);
            s[m].z = h.z; s[m].u = uv.x; s[m].v = uv.y;
        } else {
            float hz = __frcp_rn(h.z);
            s[m].u = uv.x * hz; s[m].v = uv.y * hz;
            float invW = __frcp_rn(h.w);
            to_screen(S, h.x * invW, h.y * invW, s[m].sx, s[m].sy);
            s[m].z = hz;
        }
        s[m].c = __float_as_uint(face ? uv.w : uv.z);
        if (S.flags & PFS_PHONG) {
            const float4 np = vw[2];
            const float2 pp = *reinterpret_cast<const float2 *>(vw + 3);
            s[m].n[0] = np.x; s[m].n[1] = np.y; s[m].n[2] = np.z;
            s[m].p[0] = np.w; s[m].p[1] = pp.x; s[m].p[2] = pp.y;
        }
    }
    const bool kept = setup_prim(S, face, !is2D, s[0], s[1], s[2], sg.state, P);
    if (O.rowInfo) store_row_info(O.rowInfo, g, P, kept);
    if (!kept) return false;
    // Who counts the record's covered pixels: k_raster, visiting them, where
    // the edge functions may wrap, where k_rows draws, and for triangles
    // within 32x32 pixels of launches with fewer than 8 items a tile, whose
    // tiles seldom hold a second batch to drop records from (with a limit of
    // 8x8 pixels sphere1080's k_items took 22.6 us, now 21.3; without
    // counting 20.0); the others here.
    on = edge_on(P, T.W, T.H);
    if (T.rows || !on || (!B.countSmall && P.xMax - P.xMin <= 4 * PF_TILE && P.yMax - P.yMin < 4 * PF_TILE)) P.flags |= PFP_COUNT;
    O.prims[g] = P;
    if (S.flags & PFS_PHONG) store_phong(&O.primsPh[g], s[0], s[1], s[2]);
    return true;
}
__global__ void __launch_bounds__(128, 6) k_items(const PFSegment *__restrict__ segs, int nSegs, const PFDrawState *__restrict__ states,
                        const PFVertexOut *__restrict__ vout, uint32_t nItems, uint32_t perWarp, ItemOut O, BinArgs B)
{
    __shared__ int sUniform, sAborted;
    __shared__ BinWarp sBin[4];
    // a warp's first perWarp lanes set up an item each, all of its lanes bin
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t g0 = blockIdx.x * 4u * perWarp;
    const uint32_t g = lane < perWarp ? g0 + warp * perWarp + lane : 0xffffffffu;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // k_vertex is done
    // Thread 0 takes the block's decisions, behind one barrier: whether an
    // overflow in this launch has flagged the abort (other blocks set it
    // while this one runs; a thread that returned alone would leave the rest
    // of the block with unset shared state), and the segment of the block's
    // items when they share one (the usual case; the others search).
    if (threadIdx.x == 0) {
        sAborted = B.cnt->abortCommand != 0xffffffffu;
        const int a = seg_of_item(segs, nSegs, g0), b = seg_of_item(segs, nSegs, min(g0 + 4u * perWarp, nItems) - 1);
        sUniform = (a == b) ? a : -1;
    }
    __syncthreads();
    if (sAborted) return;
    const int su = sUniform;
    // every lane stays to the end: binning below is warp-cooperative
    PFPrim P;
    bool kept = false, on = false;
    TileSpace T{ 0, 0, 0, 0, false };
    if (g < nItems) {
        // the segment and its draw state are read in place (one address for
        // the block: L1 serves it after the first access)
        const PFSegment &sg = segs[su >= 0 ? su : seg_of_item(segs, nSegs, g)];
        T = tile_space(B, sg.target);
        kept = item_setup(sg, nullptr, states, vout, g, O, B, T, P, on);
    }
    // one counter update per warp, its result unused (a reduction in L2, no
    // round trip, no block barrier)
    const unsigned wk = __popc(__ballot_sync(0xffffffffu, kept));
    if ((threadIdx.x & 31) == 0 && wk) atomicAdd(&B.cnt->batchRasterized, (unsigned long long)wk);
    if (O.rowInfo) {                                   // the warp's summary for k_rows (perWarp is 32)
        const uint64_t grp = row_group(g < nItems ? O.rowInfo[g] : 0ull);
        if ((threadIdx.x & 31) == 0) O.rowGroup[g >> 5] = grp;
    }
    bin_prim_warp(B, T, kept, P, on, g << PF_SUB_BITS, sBin[warp]);
}

// ---------------------------------------------------------------------------
// k_binsort and k_raster
//
// k_items appends a tile's bin entries (order keys item << 4 | sub-triangle)
// in atomic order.  k_binsort puts every bin that reached REG_SORT_MAX
// entries back into submission order, in place (one CTA per bin); shorter
// bins are sorted by the rasterizing warp itself, in registers.
//
// k_raster: one warp per 8x8 tile, two pixels per lane, warps independent
// of each other (a CTA only groups four of them).  A warp takes a tile from
// the work queue and walks its bin in batches of 32 sub-triangles in
// submission order:
//   1. every lane loads one record of the batch into the warp's shared
//      memory and derives its edge functions at the tile origin and its
//      bounding box clipped to the tile (from the second batch on, records
//      that lie behind every pixel of the tile do not get into a batch);
//   2. each lane walks the records in order at its own two pixels: coverage
//      with the reference's integer edge functions, depth, depth test and
//      depth write (triangles.c:398-438) -- which leaves, per pixel, the
//      fragments that passed and are not replaced by a later unblended one
//      (bit k of a 32-bit mask: the record's place in the batch);
//   3. the passing fragments are listed pixel by pixel in submission order
//      and shaded densely over the warp (texture, Gouraud / Phong colour:
//      the source colour does not depend on the destination);
//   4. every pixel blends its listed fragments in order into its colour,
//      held in registers with its depth for the whole tile.
// ---------------------------------------------------------------------------
// k_raster's CTAs group 2, 4 or 8 independent warps (the block shape, a
// tuning knob); each warp owns one tile at a time
#define QCHN 32                     // records per batch (bit k of a pixel's 32-bit masks)
// work-queue entries of a half tile: the tile index with one of these set
#define TILE_TOP 0x40000000u
#define TILE_BOTTOM 0x60000000u
#define TILE_HALF_MASK 0x60000000u
#define QFW 128                     // fragment window of a warp
#define SORT_THREADS 256
#define REG_SORT_MAX 128            // bins shorter than this are sorted by the raster warp (four keys a lane)
#define REG_SORT_LEVEL 2            // the heavy-level list of bins that reached REG_SORT_MAX entries

static_assert(PF_TILE == 8 && PF_TILE_PIXELS == 64, "a warp owns a tile: two pixels per lane");
static_assert(REG_SORT_MAX == (PF_HEAVY_BASE << (2 * (REG_SORT_LEVEL - 1))), "k_binsort takes one heavy-level list");

struct RasterArgs {
    const uint32_t *binCount;
    const uint32_t *tileList;
    uint32_t listStride;
    uint32_t *bins;
    uint32_t cap;
    const PFPrim *prims;
    const PFPrimPhong *primsPh;
    const float4 *planes;
    const PFPrim *pool;
    const PFPrimPhong *poolPh;
    const PFDrawState *states;
    const PFTarget *targets;
    int nTargets;
    uint32_t totalTiles;
    PFDevCounters *cnt;
    uint32_t command;
    int anyPhong;
    uint32_t sortGroups;       // k_binsort: groups of 128 items in a warp's item map, 0: no maps
};

// A batch record in shared memory, padded to 144 bytes: lane i's record
// starts 4 banks after lane i-1's, so 16-byte accesses of the records of 8
// lanes touch all 32 banks once (with 128 bytes they would all start in
// bank 0).
struct __align__(16) SPrim {
    PFPrim p;
    const PFPrimPhong *ph;     // its per-fragment lighting record (read when a fragment is shaded)
    uint64_t pad;
};

// A batch record's coverage view, three 16-byte words: edge functions at the
// tile origin and their x / y steps, the box clipped to the tile
// (x0 | width << 4 | y0 << 8 | height << 12) with the record's kind above
// (bits 16-17), the raster state and the depth-test rejection bound.
struct __align__(16) QEdge {
    int32_t e0[3], ex0;
    int32_t ex1, ex2, ey0, ey1;
    int32_t ey2;
    uint32_t box, rstate;
    float zReject;             // every covered fragment fails the depth test when zReject >= depth (NaN: never)
};

#define QE_COUNT (1u << 18)     // of box: k_raster counts the record's fragments (k_items has not; rectangles have none)

// Shared memory of one warp.
struct QWarp {
    SPrim rec[QCHN];
    QEdge edge[QCHN];
    uint32_t keys[REG_SORT_MAX];   // the queue of the next keys; a short bin's further ones, sorted in registers
    uint32_t pend[PF_TILE_PIXELS]; // per pixel (32 slot + lane) the bin key of its fragment that waits to be shaded
    uint16_t fdesc[QFW];       // listed fragments: tile pixel << 5 | record
    uint32_t fc[QFW];          // their colour
    uint32_t queued, lowering; // queue_refill: keys in the queue; no key so far may raise a depth
    uint32_t pad[2];
};

// Edge set-up of a record (its first three 16-byte words: x1 y1 x2 y2 |
// x3 y3 xMin yMin | xMax yMax flags -) for the tile at (ox, oy) of a W x H
// framebuffer (triangles.c:336-349, 398-420: the integer edge functions,
// stepped from the tile origin).
__device__ __forceinline__ void tile_edge(const int4 q0, const int4 q1, const int4 q2, uint32_t rstate, float zReject,
                                          uint32_t ox, uint32_t oy, uint32_t W, uint32_t H, QEdge &E)
{
    const int32_t X1 = q0.x, Y1 = q0.y, X2 = q0.z, Y2 = q0.w, X3 = q1.x, Y3 = q1.y;
    const uint32_t xMin = (uint32_t)q1.z, yMin = (uint32_t)q1.w, xMax = (uint32_t)q2.x, yMax = (uint32_t)q2.y;
    const uint32_t flags = (uint32_t)q2.z, face = flags & 1u;
    int32_t sx[3] = { Y3 - Y2, Y1 - Y3, Y2 - Y1 };
    int32_t sy[3] = { X2 - X3, X3 - X1, X1 - X2 };
    const int32_t rx[3] = { X2, X3, X1 }, ry[3] = { Y2, Y3, Y1 };
    int32_t e0[3];
    for (int e = 0; e < 3; e++) {
        if (face) { sx[e] = -sx[e]; sy[e] = -sy[e]; }
        e0[e] = (int32_t)((ox - (uint32_t)rx[e]) * (uint32_t)sx[e] + (oy - (uint32_t)ry[e]) * (uint32_t)sy[e]);
    }
    // pixels x in [xMin, xMax), y in [yMin, yMax] (unsigned), inside the tile and the framebuffer
    const uint32_t x0 = max(xMin, ox), x1 = min(min(xMax, ox + PF_TILE), W);
    const uint32_t y0 = max(yMin, oy);
    uint32_t y1e = min(min(yMax + 1u, oy + PF_TILE), H);
    if (yMax == 0xffffffffu) y1e = 0;                  // yMax + 1 wrapped
    const bool empty = (x0 >= x1) || (y0 >= y1e) || (xMin >= xMax) || (yMin > yMax);
    const uint32_t bx0 = empty ? 0 : x0 - ox, by0 = empty ? 0 : y0 - oy;
    const uint32_t bw = empty ? 0 : x1 - x0, bh = empty ? 0 : y1e - y0;
    E.e0[0] = e0[0]; E.e0[1] = e0[1]; E.e0[2] = e0[2];
    E.ex0 = sx[0]; E.ex1 = sx[1]; E.ex2 = sx[2];
    E.ey0 = sy[0]; E.ey1 = sy[1]; E.ey2 = sy[2];
    E.box = bx0 | (bw << 4) | (by0 << 8) | (bh << 12) | (((flags & PFP_KIND) >> 6) << 16) |
            (((flags & PFP_KIND) ? (flags & PFP_KIND) != PFP_BLIT : (flags & PFP_COUNT) != 0) ? QE_COUNT : 0u);
    E.rstate = rstate;
    E.zReject = zReject;
}

// Order-preserving integer key of a depth: keys compare as the depths do,
// NaN above everything.
__device__ __forceinline__ uint32_t depth_key(float d)
{
    const uint32_t u = (uint32_t)__float_as_int(d);
    return d != d ? 0xffffffffu : u ^ ((int32_t)u < 0 ? 0xffffffffu : 0x80000000u);
}

// Normalised weights and depth of a covered fragment at tile pixel (X, Y)
// (triangles.c:421-438).
__device__ __forceinline__ float tile_depth(const QEdge &E, const PFPrim &P, uint32_t X, uint32_t Y, float *wn)
{
    const int32_t w1 = (int32_t)((uint32_t)E.e0[0] + X * (uint32_t)E.ex0 + Y * (uint32_t)E.ey0);
    const int32_t w2 = (int32_t)((uint32_t)E.e0[1] + X * (uint32_t)E.ex1 + Y * (uint32_t)E.ey1);
    const int32_t w3 = (int32_t)((uint32_t)E.e0[2] + X * (uint32_t)E.ex2 + Y * (uint32_t)E.ey2);
    wn[0] = (float)w1 * P.wInvSum; wn[1] = (float)w2 * P.wInvSum; wn[2] = (float)w3 * P.wInvSum;
    float zs = P.z1 * wn[0] + P.z2 * wn[1];
    zs = zs + P.z3 * wn[2];
    return __frcp_rn(zs);          // 1 / zs, correctly rounded
}

// Source colour of one fragment (triangles.c:500-521): colour interpolation,
// texturing, per-fragment lighting.  Independent of the destination pixel.
// texOn false: a pixel outside the mask, whose texture coordinates the
// reference replaces by zero before sampling (triangles.c:508-513);
// anyWeights: the pixel may lie outside the triangle (weights outside
// [0, 1]), so the weight conversions follow CVTPS2DQ out of range too.
template <bool PHONG>
__device__ __forceinline__ uint32_t shade_fragment(const PFPrim &P, const PFPrimPhong *Q, const PFDrawState *states,
                                                   float wn1, float wn2, float wn3, float z,
                                                   bool texOn = true, bool anyWeights = false)
{
    const uint32_t fl = P.rstate;
    uint32_t frag;
    if (fl & PFS_SMOOTH) {
        // covered pixels have weights in [0, 1]: the conversions are in range
        const float s1 = wn1 * 255.0f, s2 = wn2 * 255.0f, s3 = wn3 * 255.0f;
        const uint32_t u1 = anyWeights ? pff_cvt_rne(s1) : (uint32_t)__float2int_rn(s1);
        const uint32_t u2 = anyWeights ? pff_cvt_rne(s2) : (uint32_t)__float2int_rn(s2);
        const uint32_t u3 = anyWeights ? pff_cvt_rne(s3) : (uint32_t)__float2int_rn(s3);
        int32_t o[4];
        for (int i = 0; i < 4; i++) {
            uint32_t s = u1 * chn(P.c1, i) + u2 * chn(P.c2, i);
            s = s + u3 * chn(P.c3, i);
            o[i] = (int32_t)((s * 257u) >> 16);
        }
        frag = pack4(o);
    } else {
        const float mx = x86_max(wn1, x86_max(wn2, wn3));
        frag = ((mx == wn1) ? P.c1 : 0u) | (((mx == wn2) ? P.c2 : 0u) | ((mx == wn3) ? P.c3 : 0u));
    }
    if (fl & PFS_TEXTURE) {
        float tu = 0.0f, tv = 0.0f;
        if (texOn) {
            tu = P.u1 * wn1 + P.u2 * wn2;
            tu = tu + P.u3 * wn3;
            tv = P.v1 * wn1 + P.v2 * wn2;
            tv = tv + P.v3 * wn3;
            if (P.flags & 2) { tu = tu * z; tv = tv * z; }
        }
        frag = blend_simd(4, tex_sample(tex_desc(P, states), tu, tv), frag);
    }
    if (PHONG && (fl & PFS_PHONG)) {
        const PFDrawState &S = states[P.flags >> 8];
        PFPrimPhong q;                                  // (80 bytes, five 16-byte loads)
        for (int i = 0; i < 5; i++) reinterpret_cast<float4 *>(&q)[i] = __ldg(reinterpret_cast<const float4 *>(Q) + i);
        float N[3], Pp[3];
        for (int i = 0; i < 3; i++) {
            float t0 = q.n1[i] * wn1 + q.n2[i] * wn2; N[i] = t0 + q.n3[i] * wn3;
            float t1 = q.p1[i] * wn1 + q.p2[i] * wn2; Pp[i] = t1 + q.p3[i] * wn3;
        }
        frag = light_phong(S, frag, S.mat[P.flags & 1], Pp, N);
    }
    return frag;
}

// ---------------------------------------------------------------------------
// points and lines (src/internal/primitives/points.c, lines.c), set up on
// the host into PFPrim records:
//   line   x1, y1 first pixel; x2 endVal (signed pixel count along the long
//          axis); y2 decInc (16.16 step of the short axis); x3 sgnInc;
//          wInvSum 1 / endVal; z1, z2 and c1, c2 at the ends
//   point  x1, y1 centre; x2 radius in pixels (-1: the single centre
//          pixel); wInvSum the squared radius; z1, c1
// Pixels are absolute framebuffer coordinates.  These run out of line: the
// triangle path stays free of their registers.
// ---------------------------------------------------------------------------
__device__ __noinline__ bool lp_covers(const PFPrim &P, int32_t X, int32_t Y)
{
    if ((P.flags & PFP_KIND) == PFP_BLIT) return true;          // every pixel of its box
    if ((P.flags & PFP_KIND) == PFP_POINT) {                     // points.c:106-183
        const int32_t dx = X - P.x1, dy = Y - P.y1;
        if (P.x2 < 0) return dx == 0 && dy == 0;
        if (dx < -P.x2 || dx > P.x2 || dy < -P.x2 || dy > P.x2) return false;
        return (float)(dy * dy + dx * dx) <= P.wInvSum;
    }
    // lines.c:304-431: step i of the DDA lands on long-axis coordinate a1 + i
    const bool yl = (P.flags & PFP_Y_LONGER) != 0;
    const int32_t a = yl ? Y : X, b = yl ? X : Y, a1 = yl ? P.y1 : P.x1, b1 = yl ? P.x1 : P.y1;
    const uint32_t k = ((uint32_t)a - (uint32_t)a1) * (uint32_t)P.x3;          // steps taken
    const uint32_t steps = P.x2 < 0 ? 0u - (uint32_t)P.x2 : (uint32_t)P.x2;
    if (k >= steps) return false;
    const int32_t j = (int32_t)(k * (uint32_t)P.y2);
    return (uint32_t)b == (uint32_t)b1 + (uint32_t)(j >> 16);
}

// Interpolation parameter of a line pixel: t = i / endVal (lines.c:366).
__device__ __forceinline__ float lp_t(const PFPrim &P, int32_t X, int32_t Y)
{
    const bool yl = (P.flags & PFP_Y_LONGER) != 0;
    const int32_t i = (int32_t)((uint32_t)(yl ? Y : X) - (uint32_t)(yl ? P.y1 : P.x1));
    return (float)i * P.wInvSum;
}

// (PFsizei)(float) as the reference's x86-64 build converts it: a 64-bit
// truncating conversion whose low 32 bits are kept; 0 for NaN / out of range.
__device__ __forceinline__ uint32_t x86_ftou32(float x)
{
    if (!(x > -9.2e18f && x < 9.2e18f)) return 0u;
    return (uint32_t)(unsigned long long)__float2ll_rz(x);
}

// A pfRectf record's colour, or the pfDrawPixels source pixel that lands on
// (X, Y) (context.c:2044-2082): x1, y1 the raster position on screen, x2 the
// image width, y2 / x3 width - 1 / height - 1, wInvSum / z2 the inverse
// zoomed width / height.  Elements past the image read as 0.
__device__ __forceinline__ uint32_t blit_color(const PFPrim &P, int32_t X, int32_t Y)
{
    if (!P.src) return P.c1;
    const float v = (float)(int32_t)((uint32_t)Y - (uint32_t)P.y1) * P.z2;
    const uint32_t ySrc = x86_ftou32(v * (float)(uint32_t)P.x3) * (uint32_t)P.x2;
    const float u = (float)(int32_t)((uint32_t)X - (uint32_t)P.x1) * P.wInvSum;
    const uint32_t o = ySrc + x86_ftou32(u * (float)(uint32_t)P.y2);
    return o < P.nSrc ? __ldg(reinterpret_cast<const uint32_t *>(P.src) + o) : 0u;
}

__device__ __noinline__ float lp_depth(const PFPrim &P, int32_t X, int32_t Y)
{
    if ((P.flags & PFP_KIND) != PFP_LINE) return P.z1;
    const float t = lp_t(P, X, Y);
    return P.z1 + t * (P.z2 - P.z1);
}

// pfiColorLerpSmooth (src/internal/color.h): (PFubyte)(a + t (b - a)) per channel
__device__ __noinline__ uint32_t lp_color(const PFPrim &P, int32_t X, int32_t Y)
{
    if ((P.flags & PFP_KIND) == PFP_POINT) return P.c1;
    if ((P.flags & PFP_KIND) == PFP_BLIT) return blit_color(P, X, Y);
    const float t = lp_t(P, X, Y);
    int32_t o[4];
    for (int i = 0; i < 4; i++) {
        const int32_t a = (int32_t)chn(P.c1, i), b = (int32_t)chn(P.c2, i);
        o[i] = x86_cvt_trunc((float)a + t * (float)(b - a)) & 255;
    }
    return pack4(o);
}

// Scalar depth test of points and lines (src/internal/depth.h:27-74):
// NOTEQUAL is a real !=.
__device__ __forceinline__ bool depth_sisd(int f, float src, float dst)
{
    switch (f) {
    case 0: return src == dst;                                   // EQUAL
    case 1: return src != dst;                                   // NOTEQUAL
    case 2: return src < dst;                                    // LESS
    case 3: return src <= dst;                                   // LEQUAL
    case 4: return src > dst;                                    // GREATER
    default: return src >= dst;                                  // GEQUAL
    }
}

// Scalar blending of points and lines (src/internal/blend.h:27-126): SUB
// subtracts, MUL divides by 255, ALPHA weighs with a + 1.
__device__ __noinline__ uint32_t blend_sisd(int mode, uint32_t src, uint32_t dst)
{
    int32_t o[4];
    for (int i = 0; i < 4; i++) {
        const int32_t s = (int32_t)chn(src, i), d = (int32_t)chn(dst, i);
        int32_t v;
        switch (mode) {
        case 0: v = (s + d) >> 1; break;                         // AVERAGE
        case 1: {                                                // ALPHA
            const uint32_t al = chn(src, 3) + 1u, ia = 256u - al;
            v = (int32_t)((al * (uint32_t)(i == 3 ? 255 : s) + ia * (uint32_t)d) >> 8);
            break;
        }
        case 2: v = min(d + s, 255); break;                      // ADD
        case 3: v = max(d - s, 0); break;                        // SUB
        case 4: v = (s * d) / 255; break;                        // MUL
        case 5: v = min(((d * (255 - s)) >> 8) + s, 255); break; // SCREEN
        case 6: v = max(s, d); break;                            // LIGHTEN
        default: v = min(s, d); break;                           // DARKEN
        }
        o[i] = v & 255;
    }
    return pack4(o);
}

// The colour of the pixel a k_raster thread owns, as the framebuffer holds
// it.  RGBA / unsigned byte: the packed colour, whose getters and setters
// are the identity.  Other formats: the raw pixel, read for blending through
// the SIMD getter (triangles) or the scalar one (points, lines, rectangles,
// images) and written through the matching setter.
template <bool GEN> struct FbPixel;
template <> struct FbPixel<false> {
    uint32_t c;
    __device__ __forceinline__ void load(const PFTarget &T, size_t i) { c = ((const uint32_t *)T.color)[i]; }
    __device__ __forceinline__ void clear(const PFTarget &T) { c = T.clearRaw[0]; }
    __device__ __forceinline__ void store(const PFTarget &T, size_t i) const { ((uint32_t *)T.color)[i] = c; }
    __device__ __forceinline__ uint32_t get(bool) const { return c; }
    __device__ __forceinline__ void set(bool, uint32_t v) { c = v; }
};
template <> struct FbPixel<true> {
    uint32_t r[4];
    uint32_t f;
    __device__ __forceinline__ void load(const PFTarget &T, size_t i) { f = T.fmt; pff_load(f, T.color, i, r); }
    __device__ __forceinline__ void clear(const PFTarget &T)
    {
        f = T.fmt; r[0] = T.clearRaw[0]; r[1] = T.clearRaw[1]; r[2] = T.clearRaw[2]; r[3] = T.clearRaw[3];
    }
    __device__ __forceinline__ void store(const PFTarget &T, size_t i) const { pff_store(f, T.color, i, r); }
    __device__ __forceinline__ uint32_t get(bool scalar) const { return scalar ? pff_get_sisd(f, r) : pff_get_simd(f, r); }
    __device__ __forceinline__ void set(bool scalar, uint32_t v) { if (scalar) pff_set_sisd(f, v, r); else pff_set_simd(f, v, r); }
};

// k_binsort: one CTA per bin that reached REG_SORT_MAX entries (a
// heavy-level list), taken from a queue: its keys are put back into
// submission order in place by a merge sort in shared memory.  A bin is a
// concatenation of runs that are each in order already (a warp of k_items
// appends its lanes' entries of a tile in lane order): each warp first
// sorts 32-key chunks in registers, then chunks are merged pairwise, level
// by level -- a key's place in the merged run is its place in its own run
// plus the number of smaller keys in the partner run, found by binary
// search.  Keys are unique (item << PF_SUB_BITS | sub-triangle, below 2^31);
// the padding to a whole chunk is unique too (2^31 + place), so every level
// is a permutation.
//
// Where one target's items fit a map of a bit each in a warp's shared memory
// (SORT_MAP_ITEMS) and none was clipped into several sub-triangles, a warp
// sorts a bin by setting its items' bits and reading the map back in order:
// one pass over the keys and one over the bits, whatever the bin's length,
// and no barriers.  The merge sort is bound by the latency of its levels and
// their barriers: the 64-soup batch's 83,000 bins, 130 to 2,000 entries
// each, 335 us, with the maps 93; soup256 9 -> 7.6.  (A warp's bitonic sort
// in registers for bins below 512, the merge sort for the others: 322.)
#define SORT_MAP_ITEMS 65536
__device__ void map_sort(uint32_t *bin, uint32_t n, uint4 *map, uint32_t groups)
{
    const uint32_t lane = threadIdx.x & 31u, all = 0xffffffffu;
    uint32_t *words = reinterpret_cast<uint32_t *>(map);
    // (the items of a bin lie within `groups` groups of 128, at their number
    // modulo that many)
    uint32_t lo = 0xffffffffu, hi = 0;
    for (uint32_t i0 = 0; i0 < n; i0 += 128u) {
        uint32_t key[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) { const uint32_t i = i0 + 32u * u + lane; key[u] = i < n ? bin[i] : 0xffffffffu; }
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            if (key[u] == 0xffffffffu) continue;
            const uint32_t item = key[u] >> PF_SUB_BITS;
            lo = min(lo, item); hi = max(hi, item);
            atomicOr(&words[(item >> 5) & (4u * groups - 1u)], 1u << (item & 31u));
        }
    }
    __syncwarp();
    const uint32_t last = __reduce_max_sync(all, hi) >> 7;
    uint32_t out = 0;
    for (uint32_t g0 = __reduce_min_sync(all, lo) >> 7; g0 <= last; g0 += 32u) {
        const uint32_t g = g0 + lane;
        uint4 m = make_uint4(0, 0, 0, 0);
        if (g <= last) { m = map[g & (groups - 1u)]; map[g & (groups - 1u)] = make_uint4(0, 0, 0, 0); }
        const uint32_t w[4] = { m.x, m.y, m.z, m.w };
        uint32_t total;
        uint32_t *o = bin + out + warp_offsets((uint32_t)(__popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w)), total);
#pragma unroll
        for (uint32_t k = 0; k < 4; k++)
            for (uint32_t b = w[k]; b; b &= b - 1u) *o++ = (g * 128u + 32u * k + (uint32_t)(__ffs(b) - 1)) << PF_SUB_BITS;
        out += total;
    }
    __syncwarp();                                      // the map is clear again
}

__device__ __forceinline__ uint32_t warp_sort32(uint32_t key)
{
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t k = 2; k <= 32; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const uint32_t o = __shfl_xor_sync(0xffffffffu, key, (int)j);
            const bool asc = (lane & k) == 0, low = (lane & j) == 0;
            key = (asc == low) ? min(key, o) : max(key, o);
        }
    return key;
}

// (MAPS: the launch's targets fit the maps; the merge sort is there for
// launches that clip)
template <bool MAPS>
__global__ void __launch_bounds__(SORT_THREADS) k_binsort(RasterArgs a)
{
    extern __shared__ __align__(16) uint32_t sbuf[];  // two buffers of a bin's keys (merge source and target), or the warps' maps
    __shared__ uint32_t sTile;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // k_items is done
    if (a.cnt->abortCommand <= a.command) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nList = min(a.cnt->heavyCount[REG_SORT_LEVEL - 1], a.totalTiles);
    if (MAPS && a.cnt->clipCount == 0) {
        // a bin a warp; the next one's count is read while one is sorted
        const uint32_t warps = gridDim.x * (SORT_THREADS / 32);
        const uint32_t *list = a.tileList + (size_t)REG_SORT_LEVEL * a.listStride;
        uint32_t e = blockIdx.x * (SORT_THREADS / 32) + (uint32_t)warp;
        if (e >= nList) return;
        uint4 *map = reinterpret_cast<uint4 *>(sbuf) + (size_t)warp * a.sortGroups;
        for (uint32_t i = (uint32_t)lane; i < a.sortGroups; i += 32u) map[i] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        uint32_t t = __ldg(list + e), n = __ldg(a.binCount + t);
        for (; e < nList; e += warps) {
            const uint32_t tn = e + warps < nList ? __ldg(list + e + warps) : 0u;
            const uint32_t nn = e + warps < nList ? __ldg(a.binCount + tn) : 0u;
            map_sort(a.bins + (size_t)t * a.cap, min(n, a.cap), map, a.sortGroups);
            t = tn;
            n = nn;
        }
        return;
    }
    uint32_t capPad = 32; while (capPad < a.cap) capPad <<= 1;   // each buffer's room
    // a CTA's first entry is its index in the grid, the counter hands out
    // the entries after those (no atomics at all when no bin needs sorting)
    for (uint32_t first = 1;; first = 0) {
        if (tid == 0) {
            const uint32_t q = first ? blockIdx.x : (blockIdx.x < nList ? gridDim.x + atomicAdd(&a.cnt->sortQueue, 1u) : nList);
            sTile = q < nList ? __ldg(a.tileList + (size_t)REG_SORT_LEVEL * a.listStride + q) : 0xffffffffu;
        }
        __syncthreads();
        const uint32_t t = sTile;
        if (t == 0xffffffffu) break;
        const uint32_t n = min(__ldg(a.binCount + t), a.cap);
        const uint32_t nPad = (n + 31u) & ~31u;
        uint32_t *bin = a.bins + (size_t)t * a.cap;
        // 1. chunks of 32 keys sorted in registers (padding 2^31 + place);
        //    whether the bin is in order already
        int unsorted = 0;
        for (uint32_t c = (uint32_t)warp * 32u; c < nPad; c += SORT_THREADS) {
            const uint32_t i = c + (uint32_t)lane;
            const uint32_t key = i < n ? bin[i] : 0x80000000u + i;
            const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
            unsorted |= (lane > 0 && prev > key) || (lane == 0 && c > 0 && i < n && bin[i - 1] > key);
            sbuf[i] = warp_sort32(key);
        }
        if (__syncthreads_or(unsorted)) {
            // 2. merge levels: runs of w keys, pairwise, into the other buffer
            uint32_t *src = sbuf, *dst = sbuf + capPad;
            for (uint32_t w = 32; w < nPad; w <<= 1) {
                for (uint32_t i = tid; i < nPad; i += SORT_THREADS) {
                    const uint32_t run = i / w, s0 = run * w;
                    const uint32_t oStart = (run & 1u) ? s0 - w : s0 + w;      // the partner run
                    const uint32_t oLen = oStart < nPad ? min(w, nPad - oStart) : 0u;
                    const uint32_t key = src[i];
                    uint32_t lo = 0, hi = oLen;                                  // partner keys below key
                    while (lo < hi) { const uint32_t mid = (lo + hi) >> 1; if (src[oStart + mid] < key) lo = mid + 1; else hi = mid; }
                    dst[(run & ~1u) * w + (i - s0) + lo] = key;
                }
                __syncthreads();
                uint32_t *tmp = src; src = dst; dst = tmp;
            }
            for (uint32_t i = tid; i < n; i += SORT_THREADS) bin[i] = src[i];
        }
        __syncthreads();                               // sTile and the buffers are free
    }
}

// List this lane's fragments (bit 32 s + k of m: record k at its pixel of
// slot s), in order, as entries off, off + 1, ... of the warp's fragment
// list, as far as they fall in the window [b0, bEnd).
__device__ __forceinline__ void tile_list(unsigned long long m, uint32_t off, uint32_t b0, uint32_t bEnd,
                                          uint16_t *fdesc)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t cnt = __popcll(m);
    if (!cnt || off >= bEnd || off + cnt <= b0) return;
    uint32_t f = off;
    for (unsigned long long mm = m; mm && f < bEnd; mm &= mm - 1, f++) {
        if (f < b0) continue;
        const uint32_t b = (uint32_t)(__ffsll(mm) - 1);
        fdesc[f - b0] = (uint16_t)(((lane + 32u * (b >> 5)) << 5) | (b & 31u));
    }
}

// Refill the queue of a tile's next keys at Q.keys (`left` of them at
// Q.keys[taken] on) from the bin's keys c0 .. n - 1 (at Q.keys too when bin
// is null) up to a batch, leaving out the records that lie behind every
// pixel of the tile -- its farthest depth is farKey -- by their depth planes
// alone: 16 bytes and a dozen operations a key, where copying the record,
// its set-up and its coverage take 30.  Their covered pixels need no visit,
// k_items has counted them.  Nothing is left out once a key came that may
// raise a depth.  Returns the next key.  Against dropping them after their
// set-up: 64-soup batch 1,458 -> 1,160 us, phong1080 315 -> 256, the
// 2,000-triangle soup at 256x256 50 -> 47, sphere1080, whose tiles hold one
// batch, unchanged; k_items pays for the counting (batch 326 -> 331,
// phong1080 190 -> 230, sphere1080 20 -> 21.3).  Two groups of 32 keys a
// step: 1,209 -> 1,259; out of line: 1,190.
__device__ __forceinline__ uint32_t queue_refill(QWarp &Q, const uint32_t *bin, const float4 *planes, uint32_t n, uint32_t c0,
                                              uint32_t left, uint32_t taken, uint32_t farKey, uint32_t ox, uint32_t oy)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t k = lane < left ? Q.keys[taken + lane] : 0u;
    __syncwarp();
    if (lane < left) Q.keys[lane] = k;
    uint32_t queued = left;
    bool lowering = Q.lowering != 0;
    const float farDepth = __int_as_float((int32_t)((farKey & 0x80000000u) ? farKey ^ 0x80000000u : ~farKey));
    // No bound below 3e38: a record without one has none either; NaN, which
    // hides nothing, for a zero.  (Before an infinity lies every depth, and
    // its reciprocal has no sign: that is compared by the depth itself.)
    const float inv = farDepth > 0.0f ? fminf(__frcp_rn(farDepth) * 0.99999f, 3e38f) :
                      farDepth < 0.0f ? __frcp_rn(farDepth) * 1.00001f : __int_as_float(0x7fffffff);
    const float fx = (float)ox, fy = (float)oy;
    while (queued < QCHN && c0 < n) {
        const uint32_t i = c0 + lane;
        uint32_t key = 0;
        float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < n) {
            key = bin ? __ldg(bin + i) : Q.keys[i];
            p = __ldg(planes + (key >> PF_SUB_BITS));
        }
        lowering = __all_sync(0xffffffffu, p.w == p.w) && lowering;
        const float top = fminf(((p.x + p.y * fx) + p.z * fy) + (fmaxf(p.y * 7.0f, 0.0f) + fmaxf(p.z * 7.0f, 0.0f)), p.w);
        const bool behind = lowering && top <= inv && (p.w > 0.0f) == (farDepth > 0.0f) && (key & ((1u << PF_SUB_BITS) - 1u)) == 0;
        const uint32_t m = __ballot_sync(0xffffffffu, i < n && !behind);
        if ((m >> lane) & 1u) Q.keys[queued + __popc(m & ((1u << lane) - 1u))] = key;
        queued += __popc(m);
        c0 += 32u;
        __syncwarp();
    }
    if (lane == 0) { Q.queued = queued; Q.lowering = lowering; }
    __syncwarp();
    return c0;
}

// GEN: a target is not RGBA / unsigned byte.  PHONG: a draw state lights per
// fragment; launches without one do without that code: sphere1080 58 -> 56
// us, 64-soup batch 1,925 -> 1,780.  Warps an SM, as measured: plain 28
// (against 24: 64-soup batch 1,555 -> 1,455, 8,192 small triangles 32 -> 28;
// 32 warps: 1,505), GEN 24 (28: 35 -> 36.5 on RGBA half), PHONG 20 (against
// 24: phong1080 340 -> 312; 16: 362).  That leaves 72, 80 and 96 registers;
// of the variants of 4 warps a CTA only the plain one does not spill (bytes
// stored and loaded: GEN 8 and 16, PHONG 8 and 16, both 68 and 76).  Bound by
// instruction issue and the round trips of claims, bin keys and records.
template <bool GEN, int WARPS, bool PHONG>
__global__ void __launch_bounds__(WARPS * 32, (PHONG ? 20 : GEN ? 24 : 28) / WARPS) k_raster(RasterArgs a)
{
    extern __shared__ __align__(16) unsigned char rsmem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    QWarp &Q = reinterpret_cast<QWarp *>(rsmem)[warp];

    asm volatile("griddepcontrol.wait;" ::: "memory");   // k_binsort is done
    if (a.cnt->abortCommand <= a.command) return;
    // the batch completed set-up without overflow: its sub-triangles count
    if (blockIdx.x == 0 && tid == 0) {
        atomicAdd(&a.cnt->rasterized, a.cnt->batchRasterized);
        atomicAdd(&a.cnt->fragments, a.cnt->batchFragments);
    }
    const uint32_t lx = (uint32_t)lane & 7u, ly = (uint32_t)lane >> 3;     // my pixels: (lx, ly) and (lx, ly + 4)
    uint32_t frags = 0;                                // (at most 64 a bin entry and tile)

    // persistent: warps take tiles from a shared work queue -- the tiles the
    // binning listed as non-empty, those of the heaviest level first, then
    // of each lighter level, then the rest (a tile is rasterized from the
    // first list it is on and skipped on the later ones); then the groups of
    // 32 tiles whose empty bins only get their fused clear, if any, one tile
    // a lane
    // A heavy level with few tiles against the grid's warps sets the end of
    // the launch (its tiles start first but run longest): each of its tiles
    // is then two work items, its top and bottom halves, each a warp with
    // one pixel a lane, which take about half as long.  Where heavy tiles
    // are many the launch is bound by the total work, which halves would
    // only add to (each half walks the whole bin).  A launch of at most half
    // as many tiles as warps has idle warps for every level (the 64 tiles of
    // a 64x64 context 57 -> 31 us, the 1,024 of soup256 56 -> 50; taking
    // halves of all levels up to half the warps instead, phong1080 335 -> 357).
    // (in shared memory, like the fragment count: read by lane 0 between
    // tiles only, they would cost the tile's loops registers)
    __shared__ uint32_t sLevelEnd[PF_HEAVY_LEVELS + 1];    // queue index past level l's entries, heaviest first
    __shared__ uint32_t sSplit;
    __shared__ unsigned long long sFrags;
    if (tid == 0) {
        uint32_t nQueue = 0, split = 0;
        for (int l = PF_HEAVY_LEVELS; l >= 1; l--) {
            const uint32_t c = min(a.cnt->heavyCount[l - 1], a.totalTiles);
            const bool sp = 4u * c <= gridDim.x * (uint32_t)WARPS || 2u * a.totalTiles <= gridDim.x * (uint32_t)WARPS;
            split |= sp ? 1u << l : 0u;
            nQueue += sp ? 2u * c : c;
            sLevelEnd[l] = nQueue;
        }
        sLevelEnd[0] = nQueue + min(a.cnt->tileListCount, a.totalTiles);
        sSplit = split;
        sFrags = 0;
    }
    __syncthreads();
    // each warp's first entry is its own index in the grid; the counter
    // hands out the entries after those (3,648 warps claiming their first
    // entry with one atomic each would serialise at the start)
    uint32_t claim = blockIdx.x * (uint32_t)WARPS + (uint32_t)warp;
    for (;;) {
    uint32_t next = 0xffffffffu, nextCount = 0;
    if (lane == 0) {
        const uint32_t q = claim, nQueue = sLevelEnd[0];
        if (q < nQueue + (a.totalTiles + 31u) / 32u) {
            claim = gridDim.x * (uint32_t)WARPS + atomicAdd(&a.cnt->tileQueue, 1u);
            if (q >= nQueue) next = 0x80000000u | (q - nQueue);      // a group of tiles to clear
            else {
                uint32_t level = PF_HEAVY_LEVELS, begin = 0;
                while (q >= sLevelEnd[level]) { begin = sLevelEnd[level]; level--; }
                const uint32_t e = q - begin;
                const bool split = (sSplit >> level) & 1u;
                next = __ldg(a.tileList + (size_t)level * a.listStride + (split ? e >> 1 : e));
                nextCount = __ldg(a.binCount + next);
                if (heavy_level(nextCount) != level) next = 0xfffffffeu;   // rasterized from an earlier list
                else if (split) next |= (e & 1u) ? TILE_BOTTOM : TILE_TOP;
            }
        }
    }
    const uint32_t gt = __shfl_sync(0xffffffffu, next, 0);
    const uint32_t gtCount = __shfl_sync(0xffffffffu, nextCount, 0);   // (its bin count, read for the check)
    if (gt == 0xffffffffu) break;
    if (gt == 0xfffffffeu) continue;
    if (gt & 0x80000000u) {
        // the fused clear of the empty tiles of group gt: one tile a lane,
        // each row of pixels and depths in 16-byte stores
        const uint32_t t = 32u * (gt & 0x7fffffffu) + (uint32_t)lane;
        if (t < a.totalTiles && __ldg(a.binCount + t) == 0) {
            int clo = 0, chi = a.nTargets - 1;
            while (clo < chi) { int mid = (clo + chi + 1) >> 1; if (a.targets[mid].tileBase <= t) clo = mid; else chi = mid - 1; }
            const PFTarget &C = a.targets[clo];
            if (C.clearMode != 0 && !(GEN && C.fmt == PFF_BGRA8)) {     // (k_rows clears those)
                const uint32_t tile = t - C.tileBase;
                const uint32_t cx = (tile % C.tilesX) * PF_TILE, cy = (tile / C.tilesX) * PF_TILE;
                const uint32_t xe = min(cx + PF_TILE, C.W);
                // (GEN: pixels of 2, 4, 8 or 16 bytes, the others pixel by pixel.
                // Bound by the sectors L2 takes: a word a store, the sphere
                // frame's raster sent it 14 M of RGBA float, most of them in part,
                // and took 200 us with L2 full of written lines, 100 now; RGBA
                // half 119 -> 101, 5-6-5 79 -> 71.  Apart from the plain clear:
                // one body for both cost that 0.5 % of the 64-soup batch)
                uint4 v = make_uint4(0, 0, 0, 0);
                uint32_t bytes = 0;
                if (GEN) {
                    const uint32_t b = (uint32_t)pff_bytes(C.fmt), c0 = C.clearRaw[0];
                    if (b == 2u) { const uint32_t two = (c0 & 0xffffu) * 0x10001u; v = make_uint4(two, two, two, two); }
                    else if (b == 4u) v = make_uint4(c0, c0, c0, c0);
                    else if (b == 8u) v = make_uint4(c0, C.clearRaw[1], c0, C.clearRaw[1]);
                    else v = make_uint4(c0, C.clearRaw[1], C.clearRaw[2], C.clearRaw[3]);
                    bytes = (b & (b - 1u)) == 0 ? b : 0u;
                }
                for (uint32_t py = cy; py < min(cy + PF_TILE, C.H); py++) {
                    const size_t row = (size_t)py * C.W;
                    if (!GEN && xe == cx + 8u && ((row + cx) & 3u) == 0 && !(C.clearMode == 1 && row + cx < 8) &&
                        (((uintptr_t)C.color | (uintptr_t)C.depth) & 15u) == 0) {
                        const uint32_t cr = C.clearRaw[0];
                        const float cd = C.clearDepth;
                        uint4 *cp = reinterpret_cast<uint4 *>((uint32_t *)C.color + row + cx);
                        float4 *dp = reinterpret_cast<float4 *>(C.depth + row + cx);
                        cp[0] = make_uint4(cr, cr, cr, cr); cp[1] = make_uint4(cr, cr, cr, cr);
                        dp[0] = make_float4(cd, cd, cd, cd); dp[1] = make_float4(cd, cd, cd, cd);
                        continue;
                    }
                    if (GEN && bytes && xe == cx + 8u && !(C.clearMode == 1 && row + cx < 8)) {
                        uint4 *cp = reinterpret_cast<uint4 *>((unsigned char *)C.color + (row + cx) * bytes);
                        float4 *dp = reinterpret_cast<float4 *>(C.depth + row + cx);
                        if ((((uintptr_t)cp | (uintptr_t)dp) & 15u) == 0) {
                            const float cd = C.clearDepth;
                            for (uint32_t k = 0; k < bytes / 2u; k++) cp[k] = v;
                            dp[0] = make_float4(cd, cd, cd, cd); dp[1] = make_float4(cd, cd, cd, cd);
                            continue;
                        }
                    }
                    for (uint32_t px = cx; px < xe; px++) {
                        const size_t pidx = row + px;
                        if (C.clearMode == 1 && pidx < 8) continue;  // pfClear keeps pixels 0..7
                        if (GEN) pff_store(C.fmt, C.color, pidx, C.clearRaw);
                        else ((uint32_t *)C.color)[pidx] = C.clearRaw[0];
                        C.depth[pidx] = C.clearDepth;
                    }
                }
            }
        }
        continue;
    }
    // whole tile: my pixels are rows ly and ly + 4; half tile: row ly of
    // the top half or ly + 4 of the bottom half only
    const uint32_t gtile = gt & ~TILE_HALF_MASK;
    const bool whole = (gt & TILE_HALF_MASK) == 0;
    const uint32_t rowA = ly + ((gt & TILE_HALF_MASK) == TILE_BOTTOM ? 4u : 0u);
    int tlo = 0, thi = a.nTargets - 1;
    while (tlo < thi) { int mid = (tlo + thi + 1) >> 1; if (a.targets[mid].tileBase <= gtile) tlo = mid; else thi = mid - 1; }
    const PFTarget &T = a.targets[tlo];
    if (GEN && T.fmt == PFF_BGRA8) continue;                 // rasterized by k_rows
    const uint32_t tile = gtile - T.tileBase;
    const uint32_t n = min(gtCount, a.cap);
    if (n == 0 && T.clearMode == 0) continue;
    const uint32_t ox = (tile % T.tilesX) * PF_TILE, oy = (tile / T.tilesX) * PF_TILE;
    const uint32_t W = T.W, H = T.H;

    FbPixel<GEN> col0{}, col1{};
    float dep0 = 0.0f, dep1 = 0.0f;
    const uint32_t X0 = ox + lx, Y0 = oy + rowA, Y1 = Y0 + 4u;
    const bool in0 = X0 < W && Y0 < H, in1 = whole && X0 < W && Y1 < H;
    const size_t pidx0 = (size_t)Y0 * W + X0, pidx1 = (size_t)Y1 * W + X0;
    {
        auto init = [&](FbPixel<GEN> &c, float &d, bool in, size_t pi) {
            if (!in) return;
            if (T.clearMode == 2 || (T.clearMode == 1 && pi >= 8)) { c.clear(T); d = T.clearDepth; }
            else { c.load(T, pi); d = T.depth[pi]; }
        };
        init(col0, dep0, in0, pidx0);
        init(col1, dep1, in1, pidx1);
    }

    // a bin shorter than REG_SORT_MAX is put into submission order here, in
    // registers: a bitonic network over 32, 64 or 128 places, place
    // 32 r + lane in key r of the lane; longer bins were sorted by k_binsort
    const uint32_t *bin = a.bins + (size_t)gtile * a.cap;
    const bool regSort = n < REG_SORT_MAX;
    uint32_t sk[4] = { 0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu };
    if (regSort) {
        const uint32_t nk = n <= 32 ? 1u : n <= 64 ? 2u : 4u;    // keys a lane sorts: a power-of-two network
        for (uint32_t r = 0; r < 4; r++)
            if (32 * r + (uint32_t)lane < n) sk[r] = __ldg(bin + 32 * r + lane);
        // keys binned by one warp of k_items arrive in order: check first
        bool ordered = true;
#pragma unroll
        for (uint32_t r = 0; r < 4; r++) {
            if (r >= nk) break;                               // uniform over the warp
            const uint32_t o = __shfl_down_sync(0xffffffffu, sk[r], 1);
            const uint32_t b = __shfl_sync(0xffffffffu, sk[r < 3 ? r + 1 : 3], 0);
            ordered = ordered && (lane < 31 ? sk[r] <= o : (r + 1 < nk ? sk[r] <= b : true));
        }
        if (!__all_sync(0xffffffffu, ordered))
        for (uint32_t k = 2; k <= 32 * nk; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                if (j >= 32) {
                    // partners are keys of the same lane: places i and i + j
                    const uint32_t dr = j >> 5;
#pragma unroll
                    for (uint32_t r = 0; r < 4; r++) {
                        if (r >= nk) break;
                        if (r & dr) continue;
                        const uint32_t i = 32 * r + (uint32_t)lane;
                        const uint32_t x = sk[r], y = sk[r + dr];
                        const bool asc = (i & k) == 0;
                        sk[r] = asc ? min(x, y) : max(x, y);
                        sk[r + dr] = asc ? max(x, y) : min(x, y);
                    }
                } else {
#pragma unroll
                    for (uint32_t r = 0; r < 4; r++) {
                        if (r >= nk) break;                       // uniform over the warp
                        const uint32_t i = 32 * r + (uint32_t)lane;
                        const uint32_t o = __shfl_xor_sync(0xffffffffu, sk[r], j);
                        sk[r] = (((i & k) == 0) == ((i & j) == 0)) ? min(sk[r], o) : max(sk[r], o);
                    }
                }
            }
        // (kept in shared memory for the batches: the registers are free)
        for (uint32_t r = 0; r < 4; r++) Q.keys[32 * r + (uint32_t)lane] = sk[r];
        __syncwarp();
    }

    // Where fragments are lit one by one (PHONG), unblended ones wait: in a
    // tile of several batches, a pixel's fragment that nothing of its batch
    // blends over is kept as its bin key (Q.pend) and shaded only when a
    // batch with blended records comes, or at the end -- most are replaced
    // before that (phong1080: about three of a pixel's fragments pass, one
    // is seen; k_raster 520 -> 405 us).  Without per-fragment lighting the
    // bookkeeping costs more than it saves (64-soup batch 1,925 -> 2,255 us,
    // sphere1080 58 -> 65).  Shading those that wait is a
    // batch of its own per pixel slot (phase 1 and 2), whose records are the
    // lanes' own; it ends the waiting, so that draws that alternate between
    // blended and unblended records pay for it once a tile.
    bool defer = n > QCHN, pending = false;
    uint32_t ph = 0;
    // The bin's next keys, in order, are a queue at Q.keys: a batch is its
    // first 32 (queue_refill).  A short bin's keys wait behind the queue:
    // c0, the next one, is never below its room.
    uint32_t c0 = min(n, (uint32_t)QCHN), queued = c0, taken = 0;
    if (lane == 0) Q.lowering = 1;
    if (!regSort) Q.keys[lane] = __ldg(bin + lane);
    __syncwarp();
    for (;;) {
        if ((!PHONG || ph == 0) && taken) {
            if ((!PHONG || !pending) && queued == taken && c0 >= n) break;
            const uint32_t farKey = __reduce_max_sync(0xffffffffu, max(in0 ? depth_key(dep0) : 0u, in1 ? depth_key(dep1) : 0u));
            c0 = queue_refill(Q, regSort ? nullptr : bin, a.planes, n, c0, queued - taken, taken, farKey, ox, oy);
            queued = Q.queued; taken = 0;
        }
        if (ph == 0 && queued == 0) {
            if (!PHONG || !pending) break;
            ph = 1;
        }
        const uint32_t phase = PHONG ? ph : 0u;
        // 1. my record: load, stage, derive its tile set-up and coverage
        uint32_t kind = 0;
        uint32_t covLo = 0, covHi = 0;                  // its coverage, rows 0-3 and 4-7 (bit 8 y + x of the 64)
        bool blends = false;
        uint32_t key = 0xffffffffu;
        if (phase != 0) key = Q.pend[32u * (phase - 1u) + (uint32_t)lane];
        else if ((uint32_t)lane < queued) key = Q.keys[lane];
        const bool have = key != 0xffffffffu;
        if (have) {
            const uint32_t item = key >> PF_SUB_BITS, sub = key & ((1u << PF_SUB_BITS) - 1);
            const PFPrim *src = &a.prims[item];
            uint32_t pi = item;
            if (sub != 0) { pi = (uint32_t)__ldg(&a.prims[item].poolBase) + sub - 1; src = &a.pool[pi]; }
            // (straight into shared memory: through registers, the record's 32
            // words would spill what the tile holds)
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&Q.rec[lane].p);
#pragma unroll
            for (int i = 0; i < 8; i++)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst + 16u * i), "l"((const char *)src + 16 * i) : "memory");
            if (PHONG) Q.rec[lane].ph = sub != 0 ? &a.poolPh[pi] : &a.primsPh[item];
            asm volatile("cp.async.wait_all;" ::: "memory");
            const int4 *r = reinterpret_cast<const int4 *>(&Q.rec[lane].p);
            const int4 r1 = r[1], r2 = r[2];
            QEdge E;
            tile_edge(r[0], r1, r2, Q.rec[lane].p.rstate, Q.rec[lane].p.zReject, ox, oy, W, H, E);
            kind = (uint32_t)r2.z & PFP_KIND;
            blends = (E.rstate & PFS_BLEND) != 0;
            // my record's coverage of the tile: the pixels of its box that
            // pass the integer edge test (triangles.c:398-424) or, for a
            // point, line or rectangle, its own rule
            const uint32_t bx0 = E.box & 15u, bw = (E.box >> 4) & 15u, by0 = (E.box >> 8) & 15u, bh = (E.box >> 12) & 15u;
            if (phase != 0) {
                // (covered and visible already)
            } else if (kind == 0) {
                // the whole box when no edge function is negative at its
                // least corner; values in [-2^30, 2^30) and steps in
                // [-2^26, 2^26), of which none wraps inside the tile (-2^31,
                // which has no absolute value, is outside as well)
                bool full = bw + bh >= 12u;
                if (full) {
                    uint32_t sign = 0, steps = 0;
#pragma unroll
                    for (int e = 0; e < 3; e++) {
                        const uint32_t e0 = (uint32_t)E.e0[e], ex = (uint32_t)(e == 0 ? E.ex0 : e == 1 ? E.ex1 : E.ex2);
                        const uint32_t ey = (uint32_t)(e == 0 ? E.ey0 : e == 1 ? E.ey1 : E.ey2);
                        sign |= (e0 + (1u << 30)) | (e0 + ((int32_t)ex > 0 ? bx0 : bx0 + bw - 1u) * ex + ((int32_t)ey > 0 ? by0 : by0 + bh - 1u) * ey);
                        steps |= (ex + (1u << 26)) | (ey + (1u << 26));
                    }
                    full = (sign >> 31 | steps >> 27) == 0;
                }
                const uint32_t cols = ((1u << bw) - 1u) << bx0;
                if (full) {
                    const unsigned long long rows = (~0ull >> (64u - 8u * bh)) << (8u * by0);
                    covLo = cols * 0x01010101u & (uint32_t)rows;
                    covHi = cols * 0x01010101u & (uint32_t)(rows >> 32);
                } else {
                    // a row at a time, from column 7 down: the sign of the three
                    // edge functions' OR, shifted in (they are not all zero
                    // together: their sum is the area, and records without any
                    // were culled).  Straight-line code for the eight columns
                    // beats a loop over the box's, as the lanes' boxes differ:
                    // 64-soup batch 1,774 -> 1,555 us, phong1080 405 -> 340,
                    // sphere1080 54 -> 51.
                    uint32_t r0 = (uint32_t)E.e0[0] + 7u * (uint32_t)E.ex0 + by0 * (uint32_t)E.ey0;
                    uint32_t r1 = (uint32_t)E.e0[1] + 7u * (uint32_t)E.ex1 + by0 * (uint32_t)E.ey1;
                    uint32_t r2 = (uint32_t)E.e0[2] + 7u * (uint32_t)E.ex2 + by0 * (uint32_t)E.ey2;
                    for (uint32_t y = by0; y < by0 + bh; y++) {
                        uint32_t w0 = r0, w1 = r1, w2 = r2, row = 0;
#pragma unroll
                        for (int x = 0; x < 8; x++) {
                            row = __funnelshift_l(~(w0 | w1 | w2), row, 1);
                            w0 -= (uint32_t)E.ex0; w1 -= (uint32_t)E.ex1; w2 -= (uint32_t)E.ex2;
                        }
                        row = (row & cols) << (8u * (y & 3u));
                        if (y < 4u) covLo |= row; else covHi |= row;
                        r0 += (uint32_t)E.ey0; r1 += (uint32_t)E.ey1; r2 += (uint32_t)E.ey2;
                    }
                }
            } else {
                const PFPrim &P = Q.rec[lane].p;
                for (uint32_t y = by0; y < by0 + bh; y++)
                    for (uint32_t x = bx0; x < bx0 + bw; x++)
                        if (lp_covers(P, (int32_t)(ox + x), (int32_t)(oy + y))) {
                            if (y < 4u) covLo |= 1u << (8u * y + x); else covHi |= 1u << (8u * (y - 4u) + x);
                        }
            }
            Q.edge[lane] = E;
        }
        const bool anyLP = __any_sync(0xffffffffu, kind != 0);
        uint32_t vis0 = 0, vis1 = 0;                    // bit k: record k passed at my pixel of slot 0 / 1
        if (phase != 0) {
            if (phase == 1) vis0 = have ? 1u << lane : 0u; else vis1 = have ? 1u << lane : 0u;
            __syncwarp();
        } else {
        const bool live = (covLo | covHi) != 0;
        if (PHONG && pending && __any_sync(0xffffffffu, live && blends)) { ph = 1; __syncwarp(); continue; }
        if (!__any_sync(0xffffffffu, live)) { taken = min(queued, (uint32_t)QCHN); __syncwarp(); continue; }
        __syncwarp();
        // 2a. coverage per pixel: bit k of cm0 / cm1 -- record k covers my
        //     pixel of slot 0 / 1 -- the records' masks transposed over the
        //     warp (rows 0-3 of the tile are bits 0-31: bit 8 y + x is lane
        //     8 y + x's pixel of slot 0; rows 4-7 its pixel of slot 1)
        const uint32_t cmLo = warp_transpose32(covLo);
        const uint32_t cmHi = warp_transpose32(covHi);
        const uint32_t cm0 = (rowA == ly) ? cmLo : cmHi, cm1 = whole ? cmHi : 0u;
        // 2b. depth: each of my pixels walks its covering records in
        //     submission order -- depth (the correctly rounded reciprocal),
        //     the depth-test rejection bound, the depth test and write
        uint32_t cov = 0;
        auto depth_walk = [&](uint32_t cm, float &d, uint32_t &vis, uint32_t row, uint32_t Y) {
            for (; cm; cm &= cm - 1) {
                const uint32_t k = (uint32_t)(__ffs(cm) - 1);
                const int4 *e4 = reinterpret_cast<const int4 *>(&Q.edge[k]);
                const int4 q2 = e4[2];
                const uint32_t box = (uint32_t)q2.y, rs = (uint32_t)q2.z;
                const int func = (int)((rs >> 16) & 255u);
                float z;
                cov += (box >> 18) & 1u;
                if (((box >> 16) & 3u) == 0) {
                    if (__int_as_float(q2.w) >= d) continue;  // every fragment of it fails the depth test
                    const int4 q0 = e4[0], q1 = e4[1];
                    const uint32_t w1 = (uint32_t)q0.x + lx * (uint32_t)q0.w + row * (uint32_t)q1.z;
                    const uint32_t w2 = (uint32_t)q0.y + lx * (uint32_t)q1.x + row * (uint32_t)q1.w;
                    const uint32_t w3 = (uint32_t)q0.z + lx * (uint32_t)q1.y + row * (uint32_t)q2.x;
                    const float4 zq = reinterpret_cast<const float4 *>(&Q.rec[k].p)[3];     // wInvSum z1 z2 z3
                    const float wn1 = (float)(int32_t)w1 * zq.x, wn2 = (float)(int32_t)w2 * zq.x;
                    const float wn3 = (float)(int32_t)w3 * zq.x;
                    float zs = zq.y * wn1 + zq.z * wn2;
                    zs = zs + zq.w * wn3;
                    z = __frcp_rn(zs);
                    if ((rs & PFS_DEPTH_TEST) && !depth_simd(func, z, d)) continue;
                } else {
                    // a point, line or rectangle set up on the host: its own
                    // depth, the scalar depth test (rectangles are not fragments)
                    const PFPrim &P = Q.rec[k].p;
                    z = lp_depth(P, (int32_t)X0, (int32_t)Y);
                    if ((rs & PFS_DEPTH_TEST) && !depth_sisd(func, z, d)) continue;
                }
                // (an unblended fragment replaces what the batch drew here before:
                // those fragments are never shaded)
                vis = ((rs & PFS_BLEND) ? vis : 0u) | 1u << k;
                if (rs & PFS_DEPTH_MASK) d = z;
            }
        };
        depth_walk(cm0, dep0, vis0, rowA, Y0);
        depth_walk(cm1, dep1, vis1, ly + 4u, Y1);
        frags += cov;
        if (PHONG && defer) {
            auto waits = [&](uint32_t vis) {
                return vis && !(vis & (vis - 1u)) && !(Q.edge[__ffs(vis) - 1].rstate & PFS_BLEND);
            };
            const bool d0 = waits(vis0), d1 = waits(vis1);
            if (__any_sync(0xffffffffu, d0 || d1)) {
                auto key_of = [&](uint32_t vis) {
                    return Q.keys[__ffs(vis) - 1];
                };
                if (d0 || !pending) Q.pend[lane] = d0 ? key_of(vis0) : 0xffffffffu;
                if (d1 || !pending) Q.pend[32 + lane] = d1 ? key_of(vis1) : 0xffffffffu;
                if (d0) vis0 = 0;
                if (d1) vis1 = 0;
                pending = true;
            }
        }
        }
        // 3+4. shade the fragments that passed, densely over the warp, and
        //      blend each pixel's in submission order
        uint32_t totalv;
        const uint32_t cntv = __popc(vis0) + __popc(vis1);
        const uint32_t offv = warp_offsets(cntv, totalv);
        for (uint32_t b0 = 0; b0 < totalv; b0 += QFW) {
            const uint32_t bEnd = min(totalv, b0 + QFW);
            tile_list(vis0 | ((unsigned long long)vis1 << 32), offv, b0, bEnd, Q.fdesc);
            __syncwarp();
            for (uint32_t f = b0 + (uint32_t)lane; f < bEnd; f += 32) {
                const uint32_t d = Q.fdesc[f - b0], p = d >> 5, k = d & 31u;
                const uint32_t X = p & 7u, Y = (p >> 3) + (rowA - ly);     // (a bottom half's slot 0 is row ly + 4)
                const PFPrim &P = Q.rec[k].p;
                if (anyLP && (P.flags & PFP_KIND)) {
                    Q.fc[f - b0] = lp_color(P, (int32_t)(ox + X), (int32_t)(oy + Y));
                    continue;
                }
                float wn[3];
                const float z = tile_depth(Q.edge[k], P, X, Y, wn);
                Q.fc[f - b0] = shade_fragment<PHONG>(P, Q.rec[k].ph, a.states, wn[0], wn[1], wn[2], z);
            }
            __syncwarp();
            if (cntv && offv < bEnd && offv + cntv > b0) {
                uint32_t f = offv;
                auto blend = [&](FbPixel<GEN> &c, uint32_t mm) {
                    for (; mm && f < bEnd; mm &= mm - 1, f++) {
                        if (f < b0) continue;
                        const uint32_t k = (uint32_t)(__ffs(mm) - 1);
                        const uint32_t rs = Q.edge[k].rstate;
                        const bool lpk = anyLP && (Q.rec[k].p.flags & PFP_KIND);
                        uint32_t frag = Q.fc[f - b0];
                        if (rs & PFS_BLEND)
                            frag = lpk ? blend_sisd((int)(rs >> 24), frag, c.get(true))
                                       : blend_simd((int)(rs >> 24), frag, c.get(false));
                        c.set(lpk, frag);
                    }
                };
                blend(col0, vis0);
                blend(col1, vis1);
            }
            __syncwarp();                                  // the window's lists are free
        }
        __syncwarp();                                      // the batch's records are free
        if (phase == 0) taken = min(queued, (uint32_t)QCHN);
        else if (phase == 1 && whole) ph = 2;
        else { ph = 0; pending = false; defer = false; }
    }
    {
        // (indices from the target again: held through the batches they
        // would cost registers)
        const size_t p0 = (size_t)(oy + rowA) * T.W + ox + lx;
        if (in0) { col0.store(T, p0); T.depth[p0] = dep0; }
        const size_t p1 = (size_t)(oy + rowA + 4u) * T.W + ox + lx;
        if (in1) { col1.store(T, p1); T.depth[p1] = dep1; }
    }
    if (frags >= 0x40000000u) { atomicAdd(&sFrags, (unsigned long long)frags); frags = 0; }
    }   // tile loop

    // fragment counter: one atomic per CTA (same-address atomics serialise)
    unsigned long long all = frags;
    for (int o = 16; o > 0; o >>= 1) all += __shfl_down_sync(0xffffffffu, all, o);
    if (lane == 0 && all) atomicAdd(&sFrags, all);
    __syncthreads();
    if (tid == 0 && sFrags) atomicAdd(&a.cnt->fragments, sFrags);
}

// ---------------------------------------------------------------------------
// k_rows: targets of BGRA / unsigned-byte format, row by row in submission
// order.
//
// The reference writes such a framebuffer through a SIMD getter and setter
// that shuffle each 4-pixel half of the 8-pixel vector with the bytes of
// the half's first pixel (pixel.h:2070-2078, 2916-2921; simd.h:564-583):
// every pixel of a half that a triangle's mask lets through takes the value
// computed at the half's first pixel -- that pixel's own colour (texture
// coordinates zero when it is outside the mask, triangles.c:508-513)
// blended with that pixel's destination.  The halves start at xMin + 4k of
// the triangle's box (x steps by 8 from xMin, triangles.c:409), so a half's
// first pixel may lie in the tile to the left, whose colour when the
// triangle is drawn depends on everything drawn there before it: the tiles
// of a row are not independent.  Rows are.  Points, lines and rectangles use
// the scalar getter and setter (a plain R / B swap, pixel.h:356-363,
// 703-707), pixel by pixel.
//
// A CTA owns one row of such a target for the whole launch and keeps its
// colour and depth in shared memory.  Only the depth test and the blend need
// the row as it is when a record is drawn; a half's coverage, its pixels'
// depths and both colours its first pixel can give (inside the mask or
// outside) do not.  So the row's records pass through a pipeline, a batch of
// up to 32 records a step, one block barrier between steps: one warp looks
// for records that reach the row (8-byte summaries -- row_info: the records
// an item has and the rows they span -- so that items off the row cost a
// coalesced load), one makes the next batch and loads its records, two work
// out the halves of the batch before, and one draws the batch before that,
// record by record, a lane a pixel.  Bound by that last chain: a record's
// step reads its pixels, compares, blends and writes.  With one warp doing
// all of it a record at a time (its load and its texels waited for in every
// step) the sphere frame's launch at 1080p took 1,210 us, now 210, and 798
// now 177 with the mesh turned, so that the small triangles around its poles
// share no rows; with a lane a half in the drawing warp and one finding warp
// 240 (turned).  Five CTAs an SM were chosen without per-fragment lighting
// (six: 184), where 72 registers do.  With it they spill 136 bytes: a lit
// frame (81,920 triangles, four lights, 1280x720) takes 1,113 us on the
// device (3,002 before), and 1,060 with four CTAs, whose 96 registers do not
// spill.
// ---------------------------------------------------------------------------
#define ROW_THREADS 160
#define ROW_BATCH 32                // records of a batch
#define ROW_HALVES 96               // halves of a batch (a wider record is drawn in parts)
#define ROW_AHEAD 128               // records the looking warp keeps in the queue
#define ROW_QUEUE 2048              // its room: those and what four groups of 32 items may add

struct __align__(16) RowHalf {
    float z[4];                     // its pixels' depths
    uint32_t cov;                   // bit j: pixel j is covered
    uint32_t in, out;               // its colour when its first pixel passes, and when it does not
    uint32_t pad;                   // (R and B swapped as they are stored, but for modes that blend in RGBA order)
};
struct __align__(16) RowEntry {
    uint32_t x;                     // first pixel of its first half in the batch
    uint32_t n;                     // halves | place of the first in the batch << 8 | kind << 16
    uint32_t rstate;
    uint32_t ref;                   // item, or pool index with the top bit
};
struct RowShared {
    SPrim rec[2][ROW_BATCH];
    RowHalf half[2][ROW_HALVES];
    RowEntry entry[3][ROW_BATCH];
    uint32_t queue[ROW_QUEUE];
    uint32_t nEntries[3], nHalves[3];
    uint32_t tail[2], head[2];      // of the queue, as of the last steps
    uint32_t found[2];              // whether nothing more comes
    uint32_t last;                  // the step that made the last batch
};
static_assert(ROW_AHEAD + 4 * 32 * PF_MAX_SUBTRIS <= ROW_QUEUE && (ROW_QUEUE & (ROW_QUEUE - 1)) == 0, "room for four groups' records");
static_assert(ROW_HALVES < 256 && PFP_KIND < 256, "fields of RowEntry.n");

// Blending in the stored order is the same for the modes that treat R and B
// alike: none, and alpha.  (SUB's channels are ORed without masks.)
__device__ __forceinline__ bool row_swapped(uint32_t rs) { return !(rs & PFS_BLEND) || (rs >> 24) == 1u; }

__device__ __forceinline__ const PFPrim *row_prim(const RasterArgs &a, uint32_t ref)
{
    return (ref & 0x80000000u) ? a.pool + (ref & 0x7fffffffu) : a.prims + ref;
}

// Half (xf, y) of a set-up triangle: everything that does not depend on the
// row's contents.  Returns the covered pixels.
template <bool PHONG>
__device__ __forceinline__ uint32_t row_half(const SPrim &R, const PFDrawState *states, uint32_t xf, uint32_t y, uint32_t W, RowHalf &H)
{
    const PFPrim &P = R.p;
    const uint32_t xEnd = min((uint32_t)P.xMax, W), rs = P.rstate;
    // edge functions at pixel (x, y): (x - rx) sx + (y - ry) sy, 32-bit
    // wrapping (triangles.c:336-349, 398-420)
    int32_t sx[3] = { P.y3 - P.y2, P.y1 - P.y3, P.y2 - P.y1 };
    int32_t sy[3] = { P.x2 - P.x3, P.x3 - P.x1, P.x1 - P.x2 };
    const int32_t rx[3] = { P.x2, P.x3, P.x1 }, ry[3] = { P.y2, P.y3, P.y1 };
    if (P.flags & 1u)
        for (int e = 0; e < 3; e++) { sx[e] = -sx[e]; sy[e] = -sy[e]; }
    uint32_t w[3];
    for (int e = 0; e < 3; e++)
        w[e] = (xf - (uint32_t)rx[e]) * (uint32_t)sx[e] + (y - (uint32_t)ry[e]) * (uint32_t)sy[e];
    float wf[3] = { 0.0f, 0.0f, 0.0f }, zl[4];
    uint32_t cov = 0;
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
        const float wn1 = (float)(int32_t)w[0] * P.wInvSum, wn2 = (float)(int32_t)w[1] * P.wInvSum;
        const float wn3 = (float)(int32_t)w[2] * P.wInvSum;
        float zs = P.z1 * wn1 + P.z2 * wn2;
        zs = zs + P.z3 * wn3;
        zl[j] = __frcp_rn(zs);
        if (j == 0) { wf[0] = wn1; wf[1] = wn2; wf[2] = wn3; }
        if (xf + j < xEnd && (int32_t)(w[0] | w[1] | w[2]) > 0) cov |= 1u << j;
        for (int e = 0; e < 3; e++) w[e] += (uint32_t)sx[e];
    }
    H.z[0] = zl[0]; H.z[1] = zl[1]; H.z[2] = zl[2]; H.z[3] = zl[3];
    H.cov = cov;
    if (cov) {
        // the colours of the outcomes there can be: the first pixel outside
        // the mask unless it is covered and no depth test can take it out
        const bool in = (cov & 1u) != 0, out = !in || (rs & PFS_DEPTH_TEST);
        uint32_t c = 0;
        if (in) c = shade_fragment<PHONG>(P, R.ph, states, wf[0], wf[1], wf[2], zl[0], true, true);
        H.in = row_swapped(rs) ? pff_swap_rb(c) : c;
        if (out && (!in || (rs & PFS_TEXTURE))) c = shade_fragment<PHONG>(P, R.ph, states, wf[0], wf[1], wf[2], zl[0], false, true);
        H.out = row_swapped(rs) ? pff_swap_rb(c) : c;
    }
    return (uint32_t)__popc(cov);
}

// The pixels of a row, colour and depth bits: in shared memory, or in place.
template <bool SMEM> struct RowPixels;
template <> struct RowPixels<true> {
    uint2 *p;
    __device__ __forceinline__ uint2 get(uint32_t x) const { return p[x]; }
    __device__ __forceinline__ void set(uint32_t x, uint32_t c, uint32_t d) const { p[x] = make_uint2(c, d); }
};
template <> struct RowPixels<false> {
    uint32_t *c;
    float *d;
    __device__ __forceinline__ uint2 get(uint32_t x) const { return make_uint2(c[x], __float_as_uint(d[x])); }
    __device__ __forceinline__ void set(uint32_t x, uint32_t cv, uint32_t dv) const { c[x] = cv; d[x] = __uint_as_float(dv); }
};

// A point, line or rectangle over n halves of row y from pixel x on; returns
// the fragments it counted.
template <bool SMEM>
__device__ __noinline__ uint32_t row_scalar(const PFPrim &P, uint32_t rs, uint32_t x0, uint32_t n, RowPixels<SMEM> row,
                                            uint32_t W, uint32_t y, uint32_t lane)
{
    const uint32_t xEnd = min(min((uint32_t)P.xMax, W), x0 + 4u * n);
    uint32_t cov = 0;
    for (uint32_t x = x0 + lane; x < xEnd; x += 32) {
        if (!lp_covers(P, (int32_t)x, (int32_t)y)) continue;
        if ((P.flags & PFP_KIND) != PFP_BLIT) cov++;
        const float z = lp_depth(P, (int32_t)x, (int32_t)y);
        const uint2 p = row.get(x);
        if ((rs & PFS_DEPTH_TEST) && !depth_sisd((int)((rs >> 16) & 255u), z, __uint_as_float(p.y))) continue;
        uint32_t c = lp_color(P, (int32_t)x, (int32_t)y);
        if (rs & PFS_BLEND) c = blend_sisd((int)(rs >> 24), c, pff_swap_rb(p.x));
        row.set(x, pff_swap_rb(c), (rs & PFS_DEPTH_MASK) ? __float_as_uint(z) : p.y);
    }
    return cov;
}

// The warp that looks for the row's records, in order.
struct RowFinder {
    int si;                         // segment
    uint32_t gBegin, gEnd;          // its items
    uint32_t cb, cEnd;              // next group of 32 items to look at
    uint32_t base, m[4];            // groups that reach the row, of the 128 from base on
    uint32_t tail;                  // of the queue
    bool done;                      // no group left
};

__device__ __forceinline__ bool on_row(uint64_t w, uint64_t some, uint32_t y)
{
    return (w & some) && ((w >> 16) & 0xffffffu) <= y && (w >> 40) >= y;
}

// Puts records that may reach row y of target t on the queue until it holds
// ROW_AHEAD.  The whole warp calls it.
__device__ __forceinline__ void row_find(const RasterArgs &a, RowFinder &F, RowShared &S, const PFSegment *__restrict__ segs, int nSegs,
                                         const uint64_t *__restrict__ rowInfo, const uint64_t *__restrict__ rowGroup,
                                         int t, uint32_t y, uint32_t head)
{
    const uint32_t lane = threadIdx.x & 31u, all = 0xffffffffu;
    while (F.tail - head < (uint32_t)ROW_AHEAD && !F.done) {
        if (!(F.m[0] | F.m[1] | F.m[2] | F.m[3])) {
            // the next 128 groups
            while (F.cb >= F.cEnd && !F.done) {
                do F.si++; while (F.si < nSegs && (segs[F.si].target != t || segs[F.si].nItems == 0));
                if (F.si >= nSegs) { F.done = true; break; }
                F.gBegin = segs[F.si].itemBase; F.gEnd = F.gBegin + segs[F.si].nItems;
                F.cb = F.gBegin >> 5; F.cEnd = ((F.gEnd - 1u) >> 5) + 1u;
            }
            if (F.done) break;
            uint64_t w[4];
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) { const uint32_t c = F.cb + 32u * i + lane; w[i] = c < F.cEnd ? __ldg(rowGroup + c) : 0ull; }
#pragma unroll
            for (uint32_t i = 0; i < 4; i++) F.m[i] = __ballot_sync(all, on_row(w[i], 1ull, y));
            F.base = F.cb;
            F.cb += 128u;
            continue;
        }
        // the items' records of the next four groups that may reach the row
        // (four loads under way instead of one)
        uint32_t g[4];
        uint64_t w[4];
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) {
            uint32_t at = 0xffffffffu;
#pragma unroll
            for (uint32_t i = 0; i < 4; i++)
                if (at == 0xffffffffu && F.m[i]) {
                    at = F.base + 32u * i + (uint32_t)(__ffs(F.m[i]) - 1);
                    F.m[i] &= F.m[i] - 1u;
                }
            g[q] = at == 0xffffffffu ? 0xffffffffu : (at << 5) + lane;
            w[q] = (g[q] >= F.gBegin && g[q] < F.gEnd) ? __ldg(rowInfo + g[q]) : 0ull;
        }
#pragma unroll
        for (uint32_t q = 0; q < 4; q++) {
            const uint32_t subs = on_row(w[q], 0xffffull, y) ? (uint32_t)w[q] & 0xffffu : 0u;
            uint32_t total;
            uint32_t at = F.tail + warp_offsets((uint32_t)__popc(subs), total);
            const uint32_t pb = (subs & ~1u) ? (uint32_t)__ldg(&a.prims[g[q]].poolBase) : 0u;
            for (uint32_t mm = subs; mm; mm &= mm - 1u, at++) {
                const uint32_t sub = (uint32_t)(__ffs(mm) - 1);
                S.queue[at & (ROW_QUEUE - 1)] = sub ? 0x80000000u | (pb + sub - 1u) : g[q];
            }
            F.tail += total;
        }
    }
}

// Makes the next batch of row y from the queue's records [head, tail) and
// loads its records into slot `step` of the buffers; part: halves of the
// first one that are in an earlier batch.  The whole warp calls it.
template <bool PHONG>
__device__ __forceinline__ void row_batch(const RasterArgs &a, RowShared &S, uint32_t &head, uint32_t tail, uint32_t &part, bool found,
                                          uint32_t W, uint32_t y, uint32_t step)
{
    const uint32_t lane = threadIdx.x & 31u, all = 0xffffffffu;
    // whole records while their halves fit, and part of the next
    const uint32_t n = min((uint32_t)ROW_BATCH, tail - head);
    uint32_t ref = 0, x = 0, len = 0, rs = 0, kind = 0;
    const uint32_t t0 = lane == 0 ? part : 0u;
    if (lane < n) {
        ref = S.queue[(head + lane) & (ROW_QUEUE - 1)];
        SPrim &R = S.rec[step & 1u][lane];
        const int4 *src = reinterpret_cast<const int4 *>(row_prim(a, ref));
        int4 r[8];
        for (int i = 0; i < 8; i++) r[i] = __ldg(src + i);
        for (int i = 0; i < 8; i++) reinterpret_cast<int4 *>(&R.p)[i] = r[i];
        if (PHONG) R.ph = (ref & 0x80000000u) ? a.poolPh + (ref & 0x7fffffffu) : a.primsPh + ref;
        rs = (uint32_t)r[4].w; kind = (uint32_t)r[2].z & PFP_KIND;
        // the row and columns as tile_edge clips a box: y in [yMin, yMax], x
        // in [xMin, xMax), inside the framebuffer (unsigned)
        const uint32_t xMin = (uint32_t)r[1].z, xEnd = min((uint32_t)r[2].x, W);
        if (xMin < xEnd && y >= (uint32_t)r[1].w && y <= (uint32_t)r[2].y) {
            len = (xEnd - xMin + 3u) / 4u - t0;
            x = xMin + 4u * t0;
        }
    }
    uint32_t total;
    const uint32_t h0 = warp_offsets(min(len, (uint32_t)ROW_HALVES + 1u), total);
    const uint32_t fit = h0 >= (uint32_t)ROW_HALVES ? 0u : min(len, (uint32_t)ROW_HALVES - h0);
    const uint32_t over = __ballot_sync(all, lane < n && fit < len);
    const uint32_t whole = over ? (uint32_t)(__ffs(over) - 1) : n;             // records finished by this batch
    uint32_t cut = __shfl_sync(all, fit, (int)(whole & 31u));
    if (!over) cut = 0u;                                                        // halves taken of the next
    const uint32_t entries = whole + (cut ? 1u : 0u), s3 = step % 3u;
    if (lane < entries) S.entry[s3][lane] = RowEntry{ x, fit | h0 << 8 | kind << 16, rs, ref };
    const uint32_t end = __shfl_sync(all, h0 + fit, (int)((entries - 1u) & 31u));
    part = over ? (whole == 0 ? part : 0u) + cut : 0u;
    head += whole;
    if (lane == 0) {
        S.nEntries[s3] = entries; S.nHalves[s3] = entries ? end : 0u;
        if (found && head == tail) S.last = step;
    }
}

// SMEM: the row's colour and depth are kept in shared memory (rows up to
// ROW_SMEM_MAX_W pixels), else they are drawn in place.
#define ROW_SMEM_MAX_W 2048
template <bool SMEM, bool PHONG>
__global__ void __launch_bounds__(ROW_THREADS, 5) k_rows(RasterArgs a, const PFSegment *__restrict__ segs, int nSegs,
                                                         const uint64_t *__restrict__ rowInfo,
                                                         const uint64_t *__restrict__ rowGroup, uint32_t rowW)
{
    extern __shared__ __align__(16) unsigned char rowSmem[];
    RowShared &S = *reinterpret_cast<RowShared *>(rowSmem);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // k_raster is done
    if (a.cnt->abortCommand <= a.command) return;
    // my row: row y of the BGRA / unsigned-byte targets, in target order
    uint32_t y = blockIdx.x;
    int t = 0;
    for (; t < a.nTargets; t++) {
        if (a.targets[t].fmt != PFF_BGRA8) continue;
        if (y < a.targets[t].H) break;
        y -= a.targets[t].H;
    }
    if (t >= a.nTargets) return;
    const PFTarget &T = a.targets[t];
    const uint32_t W = T.W;
    uint32_t *gcol = static_cast<uint32_t *>(T.color) + (size_t)y * W;
    float *gdep = T.depth + (size_t)y * W;
    RowPixels<SMEM> row;
    if constexpr (SMEM) row.p = reinterpret_cast<uint2 *>(rowSmem + sizeof(RowShared));
    else { row.c = gcol; row.d = gdep; }
    // the row as the draws find it: the fused clear (pfClear keeps pixels
    // 0..7), or the framebuffer's contents
    for (uint32_t x = tid; x < W; x += ROW_THREADS) {
        const bool clr = T.clearMode == 2 || (T.clearMode == 1 && (size_t)y * W + x >= 8);
        if (clr) row.set(x, T.clearRaw[0], __float_as_uint(T.clearDepth));
        else if (SMEM) row.set(x, gcol[x], __float_as_uint(gdep[x]));
    }
    if (tid == 0) {
        S.last = 0xffffffffu;
        for (int i = 0; i < 2; i++) S.head[i] = S.tail[i] = S.found[i] = 0u;
    }
    __syncthreads();
    RowFinder F{ -1, 0, 0, 0, 0, 0, { 0, 0, 0, 0 }, 0, false };
    uint32_t head = 0, part = 0;
    unsigned long long frags = 0;
    // step s looks ahead, makes batch s of the records found before it, works
    // out the halves of batch s - 1 and draws batch s - 2
    for (uint32_t step = 0;; step++) {
        const uint32_t last = S.last;                      // (this step may write it: nothing differs before two steps on)
        if (last != 0xffffffffu && step > last + 2u) break;
        if (warp == 4) {
            if (!S.found[(step + 1u) & 1u]) row_find(a, F, S, segs, nSegs, rowInfo, rowGroup, t, y, S.head[(step + 1u) & 1u]);
            __syncwarp();
            if (lane == 0) { S.tail[step & 1u] = F.tail; S.found[step & 1u] = F.done; }
        } else if (warp == 1) {
            if (last == 0xffffffffu)
                row_batch<PHONG>(a, S, head, S.tail[(step + 1u) & 1u], part, S.found[(step + 1u) & 1u] != 0, W, y, step);
            if (lane == 0) S.head[step & 1u] = head;
        } else if (warp >= 2) {
            if (step >= 1 && step - 1u <= last) {
                const uint32_t b = step - 1u, nE = S.nEntries[b % 3u], nH = S.nHalves[b % 3u];
                const RowEntry *E = S.entry[b % 3u];
                for (uint32_t h = tid - 64u; h < nH; h += 64u) {
                    // its entry: the last one that starts at or before it
                    uint32_t lo = 0, hi = nE - 1u;
                    while (lo < hi) { const uint32_t mid = (lo + hi + 1u) >> 1; if (((E[mid].n >> 8) & 255u) <= h) lo = mid; else hi = mid - 1u; }
                    const RowEntry e = E[lo];
                    if (!(e.n >> 16))
                        frags += row_half<PHONG>(S.rec[b & 1u][lo], a.states, e.x + 4u * (h - ((e.n >> 8) & 255u)), y, W, S.half[b & 1u][h]);
                }
            }
        } else if (step >= 2 && step - 2u <= last) {
            const uint32_t b = step - 2u, nE = S.nEntries[b % 3u];
            const RowEntry *E = S.entry[b % 3u];
            const RowHalf *H = S.half[b & 1u];
            // a lane a pixel, eight halves at a time; the next record's entry
            // and halves are read while one is drawn.  A lane reads and
            // writes its own pixel only: the first pixel's colour and its
            // outcome come from its lane.
            const uint32_t j = lane & 3u, k0 = lane >> 2, quad = lane & 28u;
            RowEntry e{};
            float z = 0.0f;
            uint4 c = make_uint4(0, 0, 0, 0);                  // cov, in, out
            auto fetch = [&](uint32_t i, RowEntry &en, float &zn, uint4 &cn) {
                en.n = 0;
                cn.x = 0;
                if (i < nE) {
                    en = E[i];
                    if (k0 < (en.n & 255u) && !(en.n >> 16)) {
                        const RowHalf &h = H[((en.n >> 8) & 255u) + k0];
                        zn = h.z[j];
                        cn = *reinterpret_cast<const uint4 *>(&h.cov);
                    }
                }
            };
            fetch(0, e, z, c);
            for (uint32_t i = 0; i < nE; i++) {
                RowEntry en;
                float zn = 0.0f;
                uint4 cn;
                fetch(i + 1u, en, zn, cn);
                const uint32_t rs = e.rstate, n = e.n & 255u;
                if (e.n >> 16) {
                    frags += row_scalar<SMEM>(*row_prim(a, e.ref), rs, e.x, n, row, W, y, lane);
                } else {
                    for (uint32_t h = 0;;) {
                        const uint32_t x = e.x + 4u * (h + k0) + j;
                        uint2 p = make_uint2(0, 0);
                        if (c.x && x < W) p = row.get(x);
                        bool pass = (c.x >> j) & 1u;
                        if (rs & PFS_DEPTH_TEST) {
                            const uint32_t func = (rs >> 16) & 255u;
                            const float d = __uint_as_float(p.y);
                            pass = pass && (func == 2u ? z < d : depth_simd((int)func, z, d));
                        }
                        const uint32_t m = __ballot_sync(0xffffffffu, pass) >> quad;
                        // the half's value: its first pixel's colour and destination
                        uint32_t frag = (m & 1u) ? c.y : c.z;
                        if (rs & PFS_BLEND) {
                            const uint32_t dst = __shfl_sync(0xffffffffu, p.x, (int)quad);
                            const uint32_t mode = rs >> 24;
                            frag = mode == 1u ? blend_simd(1, frag, dst) : pff_swap_rb(blend_simd((int)mode, frag, pff_swap_rb(dst)));
                        }
                        if (pass) row.set(x, frag, (rs & PFS_DEPTH_MASK) ? __float_as_uint(z) : p.y);
                        h += 8u;
                        if (h >= n) break;
                        c.x = 0;                               // (more than eight halves)
                        if (h + k0 < n) {
                            const RowHalf &q = H[((e.n >> 8) & 255u) + h + k0];
                            z = q.z[j];
                            c = *reinterpret_cast<const uint4 *>(&q.cov);
                        }
                    }
                }
                __syncwarp();                                  // the record's pixels are written
                e = en;
                z = zn;
                c = cn;
            }
        }
        __syncthreads();
    }
    if (SMEM)
        for (uint32_t x = tid; x < W; x += ROW_THREADS) { const uint2 p = row.get(x); gcol[x] = p.x; gdep[x] = __uint_as_float(p.y); }
    for (int o = 16; o > 0; o >>= 1) frags += __shfl_down_sync(0xffffffffu, frags, o);
    if (lane == 0 && frags) atomicAdd(&a.cnt->fragments, frags);
}

// ---------------------------------------------------------------------------
// framebuffer-wide passes
// ---------------------------------------------------------------------------
// pfClear, SIMD build (context.c:680-745): pixels [8, n - n%8) take the clear
// value (as the SIMD setter stores it), the tail copies pixel 0's bytes,
// pixels 0..7 are left as they are.  For the packed 16-bit formats the
// reference steps the tail copy by components x 2 bytes (pixel.h:3156-3210),
// past the pixels: their tail keeps its colour (the depth tail is copied).
__global__ void k_clear(void *color, uint32_t fmt, float *depth, size_t n, uint4 cc, float cd,
                        const PFDevCounters *cnt, uint32_t command)
{
    if (cnt->abortCommand <= command) return;
    const size_t aligned = n - (n % 8);
    const uint32_t craw[4] = { cc.x, cc.y, cc.z, cc.w };
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        // the vector loop starts at pixel 8; the tail starts at `aligned`,
        // which is 0 below 8 pixels (then every pixel takes pixel 0's value)
        if (i < aligned ? i < 8 : i == 0) continue;
        if (fmt == PFF_RGBA8) {
            uint32_t *c32 = (uint32_t *)color;
            if (i < aligned) c32[i] = cc.x; else c32[i] = c32[0];
        } else if (i < aligned) pff_store(fmt, color, i, craw);
        else if (pff_bytes(fmt) != 2) { uint32_t r[4]; pff_load(fmt, color, 0, r); pff_store(fmt, color, i, r); }
        depth[i] = (i < aligned) ? cd : depth[0];
    }
}

// pfClearFramebuffer (framebuffer.c:89-102): every pixel, through the
// scalar setter.
__global__ void k_fill(void *color, uint32_t fmt, float *depth, size_t n, uint4 cc, float cd,
                       const PFDevCounters *cnt, uint32_t command)
{
    if (cnt->abortCommand <= command) return;
    const uint32_t craw[4] = { cc.x, cc.y, cc.z, cc.w };
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        if (fmt == PFF_RGBA8) ((uint32_t *)color)[i] = cc.x;
        else pff_store(fmt, color, i, craw);
        depth[i] = cd;
    }
}

// Post-process hooks (pfPostProcess, context.c:2397-2441) and pfFogProcess
// (context.c:2288-2351) on the colour c of pixel i, as the scalar getter
// reads it.  The hooks rewrite every pixel; the fog writes only the pixels
// past its start (false: keep the pixel).
__device__ __forceinline__ bool hook_pixel(uint32_t &c, float depth, size_t i, int hook, const PFHookParams &hp)
{
    bool write = true;
    if (hook == 1) {          // linear fog on depth
        float d = (depth + hp.znear) / (hp.zfar + hp.znear);
        float f = (hp.end - d) / (hp.end - hp.start);
        f = x86_min(x86_max(f, 0.0f), 1.0f);
        uint32_t k = (uint32_t)x86_cvt_trunc(f * 255.0f);
        uint32_t r = 0;
        for (int ch = 0; ch < 4; ch++) r |= (((chn(c, ch) * k + chn(hp.color, ch) * (255u - k)) / 255u) & 255u) << (8 * ch);
        c = r;
    } else if (hook == 3) {   // pfFogProcess (context.c:2288-2351)
        const float d = depth;
        write = d > hp.start;
        const uint32_t alpha = hp.color >> 24, fc = hp.color & 0x00ffffffu;
        if (d >= hp.end) {
            const uint32_t f = fc | (alpha << 24);
            c = alpha == 255u ? f : blend_sisd(1, f, c);
        } else if (d > hp.start) {
            float t = 0.0f;
            const float invLen = __frcp_rn(hp.end - hp.start);
            if (hp.mode == 0) t = (d - hp.start) * invLen;
            else if (hp.mode == 1) t = 1.0f - (float)exp((double)(-hp.density * (d - hp.start)));
            else if (hp.mode == 2) t = 1.0f - (float)exp2((double)(-hp.density * (d - hp.start)));
            const uint32_t a = (uint32_t)x86_cvt_trunc(t * (float)alpha) & 255u;
            c = blend_sisd(1, fc | (a << 24), c);
        }
    } else if (hook == 2) {   // grayscale
        uint32_t gy = (77u * chn(c, 0) + 150u * chn(c, 1) + 29u * chn(c, 2)) >> 8;
        c = gy | (gy << 8) | (gy << 16) | (c & 0xff000000u);
    } else if (hook == 4) {   // ordered 3x3 dither (examples/raylib/raylib_PostProcess.c:7-19)
        const uint32_t x = (uint32_t)(i % hp.width), y = (uint32_t)(i / hp.width);
        // the matrix {{230, 51, 128}, {25, 102, 179}, {154, 205, 77}}, row
        // x % 3, column y % 3: its first eight bytes packed low to high
        const uint32_t m = x % 3u * 3u + y % 3u;
        const uint32_t dv = m < 8u ? (uint32_t)((0xCD9AB366198033E6ull >> (8u * m)) & 255u) : 77u;
        const uint32_t avg = (chn(c, 0) + chn(c, 1) + chn(c, 2)) / 3u;
        c = (avg >= dv) ? 0xffffffffu : 0u;
    }
    return write;
}

// RGBA / unsigned byte (whose scalar getter and setter are the identity):
// four pixels a thread in 16-byte accesses, a thread's loads all under way at
// once.  Bound by its loads' latency: one pixel a thread and step, 20 us for
// the 1080p linear fog, now 8.7 (24.9 MB read and written).
__global__ void k_hook(void *color, uint32_t fmt, const float *depth, size_t n, int hook, PFHookParams hp,
                       const PFDevCounters *cnt, uint32_t command)
{
    if (cnt->abortCommand <= command) return;
    const size_t first = blockIdx.x * (size_t)blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
    size_t done = 0;
    if (fmt == PFF_RGBA8 && (((uintptr_t)color | (uintptr_t)depth) & 15u) == 0) {
        const size_t n4 = n / 4;
        for (size_t q = first; q < n4; q += stride) {
            uint4 v = reinterpret_cast<const uint4 *>(color)[q];
            const float4 z = reinterpret_cast<const float4 *>(depth)[q];
            // (a pixel the hook leaves is stored as it was read)
            const uint4 o = v;
            if (!hook_pixel(v.x, z.x, 4 * q, hook, hp)) v.x = o.x;
            if (!hook_pixel(v.y, z.y, 4 * q + 1, hook, hp)) v.y = o.y;
            if (!hook_pixel(v.z, z.z, 4 * q + 2, hook, hp)) v.z = o.z;
            if (!hook_pixel(v.w, z.w, 4 * q + 3, hook, hp)) v.w = o.w;
            reinterpret_cast<uint4 *>(color)[q] = v;
        }
        done = 4 * n4;
    }
    for (size_t i = done + first; i < n; i += stride) {
        uint32_t raw[4];
        pff_load(fmt, color, i, raw);
        uint32_t c = pff_get_sisd(fmt, raw);
        if (hook_pixel(c, depth[i], i, hook, hp)) {
            pff_set_sisd(fmt, c, raw);
            pff_store(fmt, color, i, raw);
        }
    }
}

// The largest of n u32 indices (already on the device, 16-byte aligned):
// per-warp maxima folded into *out with one atomic per warp.
__global__ void k_max_u32(const uint32_t *src, size_t n, unsigned *out)
{
    const size_t n4 = n / 4;
    const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
    unsigned m = 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n4; i += stride) {
        const uint4 v = __ldg(s4 + i);
        m = max(m, max(max(v.x, v.y), max(v.z, v.w)));
    }
    for (size_t i = n4 * 4 + blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += stride) m = max(m, __ldg(src + i));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers (called by pf_host.cpp)
// ---------------------------------------------------------------------------
static inline unsigned grid_for(size_t n, unsigned block) { return (unsigned)((n + block - 1) / block); }

// The three pipeline kernels are launched with programmatic stream
// serialization: a kernel's CTAs may be scheduled as the previous kernel's
// last CTAs exit (no early trigger is issued, so every CTA of the previous
// grid has left its SM by then), and each kernel starts with
// griddepcontrol.wait, which returns once the previous grid has completed
// and its memory is visible.  What this hides is the launch gap between
// the kernels of a frame.
template <typename... KArgs, typename... Args>
static cudaError_t launch_serialized(void (*kernel)(KArgs...), unsigned grid, unsigned block, size_t smem,
                                     cudaStream_t st, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

int pfd_sm_count(void)
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
            cudaGetLastError();
            sms = 152;
        }
    }
    return sms;
}

// k_vertex starts a launch's chain: its predecessors in the stream are the
// uploads, the counter reset and the wait for the draw-time copies, so it
// is launched without programmatic serialization (its griddepcontrol.wait
// then returns at once).
cudaError_t pfd_launch_vertex(const PFBatchLaunch &L, cudaStream_t st)
{
    const uint32_t nTiles = L.totalTiles;
    const size_t work = L.nVerts > nTiles ? L.nVerts : nTiles;
    k_vertex<<<grid_for(work, 128), 128, 0, st>>>(L.segs, L.nSegs, L.states, L.vout, L.nVerts, L.cnt, L.binCount, nTiles,
                                               L.targets, L.nTargets);
    return cudaGetLastError();
}

cudaError_t pfd_launch_items(const PFBatchLaunch &L, cudaStream_t st)
{
    if (L.nItems == 0) return cudaSuccess;
    BinArgs B{ L.binCount, L.tileList, L.listStride, L.bins, L.cap, L.targets, L.cnt, L.command, L.planes,
               L.nItems / 8u >= L.totalTiles };
    ItemOut O{ L.prims, L.primsPh, L.pool, L.poolPh, L.poolCap, L.rowCount ? L.rowInfo : nullptr, L.rowGroup };
    // Items a warp: a full warp of 32 sets up fastest, but a small launch
    // then leaves most of the GPU idle while a few warps bin all its tiles.
    // Fewer items a warp until there are 12 warps an SM (half of what is
    // resident; all 24 measured slower): 2,000 soup triangles 66 (32 a warp)
    // -> 16 us (1), 8,192 small ones 20 -> 12 us (4; 2: 15.5), 20,480 mesh
    // items 22.5 -> 12.5 us (8; 4: 15); 131,072 stay at 32 (20.6 us; 16: 22).
    // k_rows' summaries are one a warp of 32.
    uint32_t perWarp = 32;
    if (!O.rowInfo)
        while (perWarp > 1 && L.nItems / perWarp < (uint32_t)pfd_sm_count() * 12u) perWarp >>= 1;
    return launch_serialized(k_items, grid_for(L.nItems, 4 * perWarp), 128, 0, st, L.segs, L.nSegs, L.states,
                             (const PFVertexOut *)L.vout, L.nItems, perWarp, O, B);
}

// Dynamic shared memory of k_raster: the warps' batch buffers (a record's
// per-fragment lighting data is read through L1 when a fragment is shaded,
// not staged: the CTAs' shared memory would bound how many fit on an SM).
static size_t raster_smem(int warps)
{
    return (size_t)warps * sizeof(QWarp);
}

static RasterArgs raster_args(const PFBatchLaunch &L)
{
    return RasterArgs{ L.binCount, L.tileList, L.listStride, L.bins, L.cap, L.prims, L.primsPh, L.planes, L.pool, L.poolPh, L.states,
                       L.targets, L.nTargets, L.totalTiles, L.cnt, L.command, L.anyPhong, 0 };
}

// Persistent grid of `kernel`: as many CTAs as fit on the GPU at once, at
// most `perSM` per SM (0: as many as fit), at most `units`.
static cudaError_t persistent_grid(const void *kernel, int block, size_t smem, bool maxShared, int perSM, uint32_t units, uint32_t &grid)
{
    int fit = 0;
    cudaError_t e = pfd_ctas_per_sm(kernel, block, smem, maxShared, fit);
    if (e != cudaSuccess) return e;
    uint32_t per = (uint32_t)(fit > 0 ? fit : 1);
    if (perSM > 0) per = min(per, (uint32_t)perSM);
    grid = max(1u, min(units, (uint32_t)pfd_sm_count() * per));
    return cudaSuccess;
}

cudaError_t pfd_launch_binsort(const PFBatchLaunch &L, cudaStream_t st)
{
    if (L.totalTiles == 0) return cudaSuccess;
    uint32_t N = 32; while (N < L.cap) N <<= 1;
    size_t smem = 2 * (size_t)N * sizeof(uint32_t);                   // merge source and target
    RasterArgs A = raster_args(L);
    if (L.itemSpan > 0 && L.itemSpan <= SORT_MAP_ITEMS) {
        A.sortGroups = 16;
        while (A.sortGroups < L.itemSpan / 128u + 2u) A.sortGroups <<= 1;
        const size_t maps = (SORT_THREADS / 32) * (size_t)A.sortGroups * sizeof(uint4);
        smem = smem > maps ? smem : maps;
    }
    uint32_t grid = 0;
    void (*kernel)(RasterArgs) = A.sortGroups ? k_binsort<true> : k_binsort<false>;
    cudaError_t e = persistent_grid((const void *)kernel, SORT_THREADS, smem, false, 0, L.totalTiles, grid);
    if (e != cudaSuccess) return e;
    return launch_serialized(kernel, grid, SORT_THREADS, smem, st, A);
}

template <bool GEN, bool PHONG> static void (*raster_kernel(int warps))(RasterArgs)
{
    return warps == 2 ? k_raster<GEN, 2, PHONG> : warps == 8 ? k_raster<GEN, 8, PHONG> : k_raster<GEN, 4, PHONG>;
}

cudaError_t pfd_launch_raster(const PFBatchLaunch &L, cudaStream_t st)
{
    if (L.totalTiles == 0) return cudaSuccess;
    const int warps = (L.rasterWarps == 2 || L.rasterWarps == 8) ? L.rasterWarps : 4;
    const size_t smem = raster_smem(warps);
    void (*kernel)(RasterArgs) =
        L.generic ? (L.anyPhong ? raster_kernel<true, true>(warps) : raster_kernel<true, false>(warps))
                  : (L.anyPhong ? raster_kernel<false, true>(warps) : raster_kernel<false, false>(warps));
    uint32_t grid = 0;
    cudaError_t e = persistent_grid((const void *)kernel, warps * 32, smem, true, L.rasterCtasPerSM,
                                    (2u * L.totalTiles + (uint32_t)warps - 1) / (uint32_t)warps, grid);       // half tiles
    if (e != cudaSuccess) return e;
    e = launch_serialized(kernel, grid, (unsigned)(warps * 32), smem, st, raster_args(L));
    if (e != cudaSuccess || L.rowCount == 0 || !L.rowInfo || !L.rowGroup) return e;
    const bool inSmem = L.rowMaxW <= ROW_SMEM_MAX_W;
    const uint32_t rowW = (L.rowMaxW + 255u) & ~255u;                                   // (few sizes: pfd_ctas_per_sm keeps them)
    const size_t rsm = sizeof(RowShared) + (inSmem ? (size_t)rowW * 8 : 0);            // colour and depth of the row
    auto rows = inSmem ? (L.anyPhong ? k_rows<true, true> : k_rows<true, false>)
                       : (L.anyPhong ? k_rows<false, true> : k_rows<false, false>);
    int fit = 0;
    e = pfd_ctas_per_sm((const void *)rows, ROW_THREADS, rsm, false, fit);
    if (e != cudaSuccess) return e;
    return launch_serialized(rows, L.rowCount, ROW_THREADS, rsm, st, raster_args(L), L.segs, L.nSegs,
                             (const uint64_t *)L.rowInfo, (const uint64_t *)L.rowGroup, rowW);
}

cudaError_t pfd_launch_clear(void *color, uint32_t fmt, float *depth, size_t n, const uint32_t cc[4], float cd, bool all,
                             const PFDevCounters *cnt, uint32_t command, cudaStream_t st)
{
    unsigned grid = (unsigned)min((size_t)152 * 8, (n + 255) / 256);
    if (grid == 0) return cudaSuccess;
    const uint4 c4 = make_uint4(cc[0], cc[1], cc[2], cc[3]);
    if (all) k_fill<<<grid, 256, 0, st>>>(color, fmt, depth, n, c4, cd, cnt, command);
    else k_clear<<<grid, 256, 0, st>>>(color, fmt, depth, n, c4, cd, cnt, command);
    return cudaGetLastError();
}

cudaError_t pfd_launch_hook(void *color, uint32_t fmt, const float *depth, size_t n, int hook, const PFHookParams &hp,
                            const PFDevCounters *cnt, uint32_t command, cudaStream_t st)
{
    unsigned grid = (unsigned)min((size_t)pfd_sm_count() * 16, (n / 4 + 127) / 128 + 1);
    if (n == 0) return cudaSuccess;
    k_hook<<<grid, 128, 0, st>>>(color, fmt, depth, n, hook, hp, cnt, command);
    return cudaGetLastError();
}

cudaError_t pfd_max_u32(const uint32_t *d, size_t n, unsigned *dWord, unsigned *hWord, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(dWord, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    if (n) {
        const unsigned grid = (unsigned)min((size_t)pfd_sm_count() * 2, (n / 4 + 255) / 256 + 1);
        k_max_u32<<<grid, 256, 0, st>>>(d, n, dWord);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaMemcpyAsync(hWord, dWord, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
}


