// pf_grad.cu -- differentiable float relaxation of the triangle pipeline
// (the pfgrad* entry points of include/pixelforge_grad.h).
//
// Scene set-up (once per mesh and set of views):
//   k_gsetup    one thread per (view, triangle, face) item, in the reference's
//               order (triangle-major, FRONT pass before BACK): projection,
//               2D/3D decision and the reference's integer set-up and cull --
//               the same device code as the pipeline's k_items -- and a count
//               of the 16x16 tiles each set-up triangle overlaps
//   k_gscan     exclusive scan of the tile counts (one CTA)
//   k_gorder    the tiles that have triangles, and those that have none
//   k_gfill     item numbers into the tile lists (atomic slots)
//   k_gsort     per tile: restores item order (bitonic sort in shared memory)
// Every evaluation:
//   k_glight          one thread per (view, vertex): Gouraud Blinn-Phong in float
//   k_gforward        one CTA per tile, one warp per 8x8 block: coverage and
//                     depth test exactly as the reference list the block's
//                     visible fragments, then float shading densely over the
//                     warp and alpha-over in item order
//   k_gadjoint        the same list; per pixel the colour under each fragment
//                     and, from the front, the gradients of its colour and
//                     opacity; then texel gradients (vector atomics, pairs of
//                     neighbours on one texel combined first) and vertex
//                     gradients (summed per triangle and step)
//   k_glight_adjoint  one thread per (vertex, 8 views): back through the
//                     Gouraud Blinn-Phong formula; scalar gradients reduced per CTA
//   k_gfinish         light-direction normalisation adjoint
//
// The file is compiled with -fmad=false: coverage, depth and texel addressing
// use the same separately rounded arithmetic as the u8 pipeline.

#include <cuda_runtime.h>
#include <stdint.h>
#include <float.h>
#include <math.h>
#include <string.h>
#include <new>
#include "pf_layout.h"
#include "pixelforge_grad.h"

namespace {

#include "pf_common.cuh"

constexpr int GTILE = 16;
constexpr int GBLOCK = 8;          // a warp's block of pixels: 8x8, two a lane
constexpr int GTHREADS = 32 * (GTILE / GBLOCK) * (GTILE / GBLOCK);
constexpr int GCHUNK = 64;         // list entries staged at a time
constexpr int GFW = 128;           // fragments a block lists before they are blended
constexpr int RING = 4;            // visible fragments walked back per pixel per replay (blocks of more than GFW)
constexpr uint32_t GP_VALID = 1u << 31;

// A set-up triangle of one view, seven 16-byte words: the first six are what
// a fragment is shaded from, the last its box.
struct __align__(16) GPrim {
    int32_t ex[3];                 // edge functions x ex + y ey + c of pixel (x, y), in 32-bit wrap-around
    float wInvSum;                 // arithmetic: the reference's row starts and steps give the same values
    int32_t ey[3];
    uint32_t flags;                // bit0 face (1 = BACK), bit1 3D path, bit31 valid
    int32_t c[3];
    uint32_t v0;                   // vertex indices
    float z[3];                    // depth terms: 1/z_clip on the 3D path, z on the 2D path
    uint32_t v1;
    float su[3];                   // texture coordinates, times 1/z_clip on the 3D path
    uint32_t v2;
    float sv[3];
    uint32_t pad;
    int32_t xMin, yMin, xMax, yMax;  // pixels x in [xMin, xMax), y in [yMin, yMax] (unsigned compares)
};
static_assert(sizeof(GPrim) == 112, "GPrim is seven 16-byte words");

struct GTex {
    const float4 *tex;
    uint32_t w, h;
    int32_t wrap, filter;
    float tx, ty;
};

struct GView {
    uint32_t W, H, tilesX, tilesPerView;
    uint32_t nv;
    float bg[3];
    float clearDepth;
};

// ---------------------------------------------------------------------------
// set-up and binning
// ---------------------------------------------------------------------------
struct SetupArgs {
    const float *pos, *uv;
    const uint32_t *idx;
    uint32_t nv, nt, nViews, nFaces;
    int32_t face0;
    const float *mvp;              // nViews x 16
    const PFDrawState *S;          // viewport of the views
    GView view;
    GPrim *prims;
    uint32_t *tileCount;
    uint32_t *status;              // [0] items needing clipping, [1] valid prims
};

__device__ __forceinline__ bool gtile_range(const GView &V, const GPrim &P, uint32_t &tx0, uint32_t &ty0,
                                            uint32_t &ntx, uint32_t &nty)
{
    uint32_t x0 = (uint32_t)P.xMin, x1 = (uint32_t)P.xMax, y0 = (uint32_t)P.yMin, y1 = (uint32_t)P.yMax;
    if (x1 > V.W) x1 = V.W;
    if (y1 >= V.H) y1 = V.H - 1;
    if (x0 >= x1 || y0 > y1) return false;
    tx0 = x0 / GTILE; ty0 = y0 / GTILE;
    ntx = (x1 - 1) / GTILE - tx0 + 1; nty = y1 / GTILE - ty0 + 1;
    return true;
}

__global__ void k_gsetup(SetupArgs a)
{
    const uint32_t perView = a.nt * a.nFaces;
    const uint64_t total = (uint64_t)perView * a.nViews;
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    const uint32_t view = (uint32_t)(g / perView), r = (uint32_t)(g % perView);
    const uint32_t tri = r / a.nFaces;
    const int face = (a.nFaces == 2) ? (int)(r & 1u) : a.face0;
    GPrim &out = a.prims[g];
    out.flags = 0;
    const float *M = a.mvp + 16 * (size_t)view;
    uint32_t vi[3];
    float4 hv[3];
    for (int m = 0; m < 3; m++) {
        vi[m] = min(a.idx[3 * (size_t)tri + m], a.nv - 1);
        const float p[4] = { a.pos[3 * (size_t)vi[m]], a.pos[3 * (size_t)vi[m] + 1], a.pos[3 * (size_t)vi[m] + 2], 1.0f };
        float h[4];
        v4_transform(h, p, M);
        hv[m] = make_float4(h[0], h[1], h[2], h[3]);
    }
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
        if (!inside) { atomicAdd(&a.status[0], 1u); return; }
    }
    const PFDrawState &S = *a.S;
    SVert s[3];
    for (int m = 0; m < 3; m++) {
        const float4 h = hv[m];
        const float u = a.uv[2 * (size_t)vi[m]], v = a.uv[2 * (size_t)vi[m] + 1];
        if (is2D) {
            to_screen(S, h.x, h.y, s[m].sx, s[m].sy);
            s[m].z = h.z; s[m].u = u; s[m].v = v;
        } else {
            const float hz = 1.0f / h.z;
            s[m].u = u * hz; s[m].v = v * hz;
            const float invW = 1.0f / h.w;
            to_screen(S, h.x * invW, h.y * invW, s[m].sx, s[m].sy);
            s[m].z = hz;
        }
        s[m].c = 0;
    }
    PFPrim P;
    if (!setup_prim(S, face, !is2D, s[0], s[1], s[2], 0, P)) return;
    GPrim q;
    {
        // (triangles.c:331-349, 404-424)
        const int32_t rx[3] = { P.x2, P.x3, P.x1 }, ry[3] = { P.y2, P.y3, P.y1 };
        const int32_t sx[3] = { P.y3 - P.y2, P.y1 - P.y3, P.y2 - P.y1 }, sy[3] = { P.x2 - P.x3, P.x3 - P.x1, P.x1 - P.x2 };
        for (int e = 0; e < 3; e++) {
            q.ex[e] = face ? -sx[e] : sx[e];
            q.ey[e] = face ? -sy[e] : sy[e];
            q.c[e] = (int32_t)(0u - ((uint32_t)rx[e] * (uint32_t)q.ex[e] + (uint32_t)ry[e] * (uint32_t)q.ey[e]));
        }
    }
    q.xMin = P.xMin; q.yMin = P.yMin; q.xMax = P.xMax; q.yMax = P.yMax;
    q.wInvSum = P.wInvSum;
    q.flags = (uint32_t)face | (is2D ? 0u : 2u);
    q.v0 = vi[0]; q.v1 = vi[1]; q.v2 = vi[2]; q.pad = 0;
    for (int m = 0; m < 3; m++) { q.z[m] = s[m].z; q.su[m] = s[m].u; q.sv[m] = s[m].v; }
    uint32_t tx0, ty0, ntx, nty;
    if (!gtile_range(a.view, q, tx0, ty0, ntx, nty)) { out = q; return; }
    q.flags |= GP_VALID;
    out = q;
    atomicAdd(&a.status[1], 1u);
    const uint32_t base = view * a.view.tilesPerView;
    for (uint32_t ty = ty0; ty < ty0 + nty; ty++)
        for (uint32_t tx = tx0; tx < tx0 + ntx; tx++) atomicAdd(&a.tileCount[base + ty * a.view.tilesX + tx], 1u);
}

// Exclusive scan of n counts into off[0..n]; info[0] = longest list.
__global__ void __launch_bounds__(1024) k_gscan(const uint32_t *cnt, uint32_t *off, uint32_t n, uint32_t *info)
{
    __shared__ uint32_t warpSum[32];
    __shared__ uint32_t carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) carry = 0;
    uint32_t mx = 0;
    for (uint32_t b = 0; b < n; b += 1024) {
        __syncthreads();
        const uint32_t i = b + tid;
        const uint32_t v = i < n ? cnt[i] : 0u;
        mx = max(mx, v);
        uint32_t s = v;
        for (int o = 1; o < 32; o <<= 1) { uint32_t t = __shfl_up_sync(0xffffffffu, s, o); if (lane >= o) s += t; }
        if (lane == 31) warpSum[warp] = s;
        __syncthreads();
        if (warp == 0) {
            uint32_t w = warpSum[lane];
            for (int o = 1; o < 32; o <<= 1) { uint32_t t = __shfl_up_sync(0xffffffffu, w, o); if (lane >= o) w += t; }
            warpSum[lane] = w;
        }
        __syncthreads();
        const uint32_t excl = carry + (warp ? warpSum[warp - 1] : 0u) + s - v;
        if (i < n) off[i] = excl;
        __syncthreads();
        if (tid == 1023) carry = excl + v;
    }
    __syncthreads();
    if (tid == 0) off[n] = carry;
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) atomicMax(&info[0], mx);
}

// The tiles with a non-empty list into order[0 ..), the others from its end;
// nFull[0] and nFull[1] (zero before) count them.  Roughly in tile order.
__global__ void k_gorder(const uint32_t *off, uint32_t nTiles, uint32_t *order, uint32_t *nFull)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    const bool in = t < nTiles, full = in && off[t + 1] > off[t];
    const uint32_t m = __ballot_sync(0xffffffffu, full);
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(nFull, (unsigned)__popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (full) order[at + __popc(m & ((1u << lane) - 1u))] = t;
    const uint32_t e = __ballot_sync(0xffffffffu, in && !full);
    uint32_t ae = 0;
    if (lane == 0) ae = atomicAdd(nFull + 1, (unsigned)__popc(e));
    ae = __shfl_sync(0xffffffffu, ae, 0);
    if (in && !full) order[nTiles - 1u - (ae + __popc(e & ((1u << lane) - 1u)))] = t;
}

__global__ void k_gfill(const GPrim *prims, uint64_t total, GView V, uint32_t perView, const uint32_t *off,
                        uint32_t *fillCount, uint32_t *list)
{
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    const GPrim &P = prims[g];
    if (!(P.flags & GP_VALID)) return;
    uint32_t tx0, ty0, ntx, nty;
    if (!gtile_range(V, P, tx0, ty0, ntx, nty)) return;
    const uint32_t base = (uint32_t)(g / perView) * V.tilesPerView;
    for (uint32_t ty = ty0; ty < ty0 + nty; ty++)
        for (uint32_t tx = tx0; tx < tx0 + ntx; tx++) {
            const uint32_t t = base + ty * V.tilesX + tx;
            list[off[t] + atomicAdd(&fillCount[t], 1u)] = (uint32_t)g;
        }
}

// Sorts each tile's list ascending (item order).  Lists are at most `cap`
// long (a power of two, checked by the host).
__global__ void k_gsort(const uint32_t *off, uint32_t *list, uint32_t cap)
{
    extern __shared__ uint32_t sk[];
    const uint32_t t = blockIdx.x;
    const uint32_t beg = off[t], n = off[t + 1] - beg;
    if (n < 2) return;
    uint32_t *L = list + beg;
    int unsorted = 0;
    for (uint32_t i = threadIdx.x; i + 1 < n; i += blockDim.x) unsorted |= (L[i] > L[i + 1]);
    if (!__syncthreads_or(unsorted)) return;
    uint32_t N = 1; while (N < n) N <<= 1;
    if (N > cap) return;
    for (uint32_t i = threadIdx.x; i < N; i += blockDim.x) sk[i] = i < n ? L[i] : 0xffffffffu;
    __syncthreads();
    for (uint32_t k = 2; k <= N; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < N; i += blockDim.x) {
                const uint32_t ixj = i ^ j;
                if (ixj > i) {
                    const uint32_t x = sk[i], y = sk[ixj];
                    const bool up = (i & k) == 0;
                    if ((x > y) == up) { sk[i] = y; sk[ixj] = x; }
                }
            }
            __syncthreads();
        }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) L[i] = sk[i];
}

// ---------------------------------------------------------------------------
// vertex lighting (float relaxation of lighting.c:24-134, one directional
// light, Blinn half vector)
// ---------------------------------------------------------------------------
struct LightArgs {
    const float *pos, *nrm, *col, *alpha;
    const float *material;         // diffuse, specular, shininess
    const float *light;            // direction towards the light
    const float *eye;              // nViews x 3
    uint32_t nv, nViews;
    float ambient;
};

struct VertexTerms {
    float N[3], L[3], H[3];
    float hlen;                    // |L + V|
    float nl, nh, spec;
};

__device__ __forceinline__ void vertex_terms(const LightArgs &a, uint32_t v, uint32_t view, const float *Ldir,
                                             VertexTerms &t)
{
    float N[3] = { a.nrm[3 * (size_t)v], a.nrm[3 * (size_t)v + 1], a.nrm[3 * (size_t)v + 2] };
    v3_normalize(N);
    const float *E = a.eye + 3 * (size_t)view;
    float V[3] = { E[0] - a.pos[3 * (size_t)v], E[1] - a.pos[3 * (size_t)v + 1], E[2] - a.pos[3 * (size_t)v + 2] };
    v3_normalize(V);
    float Hu[3] = { Ldir[0] + V[0], Ldir[1] + V[1], Ldir[2] + V[2] };
    const float hl = sqrtf(Hu[0] * Hu[0] + Hu[1] * Hu[1] + Hu[2] * Hu[2]);
    const float ih = hl > 0.0f ? 1.0f / hl : 0.0f;
    for (int i = 0; i < 3; i++) { t.N[i] = N[i]; t.L[i] = Ldir[i]; t.H[i] = Hu[i] * ih; }
    t.hlen = hl;
    t.nl = v3_dot(t.N, t.L);
    t.nh = v3_dot(t.N, t.H);
    const float shin = a.material[2];
    t.spec = t.nh > 0.0f ? powf(t.nh, shin) : 0.0f;
}

__device__ __forceinline__ void light_dir(const float *l, float *L, float &len)
{
    len = sqrtf(l[0] * l[0] + l[1] * l[1] + l[2] * l[2]);
    const float inv = len > 0.0f ? 1.0f / len : 0.0f;
    L[0] = l[0] * inv; L[1] = l[1] * inv; L[2] = l[2] * inv;
}

__global__ void k_glight(LightArgs a, float4 *lit)
{
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= (uint64_t)a.nv * a.nViews) return;
    const uint32_t view = (uint32_t)(g / a.nv), v = (uint32_t)(g % a.nv);
    float L[3], llen;
    light_dir(a.light, L, llen);
    VertexTerms t;
    vertex_terms(a, v, view, L, t);
    const float kd = a.material[0], ks = a.material[1];
    const float diff = fmaxf(t.nl, 0.0f);
    float o[3];
    for (int c = 0; c < 3; c++) {
        const float D = a.col[3 * (size_t)v + c] * kd;
        o[c] = fminf(D * (a.ambient + diff) + ks * t.spec, 1.0f);
    }
    lit[g] = make_float4(o[0], o[1], o[2], a.alpha[v]);
}

// ---------------------------------------------------------------------------
// fragments
// ---------------------------------------------------------------------------
struct FragIn {                    // a covered pixel of a set-up triangle
    float wn[3];                   // screen-space weights
    float z;                       // interpolated depth
};

// Weights and depth of a covered pixel (px, py).
template <typename Prim>
__device__ __forceinline__ void fragment(const Prim &P, uint32_t px, uint32_t py, FragIn &f)
{
    int32_t w[3];
    for (int e = 0; e < 3; e++)
        w[e] = (int32_t)(px * (uint32_t)P.ex[e] + py * (uint32_t)P.ey[e] + (uint32_t)P.c[e]);
    f.wn[0] = (float)w[0] * P.wInvSum; f.wn[1] = (float)w[1] * P.wInvSum; f.wn[2] = (float)w[2] * P.wInvSum;
    float zs = P.z[0] * f.wn[0] + P.z[1] * f.wn[1];
    zs = zs + P.z[2] * f.wn[2];
    f.z = 1.0f / zs;
}

// Whether the triangle covers the pixel: inside its box with no edge
// function negative (the three never vanish together: they add up to twice
// the area, and triangles without any were culled).
__device__ __forceinline__ bool covers(const GPrim &P, uint32_t px, uint32_t py)
{
    if (!(px >= (uint32_t)P.xMin && px < (uint32_t)P.xMax && py >= (uint32_t)P.yMin && py <= (uint32_t)P.yMax)) return false;
    uint32_t any = 0;
    for (int e = 0; e < 3; e++) any |= px * (uint32_t)P.ex[e] + py * (uint32_t)P.ey[e] + (uint32_t)P.c[e];
    return (int32_t)any > 0;
}

struct Taps {                      // texel offsets (-1: none) and weights of a texture sample
    int32_t off[4];
    float w[4];
};

__device__ __forceinline__ int32_t texel_off(const GTex &T, int32_t x, int32_t y)
{
    const int32_t off = (int32_t)((uint32_t)y * T.w + (uint32_t)x);
    return (off < 0 || (uint32_t)off >= T.w * T.h) ? -1 : off;
}

__device__ __forceinline__ float4 texel(const GTex &T, int32_t off)
{
    return off < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldg(T.tex + off);
}

__device__ __forceinline__ float4 lerp4(float4 a, float4 b, float t)
{
    return make_float4(a.x + t * (b.x - a.x), a.y + t * (b.y - a.y), a.z + t * (b.z - a.z), a.w + t * (b.w - a.w));
}

// Texture sample with the reference's addressing (sampler.h:203-430):
// nearest, or bilinear from x0 = map(u), x1 = map(u + 1/w) and
// fx = clamp(u*w - x0, 0, 1).
__device__ __forceinline__ float4 sample(const GTex &T, float u, float v, Taps &tp)
{
    int32_t x0, y0;
    tex_map_wh(T.w, T.h, T.wrap, u, v, x0, y0);
    if (T.filter == 0) {
        tp.off[0] = texel_off(T, x0, y0); tp.w[0] = 1.0f;
        tp.off[1] = tp.off[2] = tp.off[3] = -1; tp.w[1] = tp.w[2] = tp.w[3] = 0.0f;
        return texel(T, tp.off[0]);
    }
    int32_t x1, y1;
    tex_map_wh(T.w, T.h, T.wrap, u + T.tx, v + T.ty, x1, y1);
    float fx = u * (float)T.w - (float)x0;
    float fy = v * (float)T.h - (float)y0;
    fx = x86_min(x86_max(fx, 0.0f), 1.0f);
    fy = x86_min(x86_max(fy, 0.0f), 1.0f);
    tp.off[0] = texel_off(T, x0, y0); tp.off[1] = texel_off(T, x1, y0);
    tp.off[2] = texel_off(T, x0, y1); tp.off[3] = texel_off(T, x1, y1);
    tp.w[0] = (1.0f - fx) * (1.0f - fy); tp.w[1] = fx * (1.0f - fy);
    tp.w[2] = (1.0f - fx) * fy;          tp.w[3] = fx * fy;
    const float4 r0 = lerp4(texel(T, tp.off[0]), texel(T, tp.off[1]), fx);
    const float4 r1 = lerp4(texel(T, tp.off[2]), texel(T, tp.off[3]), fx);
    return lerp4(r0, r1, fy);
}

struct Shade {
    float4 c;                      // interpolated lit colour (rgb) and alpha
    float4 t;                      // texel
    float src[3], a;               // fragment colour and opacity
    Taps tp;
};

// l1, l2, l3: its vertices' lit colours
template <typename Prim>
__device__ __forceinline__ void shade(const Prim &P, const FragIn &f, const float4 l1, const float4 l2, const float4 l3, const GTex &T, Shade &s)
{
    s.c.x = (f.wn[0] * l1.x + f.wn[1] * l2.x) + f.wn[2] * l3.x;
    s.c.y = (f.wn[0] * l1.y + f.wn[1] * l2.y) + f.wn[2] * l3.y;
    s.c.z = (f.wn[0] * l1.z + f.wn[1] * l2.z) + f.wn[2] * l3.z;
    s.c.w = (f.wn[0] * l1.w + f.wn[1] * l2.w) + f.wn[2] * l3.w;
    float tu = P.su[0] * f.wn[0] + P.su[1] * f.wn[1];
    tu = tu + P.su[2] * f.wn[2];
    float tv = P.sv[0] * f.wn[0] + P.sv[1] * f.wn[1];
    tv = tv + P.sv[2] * f.wn[2];
    if (P.flags & 2u) { tu = tu * f.z; tv = tv * f.z; }
    s.t = sample(T, tu, tv, s.tp);
    s.src[0] = s.t.x * s.c.x; s.src[1] = s.t.y * s.c.y; s.src[2] = s.t.z * s.c.z;
    s.a = s.t.w * s.c.w;
}

struct RasterArgsG {
    const GPrim *prims;
    const uint32_t *off, *list;
    const float4 *lit;             // nViews x nv
    GTex T;
    GView V;
    float *image;                  // nViews x H x W x 3
    const float *dImage;
    float4 *dTex;
    float4 *dLit;                  // nViews x nv
    const uint32_t *order;         // the tiles that have triangles, then the others from the end
    uint32_t nFull, nTiles;        // how many there are of the former, and of all
};

// ---------------------------------------------------------------------------
// One CTA per tile; its list is staged in shared memory, GCHUNK entries at a
// time, with their vertices' lit colours.  Each warp takes an 8x8 block,
// pixels (lane % 8, lane / 8) and four rows below it a lane: of the staged
// triangles that reach the block, 32 at a time, lane k finds triangle k's
// covered pixels, the masks are transposed over the warp, and each pixel
// walks its covering triangles in order (depth test).  The visible fragments
// go on a list of the block, linked per pixel in order, and are shaded
// densely over the warp.
//
// Bound by the chain of loads a tile starts with (list range, entries,
// triangles, lit vertices) and by instruction issue.  Every pixel walking
// the tile's whole list from global memory and shading as it went (31
// entries a list; a pixel on a vertex of the mesh has six covering triangles
// and two or three visible ones, so few lanes of a shading step were busy)
// took 551 us for 64 views of 512x512 and 922 us for their adjoint; with a
// list of each block's triangles staged per warp 232 and 408; this takes
// 200 and 363.
// ---------------------------------------------------------------------------
// A staged triangle (a stride of 36 banks: 16-byte reads of eight of them
// touch every bank once).
struct __align__(16) GStage {
    int32_t ex[3];
    float wInvSum;
    int32_t ey[3];
    uint32_t flags;
    int32_t c[3];
    uint32_t v0;
    float z[3];
    uint32_t v1;
    float su[3];
    uint32_t v2;
    float sv[3];
    uint32_t id;                   // its index
    float4 lit[3];
};
static_assert(sizeof(GStage) == 144, "nine 16-byte words, the first six as GPrim's");

struct GTileStage {
    GStage rec[GCHUNK];
    int4 box[GCHUNK];              // xMin yMin xMax yMax
};

constexpr uint32_t GNONE = 0xffffu;

struct GWarp {
    float4 fs[GFW];                // per listed fragment: colour and opacity, then what the passes make of it
    uint16_t fnext[GFW];           // the pixel's next fragment
    uint8_t fpix[GFW];             // its pixel: 32 slot + lane
    uint8_t frec[GFW];             // its staged triangle
    uint8_t ids[GCHUNK];           // the staged triangles that reach the block
};
struct GWarpAdjoint {
    GWarp w;
    float4 dc[32];                 // a step's fragments: d(lit) of the interpolated colour
    float wn[3][32];               // and their weights
    uint32_t fid[GFW];             // per listed fragment: its triangle
    uint16_t fprev[GFW];           // the pixel's previous fragment
};
template <typename Warp> struct GShared {
    GTileStage tile;
    Warp warp[GTHREADS / 32];
};

struct Block {
    uint32_t view, bx, by;
    uint32_t beg, n;               // its tile's list
};
__device__ __forceinline__ Block block_of(const RasterArgsG &a, uint32_t gt)
{
    const uint32_t warp = threadIdx.x >> 5, tile = gt % a.V.tilesPerView;
    Block b;
    b.view = gt / a.V.tilesPerView;
    b.bx = (tile % a.V.tilesX) * GTILE + (warp & 1u) * GBLOCK;
    b.by = (tile / a.V.tilesX) * GTILE + (warp >> 1) * GBLOCK;
    b.beg = a.off[gt]; b.n = a.off[gt + 1] - b.beg;
    return b;
}

// Stages list entries [c0, c0 + GCHUNK) of the tile, two threads an entry.
// The whole CTA calls it; what was staged before is no longer read.
__device__ __forceinline__ void stage_chunk(const RasterArgsG &a, const Block &b, const float4 *lit, uint32_t c0, GTileStage &T)
{
    static_assert(GTHREADS == 2 * GCHUNK, "two threads an entry");
    const uint32_t r = threadIdx.x >> 1;
    if (c0 + r < b.n) {
        const uint32_t id = __ldg(a.list + b.beg + c0 + r);
        const int4 *src = reinterpret_cast<const int4 *>(a.prims + id);
        GStage &R = T.rec[r];
        int4 *dst = reinterpret_cast<int4 *>(&R);
        if ((threadIdx.x & 1u) == 0) {
            const int4 q2 = __ldg(src + 2), q0 = __ldg(src), q1 = __ldg(src + 1), q6 = __ldg(src + 6);
            const float4 l0 = __ldg(lit + (uint32_t)q2.w);
            dst[0] = q0; dst[1] = q1; dst[2] = q2;
            T.box[r] = q6;
            R.lit[0] = l0;
        } else {
            const int4 q3 = __ldg(src + 3), q4 = __ldg(src + 4);
            int4 q5 = __ldg(src + 5);
            const float4 l1 = __ldg(lit + (uint32_t)q3.w), l2 = __ldg(lit + (uint32_t)q4.w);
            q5.w = (int)id;
            dst[3] = q3; dst[4] = q4; dst[5] = q5;
            R.lit[1] = l1; R.lit[2] = l2;
        }
    }
}

// A pixel's fragments on the block's list.
struct Chain {
    uint32_t head, tail;
};

// Shades the fragment of pixel p of block b of a staged triangle.
__device__ __forceinline__ void shade_staged(const RasterArgsG &a, const Block &b, const GStage &r, uint32_t p, FragIn &f, Shade &s)
{
    fragment(r, b.bx + (p & 7u), b.by + (p >> 3), f);
    shade(r, f, r.lit[0], r.lit[1], r.lit[2], a.T, s);
}

// Lists the visible fragments of the block's pixels (in0 / in1: whether my
// two take part) into S, linked per pixel, with the colour and opacity of
// each in S.fs; `full` is called when the list has no room (it makes room
// and returns true, or returns false: the block's walk ends), listed(i, k,
// prev) for each fragment put on the list.  nf: fragments on the list.
// staged: whether the tile's only chunk is staged already.  Returns whether
// the walk came to its end.  The whole CTA calls it.
template <typename Full, typename Listed>
__device__ __forceinline__ bool list_block(const RasterArgsG &a, const Block &b, const float4 *lit, GTileStage &T, GWarp &S,
                                           bool staged, bool in0, bool in1, Chain &ch0, Chain &ch1, uint32_t &nf, Full full, Listed listed)
{
    const uint32_t all = 0xffffffffu, lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const uint32_t px = b.bx + (lane & 7u), py = b.by + (lane >> 3);
    float D0 = a.V.clearDepth, D1 = a.V.clearDepth;
    ch0.head = ch0.tail = ch1.head = ch1.tail = GNONE;
    nf = 0;
    bool open = __any_sync(all, in0 || in1);
    for (uint32_t c0 = 0; c0 < b.n; c0 += GCHUNK) {
        if (!staged) {
            if (c0) __syncthreads();                   // the last chunk is no longer read
            stage_chunk(a, b, lit, c0, T);
            __syncthreads();
        }
        if (!open) continue;
        uint32_t hits = 0;
        for (uint32_t k0 = 0; k0 < GCHUNK; k0 += 32u) {
            bool hit = false;
            if (c0 + k0 + lane < b.n) {
                const int4 q = T.box[k0 + lane];
                hit = (uint32_t)q.x < b.bx + GBLOCK && (uint32_t)q.z > b.bx && (uint32_t)q.y < b.by + GBLOCK && (uint32_t)q.w >= b.by;
            }
            const uint32_t m = __ballot_sync(all, hit);
            if (hit) S.ids[hits + __popc(m & lt)] = (uint8_t)(k0 + lane);
            hits += __popc(m);
        }
        __syncwarp();
        for (uint32_t h0 = 0; h0 < hits && open; h0 += 32u) {
            // my triangle's covered pixels, rows 0-3 and 4-7 of the block
            uint32_t lo = 0, hi = 0;
            if (h0 + lane < hits) {
                const uint32_t k = S.ids[h0 + lane];
                const GStage &r = T.rec[k];
                const int4 q6 = T.box[k];
                const uint32_t x0 = max((uint32_t)q6.x, b.bx), x1 = min((uint32_t)q6.z, b.bx + GBLOCK);
                const uint32_t y0 = max((uint32_t)q6.y, b.by), y1 = min((uint32_t)q6.w, b.by + GBLOCK - 1u);
                if (x0 < x1 && y0 <= y1) {
                    const uint32_t cols = ((1u << (x1 - x0)) - 1u) << (x0 - b.bx);
                    // the edge functions at column 7 of row y0
                    const uint32_t xr = b.bx + GBLOCK - 1u;
                    const uint32_t ex0 = (uint32_t)r.ex[0], ex1 = (uint32_t)r.ex[1], ex2 = (uint32_t)r.ex[2];
                    const uint32_t ey0 = (uint32_t)r.ey[0], ey1 = (uint32_t)r.ey[1], ey2 = (uint32_t)r.ey[2];
                    uint32_t r0 = xr * ex0 + y0 * ey0 + (uint32_t)r.c[0];
                    uint32_t r1 = xr * ex1 + y0 * ey1 + (uint32_t)r.c[1];
                    uint32_t r2 = xr * ex2 + y0 * ey2 + (uint32_t)r.c[2];
                    for (uint32_t y = y0 - b.by; y <= y1 - b.by; y++) {
                        uint32_t w0 = r0, w1 = r1, w2 = r2, row = 0;
#pragma unroll
                        for (int x = GBLOCK - 1; x >= 0; x--) {
                            row = __funnelshift_l(~(w0 | w1 | w2), row, 1);      // no sign bit: covered
                            w0 -= ex0; w1 -= ex1; w2 -= ex2;
                        }
                        row = (row & cols) << (8u * (y & 3u));
                        if (y < 4u) lo |= row; else hi |= row;
                        r0 += ey0; r1 += ey1; r2 += ey2;
                    }
                }
            }
            lo = warp_transpose32(lo);
            hi = warp_transpose32(hi);
            // depth test, PF_LESS with depth written
            uint32_t vis0 = 0, vis1 = 0;
            auto walk = [&](uint32_t m, uint32_t y, float &D, uint32_t &vis) {
                for (; m; m &= m - 1u) {
                    const uint32_t k = (uint32_t)(__ffs(m) - 1);
                    FragIn f;
                    fragment(T.rec[S.ids[h0 + k]], px, y, f);
                    if (f.z < D) { D = f.z; vis |= 1u << k; }
                }
            };
            if (in0) walk(lo, py, D0, vis0);
            if (in1) walk(hi, py + 4u, D1, vis1);
            // onto the list: the fragments of all slot-0 pixels in order, then
            // those of the slot-1 pixels (neighbouring entries are neighbouring
            // pixels); 32 triangles of 32 pixels stay below 2^16 a slot
            uint32_t total;
            uint32_t o0 = warp_offsets((uint32_t)__popc(vis0) | (uint32_t)__popc(vis1) << 16, total);
            uint32_t o1 = (o0 >> 16) + (total & 0xffffu);
            o0 &= 0xffffu;
            total = (total & 0xffffu) + (total >> 16);
            for (uint32_t done = 0; done < total;) {
                if (nf == (uint32_t)GFW && !full()) { open = false; break; }
                const uint32_t end = min(total, done + (uint32_t)GFW - nf);
                auto emit = [&](uint32_t &vis, uint32_t &o, Chain &ch, uint32_t pix) {
                    for (; vis && o < end; vis &= vis - 1u, o++) {
                        const uint32_t i = nf + o - done, k = S.ids[h0 + (uint32_t)(__ffs(vis) - 1)];
                        S.fpix[i] = (uint8_t)pix;
                        S.frec[i] = (uint8_t)k;
                        S.fnext[i] = (uint16_t)GNONE;
                        if (ch.tail == GNONE) ch.head = i; else S.fnext[ch.tail] = (uint16_t)i;
                        listed(i, k, ch.tail);
                        ch.tail = i;
                    }
                };
                emit(vis0, o0, ch0, lane);
                emit(vis1, o1, ch1, 32u + lane);
                __syncwarp();
                for (uint32_t i = nf + lane; i < nf + end - done; i += 32u) {
                    FragIn f; Shade s;
                    shade_staged(a, b, T.rec[S.frec[i]], S.fpix[i], f, s);
                    S.fs[i] = make_float4(s.src[0], s.src[1], s.src[2], s.a);
                }
                __syncwarp();
                nf += end - done;
                done = end;
            }
        }
        __syncwarp();                                  // S.ids is free
    }
    return open || !__any_sync(all, in0 || in1);
}

// The background of an empty tile, by one warp: 16 rows of 48 floats, in
// 16-byte stores where the rows start on 16 bytes.
__device__ __forceinline__ void clear_tile(const RasterArgsG &a, uint32_t gt)
{
    const uint32_t lane = threadIdx.x & 31u, view = gt / a.V.tilesPerView, tile = gt % a.V.tilesPerView;
    const uint32_t x0 = (tile % a.V.tilesX) * GTILE * 3u, y0 = (tile / a.V.tilesX) * GTILE;
    float *o = a.image + ((size_t)view * a.V.H + y0) * a.V.W * 3 + x0;
    const float bg0 = a.V.bg[0], bg1 = a.V.bg[1], bg2 = a.V.bg[2];
    auto bg = [&](uint32_t c) { return c == 0 ? bg0 : c == 1 ? bg1 : bg2; };
    if ((a.V.W & 3u) == 0 && ((uintptr_t)a.image & 15u) == 0 && x0 + 48u <= a.V.W * 3u) {
#pragma unroll
        for (uint32_t i = 0; i < 6; i++) {
            const uint32_t e = 32u * i + lane, y = e / 12u, x = 4u * (e % 12u), c = x % 3u;
            const float v0 = bg(c), v1 = bg((c + 1u) % 3u), v2 = bg((c + 2u) % 3u);
            if (y0 + y < a.V.H) *reinterpret_cast<float4 *>(o + (size_t)y * a.V.W * 3 + x) = make_float4(v0, v1, v2, v0);
        }
        return;
    }
    for (uint32_t e = lane; e < 48u * GTILE; e += 32u) {
        const uint32_t y = e / 48u, x = e % 48u;
        if (y0 + y < a.V.H && x0 + x < a.V.W * 3u) o[(size_t)y * a.V.W * 3 + x] = bg(x % 3u);
    }
}

// The first nFull CTAs take a tile with triangles each, the others
// GCLEAR empty tiles (one a warp).  A CTA for each of the 65,536 tiles of 64
// views of 512x512, two thirds of them empty, took 215 us.
constexpr uint32_t GCLEAR = 4;
__global__ void __launch_bounds__(GTHREADS, 8) k_gforward(RasterArgsG a)
{
    if (blockIdx.x >= a.nFull) {
        const uint32_t first = a.nFull + (blockIdx.x - a.nFull) * GCLEAR, warp = threadIdx.x >> 5;
        for (uint32_t i = first + warp; i < min(first + GCLEAR, a.nTiles); i += GTHREADS / 32) clear_tile(a, __ldg(a.order + i));
        return;
    }
    __shared__ GShared<GWarp> sh;
    GWarp &S = sh.warp[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const Block b = block_of(a, __ldg(a.order + blockIdx.x));
    const uint32_t px = b.bx + (lane & 7u), py = b.by + (lane >> 3);
    const bool in0 = px < a.V.W && py < a.V.H, in1 = px < a.V.W && py + 4u < a.V.H;
    float C0[3] = { a.V.bg[0], a.V.bg[1], a.V.bg[2] }, C1[3] = { a.V.bg[0], a.V.bg[1], a.V.bg[2] };
    {
        const float4 *lit = a.lit + (size_t)b.view * a.V.nv;
        Chain ch0, ch1;
        uint32_t nf;
        // each pixel's fragments over its colour, in order
        auto resolve = [&]() {
            auto over = [&](Chain &ch, float *C) {
                for (uint32_t i = ch.head; i != GNONE; i = S.fnext[i]) {
                    const float4 v = S.fs[i];
                    C[0] = v.w * v.x + (1.0f - v.w) * C[0];
                    C[1] = v.w * v.y + (1.0f - v.w) * C[1];
                    C[2] = v.w * v.z + (1.0f - v.w) * C[2];
                }
                ch.head = ch.tail = GNONE;
            };
            over(ch0, C0);
            over(ch1, C1);
            nf = 0;
            __syncwarp();
            return true;
        };
        list_block(a, b, lit, sh.tile, S, false, in0, in1, ch0, ch1, nf, resolve, [](uint32_t, uint32_t, uint32_t) {});
        resolve();
    }
    // the block's rows of 24 floats, consecutive floats in consecutive lanes
    // (three floats a lane and pixel would touch every sector three times)
    float *stage = reinterpret_cast<float *>(S.fs);
    for (int c = 0; c < 3; c++) { stage[lane * 3u + c] = C0[c]; stage[96u + lane * 3u + c] = C1[c]; }
    __syncwarp();
    float *o = a.image + ((size_t)b.view * a.V.H + b.by) * a.V.W * 3;
#pragma unroll
    for (uint32_t i = 0; i < 6; i++) {
        const uint32_t e = 32u * i + lane, y = e / 24u, x = b.bx * 3u + e % 24u;
        if (b.by + y < a.V.H && x < a.V.W * 3u) o[(size_t)y * a.V.W * 3 + x] = stage[e];
    }
}

__device__ __forceinline__ void add4(float4 *p, float4 v) { atomicAdd(p, v); }

// Gradients of one fragment with respect to its texel and lit colour:
// ds = g a per colour channel, da that of the opacity.
__device__ __forceinline__ void fragment_grads(const Shade &s, const float4 d, float4 &dt, float4 &dc)
{
    dt = make_float4(d.x * s.c.x, d.y * s.c.y, d.z * s.c.z, d.w * s.c.w);
    dc = make_float4(d.x * s.t.x, d.y * s.t.y, d.z * s.t.z, d.w * s.t.w);
}

// The adjoint of one pixel a lane, of blocks whose pixels have more visible
// fragments than fit the list (hundreds of layers in far-to-near order): a
// replay of the tile's list finds the pixel's visible fragments, the last
// RING of them recorded with the colour under each; they are walked back
// from the front, older ones by further replays.
__device__ __noinline__ void adjoint_pixel(const RasterArgsG &a, const Block b, uint32_t px, uint32_t py,
                                           float gx, float gy, float gz)
{
    float g[3] = { gx, gy, gz };
    const float4 *lit = a.lit + (size_t)b.view * a.V.nv;
    float4 *dLit = a.dLit + (size_t)b.view * a.V.nv;
    uint32_t hi = 0xffffffffu;       // visible fragments at or above this index are done
    do {
        float C[3] = { a.V.bg[0], a.V.bg[1], a.V.bg[2] };
        float D = a.V.clearDepth;
        uint32_t rpos[RING], j = 0;
        float rc[RING][3];
        for (uint32_t k = 0; k < b.n && j < hi; k++) {
            const GPrim &P = a.prims[__ldg(a.list + b.beg + k)];
            if (!covers(P, px, py)) continue;
            FragIn f;
            fragment(P, px, py, f);
            if (!(f.z < D)) continue;
            D = f.z;
            Shade s;
            shade(P, f, lit[P.v0], lit[P.v1], lit[P.v2], a.T, s);
            const uint32_t slot = j % RING;
            rpos[slot] = k;
            for (int c = 0; c < 3; c++) { rc[slot][c] = C[c]; C[c] = s.a * s.src[c] + (1.0f - s.a) * C[c]; }
            j++;
        }
        hi = min(hi, j);
        const uint32_t lo = hi > (uint32_t)RING ? hi - RING : 0u;
        for (; hi > lo; hi--) {
            const uint32_t slot = (hi - 1u) % RING;
            const GPrim &P = a.prims[__ldg(a.list + b.beg + rpos[slot])];
            FragIn f;
            Shade s;
            fragment(P, px, py, f);
            shade(P, f, lit[P.v0], lit[P.v1], lit[P.v2], a.T, s);
            float4 d = make_float4(g[0] * s.a, g[1] * s.a, g[2] * s.a, 0.0f), dt, dc;
            for (int c = 0; c < 3; c++) { d.w += g[c] * (s.src[c] - rc[slot][c]); g[c] = g[c] * (1.0f - s.a); }
            fragment_grads(s, d, dt, dc);
            for (int k = 0; k < 4; k++) {
                const float w = s.tp.w[k];
                if (s.tp.off[k] >= 0) add4(a.dTex + s.tp.off[k], make_float4(dt.x * w, dt.y * w, dt.z * w, dt.w * w));
            }
            const uint32_t v[3] = { P.v0, P.v1, P.v2 };
            for (int m = 0; m < 3; m++) {
                const float w = f.wn[m];
                add4(dLit + v[m], make_float4(dc.x * w, dc.y * w, dc.z * w, dc.w * w));
            }
        }
    } while (hi > 0);
}

__global__ void __launch_bounds__(GTHREADS, 7) k_gadjoint(RasterArgsG a)
{
    __shared__ GShared<GWarpAdjoint> sh;
    GWarpAdjoint &A = sh.warp[threadIdx.x >> 5];
    GWarp &S = A.w;
    const uint32_t lane = threadIdx.x & 31u, all = 0xffffffffu;
    const Block b = block_of(a, __ldg(a.order + blockIdx.x));
    const uint32_t px = b.bx + (lane & 7u), py = b.by + (lane >> 3);
    const bool in0 = px < a.V.W && py < a.V.H, in1 = px < a.V.W && py + 4u < a.V.H;
    const float4 *lit = a.lit + (size_t)b.view * a.V.nv;
    float4 *dLit = a.dLit + (size_t)b.view * a.V.nv;
    float g0[3] = { 0.f, 0.f, 0.f }, g1[3] = { 0.f, 0.f, 0.f };
    {
        const float *gi = a.dImage + (((size_t)b.view * a.V.H + py) * a.V.W + px) * 3;
        if (in0) { g0[0] = gi[0]; g0[1] = gi[1]; g0[2] = gi[2]; }
        gi += (size_t)a.V.W * 12;
        if (in1) { g1[0] = gi[0]; g1[1] = gi[1]; g1[2] = gi[2]; }
    }
    const bool one = b.n <= (uint32_t)GCHUNK;      // one chunk: it stays staged
    // a block at once (part 0) or, when its fragments do not fit the list,
    // its pixels of slot 0 (part 1) and of slot 1 (part 2), or those one by
    // one; the CTA's warps stay together for the staging
    bool again = true;
    for (uint32_t part = 0; part < 3u; part++) {
        const bool t0 = again && in0 && part != 2u, t1 = again && in1 && part != 1u;
        Chain ch0, ch1;
        uint32_t nf;
        const bool fits = list_block(a, b, lit, sh.tile, S, one && part != 0, t0, t1, ch0, ch1, nf,
                                     []() { return false; }, [&](uint32_t i, uint32_t k, uint32_t prev) {
                                         A.fid[i] = sh.tile.rec[k].id;
                                         A.fprev[i] = (uint16_t)prev;
                                     });
        if (!fits) {
            if (part == 1u && t0) adjoint_pixel(a, b, px, py, g0[0], g0[1], g0[2]);
            if (part == 2u && t1) adjoint_pixel(a, b, px, py + 4u, g1[0], g1[1], g1[2]);
        } else {
            // 1. per pixel, in order: the colour under each fragment, as its
            //    difference to the fragment's; then from the front: the
            //    gradients of its colour and opacity
            __syncwarp();
            auto chain = [&](const Chain &ch, const float *g0) {
                float g[3] = { g0[0], g0[1], g0[2] };
                float C[3] = { a.V.bg[0], a.V.bg[1], a.V.bg[2] };
                for (uint32_t i = ch.head; i != GNONE; i = S.fnext[i]) {
                    const float4 v = S.fs[i];
                    S.fs[i] = make_float4(v.x - C[0], v.y - C[1], v.z - C[2], v.w);
                    C[0] = v.w * v.x + (1.0f - v.w) * C[0];
                    C[1] = v.w * v.y + (1.0f - v.w) * C[1];
                    C[2] = v.w * v.z + (1.0f - v.w) * C[2];
                }
                for (uint32_t i = ch.tail; i != GNONE; i = A.fprev[i]) {
                    const float4 v = S.fs[i];
                    S.fs[i] = make_float4(g[0] * v.w, g[1] * v.w, g[2] * v.w, (g[0] * v.x + g[1] * v.y) + g[2] * v.z);
                    for (int c = 0; c < 3; c++) g[c] = g[c] * (1.0f - v.w);
                }
            };
            chain(ch0, g0);
            chain(ch1, g1);
            __syncwarp();
            // 2. back through texture and lit colour, 32 fragments a step
            for (uint32_t f0 = 0; f0 < nf; f0 += 32u) {
                const bool act = f0 + lane < nf;
                FragIn f; Shade s;
                const uint32_t id = act ? A.fid[f0 + lane] : 0xffffffffu;
                uint32_t v[3] = { 0, 0, 0 };
                float4 dt = make_float4(0.f, 0.f, 0.f, 0.f), dc;
                if (act) {
                    GStage r;
                    if (one) r = sh.tile.rec[S.frec[f0 + lane]];
                    else {
                        const int4 *src = reinterpret_cast<const int4 *>(a.prims + id);
                        int4 *dst = reinterpret_cast<int4 *>(&r);
                        for (int w = 0; w < 6; w++) dst[w] = __ldg(src + w);
                        r.lit[0] = __ldg(lit + r.v0); r.lit[1] = __ldg(lit + r.v1); r.lit[2] = __ldg(lit + r.v2);
                    }
                    v[0] = r.v0; v[1] = r.v1; v[2] = r.v2;
                    shade_staged(a, b, r, S.fpix[f0 + lane], f, s);
                    fragment_grads(s, S.fs[f0 + lane], dt, dc);
                    A.dc[lane] = dc;
                    for (int m = 0; m < 3; m++) A.wn[m][lane] = f.wn[m];
                }
                // texel gradients: neighbours on the list (mostly pixels side
                // by side) that read the same texel send one atomic
                const int ntap = a.T.filter == 0 ? 1 : 4;
                for (int k = 0; k < ntap; k++) {
                    const int32_t off = act ? s.tp.off[k] : -1;
                    const float w = act ? s.tp.w[k] : 0.0f;
                    const float4 u = make_float4(dt.x * w, dt.y * w, dt.z * w, dt.w * w);
                    const int32_t po = __shfl_xor_sync(all, off, 1);
                    const float4 pu = make_float4(__shfl_xor_sync(all, u.x, 1), __shfl_xor_sync(all, u.y, 1),
                                                  __shfl_xor_sync(all, u.z, 1), __shfl_xor_sync(all, u.w, 1));
                    if (off >= 0) {
                        if (po != off) add4(a.dTex + off, u);
                        else if ((lane & 1) == 0) add4(a.dTex + off, make_float4(u.x + pu.x, u.y + pu.y, u.z + pu.z, u.w + pu.w));
                    }
                }
                // vertex gradients: a lane per (triangle of the step, vertex)
                // sums the triangle's pixels from shared memory and sends one
                // atomic
                __syncwarp();
                const uint32_t peers = __match_any_sync(all, id);
                const uint32_t heads = __ballot_sync(all, act && lane == (uint32_t)(__ffs(peers) - 1));
                const uint32_t items = 3u * (uint32_t)__popc(heads);
                for (uint32_t i0 = 0; i0 < items; i0 += 32u) {
                    const uint32_t i = min(i0 + lane, items - 1u), head = nth_bit(heads, i / 3u), m = i % 3u;
                    uint32_t p = __shfl_sync(all, peers, head);
                    const uint32_t u0 = __shfl_sync(all, v[0], head), u1 = __shfl_sync(all, v[1], head), u2 = __shfl_sync(all, v[2], head);
                    if (i0 + lane < items) {
                        float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
                        for (; p; p &= p - 1u) {
                            const uint32_t l = (uint32_t)(__ffs(p) - 1);
                            const float w = A.wn[m][l];
                            const float4 c = A.dc[l];
                            d.x += c.x * w; d.y += c.y * w; d.z += c.z * w; d.w += c.w * w;
                        }
                        if (d.x != 0.0f || d.y != 0.0f || d.z != 0.0f || d.w != 0.0f)
                            add4(dLit + (m == 0 ? u0 : m == 1 ? u1 : u2), d);
                    }
                }
                __syncwarp();                      // the step's fragments are free
            }
        }
        if (part == 0) again = !fits;
        if (part == 0 && !__syncthreads_or(again)) break;
        if (part == 1 && !one) __syncthreads();        // the last chunk is no longer read
    }
}

// ---------------------------------------------------------------------------
// vertex adjoint
// ---------------------------------------------------------------------------
// One thread per (vertex, group of GVIEWS views).  Per-vertex gradients are
// added into dCol/dAlpha (zeroed first); acc: [0] d diffuse, [1] d specular,
// [2] d shininess, [3..5] d L (unit light direction), reduced per CTA.
constexpr uint32_t GVIEWS = 8;

__global__ void __launch_bounds__(256) k_glight_adjoint(LightArgs a, const float4 *dLit, float *dCol, float *dAlpha,
                                                         float *acc)
{
    const uint32_t groups = (a.nViews + GVIEWS - 1) / GVIEWS;
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = g < (uint64_t)a.nv * groups;
    const uint32_t v = valid ? (uint32_t)(g % a.nv) : 0u;
    const uint32_t v0 = valid ? (uint32_t)(g / a.nv) * GVIEWS : a.nViews;
    float L[3], llen;
    light_dir(a.light, L, llen);
    const float kd = a.material[0], ks = a.material[1], shin = a.material[2];
    float part[6] = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };
    if (valid) {
        const float C[3] = { a.col[3 * (size_t)v], a.col[3 * (size_t)v + 1], a.col[3 * (size_t)v + 2] };
        float dC[3] = { 0.f, 0.f, 0.f }, dA = 0.0f;
        const uint32_t vEnd = min(v0 + GVIEWS, a.nViews);
        for (uint32_t view = v0; view < vEnd; view++) {
            const float4 g4 = dLit[(size_t)view * a.nv + v];
            dA += g4.w;
            if (g4.x == 0.0f && g4.y == 0.0f && g4.z == 0.0f) continue;
            VertexTerms t;
            vertex_terms(a, v, view, L, t);
            const float diff = fmaxf(t.nl, 0.0f);
            const float gin[3] = { g4.x, g4.y, g4.z };
            float gdiff = 0.0f, gspec = 0.0f;
            for (int c = 0; c < 3; c++) {
                const float D = C[c] * kd;
                const float pre = D * (a.ambient + diff) + ks * t.spec;
                const float gc = pre < 1.0f ? gin[c] : 0.0f;
                dC[c] += gc * kd * (a.ambient + diff);
                part[0] += gc * C[c] * (a.ambient + diff);
                gdiff += gc * D;
                part[1] += gc * t.spec;
                gspec += gc * ks;
            }
            if (t.nl > 0.0f)
                for (int i = 0; i < 3; i++) part[3 + i] += gdiff * t.N[i];
            if (t.nh > 0.0f && t.spec > 0.0f) {
                part[2] += gspec * t.spec * logf(t.nh);
                const float gx = gspec * shin * powf(t.nh, shin - 1.0f);
                // H = (L + V) / |L + V|: dH = (I - H H^T) dHu / |L + V|
                float gH[3] = { gx * t.N[0], gx * t.N[1], gx * t.N[2] };
                const float hg = v3_dot(t.H, gH);
                for (int i = 0; i < 3; i++) part[3 + i] += (gH[i] - t.H[i] * hg) / t.hlen;
            }
        }
        if (groups == 1) {
            for (int c = 0; c < 3; c++) dCol[3 * (size_t)v + c] = dC[c];
            dAlpha[v] = dA;
        } else {
            for (int c = 0; c < 3; c++) if (dC[c] != 0.0f) atomicAdd(&dCol[3 * (size_t)v + c], dC[c]);
            if (dA != 0.0f) atomicAdd(&dAlpha[v], dA);
        }
    }
    __shared__ float red[8][6];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = 0; i < 6; i++) {
        float x = part[i];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) red[warp][i] = x;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        float x = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) x += red[w][threadIdx.x];
        if (x != 0.0f) atomicAdd(&acc[threadIdx.x], x);
    }
}

// d light = (I - L L^T) dL / |light|
__global__ void k_gfinish(const float *light, const float *acc, float *dMaterial, float *dLight)
{
    float L[3], len;
    light_dir(light, L, len);
    dMaterial[0] = acc[0]; dMaterial[1] = acc[1]; dMaterial[2] = acc[2];
    const float gl[3] = { acc[3], acc[4], acc[5] };
    const float d = v3_dot(L, gl);
    for (int i = 0; i < 3; i++) dLight[i] = len > 0.0f ? (gl[i] - L[i] * d) / len : 0.0f;
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct PFgradScene_ {
    PFgradSceneDesc desc{};
    uint32_t nFaces = 1;
    int32_t face0 = 0;
    GView V{};
    uint64_t nItems = 0;
    uint32_t nTiles = 0;
    PFgradInfo info{};
    // device
    PFDrawState *state = nullptr;
    float *mvp = nullptr, *eye = nullptr;
    GPrim *prims = nullptr;
    uint32_t *off = nullptr, *list = nullptr, *work = nullptr;   // work: tile counts, then status words
    uint32_t *order = nullptr;       // see RasterArgsG
    uint32_t nFull = 0;
    float4 *lit = nullptr, *dLit = nullptr;
    float *acc = nullptr;
};

namespace {

void scene_free(PFgradScene_ *s)
{
    cudaFree(s->state); cudaFree(s->mvp); cudaFree(s->eye); cudaFree(s->prims); cudaFree(s->off);
    cudaFree(s->list); cudaFree(s->order); cudaFree(s->work); cudaFree(s->lit); cudaFree(s->dLit); cudaFree(s->acc);
}

inline unsigned blocks(uint64_t n, unsigned b) { return (unsigned)((n + b - 1) / b); }

LightArgs light_args(const PFgradScene_ *s, const PFgradParams *p)
{
    LightArgs a;
    a.pos = s->desc.positions; a.nrm = s->desc.normals; a.col = p->colors; a.alpha = p->alphas;
    a.material = p->material; a.light = p->light; a.eye = s->eye;
    a.nv = s->desc.nVertices; a.nViews = s->desc.nViews; a.ambient = s->desc.ambient;
    return a;
}

RasterArgsG raster_args(const PFgradScene_ *s, const PFgradParams *p)
{
    RasterArgsG a;
    a.prims = s->prims; a.off = s->off; a.list = s->list; a.lit = s->lit;
    a.T.tex = reinterpret_cast<const float4 *>(p->texture);
    a.T.w = s->desc.texWidth; a.T.h = s->desc.texHeight;
    a.T.wrap = s->desc.texWrap; a.T.filter = s->desc.texFilter;
    a.T.tx = 1.0f / (float)s->desc.texWidth; a.T.ty = 1.0f / (float)s->desc.texHeight;
    a.V = s->V;
    a.image = nullptr; a.dImage = nullptr; a.dTex = nullptr; a.dLit = nullptr;
    a.order = s->order; a.nFull = s->nFull; a.nTiles = s->nTiles;
    return a;
}

bool params_ok(const PFgradParams *p)
{
    return p && p->texture && p->colors && p->alphas && p->material && p->light;
}

}  // namespace

#define PFG_CHECK(x) do { if ((x) != cudaSuccess) { cudaGetLastError(); goto fail; } } while (0)

extern "C" int pfgradSceneCreate(PFgradScene *out, const PFgradSceneDesc *d, void *stream)
{
    if (!out || !d) return PFGRAD_ERR_INVALID;
    *out = nullptr;
    if (!d->positions || !d->normals || !d->texcoords || !d->indices || !d->mvp || !d->eye) return PFGRAD_ERR_INVALID;
    if (d->nVertices == 0 || d->nViews == 0 || d->width == 0 || d->height == 0 || d->width > 16384 ||
        d->height > 16384 || d->texWidth == 0 || d->texHeight == 0 || d->texFilter < 0 || d->texFilter > 1 ||
        d->texWrap < 0 || d->texWrap > 2 || d->cullFace < -1 || d->cullFace > 1)
        return PFGRAD_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    PFgradScene_ *s = new (std::nothrow) PFgradScene_();
    if (!s) return PFGRAD_ERR_CUDA;
    s->desc = *d;
    s->nFaces = d->cullFace < 0 ? 2u : 1u;
    s->face0 = d->cullFace < 0 ? 0 : (d->cullFace == 1 ? 0 : 1);   // culling BACK draws FRONT and the reverse
    const uint32_t tilesX = (d->width + GTILE - 1) / GTILE, tilesY = (d->height + GTILE - 1) / GTILE;
    s->V = GView{ d->width, d->height, tilesX, tilesX * tilesY, d->nVertices,
                  { d->background[0], d->background[1], d->background[2] }, d->clearDepth };
    s->nItems = (uint64_t)d->nTriangles * s->nFaces * d->nViews;
    const uint64_t nTiles64 = (uint64_t)tilesX * tilesY * d->nViews;
    if (nTiles64 >= 0x7fffffffu || s->nItems >= 0xffffffffu) { delete s; return PFGRAD_ERR_INVALID; }
    s->nTiles = (uint32_t)nTiles64;
    int rc = PFGRAD_ERR_CUDA;
    uint32_t host[4] = { 0, 0, 0, 0 };
    {
        PFDrawState S;
        memset(&S, 0, sizeof(S));
        S.vpPos[0] = 0; S.vpPos[1] = 0;
        S.vpDim[0] = (int32_t)d->width - 1; S.vpDim[1] = (int32_t)d->height - 1;
        S.vpMin[0] = 0; S.vpMin[1] = 0;
        S.vpMax[0] = (int32_t)d->width - 1; S.vpMax[1] = (int32_t)d->height - 1;
        const size_t nv = d->nVertices, nV = d->nViews;
        PFG_CHECK(cudaMalloc(&s->state, sizeof(PFDrawState)));
        PFG_CHECK(cudaMalloc(&s->mvp, nV * 16 * sizeof(float)));
        PFG_CHECK(cudaMalloc(&s->eye, nV * 3 * sizeof(float)));
        PFG_CHECK(cudaMalloc(&s->prims, (s->nItems ? s->nItems : 1) * sizeof(GPrim)));
        PFG_CHECK(cudaMalloc(&s->off, ((size_t)s->nTiles + 1) * sizeof(uint32_t)));
        PFG_CHECK(cudaMalloc(&s->work, ((size_t)s->nTiles + 5) * sizeof(uint32_t)));
        PFG_CHECK(cudaMalloc(&s->order, (size_t)s->nTiles * sizeof(uint32_t)));
        PFG_CHECK(cudaMalloc(&s->lit, nv * nV * sizeof(float4)));
        PFG_CHECK(cudaMalloc(&s->dLit, nv * nV * sizeof(float4)));
        PFG_CHECK(cudaMalloc(&s->acc, 8 * sizeof(float)));
        PFG_CHECK(cudaMemcpyAsync(s->state, &S, sizeof(S), cudaMemcpyHostToDevice, st));
        PFG_CHECK(cudaMemcpyAsync(s->mvp, d->mvp, nV * 16 * sizeof(float), cudaMemcpyHostToDevice, st));
        PFG_CHECK(cudaMemcpyAsync(s->eye, d->eye, nV * 3 * sizeof(float), cudaMemcpyHostToDevice, st));
        uint32_t *cnt = s->work, *status = s->work + s->nTiles;     // status: clipped items, valid prims, longest list,
                                                                      // tiles with triangles, without
        PFG_CHECK(cudaMemsetAsync(s->work, 0, ((size_t)s->nTiles + 5) * sizeof(uint32_t), st));
        if (s->nItems) {
            SetupArgs a{ d->positions, d->texcoords, d->indices, d->nVertices, d->nTriangles, d->nViews, s->nFaces,
                         s->face0, s->mvp, s->state, s->V, s->prims, cnt, status };
            k_gsetup<<<blocks(s->nItems, 128), 128, 0, st>>>(a);
            PFG_CHECK(cudaGetLastError());
        }
        k_gscan<<<1, 1024, 0, st>>>(cnt, s->off, s->nTiles, status + 2);
        PFG_CHECK(cudaGetLastError());
        k_gorder<<<blocks(s->nTiles, 256), 256, 0, st>>>(s->off, s->nTiles, s->order, status + 3);
        PFG_CHECK(cudaGetLastError());
        PFG_CHECK(cudaMemcpyAsync(host, status, 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        uint32_t total = 0;
        PFG_CHECK(cudaMemcpyAsync(&total, s->off + s->nTiles, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        PFG_CHECK(cudaStreamSynchronize(st));
        if (host[0]) { rc = PFGRAD_ERR_CLIP; goto fail; }
        if (host[2] > PFGRAD_MAX_TILE_PRIMS) { rc = PFGRAD_ERR_CAPACITY; goto fail; }
        PFG_CHECK(cudaMalloc(&s->list, (total ? total : 1) * sizeof(uint32_t)));
        if (total) {
            PFG_CHECK(cudaMemsetAsync(cnt, 0, (size_t)s->nTiles * sizeof(uint32_t), st));
            k_gfill<<<blocks(s->nItems, 256), 256, 0, st>>>(s->prims, s->nItems, s->V,
                                                            d->nTriangles * s->nFaces, s->off, cnt, s->list);
            PFG_CHECK(cudaGetLastError());
            uint32_t cap = 2; while (cap < host[2]) cap <<= 1;
            const size_t smem = (size_t)cap * sizeof(uint32_t);
            PFG_CHECK(cudaFuncSetAttribute(k_gsort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            k_gsort<<<s->nTiles, 256, smem, st>>>(s->off, s->list, cap);
            PFG_CHECK(cudaGetLastError());
        }
        PFG_CHECK(cudaStreamSynchronize(st));
        s->nFull = host[3];
        s->info.primitives = host[1];
        s->info.tileEntries = total;
        s->info.maxTilePrims = host[2];
        s->info.tiles = s->nTiles;
    }
    *out = s;
    return 0;
fail:
    scene_free(s);
    delete s;
    return rc;
}

extern "C" int pfgradSceneDestroy(PFgradScene s)
{
    if (!s) return PFGRAD_ERR_INVALID;
    scene_free(s);
    delete s;
    return 0;
}

extern "C" int pfgradSceneInfo(PFgradScene s, PFgradInfo *info)
{
    if (!s || !info) return PFGRAD_ERR_INVALID;
    *info = s->info;
    return 0;
}

extern "C" int pfgradForward(PFgradScene s, const PFgradParams *p, float *image, void *stream)
{
    if (!s || !params_ok(p) || !image) return PFGRAD_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    const LightArgs la = light_args(s, p);
    k_glight<<<blocks((uint64_t)s->desc.nVertices * s->desc.nViews, 256), 256, 0, st>>>(la, s->lit);
    RasterArgsG ra = raster_args(s, p);
    ra.image = image;
    k_gforward<<<s->nFull + (s->nTiles - s->nFull + GCLEAR - 1) / GCLEAR, GTHREADS, 0, st>>>(ra);
    if (cudaGetLastError() != cudaSuccess) return PFGRAD_ERR_CUDA;
    return 0;
}

extern "C" int pfgradBackward(PFgradScene s, const PFgradParams *p, const float *dImage, const PFgradGrads *g,
                              void *stream)
{
    if (!s || !params_ok(p) || !dImage || !g || !g->texture || !g->colors || !g->alphas || !g->material || !g->light)
        return PFGRAD_ERR_INVALID;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t nv = s->desc.nVertices, nV = s->desc.nViews;
    if (cudaMemsetAsync(g->texture, 0, (size_t)s->desc.texWidth * s->desc.texHeight * sizeof(float4), st) != cudaSuccess ||
        cudaMemsetAsync(s->dLit, 0, nv * nV * sizeof(float4), st) != cudaSuccess ||
        cudaMemsetAsync(s->acc, 0, 8 * sizeof(float), st) != cudaSuccess ||
        cudaMemsetAsync(g->colors, 0, nv * 3 * sizeof(float), st) != cudaSuccess ||
        cudaMemsetAsync(g->alphas, 0, nv * sizeof(float), st) != cudaSuccess) {
        cudaGetLastError();
        return PFGRAD_ERR_CUDA;
    }
    const LightArgs la = light_args(s, p);
    k_glight<<<blocks((uint64_t)nv * nV, 256), 256, 0, st>>>(la, s->lit);
    RasterArgsG ra = raster_args(s, p);
    ra.dImage = dImage;
    ra.dTex = reinterpret_cast<float4 *>(g->texture);
    ra.dLit = s->dLit;
    if (s->nFull) k_gadjoint<<<s->nFull, GTHREADS, 0, st>>>(ra);
    const uint64_t groups = (nV + GVIEWS - 1) / GVIEWS;
    k_glight_adjoint<<<blocks(nv * groups, 256), 256, 0, st>>>(la, s->dLit, g->colors, g->alphas, s->acc);
    k_gfinish<<<1, 1, 0, st>>>(p->light, s->acc, g->material, g->light);
    if (cudaGetLastError() != cudaSuccess) return PFGRAD_ERR_CUDA;
    return 0;
}
