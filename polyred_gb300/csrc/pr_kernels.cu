// pr_kernels.cu — the GB300 (sm_103a) render path kernels.
//
// Frame = [shadow setup + raster per casting light] -> main setup -> raster
//         -> (NaN fix-up) -> resolve -> shade (attributes, Blinn-Phong,
//         shadow lookups, AO, gamma, RGBA8 pack).
//
// Visibility is order independent: each fragment issues a 64-bit atomicMax of
// (orderable depth << 32 | ~seq), which leaves at every pixel the first
// fragment (in the reference's single-worker draw order) with the greatest
// depth — exactly what buffer.FragmentBuffer's sequential DepthTest/Set
// (buffer/buffer.go:221-280) keeps. A NaN-depth fragment only wins when it is
// the first fragment of its pixel; a rare fix-up pass settles that.
//
// Compiled with -fmad=false -prec-div=true -prec-sqrt=true -ftz=false.
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>

#include "pr_devmath.cuh"
#include "pr_hostmath.h"
#include "pr_kernels.cuh"

using namespace prd;

namespace prk {
namespace {

constexpr float kEps = 1e-7f;  // math.Epsilon as float32 (math/math.go:31)

// The approximate units, for values whose error a bound covers (PTX ISA: rcp
// 1 ulp; rsqrt 2^-22.4, ex2 2^-22 relative; lg2 2^-22 absolute on (1/2, 2), else relative).
PR_DEV float approx_lg2(float x) { float r; asm("lg2.approx.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
PR_DEV float approx_ex2(float x) { float r; asm("ex2.approx.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
PR_DEV float approx_rsq(float x) { float r; asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
PR_DEV float approx_rcp(float x) { float r; asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

// A frame's dependent launches are programmatic: a kernel's blocks become
// resident while its predecessor drains, and wait here for it to complete (and
// its writes to be seen) before their first access. Between plain launches of
// a small frame the device idled 3 to 4 us each (frames of 800x500 to
// 1280x720: 96, 164 and 192 us, so 69, 131 and 152). A kernel releases its
// successor only past its own wait, so that completion stays transitive, and
// only a short one does so before its end: waiting blocks hold registers that
// another stream's kernels could use.
PR_DEV void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
PR_DEV void release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
PR_DEV void publish(uint32_t* p) { asm volatile("st.release.gpu.u32 [%0], %1;" ::"l"(p), "r"(1u) : "memory"); }
PR_DEV bool published(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v != 0u;
}
PR_DEV unsigned long long device_clock() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

PR_DEV V4 ld4(const float4 q) { return {q.x, q.y, q.z, q.w}; }

// Mat4.MulM (math/mat4.go:201-220), plain float32 sums left to right.
PR_DEV void mulm(const float* m, const float* n, float* r) {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            r[i * 4 + j] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[i * 4 + 0], n[0 * 4 + j]), __fmul_rn(m[i * 4 + 1], n[1 * 4 + j])),
                                               __fmul_rn(m[i * 4 + 2], n[2 * 4 + j])),
                                     __fmul_rn(m[i * 4 + 3], n[3 * 4 + j]));
}

PR_DEV bool approx_eq(float a, float b) { return fabsf(__fsub_rn(a, b)) <= kEps; }
PR_DEV bool approx_less(float a, float b) { return a < b && fabsf(__fsub_rn(a, b)) > kEps; }
PR_DEV bool le_approx(float a, float b) { return approx_eq(a, b) || approx_less(a, b); }

// Triangle.IsValid (geometry/primitive/triangle.go:63-80)
PR_DEV bool tri_is_valid(V4 p1, V4 p2, V4 p3) {
    V4 a = sub4(p2, p1), b = sub4(p3, p1);
    if (approx_eq(a.x, 0) && approx_eq(a.y, 0) && approx_eq(a.z, 0)) return false;
    if (approx_eq(b.x, 0) && approx_eq(b.y, 0) && approx_eq(b.z, 0)) return false;
    float d = __fdiv_rn(dot4(a, b), __fmul_rn(len4(a), len4(b)));
    return !approx_eq(d, 1.0f) && !approx_eq(d, -1.0f);
}

struct Box { float mnx, mny, mnz, mxx, mxy, mxz; };
// NewAABB over three points (geometry/primitive/box.go:15-27)
PR_DEV Box box3(V4 a, V4 b, V4 c) {
    Box r;
    r.mnx = pmin(pmin(pmin(3.40282347e38f, a.x), b.x), c.x);
    r.mny = pmin(pmin(pmin(3.40282347e38f, a.y), b.y), c.y);
    r.mnz = pmin(pmin(pmin(3.40282347e38f, a.z), b.z), c.z);
    r.mxx = pmax(pmax(pmax(-3.40282347e38f, a.x), b.x), c.x);
    r.mxy = pmax(pmax(pmax(-3.40282347e38f, a.y), b.y), c.y);
    r.mxz = pmax(pmax(pmax(-3.40282347e38f, a.z), b.z), c.z);
    return r;
}
// AABB.Intersect with the reference's maxZ := Min(aabb.Max.Y, aabb2.Max.Z)
// (geometry/primitive/box.go:32-41); `a` is the viewport box.
PR_DEV bool box_intersect(const Box& a, const Box& b) {
    float minX = pmax(a.mnx, b.mnx), minY = pmax(a.mny, b.mny), minZ = pmax(a.mnz, b.mnz);
    float maxX = pmin(a.mxx, b.mxx), maxY = pmin(a.mxy, b.mxy), maxZ = pmin(a.mxy, b.mxz);
    return minX <= maxX && minY <= maxY && minZ <= maxZ;
}
PR_DEV bool box_contains(const Box& a, V4 v) {
    return le_approx(a.mnx, v.x) && le_approx(a.mny, v.y) && le_approx(a.mnz, v.z) && le_approx(v.x, a.mxx) &&
           le_approx(v.y, a.mxy) && le_approx(v.z, a.mxz);
}

// Pixel rectangle of drawClipped / drawDepth (render/raster.go:473-477),
// clamped to the W x H buffer. Returns false when empty.
// The viewport box and clip extent of a pass: float32(MSAA * size), the
// reference's MSAA*buf.Bounds().Dx() with the buffer already n times the
// image (render/raster.go:414-441, render/cull.go:15-23). Pixel boxes stay
// clamped to the target (buf.In).
PR_DEV float ext_w(const SetupParams& P) { return (float)(P.msaa > 1 ? P.W * P.msaa : P.W); }
PR_DEV float ext_h(const SetupParams& P) { return (float)(P.msaa > 1 ? P.H * P.msaa : P.H); }

// The pixels of the reference's box that the inside test can accept: those
// whose centre lies within a margin m of the triangle's bounding box; every
// other pixel fails drawClipped's test bc >= -Epsilon (render/raster.go:491)
// for certain, so leaving it out changes no fragment.
//
// Why. Let S_j (j = 0..2) be the exact cross products of the exact vertex
// differences with the pixel centre p, S their sum (the exact Sabc), bc_j =
// S_j / S. If p.x >= max_x + m, then p.x - max_x = sum_j bc_j (x_j - max_x)
// <= N w_x with N the sum of the negative bc_j and w_x the box width, so
// some bc_j <= -m / (2 w_x) (at most two are negative): |S_j| >=
// m |S| / (2 w_x), opposite in sign to S (the same for the other sides and
// for y). The test's float32 values: each cross product is formed from
// rounded differences (relative error u = 2^-24 each) as fma64f(vx, wy,
// -RN(vy wx)), within 3u (|vx wy| + |vy wx|) of its rounded-input value, so
// within dS = 6u E U of the exact one, E = w_x + w_y bounding every edge's
// L1 length and U = E + 4 every |p - vertex|_1 over the box (the reference
// box lies within the bounding box padded by 1.5 px); Sabc within dA = 6u E^2.
// When L = |Sabc| - dA > 2 dA, the signs hold and the computed b_j =
// RN(S_j' / Sabc') <= -(|S_j| - dS) / (|S| + dA) (1 - u) < -Epsilon as soon
// as |S_j| - dS >= 2e-7 (|Sabc| + 2 dA), which m_x = 2 w_x (dS + 2.1e-7
// (|Sabc| + 2 dA)) / L guarantees. All in upward rounding; degenerate,
// near-degenerate and non-finite triangles keep the reference box (their
// NaN and infinite barycentrics can pass the test anywhere in it).
PR_DEV void tighten_box(V4 a, V4 b, V4 c, float sabc, long long& x0, long long& x1, long long& y0, long long& y1) {
    const float mnx = fminf(fminf(a.x, b.x), c.x), mxx = fmaxf(fmaxf(a.x, b.x), c.x);
    const float mny = fminf(fminf(a.y, b.y), c.y), mxy = fmaxf(fmaxf(a.y, b.y), c.y);
    if (!(isfinite(mnx) && isfinite(mxx) && isfinite(mny) && isfinite(mxy) && isfinite(sabc))) return;
    const float wx = __fsub_ru(mxx, mnx), wy = __fsub_ru(mxy, mny);
    const float E = __fadd_ru(wx, wy), U = __fadd_ru(E, 4.0f);
    const float k6u = 3.6e-7f;  // >= 6 * 2^-24
    const float dS = __fmul_ru(__fmul_ru(k6u, E), U), dA = __fmul_ru(__fmul_ru(k6u, E), E);
    const float as = fabsf(sabc);
    const float L = __fsub_rd(as, dA);
    if (!(L > __fmul_ru(2.0f, dA)) || !(L > 0.0f)) return;
    const float q = __fdiv_ru(__fadd_ru(dS, __fmul_ru(2.1e-7f, __fadd_ru(as, __fmul_ru(2.0f, dA)))), L);
    const float mx = __fmul_ru(__fmul_ru(2.0f, wx), q), my = __fmul_ru(__fmul_ru(2.0f, wy), q);
    // centres x + 0.5 in [mnx - mx, mxx + mx], rounded outward
    const float lx = ceilf(__fsub_rd(__fsub_rd(mnx, mx), 0.5f)), hx = floorf(__fsub_ru(__fadd_ru(mxx, mx), 0.5f));
    const float ly = ceilf(__fsub_rd(__fsub_rd(mny, my), 0.5f)), hy = floorf(__fsub_ru(__fadd_ru(mxy, my), 0.5f));
    if (!(lx <= hx && ly <= hy)) {  // no pixel centre can pass
        x0 = 1;
        x1 = 0;
        return;
    }
    // within the reference box (|coordinates| < 2^24 there): float compares, then exact conversions
    if (lx > (float)x0) x0 = (long long)lx;
    if (hx < (float)x1) x1 = (long long)hx;
    if (ly > (float)y0) y0 = (long long)ly;
    if (hy < (float)y1) y1 = (long long)hy;
}

// The reference's pixel box (rounded bounding box padded by one, clamped
// to the target), narrowed by tighten_box: its words and its area, 0 with no
// pixel to test. Any coordinates, NaN and infinities included.
struct PixBox {
    uint32_t area, bx, by;
};
PR_DEV bool pixel_range(V4 a, V4 b, V4 c, float sabc, int W, int H, long long& x0, long long& x1, long long& y0, long long& y1) {
    Box r = box3(a, b, c);
    long long xmin = go_f2i(__fsub_rn(pround(r.mnx), 1.0f));
    long long xmax = go_f2i(__fadd_rn(pround(r.mxx), 1.0f));
    long long ymin = go_f2i(__fsub_rn(pround(r.mny), 1.0f));
    long long ymax = go_f2i(__fadd_rn(pround(r.mxy), 1.0f));
    x0 = xmin < 0 ? 0 : xmin, x1 = xmax > W - 1 ? W - 1 : xmax;
    y0 = ymin < 0 ? 0 : ymin, y1 = ymax > H - 1 ? H - 1 : ymax;
    if (x0 > x1 || y0 > y1) return false;
    tighten_box(a, b, c, sabc, x0, x1, y0, y1);
    return x0 <= x1 && y0 <= y1;
}
static __device__ __noinline__ PixBox pixel_box_any(V4 a, V4 b, V4 c, float sabc, int W, int H) {
    long long x0, x1, y0, y1;
    if (!pixel_range(a, b, c, sabc, W, H, x0, x1, y0, y1)) return {0u, 0u, 0u};
    return {(uint32_t)((x1 - x0 + 1) * (y1 - y0 + 1)), (uint32_t)x0 | ((uint32_t)x1 << 16), (uint32_t)y0 | ((uint32_t)y1 << 16)};
}

// The box of three screen vertices. fin: every coordinate is finite, where the
// plain minima and maxima are box3's, and below 2^62, where the reference's
// int() of a rounded coordinate is its value (from 2^63 on it is the smallest
// int64, which leaves a box empty). The others go through the general
// functions. The setup kernels are bound by issue, and box3's special cases,
// the 64-bit conversions of the pixel box and an IEEE quotient for its margin
// were a third of a triangle's instructions.
struct ScrBox {
    float mnx, mxx, mny, mxy, mnz, mxz;
    bool fin;
};
PR_DEV ScrBox scr_box(V4 a, V4 b, V4 c) {
    const float sum = __fadd_rn(__fadd_rn(__fadd_rn(fabsf(a.x), fabsf(a.y)), __fadd_rn(fabsf(a.z), fabsf(b.x))),
                                __fadd_rn(__fadd_rn(fabsf(b.y), fabsf(b.z)),
                                          __fadd_rn(fabsf(c.x), __fadd_rn(fabsf(c.y), fabsf(c.z)))));
    return {fminf(fminf(a.x, b.x), c.x), fmaxf(fmaxf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y), fmaxf(fmaxf(a.y, b.y), c.y),
            fminf(fminf(a.z, b.z), c.z), fmaxf(fmaxf(a.z, b.z), c.z), sum < 4e18f};
}
static __device__ __noinline__ bool intersect_any(float ew, float eh, V4 a, V4 b, V4 c) {
    const Box vp = {0.0f, 0.0f, -1.0f, ew, eh, 1.0f};
    return box_intersect(vp, box3(a, b, c));
}
static __device__ __noinline__ bool contains_any(float ew, float eh, V4 a, V4 b, V4 c) {
    const Box vp = {0.0f, 0.0f, -1.0f, ew, eh, 1.0f};
    return box_contains(vp, a) && box_contains(vp, b) && box_contains(vp, c);
}
// box_intersect of the viewport box (0, 0, -1) .. (ew, eh, 1), the far end of z the reference's ew-by-eh Max.Y.
PR_DEV bool scr_intersects(const ScrBox& s, float ew, float eh, V4 a, V4 b, V4 c) {
    if (!s.fin) return intersect_any(ew, eh, a, b, c);
    return s.mxx >= 0.0f && s.mnx <= ew && s.mxy >= 0.0f && s.mny <= eh && s.mxz >= -1.0f && s.mnz <= eh;
}
// box_contains of its three vertices. Above 1 and below -1 the next float is
// already more than Epsilon away, so only the bounds at 0 keep it.
PR_DEV bool scr_contained(const ScrBox& s, float ew, float eh, V4 a, V4 b, V4 c) {
    if (!s.fin) return contains_any(ew, eh, a, b, c);
    return s.mnx >= -kEps && s.mxx <= ew && s.mny >= -kEps && s.mxy <= eh && s.mnz >= -1.0f && s.mxz <= 1.0f;
}

// pixel_box_any for a box (fin) that reaches 0 or more, in float32 (the
// coordinates, clamped to [0, 2^16], round exactly by additions of 2^23). A
// reciprocal rounded up in place of tighten_box's quotient only widens its margin.
PR_DEV PixBox pixel_box(const ScrBox& s, V4 a, V4 b, V4 c, float sabc, int W, int H) {
    if (!(s.fin && s.mxx >= 0.0f && s.mxy >= 0.0f)) return pixel_box_any(a, b, c, sabc, W, H);
    const float k23 = 8388608.0f;
    auto clip = [](float v) { return fminf(fmaxf(v, 0.0f), 65536.0f); };
    auto round_up = [&](float v) { return __fsub_rn(__fadd_rz(__fadd_rd(clip(v), 0.5f), k23), k23); };  // half away from zero
    float x0 = fmaxf(__fsub_rn(round_up(s.mnx), 1.0f), 0.0f), x1 = fminf(__fadd_rn(round_up(s.mxx), 1.0f), (float)(W - 1));
    float y0 = fmaxf(__fsub_rn(round_up(s.mny), 1.0f), 0.0f), y1 = fminf(__fadd_rn(round_up(s.mxy), 1.0f), (float)(H - 1));
    // tighten_box
    const float wx = __fsub_ru(s.mxx, s.mnx), wy = __fsub_ru(s.mxy, s.mny);
    const float E = __fadd_ru(wx, wy), U = __fadd_ru(E, 4.0f);
    const float k6u = 3.6e-7f;  // >= 6 * 2^-24
    const float dS = __fmul_ru(__fmul_ru(k6u, E), U), dA = __fmul_ru(__fmul_ru(k6u, E), E);
    const float as = fabsf(sabc), L = __fsub_rd(as, dA);
    const float inv = __fmul_ru(approx_rcp(L), 1.0000005f);
    const float q = __fmul_ru(__fadd_ru(dS, __fmul_ru(2.1e-7f, __fadd_ru(as, __fmul_ru(2.0f, dA)))), inv);
    if (L > __fmul_ru(2.0f, dA) && L > 0.0f && as < 3e38f && q < 1e30f) {
        const float mx = __fmul_ru(__fmul_ru(2.0f, wx), q), my = __fmul_ru(__fmul_ru(2.0f, wy), q);
        auto up = [&](float v) { return __fsub_rn(__fadd_ru(clip(v), k23), k23); };                           // ceil
        auto down = [&](float v) { return __fsub_rn(__fadd_rd(fminf(fmaxf(v, -4.0f), 65536.0f), k23), k23); };  // floor (v < 0: below 0)
        x0 = fmaxf(x0, up(__fsub_rd(__fsub_rd(s.mnx, mx), 0.5f)));
        x1 = fminf(x1, down(__fsub_ru(__fadd_ru(s.mxx, mx), 0.5f)));
        y0 = fmaxf(y0, up(__fsub_rd(__fsub_rd(s.mny, my), 0.5f)));
        y1 = fminf(y1, down(__fsub_ru(__fadd_ru(s.mxy, my), 0.5f)));
    }
    if (!(x0 <= x1 && y0 <= y1)) return {0u, 0u, 0u};
    auto u16 = [&](float v) { return __float_as_uint(__fadd_rn(v, k23)) - 0x4B000000u; };
    const uint32_t ix0 = u16(x0), ix1 = u16(x1), iy0 = u16(y0), iy1 = u16(y1);
    return {(ix1 - ix0 + 1u) * (iy1 - iy0 + 1u), ix0 | (ix1 << 16), iy0 | (iy1 << 16)};
}

PR_DEV uint32_t find_object(const uint32_t* first, uint32_t n_obj, uint32_t t) {
    uint32_t lo = 0, hi = n_obj - 1;
    while (lo < hi) {
        uint32_t mid = (lo + hi + 1) >> 1;
        if (first[mid] <= t)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

PR_DEV uint32_t pack_col(uchar4 c) { return (uint32_t)c.x | ((uint32_t)c.y << 8) | ((uint32_t)c.z << 16) | ((uint32_t)c.w << 24); }
PR_DEV float col_ch(uint32_t c, int k) { return small_u2f((c >> (8 * k)) & 0xffu); }

struct SubVtx {
    V4 pos;
    V4 nor;
    float u, v;
    uint32_t col;
};

// clipTriangle's re-interpolated vertex (render/clipping.go:75-102)
PR_DEV SubVtx clip_vertex(V4 cp, const SubVtx* t, float psabc) {
    float b[3];
    barycoord_s(cp.x, cp.y, t[0].pos.x, t[0].pos.y, t[1].pos.x, t[1].pos.y, t[2].pos.x, t[2].pos.y, psabc, b);
    SubVtx r;
    auto lerp3 = [&](float a0, float a1, float a2) {
        return __fadd_rn(__fadd_rn(__fmul_rn(b[0], a0), __fmul_rn(b[1], a1)), __fmul_rn(b[2], a2));
    };
    r.pos = {lerp3(t[0].pos.x, t[1].pos.x, t[2].pos.x), lerp3(t[0].pos.y, t[1].pos.y, t[2].pos.y),
             lerp3(t[0].pos.z, t[1].pos.z, t[2].pos.z), 1.0f};
    r.u = lerp3(t[0].u, t[1].u, t[2].u);
    r.v = lerp3(t[0].v, t[1].v, t[2].v);
    r.nor = {lerp3(t[0].nor.x, t[1].nor.x, t[2].nor.x), lerp3(t[0].nor.y, t[1].nor.y, t[2].nor.y),
             lerp3(t[0].nor.z, t[1].nor.z, t[2].nor.z), 0.0f};
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        float s = lerp3(col_ch(t[0].col, k), col_ch(t[1].col, k), col_ch(t[2].col, k));
        c |= go_f2u8(pclamp(s, 0.0f, 255.0f)) << (8 * k);
    }
    r.col = c;
    return r;
}

// plane.intersectSegment(v0, v1) (render/clipping.go:23-30)
PR_DEV V4 intersect_segment(V4 P, V4 N, V4 v0, V4 v1) {
    V4 u = sub4(v1, v0);
    V4 w = sub4(v0, P);
    float d = dot4(N, u);
    float nn = -dot4(N, w);
    float sc = __fdiv_rn(nn, d);
    return add4(v0, V4{__fmul_rn(u.x, sc), __fmul_rn(u.y, sc), __fmul_rn(u.z, sc), __fmul_rn(u.w, sc)});
}

// Sutherland-Hodgman against the six screen-space planes
// (render/clipping.go:31-68) over a group of kClipLanes (16) lanes, lane i
// holding polygon vertex i (n <= 9 between planes: a convex polygon gains at
// most one vertex per plane, and more means NaN coordinates broke convexity).
// For each plane every lane tests the edge from the previous vertex to its
// own, as the reference's loop does at step i, and places its 0, 1 or 2 output
// vertices at the exclusive prefix sum of the counts, so each output polygon
// is the loop's, vertex for vertex; an overflow check at step i would see the
// same prefix count. One copy of a plane's code, and a plane that cuts nothing
// is left at once: the instructions a small frame's few warps fetch are what
// the clip kernel waits for (planes 6.4 -> 3.6 us of 18 in a 641x479 frame).
// All 32 lanes of the warp call; a lane outside [0, n) holds nothing. Returns
// the vertex count (or -1) to every lane of the group, and lane i < count gets
// vertex i in *v. ring: the group's 2 x 10 vertices of shared scratch.
constexpr int kClipLanes = 16;  // >= 9 polygon vertices
PR_DEV int sutherland_hodgman_group(V4* v, int n, float w, float h, uint32_t sub, V4 (*ring)[10]) {
    const unsigned full = 0xffffffffu;
    const uint32_t gbase = (threadIdx.x & 31u) & ~(uint32_t)(kClipLanes - 1);
    int res = n;
#pragma unroll 1
    for (int pl = 0; pl < 6; pl++) {
        const V4 P = {pl == 0 ? w : 0.0f, pl == 2 ? h : 0.0f, pl == 4 ? 1.0f : pl == 5 ? -1.0f : 0.0f, 1.0f};
        const V4 N = {pl == 0 ? -1.0f : pl == 1 ? 1.0f : 0.0f, pl == 2 ? -1.0f : pl == 3 ? 1.0f : 0.0f,
                      pl == 4 ? -1.0f : pl == 5 ? 1.0f : 0.0f, 1.0f};
        const bool act = (int)sub < n;  // n == 0 (an empty polygon, or a finished group): no lane acts
        const V4 e = *v;
        const bool fe = act && dot4(sub4(e, P), N) > 0.0f;
        if (!__any_sync(full, act && !fe)) continue;  // every vertex inside: the polygons stay (res holds n)
        const int src = sub == 0u ? n - 1 : (int)sub - 1;  // the previous vertex (the last one for vertex 0)
        V4 sv;
        sv.x = __shfl_sync(full, e.x, src < 0 ? 0 : src, kClipLanes);
        sv.y = __shfl_sync(full, e.y, src < 0 ? 0 : src, kClipLanes);
        sv.z = __shfl_sync(full, e.z, src < 0 ? 0 : src, kClipLanes);
        sv.w = __shfl_sync(full, e.w, src < 0 ? 0 : src, kClipLanes);
        const bool fs = __shfl_sync(full, (int)fe, src < 0 ? 0 : src, kClipLanes) != 0;
        const int cnt = !act ? 0 : fe ? (fs ? 1 : 2) : (fs ? 1 : 0);
        int incl = cnt;
#pragma unroll
        for (int d = 1; d < kClipLanes; d <<= 1) {
            const int t = __shfl_up_sync(full, incl, d, kClipLanes);
            if ((int)sub >= d) incl += t;
        }
        const int m = incl - cnt;  // the loop's m at this step
        const int total = __shfl_sync(full, incl, kClipLanes - 1, kClipLanes);
        const bool over = act && m + (fe && !fs ? 2 : 1) > 9;
        const bool any_over = ((__ballot_sync(full, over) >> gbase) & ((1u << kClipLanes) - 1u)) != 0u;
        V4* o = ring[pl & 1];
        if (act && !any_over) {
            if (fe) {
                if (!fs) o[m] = intersect_segment(P, N, sv, e);
                o[m + (fs ? 0 : 1)] = e;
            } else if (fs) {
                o[m] = intersect_segment(P, N, sv, e);
            }
        }
        __syncwarp();
        if (n > 0) res = any_over ? -1 : total;
        n = (n > 0 && !any_over) ? total : 0;
        if ((int)sub < n) *v = o[sub];  // ring[pl & 1] is next written two planes on, after a sync
    }
    return res;
}

// Vec4.Apply kept out of line in the per-triangle setup kernels: a dozen
// inlined copies of twelve emulated float64 FMAs each overflow the
// instruction cache (no_instruction stalls dominated), one shared copy
// does not.
__device__ __noinline__ V4 apply4_outline(V4 v, const float* m) { return apply4(v, m); }
// Vec4.Apply's x, y and z (w = 0).
PR_DEV V4 apply3_try(V4 v, const float* m, bool& bad) {
    return {fma64f_try(m[0], v.x, fma64f_try(m[1], v.y, fma64f_try(m[2], v.z, __fmul_rn(m[3], v.w), bad), bad), bad),
            fma64f_try(m[4], v.x, fma64f_try(m[5], v.y, fma64f_try(m[6], v.z, __fmul_rn(m[7], v.w), bad), bad), bad),
            fma64f_try(m[8], v.x, fma64f_try(m[9], v.y, fma64f_try(m[10], v.z, __fmul_rn(m[11], v.w), bad), bad), bad), 0.0f};
}
__device__ __noinline__ V4 apply3_outline(V4 v, const float* m) {
    bool bad = false;
    const V4 r = apply3_try(v, m, bad);
    return __builtin_expect(bad, 0) ? apply4_exact(v, m) : r;
}

// A screen-space vertex back in world space (render/raster.go:467-469), x, y
// and z: pos through ViewportInv, ProjInv and ViewInv. With P.inv_std the
// first two have the zero pattern of ViewportMatrix's and of a perspective
// matrix's inverse; a zero first factor or a +-0 addend rounds alike in
// float64 and float32 (fma64f_try), so 12 of the chain's 48 FMAs need the
// float64 emulation. The matrices' own zeros stay in every term.
__device__ __noinline__ V4 world_of_exact(const SetupParams& P, V4 pos) {
    return apply4(apply4(apply4(pos, P.viewport_inv), P.proj_inv), P.view_inv);
}
PR_DEV V4 world_of(const SetupParams& P, V4 pos) {
    if (!P.inv_std) return world_of_exact(P, pos);  // uniform
    bool bad = false;
    const float *a = P.viewport_inv, *b = P.proj_inv, *c = P.view_inv;
    const V4 v = {fma64f_try(a[0], pos.x, __fmaf_rn(a[1], pos.y, __fmaf_rn(a[2], pos.z, __fmul_rn(a[3], pos.w))), bad),
                  __fmaf_rn(a[4], pos.x, fma64f_try(a[5], pos.y, __fmaf_rn(a[6], pos.z, __fmul_rn(a[7], pos.w)), bad)),
                  __fmaf_rn(a[8], pos.x, __fmaf_rn(a[9], pos.y, __fmaf_rn(a[10], pos.z, __fmul_rn(a[11], pos.w)))),
                  __fmaf_rn(a[12], pos.x, __fmaf_rn(a[13], pos.y, __fmaf_rn(a[14], pos.z, __fmul_rn(a[15], pos.w))))};
    const V4 q = {__fmaf_rn(b[0], v.x, __fmaf_rn(b[1], v.y, __fmaf_rn(b[2], v.z, __fmul_rn(b[3], v.w)))),
                  __fmaf_rn(b[4], v.x, __fmaf_rn(b[5], v.y, __fmaf_rn(b[6], v.z, __fmul_rn(b[7], v.w)))),
                  __fmaf_rn(b[8], v.x, __fmaf_rn(b[9], v.y, __fmaf_rn(b[10], v.z, __fmul_rn(b[11], v.w)))),
                  __fmaf_rn(b[12], v.x, __fmaf_rn(b[13], v.y, fma64f_try(b[14], v.z, __fmul_rn(b[15], v.w), bad)))};
    const V4 m = apply3_try(q, c, bad);
    return __builtin_expect(bad, 0) ? world_of_exact(P, pos) : m;
}

// The attribute record of record ridx (drawClipped's per-vertex inputs).
// mw: the vertices' world positions when the caller has them (the chain
// below of each vertex's screen position), else null.
PR_DEV void write_attr(const SetupParams& P, uint32_t ridx, const SubVtx* v, int matid, const V4* mw) {
    AttrRec A;
    V4 m[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        A.nor[k * 3 + 0] = v[k].nor.x;
        A.nor[k * 3 + 1] = v[k].nor.y;
        A.nor[k * 3 + 2] = v[k].nor.z;
        A.uv[k * 2 + 0] = v[k].u;
        A.uv[k * 2 + 1] = v[k].v;
        A.col[k] = v[k].col;
        // render/raster.go:467-469
        m[k] = mw ? mw[k] : world_of(P, v[k].pos);
        A.m[k * 3 + 0] = m[k].x;
        A.m[k * 3 + 1] = m[k].y;
        A.m[k * 3 + 2] = m[k].z;
    }
    V4 fn = unit4(cross4(sub4(m[1], m[0]), sub4(m[2], m[0])));  // render/raster.go:479
    A.fn[0] = fn.x; A.fn[1] = fn.y; A.fn[2] = fn.z; A.fn[3] = fn.w;
    A.matid = matid;
    const float4* as = reinterpret_cast<const float4*>(&A);
    float4* ad = reinterpret_cast<float4*>(P.arec + ridx);
#pragma unroll
    for (int k = 0; k < 8; k++) ad[k] = as[k];
}

// Build and store the records of one sub-triangle of Sabc sabc and pixel box
// pb. With P.defer_attr the attribute record is left to attr_kernel, which
// writes it only for records that win a pixel.
PR_DEV void write_sub(const SetupParams& P, uint32_t ridx, uint32_t seq, const SubVtx* v, const float* recipw, int matid,
                      float sabc, const PixBox& pb, const V4* mw = nullptr) {
    // no pixel to test: no task will name the record, no pixel can pick it
    // as its winner, so nothing reads it
    if (pb.area == 0) {
        if (P.attr_state) P.attr_state[ridx] = kAttrDone;
        return;
    }
    RasterRec R;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        R.v[3 * k + 0] = v[k].pos.x;
        R.v[3 * k + 1] = v[k].pos.y;
        R.v[3 * k + 2] = v[k].pos.z;
        R.recipw[k] = recipw ? recipw[k] : 0.0f;
    }
    R.sabc = sabc;
    R.seq = seq;
    R.bx = pb.bx;
    R.by = pb.by;
    const float4* rs = reinterpret_cast<const float4*>(&R);
    float4* rd = reinterpret_cast<float4*>(P.rrec + ridx);
#pragma unroll
    for (int k = 0; k < 4; k++) rd[k] = rs[k];
    if (P.attr_state) P.attr_state[ridx] = P.defer_attr ? kAttrDeferred : kAttrDone;
    if (P.arec && !P.defer_attr) write_attr(P, ridx, v, matid, mw);
}

// Vec4.Apply(ViewportMatrix) for a matrix of ViewportMatrix's pattern
// [sx 0 0 tx; 0 sy 0 ty; 0 0 1 0; 0 0 0 1] (P.vp_std). A zero first factor,
// or a factor 1 with a +-0 addend, rounds exactly in float64 and float32
// alike, so only the sx and sy terms need the float64-FMA emulation; the
// matrix's own entries stay in every term (signs of zero included).
__device__ __noinline__ V4 apply_viewport_exact(V4 v, const float* m) { return apply4(v, m); }
PR_DEV V4 apply_viewport(V4 v, const float* m) {
    bool bad = false;
    const V4 r = {fma64f_try(m[0], v.x, __fmaf_rn(m[1], v.y, __fmaf_rn(m[2], v.z, __fmul_rn(m[3], v.w))), bad),
                  __fmaf_rn(m[4], v.x, fma64f_try(m[5], v.y, __fmaf_rn(m[6], v.z, __fmul_rn(m[7], v.w)), bad)),
                  __fmaf_rn(m[8], v.x, __fmaf_rn(m[9], v.y, __fmaf_rn(m[10], v.z, __fmul_rn(m[11], v.w)))),
                  __fmaf_rn(m[12], v.x, __fmaf_rn(m[13], v.y, __fmaf_rn(m[14], v.z, __fmul_rn(m[15], v.w))))};
    return __builtin_expect(bad, 0) ? apply_viewport_exact(v, m) : r;
}
PR_DEV V4 viewport_apply(const SetupParams& P, V4 v) {
    return P.vp_std ? apply_viewport(v, P.viewport) : apply4_outline(v, P.viewport);
}

// ---- warp-aggregated reservations (all 32 lanes must call them) ----------

PR_DEV uint32_t lane_id() { return threadIdx.x & 31u; }

// Reserve n slots per lane from *counter with one atomic per warp; returns
// this lane's first slot. Sets *total to the warp's total.
PR_DEV uint32_t warp_reserve(uint32_t* counter, uint32_t n, uint32_t* total) {
    const uint32_t lane = lane_id();
    uint32_t incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (uint32_t)d) incl += v;
    }
    const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
    *total = tot;
    uint32_t base = 0;
    if (tot != 0 && lane == 31) base = atomicAdd(counter, tot);
    base = __shfl_sync(0xffffffffu, base, 31);
    return base + incl - n;
}

PR_DEV uint32_t n_tasks_of(uint32_t area, uint32_t shift) { return (area + (1u << shift) - 1u) >> shift; }

// Write n (per lane) tasks (r, 0), (r, 1), ... of record r at list + o; all
// lanes call. A lane with more than kWarpEmit tasks leaves their writing to
// the whole warp, which would otherwise wait on that lane's serial stores.
// need: the task capacity that would hold one of the list's tasks.
constexpr uint32_t kWarpEmit = 8;
PR_DEV void emit_run(const SetupParams& P, uint2* list, uint32_t cap, uint32_t o, uint32_t need, uint32_t r, uint32_t n) {
    const bool fits = o + n <= cap;
    if (n != 0 && !fits) {
        atomicOr(&P.cnt->overflow, 2u);
        atomicMax(&P.cnt->need_tasks, (o + n) * need);
    }
    const bool shared = fits && n > kWarpEmit;
    if (fits && !shared)
        for (uint32_t c = 0; c < n; c++) list[o + c] = make_uint2(r, c);
    for (unsigned big = __ballot_sync(0xffffffffu, shared); big; big &= big - 1u) {
        const int l = __ffs(big) - 1;
        const uint32_t lo = __shfl_sync(0xffffffffu, o, l), ln = __shfl_sync(0xffffffffu, n, l);
        const uint32_t lr = __shfl_sync(0xffffffffu, r, l);
        for (uint32_t c = lane_id(); c < ln; c += 32u) list[lo + c] = make_uint2(lr, c);
    }
}

// A record whose pixel box has kBigArea pixels or more (and a pass with
// room for them) gets one task per 32 x 32 block of its box (raster_block)
// in place of one per 32 pixels. 20 views inside their sphere fields (bound by
// the pixel tests' issue): raster 8.7 -> 4.2 ms, and the clip kernel no longer
// writes a ground plane's tasks by the ten thousand (1080p: 45 -> 24 us). From
// 1024 pixels on, a sphere of 2000-pixel boxes rastered in 18 us, from 4096 in 15.
// A box under five pixels wide or high keeps its small tasks: from five on, w h
// >= 4096 makes (w + 31)(h + 31) / 1024 blocks at most a quarter of w h / 32
// tasks, which is the room they have; a frame that cannot grow its lists must
// not need more than before.
constexpr uint32_t kBigArea = 4096;
PR_DEV bool is_big(const SetupParams& P, const PixBox& pb) {
    if (pb.area < kBigArea || P.cap_big == 0u) return false;
    return min((pb.bx >> 16) - (pb.bx & 0xffffu), (pb.by >> 16) - (pb.by & 0xffffu)) >= 4u;
}
// The block tasks of this lane's record, if it is a large one; all lanes call.
PR_DEV void emit_blocks(const SetupParams& P, uint32_t ridx, const PixBox& pb, bool big) {
    if (!__any_sync(0xffffffffu, big)) return;
    const uint32_t n = big ? (((pb.bx >> 16) - (pb.bx & 0xffffu) + 32u) >> 5) * (((pb.by >> 16) - (pb.by & 0xffffu) + 32u) >> 5) : 0u;
    uint32_t tot;
    const uint32_t o = warp_reserve(&P.cnt->n_big, n, &tot);
    emit_run(P, P.tasks + P.cap_tasks, P.cap_big, o, 4u, ridx, n);
    if (big) atomicAdd(&P.cnt->n_big_px, n_tasks_of(pb.area, P.task_shift));
}

// The first record and the first small task of this thread among its block's
// (128 threads, all call), by one 64-bit atomic per block: one per warp and
// counter, on two words every warp of the grid adds to, were what the setup
// kernels waited for (the 10M-triangle soup: 570 us whether a triangle took
// 55 or 31 instructions per lane). rec: 0 or 1; nt < 2^14.
struct ReserveSm {
    uint32_t warp[4], rec, task;
};
PR_DEV void block_reserve(const SetupParams& P, ReserveSm& S, uint32_t rec, uint32_t nt, uint32_t* o_rec, uint32_t* o_task) {
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t v = rec | (nt << 8);  // at most 128 records, 2^21 tasks a block
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (uint32_t)d) incl += u;
    }
    if (lane == 31) S.warp[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t tot = S.warp[0] + S.warp[1] + S.warp[2] + S.warp[3];
        unsigned long long b = 0;
        if (tot)
            b = atomicAdd(reinterpret_cast<unsigned long long*>(&P.cnt->n_rec),
                          (unsigned long long)(tot & 0xffu) | (unsigned long long)(tot >> 8) << 32);
        S.rec = (uint32_t)b;
        S.task = (uint32_t)(b >> 32);
    }
    __syncthreads();
    uint32_t off = incl - v;
    for (uint32_t w = 0; w < warp; w++) off += S.warp[w];
    *o_rec = S.rec + (off & 0xffu);
    *o_task = S.task + (off >> 8);
}

// draw's transform and culls for triangle t (render/raster.go:380-436):
// Proj.MulM(View).MulM(Model).MulV, -1/W, Viewport Apply + Pos, back-face,
// viewport AABB; then the per-vertex attributes of surviving triangles
// (the normal matrix Apply does not influence the culls).
// The objects of one setup block's triangles (usually one) and their
// Proj·View·Model, computed once per block in the order of Mat4.MulM.
constexpr int kBlkObj = 8;
struct ObjCache {
    uint32_t o0, n;  // first object; n > kBlkObj: not cached
    uint32_t first[kBlkObj + 1];
    float trans[kBlkObj][16];
};

// Block-wide (every thread calls): triangles [t0, t0 + blockDim.x).
PR_DEV void obj_cache_fill(const SetupParams& P, uint32_t t0, ObjCache& C) {
    if (threadIdx.x == 0) {
        const uint32_t t1 = min(t0 + blockDim.x, P.n_tris) - 1u;
        const uint32_t o0 = find_object(P.obj_first, P.n_objects, t0);
        C.o0 = o0;
        C.n = find_object(P.obj_first, P.n_objects, t1) - o0 + 1u;
    }
    __syncthreads();
    const uint32_t n = C.n, o0 = C.o0;
    if (n <= (uint32_t)kBlkObj) {
        for (uint32_t e = threadIdx.x; e < n * 16u; e += blockDim.x) {
            const uint32_t k = e >> 4, i = (e >> 2) & 3u, j = e & 3u;
            const float* m = P.pv + i * 4;
            const float* q = P.obj_model + (size_t)(o0 + k) * 16;
            C.trans[k][e & 15u] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], q[j]), __fmul_rn(m[1], q[4 + j])),
                                                      __fmul_rn(m[2], q[8 + j])),
                                           __fmul_rn(m[3], q[12 + j]));
        }
        for (uint32_t e = threadIdx.x; e <= n; e += blockDim.x) C.first[e] = P.obj_first[o0 + e];
    }
    __syncthreads();
}

// Object of triangle t and its Proj·View·Model: from the pass's table (the
// block's first object, then the few objects that start inside the block),
// else from the block cache when it holds t's block.
PR_DEV uint32_t object_trans(const SetupParams& P, const ObjCache* C, uint32_t t, float* trans) {
    if (P.obj_trans) {
        uint32_t o = P.blk_obj[t >> 7];
        while (o + 1 < P.n_objects && P.obj_first[o + 1] <= t) o++;
        const float4* q = reinterpret_cast<const float4*>(P.obj_trans + (size_t)o * 16);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float4 r = __ldg(q + e);
            trans[4 * e] = r.x;
            trans[4 * e + 1] = r.y;
            trans[4 * e + 2] = r.z;
            trans[4 * e + 3] = r.w;
        }
        return o;
    }
    if (C && C->n <= (uint32_t)kBlkObj) {
        uint32_t k = 0;
        while (k + 1 < C->n && C->first[k + 1] <= t) k++;
#pragma unroll
        for (int e = 0; e < 16; e++) trans[e] = C->trans[k][e];
        return C->o0 + k;
    }
    const uint32_t o = find_object(P.obj_first, P.n_objects, t);
    mulm(P.pv, P.obj_model + o * 16, trans);
    return o;
}

// Triangle.IsValid of triangle t (from the flags the scene upload computed).
PR_DEV bool tri_valid_of(const SetupParams& P, uint32_t t, const V4* p) {
    if (P.tri_flags) return (P.tri_flags[t] & kTriValid) != 0;
    return tri_is_valid(p[0], p[1], p[2]);
}

// A vertex through trans and the viewport (render/raster.go:398-412). Its -1/W
// and Pos()'s 1/W are one reciprocal where the viewport leaves w as it is.
PR_DEV V4 screen_vertex(const SetupParams& P, const float* trans, V4 p, float* recipw) {
    const V4 cp = mulv(trans, p), q = viewport_apply(P, cp);
    float r = 1.0f;
    *recipw = 1.0f;
    if (P.perspective) {  // uniform
        r = __frcp_rn(cp.w);
        *recipw = -r;
    }
    if (q.w == 1.0f || q.w == 0.0f) return {q.x, q.y, q.z, 1.0f};
    if (!P.perspective || __float_as_uint(q.w) != __float_as_uint(cp.w)) r = __frcp_rn(q.w);
    return {__fmul_rn(q.x, r), __fmul_rn(q.y, r), __fmul_rn(q.z, r), 1.0f};
}

// The transform and the culls of draw (screen positions, -1/W, Sabc, the box,
// the object); false when a cull drops the triangle.
PR_DEV bool transform_main_geom(const SetupParams& P, const ObjCache* C, uint32_t t, SubVtx* v, float* recipw,
                                uint32_t* obj, float* sabc, ScrBox* box, bool* contained) {
    V4 p[3];
#pragma unroll
    for (int k = 0; k < 3; k++) p[k] = ld4(P.pos[t * 3 + k]);
    if (!tri_valid_of(P, t, p)) return false;
    float trans[16];
    const uint32_t o = object_trans(P, C, t, trans);
#pragma unroll
    for (int k = 0; k < 3; k++) v[k].pos = screen_vertex(P, trans, p[k], recipw + k);
    // cullBackFace (render/cull.go:26-28): its cross product is Barycoord's Sabc
    *sabc = sabc_of(v[0].pos.x, v[0].pos.y, v[1].pos.x, v[1].pos.y, v[2].pos.x, v[2].pos.y);
    if (*sabc < 0.0f) return false;
    *box = scr_box(v[0].pos, v[1].pos, v[2].pos);
    if (!scr_intersects(*box, ext_w(P), ext_h(P), v[0].pos, v[1].pos, v[2].pos)) return false;
    *contained = scr_contained(*box, ext_w(P), ext_h(P), v[0].pos, v[1].pos, v[2].pos);
    *obj = o;
    return true;
}

// The per-vertex attributes of surviving triangle t of object o (the normal
// matrix Apply does not influence the culls).
PR_DEV void vertex_attrs(const SetupParams& P, uint32_t t, uint32_t o, SubVtx* v, int* matid) {
    const float* nm = P.obj_normal + o * 16;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        v[k].nor = apply3_outline(ld4(P.nor[t * 3 + k]), nm);
        const float2 uv = P.uv[t * 3 + k];
        v[k].u = uv.x;
        v[k].v = uv.y;
        v[k].col = pack_col(P.col[t * 3 + k]);
    }
    int m = P.mat[t];
    if (m >= 0) m += P.obj_matbase[o];
    *matid = m;
}

// cpuForwardPass + draw for triangles fully inside the viewport
// (render/raster.go:257-269, 380-436); clipped ones go to clip_kernel.
PR_DEV void setup_main_one(const SetupParams& P, const ObjCache* C, uint32_t t, uint32_t* clip_list, ReserveSm& S) {
    SubVtx v[3];
    float recipw[3];
    int matid = -1;
    bool contained = false;
    uint32_t obj = 0;
    float sabc = 0.0f;
    ScrBox box = {};
    const bool ok = t < P.n_tris && transform_main_geom(P, C, t, v, recipw, &obj, &sabc, &box, &contained);
    if (ok && !P.defer_attr) vertex_attrs(P, t, obj, v, &matid);
    if (ok && P.tri_scr) {
        float4* s = reinterpret_cast<float4*>(P.tri_scr + 12 * (size_t)t);
        s[0] = make_float4(v[0].pos.x, v[0].pos.y, recipw[0], v[1].pos.x);
        s[1] = make_float4(v[1].pos.y, recipw[1], v[2].pos.x, v[2].pos.y);
        s[2] = make_float4(recipw[2], 0.0f, 0.0f, 0.0f);
    }
    __syncwarp();
    const bool emit = ok && contained, clip = ok && !contained;
    if (__any_sync(0xffffffffu, clip)) {  // few triangles are
        uint32_t tot;
        const uint32_t ci = warp_reserve(&P.cnt->n_clipped, clip ? 1u : 0u, &tot);
        if (clip) clip_list[ci] = t;
    }
    PixBox pb = {0u, 0u, 0u};
    if (emit) pb = pixel_box(box, v[0].pos, v[1].pos, v[2].pos, sabc, P.W, P.H);
    uint32_t ridx, o;
    const bool big = is_big(P, pb);
    const uint32_t nt = big ? 0u : n_tasks_of(pb.area, P.task_shift);
    block_reserve(P, S, emit ? 1u : 0u, nt, &ridx, &o);
    if (emit) {
        if (ridx >= P.cap_rec) {
            atomicOr(&P.cnt->overflow, 1u);
            atomicMax(&P.cnt->need_rec, ridx + 1);
        } else {
            P.first_rec[t] = ridx;
            write_sub(P, ridx, t * 8u, v, recipw, matid, sabc, pb);
        }
    }
    emit_run(P, P.tasks, P.cap_tasks, o, 1u, ridx, nt);
    emit_blocks(P, ridx, pb, big);
}
// 8 blocks per SM (64 registers, a few spilled on rare paths): more warps to
// hide the per-triangle loads and stores measured faster than 80 registers at 6.
__global__ void __launch_bounds__(128, 8) setup_main_kernel(const __grid_constant__ SetupParams P, uint32_t* clip_list) {
    __shared__ ObjCache C;
    __shared__ ReserveSm S;
    const uint32_t tri_blocks = (P.n_tris + 127u) / 128u;
    if (blockIdx.x >= tri_blocks) {
        // The raster's keys to 0, beside the triangles' latency-bound chains
        // (a memset before them: 12 us of a 4K frame).
        const size_t at = ((size_t)(blockIdx.x - tri_blocks) * 128u + threadIdx.x) * 2u;
        const size_t step = (size_t)(gridDim.x - tri_blocks) * 256u;
        for (size_t i = at; i < P.n_clear; i += step) {
            if (i + 1u < P.n_clear)
                *reinterpret_cast<ulonglong2*>(P.clear + i) = make_ulonglong2(0ull, 0ull);
            else
                P.clear[i] = 0ull;
        }
        after_previous();
        return;
    }
    after_previous();
    release_next();
    if (!P.obj_trans) obj_cache_fill(P, blockIdx.x * blockDim.x, C);  // uniform
    setup_main_one(P, &C, blockIdx.x * blockDim.x + threadIdx.x, clip_list, S);
}

// clipTriangle (render/clipping.go:70-157) for the listed triangles: fan
// sub-triangles with seq = tri*8 + i, drawn with the parent's recipw; the
// work spread over a group of kClipLanes lanes per listed triangle. Lane k < 3 transforms vertex k (screen position, -1/W, normal);
// the group clips the triangle with one polygon vertex per lane
// (sutherland_hodgman_group); lane q re-interpolates polygon vertex q with
// its world position; lane `sub` assembles and writes fan sub-triangle sub.
// A warp issues each per-vertex step once instead of once per vertex (a frame's few clipped triangles are a serial chain, often on cold
// instruction caches). The group's lanes reserve their records in lane
// order, so its sub-triangles keep consecutive records from first_rec[t].
struct ClipGroupSm {
    V4 pos[3], nor[3];
    float recipw[3];
    V4 ring[2][10];  // the clipper's polygons
    SubVtx cv[9];    // the polygon's re-interpolated vertices
    V4 mw[9];        // and their world positions
};
PR_DEV void clip_one_group(const SetupParams& P, const uint32_t* clip_list, uint32_t j, uint32_t n, uint32_t sub,
                           ClipGroupSm& G) {
    SubVtx v[3];
    float recipw[3];
    int matid = -1;
    uint32_t t = 0;
    if (j < n) {
        t = clip_list[j];
        // the listed triangle passed transform_main_geom's culls in setup
        const uint32_t k = min(sub, 2u);
        float trans[16];
        const uint32_t o = object_trans(P, nullptr, t, trans);
        float rw;
        const V4 sp = screen_vertex(P, trans, ld4(P.pos[t * 3 + k]), &rw);
        const V4 nn = apply3_outline(ld4(P.nor[t * 3 + k]), P.obj_normal + o * 16);
        if (sub < 3u) {
            G.pos[k] = sp;
            G.nor[k] = nn;
            G.recipw[k] = rw;
        }
        int m = P.mat[t];
        if (m >= 0) m += P.obj_matbase[o];
        matid = m;
    }
    __syncwarp();
    V4 pv = {0.0f, 0.0f, 0.0f, 0.0f};  // this lane's polygon vertex
    if (j < n) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            v[k].pos = G.pos[k];
            v[k].nor = G.nor[k];
            recipw[k] = G.recipw[k];
            const float2 uv = P.uv[t * 3 + k];
            v[k].u = uv.x;
            v[k].v = uv.y;
            v[k].col = pack_col(P.col[t * 3 + k]);
        }
        pv = v[min(sub, 2u)].pos;
    }
    int nc = sutherland_hodgman_group(&pv, j < n ? 3 : 0, ext_w(P), ext_h(P), sub, G.ring);
    if (nc < 0) {
        if (sub == 0u) atomicOr(&P.cnt->overflow, 4u);
        nc = 0;
    }
    const bool attrs = P.arec && !P.defer_attr;
    if ((int)sub < nc && nc > 2) {
        const float psabc = sabc_of(v[0].pos.x, v[0].pos.y, v[1].pos.x, v[1].pos.y, v[2].pos.x, v[2].pos.y);
        const SubVtx cv = clip_vertex(pv, v, psabc);
        G.cv[sub] = cv;
        if (attrs) G.mw[sub] = world_of(P, cv.pos);
    }
    __syncwarp();
    const bool mine = (int)sub < nc - 2;
    uint32_t tot;
    Counters* crec = P.cnt_rec ? P.cnt_rec : P.cnt;
    uint32_t ridx = warp_reserve(&crec->n_rec, mine ? 1u : 0u, &tot);
    PixBox pb = {0u, 0u, 0u};
    if (mine) {
        if (ridx >= P.cap_rec) {
            atomicOr(&P.cnt->overflow, 1u);
            atomicMax(&P.cnt->need_rec, ridx + 1u);
        } else {
            if (sub == 0) P.first_rec[t] = ridx;
            const SubVtx s3[3] = {G.cv[0], G.cv[sub + 1], G.cv[sub + 2]};
            const V4 mw[3] = {G.mw[0], G.mw[sub + 1], G.mw[sub + 2]};
            const float sabc = sabc_of(s3[0].pos.x, s3[0].pos.y, s3[1].pos.x, s3[1].pos.y, s3[2].pos.x, s3[2].pos.y);
            pb = pixel_box(scr_box(s3[0].pos, s3[1].pos, s3[2].pos), s3[0].pos, s3[1].pos, s3[2].pos, sabc, P.W, P.H);
            write_sub(P, ridx, t * 8u + sub, s3, recipw, matid, sabc, pb, attrs ? mw : nullptr);
        }
    }
    const bool big = is_big(P, pb);
    const uint32_t nt = big ? 0u : n_tasks_of(pb.area, P.task_shift);
    const uint32_t o = warp_reserve(&P.cnt->n_tasks, nt, &tot);
    emit_run(P, P.tasks, P.cap_tasks, o, 1u, ridx, nt);
    emit_blocks(P, ridx, pb, big);
}
__global__ void __launch_bounds__(128) clip_kernel(const __grid_constant__ SetupParams P, const uint32_t* clip_list) {
    after_previous();
    Counters* cnt = P.cnt_rec ? P.cnt_rec : P.cnt;
    if (threadIdx.x == 0) {  // the raster starts on the unclipped triangles' tasks
        // release_next gives no order: it finds setup's writes by this word
        if (blockIdx.x == 0) publish(&cnt->set_up);
        release_next();
    }
    const uint32_t n = cnt->n_clipped;
    constexpr uint32_t kPerBlock = 128 / kClipLanes;
    __shared__ ClipGroupSm s_g[kPerBlock];
    // grid-stride over the list (uniform per block, so every warp calls clip_one_group whole)
    for (uint32_t b = blockIdx.x * kPerBlock; b < n; b += gridDim.x * kPerBlock) {
        clip_one_group(P, clip_list, b + threadIdx.x / kClipLanes, n, threadIdx.x % kClipLanes,
                       s_g[threadIdx.x / kClipLanes]);
        __syncwarp();  // the group's scratch is free for its next entry
    }
}

// The transform and the culls of drawDepth for one input triangle
// (render/shadow.go:137-192); false: dropped.
PR_DEV bool shadow_geom(const SetupParams& P, const ObjCache* C, uint32_t t, SubVtx* v, float* sabc, ScrBox* box) {
    V4 p[3];
#pragma unroll
    for (int k = 0; k < 3; k++) p[k] = ld4(P.pos[t * 3 + k]);
    if (!tri_valid_of(P, t, p)) return false;
    float trans[16];
    object_trans(P, C, t, trans);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float rw;
        v[k].pos = screen_vertex(P, trans, p[k], &rw);
        v[k].nor = {0, 0, 0, 0};
        v[k].u = v[k].v = 0;
        v[k].col = 0;
    }
    // cullBackFace (render/cull.go:26-28): culled iff cross.Z, Barycoord's Sabc, is below 0
    *sabc = sabc_of(v[0].pos.x, v[0].pos.y, v[1].pos.x, v[1].pos.y, v[2].pos.x, v[2].pos.y);
    if (*sabc < 0.0f) return false;
    // cullViewFrustum (render/cull.go:15-23): NewAABB((W,H,1),(0,0,0),(0,0,-1))
    *box = scr_box(v[0].pos, v[1].pos, v[2].pos);
    return scr_intersects(*box, ext_w(P), ext_h(P), v[0].pos, v[1].pos, v[2].pos);
}
PR_DEV void setup_shadow_one(const SetupParams& P, const ObjCache* C, uint32_t t, ReserveSm& S) {
    SubVtx v[3];
    float sabc = 0.0f;
    ScrBox box = {};
    const bool ok = t < P.n_tris && shadow_geom(P, C, t, v, &sabc, &box);
    __syncwarp();
    PixBox pb = {0u, 0u, 0u};
    if (ok) pb = pixel_box(box, v[0].pos, v[1].pos, v[2].pos, sabc, P.W, P.H);
    uint32_t none, o;
    const bool big = is_big(P, pb);
    const uint32_t nt = big ? 0u : n_tasks_of(pb.area, P.task_shift);
    block_reserve(P, S, 0u, nt, &none, &o);
    if (ok) {
        const float rw[3] = {1, 1, 1};
        write_sub(P, t, t, v, rw, -1, sabc, pb);
    }
    emit_run(P, P.tasks, P.cap_tasks, o, 1u, t, nt);
    emit_blocks(P, t, pb, big);
}
// 9 blocks per SM (56 registers): more warps than at 62 registers and 8.
__global__ void __launch_bounds__(128, 9) setup_shadow_kernel(const __grid_constant__ SetupParams P) {
    __shared__ ObjCache C;
    __shared__ ReserveSm S;
    after_previous();
    if (!P.obj_trans) obj_cache_fill(P, blockIdx.x * blockDim.x, C);  // uniform
    setup_shadow_one(P, &C, blockIdx.x * blockDim.x + threadIdx.x, S);
}

// What a frame's passes start from: the counter rows of `rows` at zero, and
// Proj·View·Model per (pass, object), the product obj_cache_fill forms.
__global__ void pass_init_kernel(const __grid_constant__ PassMats pm, int n_pass, const float* obj_model,
                                 uint32_t n_objects, float* out, Counters* cnt, uint32_t rows) {
    release_next();  // launched in full order itself
    if (blockIdx.x == 0) {
        constexpr uint32_t kWords = sizeof(Counters) / 4;
        for (uint32_t e = threadIdx.x; e < kWords * (uint32_t)kNumCounters; e += blockDim.x)
            if ((rows >> (e / kWords)) & 1u) reinterpret_cast<uint32_t*>(cnt)[e] = 0u;
        __syncthreads();
        if (threadIdx.x == 0 && (rows & 1u)) cnt->stamp[0] = device_clock();
    }
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)n_pass * n_objects * 16) return;
    const size_t po = e >> 4;
    const int pass = (int)(po / n_objects);
    const size_t o = po - (size_t)pass * n_objects;
    const uint32_t i = (uint32_t)(e >> 2) & 3u, j = (uint32_t)e & 3u;
    const float* m = pm.pv[pass] + i * 4;
    const float* q = obj_model + o * 16;
    out[e] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], q[j]), __fmul_rn(m[1], q[4 + j])), __fmul_rn(m[2], q[8 + j])),
                       __fmul_rn(m[3], q[12 + j]));
}

// ---------------------------------------------------------------- raster

constexpr int kRasterWarps = 8;

// One record of a warp's task batch in shared memory, laid out for 16-byte
// loads, with the per-triangle terms of the coverage test precomputed.
struct __align__(16) SmRec {
    float4 ab;  // A.x, A.y, B.x, B.y (screen vertices)
    float4 e0;  // (B-A).x, (B-A).y, (C-A).x, (C-A).y
    float4 e1;  // (C-B).x, (C-B).y, RN(1/Sabc) (0: no early reject), Sabc
    float4 zs;  // A.z, B.z, C.z, seq (bits)
    uint4 bb;   // bbox x0, bbox y0 + the task's first row, bbox width bw, ceil(2^32 / bw) (0 for bw = 1)
};

// A warp's raster scratch: its 32 records, the prefix of their pixel counts,
// and a ring of pixels that passed the early reject. The exact test runs
// only once 32 of them are queued, on all lanes, instead of on the lanes
// whose pixel happened to survive.
struct RasterWarpSm {
    SmRec rec[32];
    int start[32];    // first warp pixel of each task
    uint32_t tq[32];  // the task's first bbox index minus start (mod 2^32)
    uint32_t q[64];   // (slot << 27) | bbox index t (t < 2^17)
    uint32_t zk[32];  // early depth test: key of a bound on the record's depths (kNoEarlyZ: none)
};

// Early depth test. Visibility keeps the largest key per texel or pixel, so
// a fragment whose key cannot exceed the value already there changes
// nothing (values only grow during a pass). For a triangle with finite
// vertex depths Zi, a covered pixel (every computed barycentric b >=
// -Epsilon) gets z = RN(RN(RN(b0 Z0) + RN(b1 Z1)) + RN(b2 Z2)) with
// |sum b - 1| <= eta = (dA + 3 dS) / |Sabc| + 3u (1.06) (the sub-areas' and
// Sabc's rounding, as in tighten_box, and the divisions'), so z <= max Zi +
// M (eta + 6 Epsilon + 8u), M = max |Zi|, while eta <= 0.05 (b <= 1.06). The
// raster skips, before the exact test, every pixel whose current value is
// at least that bound's key (a stale read is only smaller: still sound).
constexpr uint32_t kNoEarlyZ = 0xFFFFFFFFu;  // no depth key reaches it (NaN depths take the NaN path)
PR_DEV uint32_t early_z_key(float ax, float ay, float bx, float by, float cx, float cy, float sabc, float4 zs) {
    const float z0 = zs.x, z1 = zs.y, z2 = zs.z;
    if (!(isfinite(z0) && isfinite(z1) && isfinite(z2) && isfinite(sabc) && sabc != 0.0f)) return kNoEarlyZ;
    const float mnx = fminf(fminf(ax, bx), cx), mxx = fmaxf(fmaxf(ax, bx), cx);
    const float mny = fminf(fminf(ay, by), cy), mxy = fmaxf(fmaxf(ay, by), cy);
    const float E = __fadd_ru(__fsub_ru(mxx, mnx), __fsub_ru(mxy, mny)), U = __fadd_ru(E, 4.0f);
    const float k6u = 3.6e-7f;  // >= 6 * 2^-24
    const float dS = __fmul_ru(__fmul_ru(k6u, E), U), dA = __fmul_ru(__fmul_ru(k6u, E), E);
    const float eta = __fdiv_ru(__fadd_ru(dA, __fmul_ru(3.0f, dS)), fabsf(sabc));
    if (!(eta <= 0.05f)) return kNoEarlyZ;
    const float M = fmaxf(fmaxf(fabsf(z0), fabsf(z1)), fabsf(z2));
    // 3u (1.06) + 6 Epsilon + 8u < 1.3e-6
    const float zb = __fadd_ru(fmaxf(fmaxf(z0, z1), z2), __fmul_ru(M, __fadd_ru(eta, 1.5e-6f)));
    return isfinite(zb) ? fkey(zb) : kNoEarlyZ;
}

// bbox index t of a record's pixel -> (px, py). t < 2^17 and bw <= 2^14, so
// t * bw < 2^32 and the multiply-high quotient is exact.
PR_DEV void rec_pixel(const uint4& bb, uint32_t t, int* px, int* py) {
    const uint32_t q = bb.w ? __umulhi(t, bb.w) : t;  // ceil(2^32 / 1) does not fit: one column, row t
    *px = (int)(bb.x + (t - q * bb.z));
    *py = (int)(bb.y + q);
}

// Conservative early reject (pixel certainly outside): the single-rounding
// estimate differs from the reference's double rounding by at most one ulp,
// so a margin of 2^-20 relative decides only pixels that are certainly out.
PR_DEV bool pixel_rejected(const SmRec& r, int px, int py) {
    const float fx = __fadd_rn(small_u2f((uint32_t)px), 0.5f), fy = __fadd_rn(small_u2f((uint32_t)py), 0.5f);
    const float4 ab = r.ab, e0 = r.e0, e1 = r.e1;
    const float apx = __fsub_rn(fx, ab.x), apy = __fsub_rn(fy, ab.y);
    const float bpx = __fsub_rn(fx, ab.z), bpy = __fsub_rn(fy, ab.w);
    const float inv = e1.z;
    const float w0 = __fmul_rn(__fmaf_rn(e1.x, bpy, -__fmul_rn(e1.y, bpx)), inv);
    const float w1 = __fmul_rn(__fmaf_rn(apx, e0.w, -__fmul_rn(apy, e0.z)), inv);
    const float w2 = __fmul_rn(__fmaf_rn(e0.x, apy, -__fmul_rn(e0.y, apx)), inv);
    const float shrink = 0.99999904632568359375f;  // 1 - 2^-20
    return __fmul_rn(w0, shrink) < -kEps || __fmul_rn(w1, shrink) < -kEps || __fmul_rn(w2, shrink) < -kEps;
}

// Coverage and depth of one pixel against one record (drawClipped's
// Barycoord / inside / z lines, render/raster.go:487-496).
PR_DEV bool pixel_depth(const SmRec& r, int px, int py, float* zout) {
    const float fx = __fadd_rn(small_u2f((uint32_t)px), 0.5f), fy = __fadd_rn(small_u2f((uint32_t)py), 0.5f);
    const float4 ab = r.ab, e0 = r.e0, e1 = r.e1;
    const float apx = __fsub_rn(fx, ab.x), apy = __fsub_rn(fy, ab.y);
    const float bpx = __fsub_rn(fx, ab.z), bpy = __fsub_rn(fy, ab.w);
    const float sabc = e1.w;
    const float sabp = cross_z(e0.x, e0.y, apx, apy);
    const float sapc = cross_z(apx, apy, e0.z, e0.w);
    const float sbcp = cross_z(e1.x, e1.y, bpx, bpy);
    const float b0 = __fdiv_rn(sbcp, sabc), b1 = __fdiv_rn(sapc, sabc), b2 = __fdiv_rn(sabp, sabc);
    if (b0 < -kEps || b1 < -kEps || b2 < -kEps) return false;
    const float4 zs = r.zs;
    *zout = __fadd_rn(__fadd_rn(__fmul_rn(b0, zs.x), __fmul_rn(b1, zs.y)), __fmul_rn(b2, zs.z));
    return true;
}

// The depth write of a covered pixel.
PR_DEV void put_fragment(const RasterParams& P, int px, int py, float z, uint32_t seq) {
    const bool zn = isnan(z);
    if (P.mode == kMain) {
        size_t i = (size_t)(P.H - 1 - py) * P.W + px;
        if (zn) {
            atomicMin(&P.nanseq[i], seq);
            atomicExch(&P.cnt_w->nan_flag, 1u);
            atomicAdd(&P.cnt_w->n_nan, 1u);
        } else {
            unsigned long long key = ((unsigned long long)fkey(z) << 32) | (unsigned long long)(0xFFFFFFFFu - seq);
            atomicMax(&P.keys[i], key);
        }
    } else if (P.mode == kMainFixup) {
        size_t i = (size_t)(P.H - 1 - py) * P.W + px;
        if (!zn) {
            uint32_t ns = P.nanseq[i];
            if (ns != kNone && seq < ns) P.beaten[i] = 1u;
        }
    } else if (P.mode == kShadow) {
        size_t i = (size_t)px + (size_t)py * P.W;
        if (zn) {
            if (P.lastnan) atomicMax(&P.lastnan[i], seq + 1u);
            atomicExch(&P.cnt_w->nan_flag, 1u);
            atomicAdd(&P.cnt_w->n_nan, 1u);
        } else {
            atomicMax(&P.smap[i], fkey(z));
        }
    } else {  // kShadowFixup
        size_t i = (size_t)px + (size_t)py * P.W;
        uint32_t ln = P.lastnan[i];
        if (!zn && ln != 0u && seq + 1u > ln) atomicMax(&P.smap[i], fkey(z));
    }
}
// The exact test and the depth write of one queued pixel.
PR_DEV void raster_pixel(const RasterParams& P, const RasterWarpSm& S, uint32_t ent) {
    const SmRec& r = S.rec[ent >> 27];
    int px, py;
    rec_pixel(r.bb, ent & 0x7FFFFFFu, &px, &py);
    float z;
    if (pixel_depth(r, px, py, &z)) put_fragment(P, px, py, z, __float_as_uint(r.zs.w));
}

// Tasks [base, base + 32) of one pass, one per lane, pixels spread over the
// warp by a prefix scan of their counts.
PR_DEV void raster_warp(const RasterParams& P, const uint2* tasks, uint32_t base, uint32_t n_tasks, RasterWarpSm& S,
                        bool early_z) {
    const int lane = threadIdx.x & 31;
    uint32_t ti = base + lane;
    int cnt = 0;
    uint32_t qx0 = 0;
    if (ti < n_tasks) {
        uint2 tk = tasks[ti];
        const float4* rp = reinterpret_cast<const float4*>(P.rrec + tk.x);
        const float4 q0 = rp[0], q1 = rp[1], q2 = rp[2], q3 = rp[3];
        // record: A.xyz, B.xyz, C.xyz, Sabc, packed bbox x and y ranges, seq
        const float ax = q0.x, ay = q0.y, bx = q0.w, by = q1.x, cx = q1.z, cy = q1.w, sabc = q2.y;
        const uint32_t bxr = __float_as_uint(q2.z), byr = __float_as_uint(q2.w);
        const uint32_t x0 = bxr & 0xffffu, x1 = bxr >> 16, y0 = byr & 0xffffu, y1 = byr >> 16;
        SmRec& s = S.rec[lane];
        s.ab = make_float4(ax, ay, bx, by);
        s.e0 = make_float4(__fsub_rn(bx, ax), __fsub_rn(by, ay), __fsub_rn(cx, ax), __fsub_rn(cy, ay));
        const float as = fabsf(sabc);
        const float inv = (as >= 1e-30f && as <= 1e30f) ? __frcp_rn(sabc) : 0.0f;
        s.e1 = make_float4(__fsub_rn(cx, bx), __fsub_rn(cy, by), inv, sabc);
        s.zs = make_float4(q0.z, q1.y, q2.x, q3.x);
        S.zk[lane] = (early_z && (P.mode == kMain || P.mode == kShadow)) ? early_z_key(ax, ay, bx, by, cx, cy, sabc, s.zs)
                                                                          : kNoEarlyZ;
        if (x0 <= x1 && y0 <= y1) {
            const uint32_t bw = x1 - x0 + 1, area = bw * (y1 - y0 + 1);
            const uint32_t k0 = tk.y << P.task_shift;
            if (k0 < area) cnt = (int)min(area - k0, 1u << P.task_shift);
            const uint32_t qy0 = k0 / bw;  // one division per task
            qx0 = k0 - qy0 * bw;
            s.bb = make_uint4(x0, y0 + qy0, bw, bw > 1u ? 0xFFFFFFFFu / bw + 1u : 0u);
        }
    }
    int incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        int v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    S.start[lane] = incl - cnt;
    S.tq[lane] = qx0 - (uint32_t)(incl - cnt);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    __syncwarp();
    const unsigned lt = (1u << lane) - 1u;
    uint32_t head = 0, tail = 0;  // warp-uniform ring positions
    for (int g0 = 0; g0 < total; g0 += 32) {
        const int g = g0 + lane;
        bool keep = false;
        uint32_t ent = 0;
        if (g < total) {
            int j = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1)
                if (S.start[j + step] <= g) j += step;
            const SmRec& r = S.rec[j];
            const uint32_t t = S.tq[j] + (uint32_t)g;
            int px, py;
            rec_pixel(r.bb, t, &px, &py);
            keep = !pixel_rejected(r, px, py);
            const uint32_t zk = S.zk[j];
            if (keep && zk != kNoEarlyZ) {
                if (P.mode == kShadow)
                    keep = __ldcg(P.smap + ((size_t)px + (size_t)py * P.W)) < zk;
                else
                    keep = __ldcg(P.keys + ((size_t)(P.H - 1 - py) * P.W + px)) <
                           (((unsigned long long)zk << 32) | 0xFFFFFFFFull);
            }
            ent = ((uint32_t)j << 27) | t;
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) S.q[(tail + __popc(m & lt)) & 63u] = ent;
        tail += __popc(m);
        if (tail - head >= 32u) {
            __syncwarp();
            raster_pixel(P, S, S.q[(head + lane) & 63u]);
            head += 32u;
            __syncwarp();
        }
    }
    __syncwarp();
    if ((uint32_t)lane < tail - head) raster_pixel(P, S, S.q[(head + lane) & 63u]);
    __syncwarp();
}

// A 32 x 32 block of one large record's pixel box, by a warp. Lane l first
// judges the block's 8 x 4 tile l: for each edge, the sub-area S at the tile's
// pixel centre where it is largest (towards Sabc's sign) bounds S over the
// tile, real S being linear; within dS of the computed value, itself and the
// reference's (tighten_box's bound over the record's box). Where even that
// corner is below -(Epsilon |Sabc| + 2 dS), no pixel of the tile passes the
// inside test (b_j = RN(S_j / Sabc) >= -Epsilon). The other tiles' pixels then
// go, 32 at a time, through raster_warp's tests, without the search for their
// task. Degenerate and non-finite records
// keep every tile. split (a power of two): this warp takes every split-th
// remaining tile, from the part-th on.
PR_DEV void raster_block(const RasterParams& P, uint2 task, uint32_t part, uint32_t split, RasterWarpSm& S, bool early_z) {
    const int lane = threadIdx.x & 31;
    const float4* rp = reinterpret_cast<const float4*>(P.rrec + task.x);
    const float4 q0 = rp[0], q1 = rp[1], q2 = rp[2], q3 = rp[3];
    const float ax = q0.x, ay = q0.y, bx = q0.w, by = q1.x, cx = q1.z, cy = q1.w, sabc = q2.y;
    const uint32_t bxr = __float_as_uint(q2.z), byr = __float_as_uint(q2.w);
    const uint32_t x0 = bxr & 0xffffu, x1 = bxr >> 16, y0 = byr & 0xffffu, y1 = byr >> 16;
    const uint32_t nbx = (x1 - x0 + 32u) >> 5, row = task.y / nbx;
    const uint32_t X0 = x0 + 32u * (task.y - row * nbx), Y0 = y0 + 32u * row;
    const float as = fabsf(sabc);
    const bool sane = as >= 1e-30f && as <= 1e30f;
    SmRec& r = S.rec[0];  // every lane's values are the same
    r.ab = make_float4(ax, ay, bx, by);
    r.e0 = make_float4(__fsub_rn(bx, ax), __fsub_rn(by, ay), __fsub_rn(cx, ax), __fsub_rn(cy, ay));
    r.e1 = make_float4(__fsub_rn(cx, bx), __fsub_rn(cy, by), sane ? __frcp_rn(sabc) : 0.0f, sabc);
    r.zs = make_float4(q0.z, q1.y, q2.x, q3.x);
    r.bb = make_uint4(X0, Y0, 32u, 1u << 27);  // ring entries: index in the block, row-major, 32 wide
    const uint32_t zk = (early_z && (P.mode == kMain || P.mode == kShadow)) ? early_z_key(ax, ay, bx, by, cx, cy, sabc, r.zs)
                                                                           : kNoEarlyZ;
    bool live = false;
    {
        const uint32_t tx = X0 + 8u * (lane & 3), ty = Y0 + 4u * (lane >> 2);
        if (tx <= x1 && ty <= y1) {
            live = true;
            const float E = __fadd_ru(__fsub_ru(fmaxf(fmaxf(ax, bx), cx), fminf(fminf(ax, bx), cx)),
                                      __fsub_ru(fmaxf(fmaxf(ay, by), cy), fminf(fminf(ay, by), cy)));
            const float dS = __fmul_ru(__fmul_ru(3.6e-7f, E), __fadd_ru(E, 16.0f));  // a tile reaches past the box
            const float lim = -__fadd_ru(__fmul_ru(1.01e-7f, as), __fmul_ru(2.0f, dS));
            const float fx0 = __fadd_rn(small_u2f(tx), 0.5f), fy0 = __fadd_rn(small_u2f(ty), 0.5f);
            const float fx1 = __fadd_rn(fx0, 7.0f), fy1 = __fadd_rn(fy0, 3.0f);
            const bool pos = sabc > 0.0f;
            // S = ex (py - oy) - ey (px - ox), times Sabc's sign, at its largest corner
            auto top = [&](float ex, float ey, float ox, float oy) {
                const float px = ((ey < 0.0f) == pos) ? fx1 : fx0, py = ((ex > 0.0f) == pos) ? fy1 : fy0;
                const float v = __fmaf_rn(ex, __fsub_rn(py, oy), -__fmul_rn(ey, __fsub_rn(px, ox)));
                return pos ? v : -v;
            };
            if (sane)
                live = !(top(r.e1.x, r.e1.y, bx, by) < lim || top(-r.e0.z, -r.e0.w, ax, ay) < lim ||
                         top(r.e0.x, r.e0.y, ax, ay) < lim);
        }
    }
    __syncwarp();
    const unsigned lt = (1u << lane) - 1u;
    uint32_t head = 0, tail = 0;  // warp-uniform ring positions
    const unsigned all = __ballot_sync(0xffffffffu, live);
    const bool mine = live && (__popc(all & lt) & (split - 1u)) == part;
    for (unsigned todo = __ballot_sync(0xffffffffu, mine); todo; todo &= todo - 1u) {
        const int t = __ffs(todo) - 1;
        const uint32_t lx = 8u * (t & 3) + (lane & 7), ly = 4u * (t >> 2) + (lane >> 3);
        const uint32_t px = X0 + lx, py = Y0 + ly;
        bool keep = px <= x1 && py <= y1 && !pixel_rejected(r, (int)px, (int)py);
        if (keep && zk != kNoEarlyZ) {
            if (P.mode == kShadow)
                keep = __ldcg(P.smap + ((size_t)px + (size_t)py * P.W)) < zk;
            else
                keep = __ldcg(P.keys + ((size_t)(P.H - 1 - (int)py) * P.W + px)) < (((unsigned long long)zk << 32) | 0xFFFFFFFFull);
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) S.q[(tail + __popc(m & lt)) & 63u] = ly * 32u + lx;
        tail += __popc(m);
        if (tail - head >= 32u) {
            __syncwarp();
            raster_pixel(P, S, S.q[(head + lane) & 63u]);
            head += 32u;
            __syncwarp();
        }
    }
    __syncwarp();
    if ((uint32_t)lane < tail - head) raster_pixel(P, S, S.q[(head + lane) & 63u]);
    __syncwarp();
}

constexpr uint32_t kSpreadShare = 33;  // lists with fewer tasks per warp than this (and than grab) are spread
__global__ void __launch_bounds__(kRasterWarps * 32, 6) raster_kernel(const __grid_constant__ RasterParams P) {
    __shared__ RasterWarpSm s_w[kRasterWarps];
    // after_clip: clip_kernel released this one past its own wait for setup. It
    // published setup's writes before (an acquire load per block finds them: a
    // fence here made the 1M-triangle field's raster 8 us longer, the soup's
    // 15); a block that does not find the word set waits. One block waits for
    // clip_kernel at the end, so that the next kernel finds the clipped list
    // complete; more of them would only keep the shadow passes off the device.
    if (P.after_clip) {
        if (threadIdx.x == 0) {
            if (!published(&P.cnt->set_up)) after_previous();
            if (blockIdx.x == 0) P.cnt_w->stamp[1] = device_clock();
        }
        __syncthreads();
    } else {
        after_previous();
    }
    if (P.mode == kMainFixup || P.mode == kShadowFixup) {
        if (P.cnt_w->nan_flag == 0) return;  // flags of every list of the pass meet in cnt_w
    }
    const Counters* c = P.cnt;
    const uint32_t n_tasks = c->n_tasks;
    if (c->overflow) {
        if (P.after_clip && blockIdx.x == 0) after_previous();
        return;
    }
    const int warp = threadIdx.x >> 5;
    const uint32_t nw = gridDim.x * kRasterWarps;
    // Block tasks by warp index (a few per warp), after the small ones (before
    // them, or out of line, the other lists ran 1 to 5% slower). A few of them
    // (one ground plane: some hundred) are shared by several warps each.
    auto drain_big = [&](const uint2* big, uint32_t n) {
        uint32_t sh = 0;
        while (sh < 5u && (n << (sh + 1u)) <= nw) sh++;
        for (uint32_t k = blockIdx.x * kRasterWarps + (uint32_t)warp; k < (n << sh); k += nw)
            raster_block(P, big[k >> sh], k & ((1u << sh) - 1u), 1u << sh, s_w[warp], n >= nw);
    };
    // Dynamic: a task's cost is its bbox chunk, and consecutive tasks of
    // one object tend to be alike, so a static stride leaves a tail.
    // P.grab tasks per atomic (one counter serves every warp of the
    // pass): four 32-task batches on long lists, two on shorter ones,
    // where larger grabs would leave warps without work
    // The early depth test pays on passes with many fragments per pixel;
    // on short lists its extra read only lengthens each warp's chain.
    // A list of fewer than kSpreadShare (and fewer than grab) tasks per
    // warp (a small frame: a few thousand tasks; a 2048^2 shadow pass) is spread
    // over every warp instead, down to one task each, by warp index: the
    // pass then lasts one or two small batches rather than grab tasks in
    // a few warps, and no warp waits on the counter. Its batches being
    // small, a block that becomes resident late adds little.
    auto drain = [&](const uint2* tasks, uint32_t* take, uint32_t n) {
        const uint32_t grab = P.grab ? P.grab : (n < nw * 256u ? 64u : 128u);
        const bool early_z = n >= nw * 32u;
        if (n / nw < min(grab, kSpreadShare)) {
            // spread: batches of max(n / nw, 1) tasks by warp index, at most two per warp
            const uint32_t g = max(n / nw, 1u);
            for (uint32_t base = (blockIdx.x * kRasterWarps + (uint32_t)warp) * g; base < n; base += nw * g)
                raster_warp(P, tasks, base, min(base + g, n), s_w[warp], early_z);  // g <= 32
            return;
        }
        for (;;) {
            uint32_t base = 0;
            if ((threadIdx.x & 31) == 0) base = atomicAdd(take, grab);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base >= n) break;
            const uint32_t end = min(base + grab, n);
            for (uint32_t b = base; b < end; b += 32u) raster_warp(P, tasks, b, end, s_w[warp], early_z);
        }
    };
    drain(P.tasks, P.take, n_tasks);
    if (P.big) drain_big(P.big, c->n_big);
    if (P.after_clip && blockIdx.x == 0) after_previous();
    if (P.tasks2 && !P.cnt2->overflow) {
        drain(P.tasks2, P.take2, P.cnt2->n_tasks);
        drain_big(P.big2, P.cnt2->n_big);
    }
}

// Thread tid's pixel in a 32 x 8 tile: each warp takes 16 x 2 of them. Its
// pixels share more records than a row of 32 (soup shading 449 -> 420 us,
// MSAA 2 446 -> 350 us) and its marches meet a silhouette within fewer groups
// of taps; 8 x 4 shaded as fast, but its depth loads touch four lines each
// (batched march 4.2 -> 4.6 ms).
PR_DEV uint32_t tile_x(uint32_t tid) { return ((tid >> 5) & 1u) * 16u + (tid & 15u); }
PR_DEV uint32_t tile_y(uint32_t tid) { return (tid >> 6) * 2u + ((tid >> 4) & 1u); }

// The winner of pixel i: its depth, its record (kNone: none) and its seq.
PR_DEV uint32_t resolve_one(const unsigned long long* keys, const uint32_t* nanseq, const uint32_t* beaten,
                            const Counters* cnt, const uint32_t* first_rec, uint32_t* win, float* depth_ao, size_t i,
                            uint32_t* ridx) {
    unsigned long long key = keys[i];
    uint32_t w = kNone, rec = kNone;
    float d = -1.0f;
    if (cnt->nan_flag && nanseq[i] != kNone && beaten[i] == 0u) {
        w = nanseq[i];
        d = __uint_as_float(0x7fc00000u);
    } else if (key != 0ull) {
        w = 0xFFFFFFFFu - (uint32_t)(key & 0xFFFFFFFFull);
        d = fkey_decode((uint32_t)(key >> 32));
    }
    if (w != kNone) rec = first_rec[w >> 3] + (w & 7u);
    win[i] = rec;
    depth_ao[i] = d;
    *ridx = rec;
    return w;
}

// The line maxima of a frame's depths, which AO's march skips taps by: plane
// 0 along x, 1 along the rows, 2 along the diagonal, 3 along the antidiagonal,
// each entry the maximum of the kLineReach + 1 cells that start at its pixel
// in memory order. One 32 x 8 tile per 256-thread block; depth(x, row) of any
// pixel of the frame. Bound by its 16 B of stores a pixel.
constexpr int kLineReach = 3;
template <class F>
PR_DEV void ao_linemax_tile(int W, int H, int x0, int r0, float* linemax, F depth) {
    constexpr int TW = 32 + 2 * kLineReach, TH = 8 + kLineReach;
    __shared__ float s_d[TH][TW];
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    for (int e = tid; e < TH * TW; e += 256) {
        const int q = e / TW, c = e - q * TW, x = x0 + c - kLineReach, r = r0 + q;
        s_d[q][c] = (x >= 0 && x < W && r < H) ? depth(x, r) : -3.40282347e38f;
    }
    __syncthreads();
    const int x = x0 + tx, r = r0 + ty;
    if (x >= W || r >= H) return;
    const int c = tx + kLineReach;
    float m[4];
    m[0] = m[1] = m[2] = m[3] = s_d[ty][c];
#pragma unroll
    for (int j = 1; j <= kLineReach; j++) {
        m[0] = fmaxf(m[0], s_d[ty][c + j]);
        m[1] = fmaxf(m[1], s_d[ty + j][c]);
        m[2] = fmaxf(m[2], s_d[ty + j][c + j]);
        m[3] = fmaxf(m[3], s_d[ty + j][c - j]);
    }
    const size_t i = (size_t)r * W + x, plane = (size_t)W * H;
#pragma unroll
    for (int q = 0; q < 4; q++) linemax[q * plane + i] = m[q];
}

// Resolve (resolve_one) that also marks the winners' deferred attribute
// records for attr_kernel (every pixel of a record stores the same byte) and,
// with ao_list, lists the frame's AO pixels: every covered pixel whose winning
// triangle's material has AO (tri_flags kTriAO; AmbientOcclusionShade's own
// condition, material/ao.go:22), appended tile by tile (32 x 8 blocks, warps
// in order) for the march's locality, and writes the line maxima of the
// frame's depths (a halo of kLineReach keys more per tile). One atomic per
// block. Bound by the latency of its chain of gathers (key, first_rec, state).
__global__ void __launch_bounds__(256) resolve_kernel(int W, int H, const unsigned long long* keys, uint32_t* nanseq,
                                                      uint32_t* beaten, Counters* cnt, uint32_t* win, float* depth_ao,
                                                      const uint32_t* first_rec, uint8_t* attr_state,
                                                      const uint8_t* tri_flags, uint32_t* ao_list, float* linemax) {
    after_previous();
    release_next();
    const int x = (int)(blockIdx.x * 32 + tile_x(threadIdx.x)), r = (int)(blockIdx.y * 8 + tile_y(threadIdx.x));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    bool ao = false;
    const size_t i = (size_t)r * W + x;
    if (x < W && r < H) {
        uint32_t ridx;
        const uint32_t w = resolve_one(keys, nanseq, beaten, cnt, first_rec, win, depth_ao, i, &ridx);
        // the NaN bookkeeping back to its rest state (resolve reads it last)
        if (cnt->nan_flag && nanseq[i] != kNone) {
            nanseq[i] = kNone;
            beaten[i] = 0u;
        }
        if (w != kNone) {
            // most pixels find their record marked already: a plain read first
            if (attr_state[ridx] == kAttrDeferred) attr_state[ridx] = kAttrWanted;
            ao = ao_list && (tri_flags[w >> 3] & kTriAO) != 0;
        }
    }
    if (!ao_list) return;  // uniform
    __shared__ uint32_t s_cnt[8];
    __shared__ uint32_t s_base;
    const unsigned ma = __ballot_sync(0xffffffffu, ao);
    if (lane == 0) s_cnt[warp] = (uint32_t)__popc(ma);
    __syncthreads();
    if (warp == 0 && lane == 0) {
        uint32_t tot = 0;
        for (int q = 0; q < 8; q++) tot += s_cnt[q];
        s_base = tot ? atomicAdd(&cnt->n_ao, tot) : 0u;
    }
    __syncthreads();
    if (ao) {
        uint32_t o = s_base + (uint32_t)__popc(ma & ((1u << lane) - 1u));
        for (int q = 0; q < warp; q++) o += s_cnt[q];
        ao_list[o] = (uint32_t)i;
    }
    if (linemax && !cnt->nan_flag)  // uniform; a frame with NaN depths marches without them
        ao_linemax_tile(W, H, blockIdx.x * 32, blockIdx.y * 8, linemax, [&](int cx, int cr) {
            const unsigned long long key = keys[(size_t)cr * W + cx];
            return key != 0ull ? fkey_decode((uint32_t)(key >> 32)) : -1.0f;
        });
}

// The deferred attribute records of the records resolve marked: everything
// comes back from the raster record (screen positions, the triangle in seq)
// and the scene, by the same functions the setup uses, so the bits are
// those an eager setup writes. A warp takes a run of consecutive records,
// packs the marked ones and writes them ten at a time, three lanes per record
// (one per vertex), the face normal from the three world positions gathered
// by shuffles. Record order follows triangle order, so the reads of the scene
// share sectors; taken in the order pixels found them (a list), the
// 10M-triangle soup's 3.6M records read 2.2 GB in 579 us, so 1.0 GB.
// Long lists go in runs of 128 records, shorter ones (under two such runs a
// warp) in 32, each taken from a queue (a static stride left the 1M-triangle
// field's clusters to a few warps: 44 us), and those under 32 records a warp
// in tens, one batch each, by warp index.
constexpr int kAttrRun = 128;
__global__ void __launch_bounds__(128) attr_kernel(const __grid_constant__ SetupParams P) {
    __shared__ __align__(16) float s_rec[4][10][36];  // each warp's ten records (36: their words in different banks)
    __shared__ uint32_t s_idx[4][kAttrRun];
    after_previous();
    release_next();
    const uint32_t n = min(P.cnt->n_rec, P.cap_rec);  // setup and clip wrote the state of each
    const int lane = threadIdx.x & 31, r = lane / 3, k = lane - 3 * r, warp = threadIdx.x >> 5;
    const uint32_t wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    const uint32_t run = n >= nw * 2u * kAttrRun ? kAttrRun : n >= nw * 32u ? 32u : 10u;
    for (uint32_t first = wid * run;; first += nw * run) {
        if (run != 10u) {  // marked records come in clusters: runs from a queue
            if (lane == 0) first = atomicAdd(&P.cnt->take_attr, run);
            first = __shfl_sync(0xffffffffu, first, 0);
        }
        if (first >= n) break;
        uint32_t m_n = 0;  // marked records of the run
        for (uint32_t c = 0; c < run; c += 32u) {
            const uint32_t q = first + c + (uint32_t)lane;
            const bool want = c + (uint32_t)lane < run && q < n && P.attr_state[q] == kAttrWanted;
            const unsigned b = __ballot_sync(0xffffffffu, want);
            if (want) s_idx[warp][m_n + __popc(b & ((1u << lane) - 1u))] = q;
            m_n += __popc(b);
        }
        __syncwarp();
        for (uint32_t at = 0; at < m_n; at += 10u) {
            const uint32_t j = at + (uint32_t)r;
            const bool act = lane < 30 && j < m_n;
            V4 m = {0.0f, 0.0f, 0.0f, 0.0f};
            uint32_t t = 0, o = 0;
            if (act) {
                const float* R = reinterpret_cast<const float*>(P.rrec + s_idx[warp][j]);
                t = __float_as_uint(R[12]) >> 3;
                o = P.blk_obj[t >> 7];
                while (o + 1 < P.n_objects && P.obj_first[o + 1] <= t) o++;
                const V4 pos = {R[3 * k], R[3 * k + 1], R[3 * k + 2], 1.0f};
                const V4 nor = apply3_outline(ld4(P.nor[t * 3 + k]), P.obj_normal + o * 16);
                const float2 uv = P.uv[t * 3 + k];
                m = world_of(P, pos);  // render/raster.go:467-469
                float* A = s_rec[warp][r];
                A[3 * k] = nor.x;
                A[1 + 3 * k] = nor.y;
                A[2 + 3 * k] = nor.z;
                A[9 + 2 * k] = uv.x;
                A[10 + 2 * k] = uv.y;
                A[15 + k] = __uint_as_float(pack_col(P.col[t * 3 + k]));
                A[18 + 3 * k] = m.x;
                A[19 + 3 * k] = m.y;
                A[20 + 3 * k] = m.z;
            }
            const float m1x = __shfl_down_sync(0xffffffffu, m.x, 1), m1y = __shfl_down_sync(0xffffffffu, m.y, 1),
                        m1z = __shfl_down_sync(0xffffffffu, m.z, 1);
            const float m2x = __shfl_down_sync(0xffffffffu, m.x, 2), m2y = __shfl_down_sync(0xffffffffu, m.y, 2),
                        m2z = __shfl_down_sync(0xffffffffu, m.z, 2);
            if (act && k == 0) {
                const V4 m1 = {m1x, m1y, m1z, 0.0f}, m2 = {m2x, m2y, m2z, 0.0f};
                const V4 fn = unit4(cross4(sub4(m1, m), sub4(m2, m)));  // render/raster.go:479
                float* A = s_rec[warp][r];
                A[27] = fn.x;
                A[28] = fn.y;
                A[29] = fn.z;
                A[30] = fn.w;
                int matid = P.mat[t];
                if (matid >= 0) matid += P.obj_matbase[o];
                A[31] = __int_as_float(matid);
            }
            __syncwarp();
            // the warp's records out as whole 16-byte words: 8 per record
            const uint32_t nr = min(10u, m_n - at);
            for (uint32_t e = (uint32_t)lane; e < nr * 8u; e += 32u)
                reinterpret_cast<float4*>(P.arec + s_idx[warp][at + (e >> 3)])[e & 7u] =
                    reinterpret_cast<const float4*>(s_rec[warp][e >> 3])[e & 7u];
            __syncwarp();
        }
    }
}

// Shadow NaN fix-up: pixels that saw a NaN-depth fragment restart from NaN
// (key 0) and take the maximum over the fragments drawn after the last one.
// (A small persistent grid: with no NaN fragment, the usual case, every block
// reads the flag and leaves.)
__global__ void shadow_fixup_reset_kernel(size_t n, const uint32_t* lastnan, uint32_t* smap, const Counters* cnt) {
    after_previous();
    release_next();
    if (cnt->nan_flag == 0) return;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        if (lastnan[i] != 0u) smap[i] = 0u;
}

// After a pass that saw a NaN-depth fragment, put its NaN bookkeeping back to
// the state a pass starts from (a[] = va, b[] = vb); untouched otherwise, as
// only NaN fragments write it.
__global__ void nan_cleanup_kernel(size_t n, uint32_t* a, uint32_t va, uint32_t* b, uint32_t vb, const Counters* cnt) {
    after_previous();
    release_next();
    if (cnt->nan_flag == 0) return;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        a[i] = va;
        if (b) b[i] = vb;
    }
}

__global__ void decode_shadow_kernel(const uint32_t* smap, float* out, size_t n) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = fkey_decode(smap[i]);
}

// ---------------------------------------------------------------- shade

// Go math.Pow(0.5, n) for an integer 0 <= n <= 16 is exactly 2^-n.
PR_DEV float pow_half(int n) { return __uint_as_float((uint32_t)(127 - n) << 23); }

// The differentiation G-buffer of one covered pixel: triangle, material,
// flags, fixed factor (shadow now, AO multiplied in later), the screen
// barycentric weights of the pixel centre in the input triangle (for a
// material-less pixel: its perspective-correct weights), alpha, world
// position and face normal.
PR_DEV void diff_gbuffer_pixel(const ShadeParams& P, size_t i, uint32_t seq, int matid, const pr_material* mat,
                               float shadow_w, uint32_t alpha, V4 wp, V4 fn, float fx, float fy) {
    const uint32_t t = seq >> 3;
    const float4* S = reinterpret_cast<const float4*>(P.tri_scr + 12 * (size_t)t);
    const float4 s0 = S[0], s1 = S[1], s2 = S[2];
    const float x0 = s0.x, y0 = s0.y, w0 = s0.z, x1 = s0.w, y1 = s1.x, w1 = s1.y, x2 = s1.z, y2 = s1.w, w2 = s2.x;
    const float den = (y1 - y2) * (x0 - x2) + (x2 - x1) * (y0 - y2);
    float b0 = ((y1 - y2) * (fx - x2) + (x2 - x1) * (fy - y2)) / den;
    float b1 = ((y2 - y0) * (fx - x2) + (x0 - x2) * (fy - y2)) / den;
    float b2 = 1.0f - b0 - b1;
    uint32_t fl;
    if (mat) {
        fl = P.n_lights ? kDgbLit : kDgbConst;
        if (mat->flags & PR_MAT_FLAT_SHADING) fl |= kDgbFlat;
    } else {
        fl = kDgbUnlit;
        const bool persp = (P.flags & PR_FRAME_PERSPECTIVE) != 0;
        const float q0 = persp ? w0 * b0 : b0, q1 = persp ? w1 * b1 : b1, q2 = persp ? w2 * b2 : b2;
        const float inv = 1.0f / (q0 + q1 + q2);
        b0 = q0 * inv;
        b1 = q1 * inv;
        b2 = q2 * inv;
        shadow_w = 1.0f;
    }
    float4* D = P.dgb + 4 * i;
    D[0] = make_float4(__uint_as_float(t), __int_as_float(matid), __uint_as_float(fl), shadow_w);
    D[1] = make_float4(b0, b1, b2, small_u2f(alpha));
    D[2] = make_float4(wp.x, wp.y, wp.z, 1.0f);
    D[3] = make_float4(fn.x, fn.y, fn.z, fn.w);
}

// The shadow test of one light (render/raster.go:339-352, render/shadow.go:230-283):
// ws (ViewportToWorld of the pixel) through the light's view, projection and
// the map viewport, then the map depth 0.03 in front of the pixel's.
__device__ __noinline__ bool shadow_hit_exact(const ShadeParams& P, const LightK& L, V4 ws, size_t plane, int li) {
    const V4 sc = pos4(apply4(apply4(apply4(ws, L.lview), L.lproj), P.shadow_vp));
    const long long lx = go_f2i(sc.x), ly = go_f2i(sc.y);
    const long long idx =
        (long long)((unsigned long long)lx + (unsigned long long)ly * (unsigned long long)(long long)P.SW);
    if (idx > 0 && idx < (long long)plane) {
        const float sz = fkey_decode(P.smaps[plane * li + (size_t)idx]);
        return sc.z < __fsub_rn(sz, 0.03f);
    }
    return false;
}

// shadow_hit_exact from one single-rounding transform (LightK::smap), when
// its bound (LightK::serr) decides every outcome (both truncated map
// coordinates and the depth compare); false: undecided, the caller runs the
// exact test. w passes through the three bottom rows (0, 0, 0, 1) unchanged,
// so the division uses the same iw = RN(1/w) in both; it scales the bound by
// |iw| and adds two roundings (2u |sc| < 2.4e-7 |sc|); 1e-30 covers underflow.
PR_DEV bool shadow_hit_fast(const ShadeParams& P, const LightK& L, V4 ws, size_t plane, int li, bool* hit) {
    const float* m = L.smap;
    const float* q = L.serr;
    const float ax = fabsf(ws.x), ay = fabsf(ws.y), az = fabsf(ws.z), aw = fabsf(ws.w);
    auto row = [&](const float* r) { return __fmaf_rn(r[0], ws.x, __fmaf_rn(r[1], ws.y, __fmaf_rn(r[2], ws.z, __fmul_rn(r[3], ws.w)))); };
    auto err = [&](const float* r) { return __fmaf_ru(r[0], ax, __fmaf_ru(r[1], ay, __fmaf_ru(r[2], az, __fmul_ru(r[3], aw)))); };
    const V4 e = {err(q), err(q + 4), err(q + 8), 0.0f};
    float sx = row(m), sy = row(m + 4), sz = row(m + 8), ia = 1.0f;
    if (!(ws.w == 1.0f || ws.w == 0.0f)) {  // pos4
        const float iw = __frcp_rn(ws.w);
        sx = __fmul_rn(sx, iw);
        sy = __fmul_rn(sy, iw);
        sz = __fmul_rn(sz, iw);
        ia = __fmul_ru(fabsf(iw), 1.0000002f);
    }
    const float dx = __fadd_ru(__fmaf_ru(ia, e.x, __fmul_ru(2.4e-7f, fabsf(sx))), 1e-30f);
    const float dy = __fadd_ru(__fmaf_ru(ia, e.y, __fmul_ru(2.4e-7f, fabsf(sy))), 1e-30f);
    const float dz = __fadd_ru(__fmaf_ru(ia, e.z, __fmul_ru(2.4e-7f, fabsf(sz))), 1e-30f);
    const float xl = __fsub_rd(sx, dx), xh = __fadd_ru(sx, dx);
    const float yl = __fsub_rd(sy, dy), yh = __fadd_ru(sy, dy);
    if (!(fabsf(xl) < 8388608.0f && fabsf(xh) < 8388608.0f && fabsf(yl) < 8388608.0f && fabsf(yh) < 8388608.0f))
        return false;
    const int lx = trunc_small(xl), ly = trunc_small(yl);
    if (lx != trunc_small(xh) || ly != trunc_small(yh)) return false;
    const long long idx = (long long)lx + (long long)ly * (long long)P.SW;
    if (!(idx > 0 && idx < (long long)plane)) {
        *hit = false;
        return true;
    }
    const float thr = __fsub_rn(fkey_decode(P.smaps[plane * li + (size_t)idx]), 0.03f);
    if (__fadd_ru(sz, dz) < thr) {
        *hit = true;
        return true;
    }
    if (__fsub_rd(sz, dz) >= thr) {
        *hit = false;
        return true;
    }
    return false;
}

// The lights whose map hides the pixel, plus those that cast none
// (render/raster.go:339-352). ViewportToWorld of the pixel, the same for
// every light, is exact: its terms cancel (a bound on its single-rounded value
// left one lookup in seven undecided).
PR_DEV int shadow_count(const ShadeParams& P, int x, int y, float z) {
    int occl = 0;
    const size_t plane = (size_t)P.SW * P.SH;
    const V4 ws = apply4(V4{small_u2f((uint32_t)x), small_u2f((uint32_t)y), z, 1.0f}, P.s2w);
    for (int li = 0; li < P.n_lights; li++) {
        const LightK& L = P.lights[li];
        if (!L.cast) {
            occl++;
            continue;
        }
        bool hit = false;
        if (!(L.sfast && shadow_hit_fast(P, L, ws, plane, li, &hit))) hit = shadow_hit_exact(P, L, ws, plane, li);
        occl += hit ? 1 : 0;
    }
    return occl;
}

// The colour of an image texture at a fragment (Texture.Query at the
// FragmentShader's lod) by the reference's own steps, for what texture_colour
// leaves; out of line: the shade kernel's other paths keep their registers.
static __device__ __noinline__ uint32_t texture_exact(const prt::TexDesc* td, const uint32_t* texels, float du,
                                                      float dv, float u, float v) {
    return prt::tex_query(*td, texels, prt::tex_lod(*td, du, dv), u, v);
}

// Four channels as floats. trunc_pos: truncation of v in [0, 2^23), as v + 2^23 rounded down.
struct Rgba {
    float c[4];
};
PR_DEV Rgba unpack_rgba(uint32_t t) {
    return {{small_u2f(t & 0xffu), small_u2f((t >> 8) & 0xffu), small_u2f((t >> 16) & 0xffu), small_u2f(t >> 24)}};
}
PR_DEV float trunc_pos(float v) { return __fsub_rn(__fadd_rz(v, 8388608.0f), 8388608.0f); }
// lerpc in floats: the channels are 0 .. 255 and t is in [0, 1), so uint8() only truncates.
PR_DEV Rgba lerp_rgba(const Rgba& a, const Rgba& b, float t) {
    Rgba r;
#pragma unroll
    for (int k = 0; k < 4; k++) r.c[k] = trunc_pos(__fadd_rn(a.c[k], __fmul_rn(t, __fsub_rn(b.c[k], a.c[k]))));
    return r;
}
// queryBilinear for finite u, v in [0, 2): the same products, floors and
// lerps, with 32-bit indexes (a level is under 2^15 wide).
PR_DEV Rgba bilinear_rgba(const prt::TexDesc& t, const uint32_t* texels, int lvl, float u, float v) {
    const int w = t.w[lvl], h = t.h[lvl];
    const uint32_t* tx = texels + t.off[lvl];
    if (w == 1 && h == 1) return unpack_rgba(tx[0]);
    const float x = __fmul_rn(u, __fsub_rn((float)w, 1.0f)), y = __fmul_rn(v, __fsub_rn((float)h, 1.0f));
    const float x0 = floorf(x), y0 = floorf(y);
    const int i = (int)x0, j = (int)y0;
    auto at = [&](int a, int b) { return (uint32_t)a < (uint32_t)w && (uint32_t)b < (uint32_t)h ? tx[b * w + a] : 0u; };
    const bool ir = i < w - 1, jr = j < h - 1;
    const uint32_t p1 = at(i, j);
    const Rgba c1 = unpack_rgba(p1), c2 = unpack_rgba(ir ? at(i + 1, j) : p1);
    const Rgba c3 = unpack_rgba(jr ? at(i, j + 1) : p1), c4 = unpack_rgba(ir && jr ? at(i + 1, j + 1) : p1);
    const float s = __fsub_rn(x, x0);
    return lerp_rgba(lerp_rgba(c1, c2, s), lerp_rgba(c3, c4, s), __fsub_rn(y, y0));
}
// Texture.Query at the FragmentShader's lod in float32 (the reference's Modf,
// Sqrt and Log2 are float64, at few lanes an SM: a textured 1920x1080 frame
// shaded in 86 us, so in 66).
//  * Modf of a float32 is exact in float32; a float32's float64 root rounded
//    to float32 is its float32 root.
//  * A size of at most 2 texels a pixel has lod <= 1: level 0 alone.
//  * Else lod = e + lg2.approx(m) of the size m 2^e, which is within 2^-22 of
//    lg2(m), and both lods' roundings, d = 3e-7 + 1.3e-7 lod in all, only
//    weight the two levels. Where d could change the levels, or a channel's
//    truncation (d and 6.5e-5 of roundings), texture_exact decides.
PR_DEV uint32_t texture_colour(const prt::TexDesc* td, const uint32_t* texels, float du, float dv, float u, float v) {
    const float big = 3.0e38f;
    auto wrap = [](float q) {
        const float ip = truncf(q);
        float f = __fsub_rn(q, ip);
        if (ip != 0.0f && f == 0.0f) f = 1.0f;
        return f < 0.0f ? __fsub_rn(1.0f, f) : f;
    };
    if (!(fabsf(u) < big && fabsf(v) < big)) return texture_exact(td, texels, du, dv, u, v);
    const float wu = wrap(u), wv = wrap(v);
    const prt::TexDesc& t = *td;
    auto pack = [](const Rgba& q) {
        auto b = [](float f) { return __float_as_uint(__fadd_rn(f, 8388608.0f)) & 0xffu; };
        return b(q.c[0]) | b(q.c[1]) << 8 | b(q.c[2]) << 16 | b(q.c[3]) << 24;
    };
    if (!t.use_mipmap) {
        const int w = t.w[0], h = t.h[0];
        if (w == 1 && h == 1) return texels[t.off[0]];
        const int x = (int)floorf(__fmul_rn(wu, __fsub_rn((float)w, 1.0f))), y = (int)floorf(__fmul_rn(wv, __fsub_rn((float)h, 1.0f)));
        return (uint32_t)x < (uint32_t)w && (uint32_t)y < (uint32_t)h ? texels[t.off[0] + y * w + x] : 0u;
    }
    const float siz = __fmul_rn((float)t.size, __fsqrt_rn(fmaxf(du, dv)));
    if (!(du < big && dv < big && siz < big)) return texture_exact(td, texels, du, dv, u, v);
    if (siz <= 2.0f) return pack(bilinear_rgba(t, texels, 0, wu, wv));
    const uint32_t bits = __float_as_uint(siz);
    const float lod = __fadd_rn((float)((int)(bits >> 23) - 127), approx_lg2(__uint_as_float((bits & 0x7fffffu) | 0x3f800000u)));
    const float d = __fmaf_rn(1.3e-7f, lod, 3e-7f), L = (float)t.n_levels;
    if (__fsub_rn(lod, d) >= L) return pack(bilinear_rgba(t, texels, max(t.n_levels - 2, 0), wu, wv));
    const float l1 = __fsub_rn(lod, 1.0f), hf = floorf(l1), p = __fsub_rn(l1, hf);
    const int hl = (int)hf;
    bool ok = __fadd_rn(lod, d) < L && hl >= 0 && p > __fadd_rn(d, 2e-7f) && p < __fsub_rn(1.0f, __fmul_rn(2.0f, d));
    Rgba c = {};
    if (ok) {
        const Rgba a = bilinear_rgba(t, texels, hl, wu, wv), b = bilinear_rgba(t, texels, hl + 1, wu, wv);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float ab = __fsub_rn(b.c[k], a.c[k]), m = __fmaf_rn(p, ab, a.c[k]), e = __fmaf_rn(fabsf(ab), d, 6.5e-5f);
            const float lo = trunc_pos(fmaxf(__fsub_rn(m, e), 0.0f)), hi = trunc_pos(__fadd_rn(m, e));
            ok = ok && (lo == hi || ab == 0.0f);
            c.c[k] = ab == 0.0f ? a.c[k] : hi;
        }
    }
    return ok ? pack(c) : texture_exact(td, texels, du, dv, u, v);
}

// The material of flat id m (shade's lookup), or null.
PR_DEV const pr_material* material_of(const ShadeParams& P, int m) {
    return (m >= 0 && (uint32_t)m < P.n_mats) ? &P.mats[m] : nullptr;
}

PR_DEV float wsum3(float a, float b, float c, float w1, float w2, float w3) {
    return __fadd_rn(__fadd_rn(__fmul_rn(w1, a), __fmul_rn(w2, b)), __fmul_rn(w3, c));
}

// Barycoord of pixel centre (fx, fy) in raster record R.
PR_DEV void rec_bary(const RasterRec& R, float fx, float fy, float bc[3]) {
    barycoord_s(fx, fy, R.v[0], R.v[1], R.v[3], R.v[4], R.v[6], R.v[7], R.sabc, bc);
}

// Fragment.U, V (drawClipped, render/raster.go:498-520) and, with deriv, Du, Dv.
PR_DEV float4 frag_uv(const ShadeParams& P, const RasterRec& R, const AttrRec& A, float fx, float fy, const float bc[3],
                      bool deriv) {
    const float wc1 = __fmul_rn(R.recipw[0], bc[0]), wc2 = __fmul_rn(R.recipw[1], bc[1]), wc3 = __fmul_rn(R.recipw[2], bc[2]);
    const float norm = (P.flags & PR_FRAME_PERSPECTIVE) ? __fdiv_rn(1.0f, __fadd_rn(__fadd_rn(wc1, wc2), wc3)) : 1.0f;
    const float uvX = __fmul_rn(wsum3(A.uv[0], A.uv[2], A.uv[4], wc1, wc2, wc3), norm);
    const float uvY = __fmul_rn(wsum3(A.uv[1], A.uv[3], A.uv[5], wc1, wc2, wc3), norm);
    float d[2] = {0.0f, 0.0f};
    if (deriv) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            float b3[3];
            rec_bary(R, k == 0 ? __fadd_rn(fx, 1.0f) : fx, k == 0 ? fy : __fadd_rn(fy, 1.0f), b3);
            const float w1 = __fmul_rn(R.recipw[0], b3[0]), w2 = __fmul_rn(R.recipw[1], b3[1]), w3 = __fmul_rn(R.recipw[2], b3[2]);
            const float nk = __fdiv_rn(1.0f, __fadd_rn(__fadd_rn(w1, w2), w3));
            const float a = __fsub_rn(__fmul_rn(wsum3(A.uv[0], A.uv[2], A.uv[4], w1, w2, w3), nk), uvX);
            const float b = __fsub_rn(__fmul_rn(wsum3(A.uv[1], A.uv[3], A.uv[5], w1, w2, w3), nk), uvY);
            d[k] = __fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b));
        }
    }
    return make_float4(uvX, uvY, d[0], d[1]);
}

// Fragment.Col: the perspective-correct vertex colour.
PR_DEV uint32_t frag_col(const ShadeParams& P, const RasterRec& R, const AttrRec& A, const float bc[3]) {
    const float wc1 = __fmul_rn(R.recipw[0], bc[0]), wc2 = __fmul_rn(R.recipw[1], bc[1]), wc3 = __fmul_rn(R.recipw[2], bc[2]);
    const float norm = (P.flags & PR_FRAME_PERSPECTIVE) ? __fdiv_rn(1.0f, __fadd_rn(__fadd_rn(wc1, wc2), wc3)) : 1.0f;
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float s = __fmul_rn(wsum3(col_ch(A.col[0], k), col_ch(A.col[1], k), col_ch(A.col[2], k), wc1, wc2, wc3), norm);
        c |= go_f2u8(pclamp(s, 0.0f, 255.0f)) << (8 * k);
    }
    return c;
}

PR_DEV V4 frag_normal(const AttrRec& A, const float bc[3]) {
    return unit4(V4{wsum3(A.nor[0], A.nor[3], A.nor[6], bc[0], bc[1], bc[2]), wsum3(A.nor[1], A.nor[4], A.nor[7], bc[0], bc[1], bc[2]),
                    wsum3(A.nor[2], A.nor[5], A.nor[8], bc[0], bc[1], bc[2]), 0.0f});
}
PR_DEV V4 frag_world(const AttrRec& A, const float bc[3]) {
    return {wsum3(A.m[0], A.m[3], A.m[6], bc[0], bc[1], bc[2]), wsum3(A.m[1], A.m[4], A.m[7], bc[0], bc[1], bc[2]),
            wsum3(A.m[2], A.m[5], A.m[8], bc[0], bc[1], bc[2]), 1.0f};
}

// FragmentShader's lighting (shader/blinn_cpu.go:24-106) of a fragment with
// normal nn at wp and texel tc: R | G << 8 | B << 16. n_lights > 0.
PR_DEV uint32_t blinn_exact(const ShadeParams& P, const pr_material* mat, uint32_t tc, V4 nn, V4 wp) {
    const float cr = col_ch(tc, 0), cg = col_ch(tc, 1), cb = col_ch(tc, 2);
    float LaR = 0, LaG = 0, LaB = 0;
    for (int e = 0; e < P.n_ambient; e++) {
        LaR = __fadd_rn(LaR, __fmul_rn(P.ambient[e], cr));
        LaG = __fadd_rn(LaG, __fmul_rn(P.ambient[e], cg));
        LaB = __fadd_rn(LaB, __fmul_rn(P.ambient[e], cb));
    }
    float LdR = 0, LdG = 0, LdB = 0, LsR = 0, LsG = 0, LsB = 0;
    const V4 cam = {P.cam[0], P.cam[1], P.cam[2], 1.0f};
    const V4 Vv = unit4(sub4(cam, wp));  // the same for every light
    for (int li = 0; li < P.n_lights; li++) {
        const LightK& L = P.lights[li];
        V4 Lv;
        float I;
        if (L.type == PR_LIGHT_POINT) {
            const V4 Ldir = sub4(V4{L.pos[0], L.pos[1], L.pos[2], 1.0f}, wp);
            // Ldir.Unit() and Ldir.Len() share one length
            const float ln = len4(Ldir);
            const float inv = __fdiv_rn(1.0f, ln);
            Lv = V4{__fmul_rn(Ldir.x, inv), __fmul_rn(Ldir.y, inv), __fmul_rn(Ldir.z, inv), __fmul_rn(Ldir.w, inv)};
            I = __fdiv_rn(L.intensity, ln);
        } else {
            Lv = V4{-L.dir[0], -L.dir[1], -L.dir[2], 0.0f};
            I = L.intensity;
        }
        V4 Hv = unit4(add4(Lv, Vv));
        float Ld = pclamp(dot4(nn, Lv), 0.0f, 1.0f);
        float Ls = go_pow_f32(pclamp(dot4(nn, Hv), 0.0f, 1.0f), mat->shininess);
        LdR = __fadd_rn(LdR, __fmul_rn(__fmul_rn(Ld, cr), I));
        LdG = __fadd_rn(LdG, __fmul_rn(__fmul_rn(Ld, cg), I));
        LdB = __fadd_rn(LdB, __fmul_rn(__fmul_rn(Ld, cb), I));
        LsR = __fadd_rn(LsR, __fmul_rn(__fmul_rn(Ls, L.color[0]), I));
        LsG = __fadd_rn(LsG, __fmul_rn(__fmul_rn(Ls, L.color[1]), I));
        LsB = __fadd_rn(LsB, __fmul_rn(__fmul_rn(Ls, L.color[2]), I));
    }
    auto fin = [&](float La, float Ld, float Ls, uint8_t kd, uint8_t ks) {
        float v = __fadd_rn(__fadd_rn(La, __fdiv_rn(__fmul_rn(small_u2f(kd), Ld), 255.0f)),
                            __fdiv_rn(__fmul_rn(small_u2f(ks), Ls), 255.0f));
        return go_f2u8(pclamp(pround(v), 0.0f, 255.0f));
    };
    return fin(LaR, LdR, LsR, mat->diffuse[0], mat->specular[0]) | fin(LaG, LdG, LsG, mat->diffuse[1], mat->specular[1]) << 8 |
           fin(LaB, LdB, LsB, mat->diffuse[2], mat->specular[2]) << 16;
}
// The same from the records, for the pixels blinn_fast leaves.
static __device__ __noinline__ uint32_t blinn_exact_px(const ShadeParams& P, uint32_t ridx, const pr_material* mat, uint32_t tc,
                                                       float fx, float fy) {
    const RasterRec& R = P.rrec[ridx];
    const AttrRec& A = P.arec[ridx];
    float bc[3];
    rec_bary(R, fx, fy, bc);
    const V4 nn = (mat->flags & PR_MAT_FLAT_SHADING) ? V4{A.fn[0], A.fn[1], A.fn[2], A.fn[3]} : frag_normal(A, bc);
    return blinn_exact(P, mat, tc, nn, frag_world(A, bc));
}


// blinn_exact_px's colour from a plain float32 evaluation and a bound on its
// distance from the reference's, when that bound decides all three bytes;
// false: undecided (or not finite). u = 2^-24 below; every bound counts the
// reference's roundings and this function's own.
//  * Sub-areas: the same differences, and float32 FMAs that differ from the
//    reference's by at most an ulp; with the quotient by a reciprocal
//    (rcp.approx, 1 ulp) a weight differs by at most 6u of itself.
//  * Interpolated vectors (normal, world position): sums of three products of
//    weights b and vertex values N: within 12u B max|N_j|, B = sum |b_j|
//    (|N_j| <= 1.7321 times its largest component).
//  * A normalised vector x with |dx| <= e: within e / |x| + 11u (the
//    reference's dot, root, reciprocal and products 5u, here the dot and
//    rsqrt.approx, 2^-22.4, 6u).
//  * n.L: within dn + dL + 8u. n.H = (n.L + n.V) / |L + V|: within dn +
//    (dL + dV + 7u) / |L + V| + 18u. A directional light's L and a face normal
//    are exact (of length about 1, or the pixel is left).
//  * Pow(x, s), 1 <= s <= 1024, x in [0, 1]: 2^(s lg2 x) with lg2.approx
//    (2^-22 absolute on (1/2, 2), relative outside) and ex2.approx (2^-22
//    relative): within (2.1e-7 s max(1, |lg2 x|) + 3.2e-7) of itself; and a
//    change dx of x moves it by at most 1.06 s dx / x of itself while s dx <=
//    0.1 x, else by x + dx.
//  * The colour is a sum of products: 2(n_lights + n_ambient) + 14 roundings
//    of at most the sum of their magnitudes. Where the lights add less than
//    half an ulp, it is the ambient term itself (often a half: 0.1 x 255).
// A left pixel costs its warp the exact path: 1.5% of the 1M-triangle field's
// pixels (17% of its warps), 0.1% of the 10M-triangle soup's and of views with
// 16 lights. Shading at 1920x1080 131 -> 113 us, 87 -> 60 M warp instructions.
PR_DEV bool blinn_fast(const ShadeParams& P, const RasterRec& R, const AttrRec& A, const pr_material* mat, uint32_t tc, float fx,
                       float fy, uint32_t* out) {
    const float u = 5.97e-8f;
    const float kTiny2 = 1e-30f, kHuge2 = 1e36f;  // squared lengths clear of underflow and overflow
    const float s = mat->shininess;
    if (!(s >= 1.0f && s <= 1024.0f)) return false;
    // weights
    const float apx = __fsub_rn(fx, R.v[0]), apy = __fsub_rn(fy, R.v[1]), bpx = __fsub_rn(fx, R.v[3]), bpy = __fsub_rn(fy, R.v[4]);
    const float abx = __fsub_rn(R.v[3], R.v[0]), aby = __fsub_rn(R.v[4], R.v[1]), acx = __fsub_rn(R.v[6], R.v[0]),
                acy = __fsub_rn(R.v[7], R.v[1]), bcx = __fsub_rn(R.v[6], R.v[3]), bcy = __fsub_rn(R.v[7], R.v[4]);
    const float inv = approx_rcp(R.sabc);
    const float b0 = __fmul_rn(__fmaf_rn(bcx, bpy, -__fmul_rn(bcy, bpx)), inv);
    const float b1 = __fmul_rn(__fmaf_rn(apx, acy, -__fmul_rn(apy, acx)), inv);
    const float b2 = __fmul_rn(__fmaf_rn(abx, apy, -__fmul_rn(aby, apx)), inv);
    const float B = __fadd_rn(__fadd_rn(fabsf(b0), fabsf(b1)), fabsf(b2));
    auto sum3 = [&](const float* q) { return __fmaf_rn(b2, q[6], __fmaf_rn(b1, q[3], __fmul_rn(b0, q[0]))); };
    auto inf9 = [&](const float* q) {
        float m = fabsf(q[0]);
#pragma unroll
        for (int k = 1; k < 9; k++) m = fmaxf(m, fabsf(q[k]));
        return m;
    };
    auto dot3 = [](float ax, float ay, float az, float bx, float by, float bz) {
        return __fmaf_rn(ax, bx, __fmaf_rn(ay, by, __fmul_rn(az, bz)));
    };
    // normal
    float nx, ny, nz, dn;
    if (mat->flags & PR_MAT_FLAT_SHADING) {
        nx = A.fn[0];
        ny = A.fn[1];
        nz = A.fn[2];
        dn = 0.0f;
        const float l2 = dot3(nx, ny, nz, nx, ny, nz);
        if (!(l2 <= 1.001f)) return false;
    } else {
        const float rx = sum3(A.nor), ry = sum3(A.nor + 1), rz = sum3(A.nor + 2);
        const float n2 = dot3(rx, ry, rz, rx, ry, rz);
        if (!(n2 > kTiny2 && n2 < kHuge2)) return false;
        const float rl = approx_rsq(n2);
        nx = __fmul_rn(rx, rl);
        ny = __fmul_rn(ry, rl);
        nz = __fmul_rn(rz, rl);
        dn = __fmul_rn(u, __fmaf_rn(__fmul_rn(22.0f, B), __fmul_rn(inf9(A.nor), rl), 12.0f));
    }
    // world position, view vector
    const float wx = sum3(A.m), wy = sum3(A.m + 1), wz = sum3(A.m + 2);
    const float dw = __fmul_rn(__fmul_rn(u, 22.0f), __fmul_rn(B, inf9(A.m)));
    float vx = __fsub_rn(P.cam[0], wx), vy = __fsub_rn(P.cam[1], wy), vz = __fsub_rn(P.cam[2], wz);
    const float v2 = dot3(vx, vy, vz, vx, vy, vz);
    if (!(v2 > kTiny2 && v2 < kHuge2)) return false;
    const float rv = approx_rsq(v2);
    vx = __fmul_rn(vx, rv);
    vy = __fmul_rn(vy, rv);
    vz = __fmul_rn(vz, rv);
    const float dv = __fmaf_rn(dw, rv, 14.0f * u);
    const float nv = dot3(nx, ny, nz, vx, vy, vz);
    float sD = 0.0f, sR = 0.0f, sG = 0.0f, sB = 0.0f;  // sums over the lights: Ld I, Ls I light colour
    float aD = 0.0f, aS = 0.0f, eD = 0.0f, eS = 0.0f;  // magnitudes and bounds of Ld I, Ls I
    for (int li = 0; li < P.n_lights; li++) {
        const LightK& L = P.lights[li];
        float lx, ly, lz, I = L.intensity, dl = 0.0f, di = 0.0f;
        if (L.type == PR_LIGHT_POINT) {
            lx = __fsub_rn(L.pos[0], wx);
            ly = __fsub_rn(L.pos[1], wy);
            lz = __fsub_rn(L.pos[2], wz);
            const float d2 = dot3(lx, ly, lz, lx, ly, lz);
            if (!(d2 > kTiny2 && d2 < kHuge2)) return false;
            const float r = approx_rsq(d2);
            lx = __fmul_rn(lx, r);
            ly = __fmul_rn(ly, r);
            lz = __fmul_rn(lz, r);
            I = __fmul_rn(I, r);
            dl = __fmaf_rn(dw, r, 14.0f * u);
            di = dl;
        } else {
            lx = -L.dir[0];
            ly = -L.dir[1];
            lz = -L.dir[2];
            if (!(dot3(lx, ly, lz, lx, ly, lz) <= 1.001f)) return false;  // uniform
        }
        const float hx = __fadd_rn(lx, vx), hy = __fadd_rn(ly, vy), hz = __fadd_rn(lz, vz);
        const float rh = approx_rsq(dot3(hx, hy, hz, hx, hy, hz));
        const float nl = dot3(nx, ny, nz, lx, ly, lz);
        const float nh = __fmul_rn(__fadd_rn(nl, nv), rh);
        const float x = fminf(fmaxf(nh, 0.0f), 1.0f), Ld = fminf(fmaxf(nl, 0.0f), 1.0f);
        const float dnl = __fadd_rn(__fadd_rn(dn, dl), 9.0f * u);
        const float dx = __fadd_rn(dn, __fmaf_rn(__fadd_rn(__fadd_rn(dl, dv), 8.0f * u), rh, 20.0f * u));
        const float lg = approx_lg2(x);
        const float Ls = approx_ex2(__fmul_rn(s, lg));
        const float sdx = __fmul_rn(s, dx);
        float ls_e = nh < -dx ? 0.0f : __fadd_rn(__fadd_rn(x, dx), 2.5e-7f);  // certainly clamped to 0, or small
        if (sdx <= __fmul_rn(0.1f, x))
            ls_e = __fmul_rn(Ls, __fadd_rn(__fmaf_rn(__fmul_rn(2.1e-7f, s), fmaxf(1.0f, -lg), 3.2e-7f),
                                           __fmul_rn(1.25f, __fmul_rn(sdx, approx_rcp(x)))));
        const float mI = fabsf(I);
        eD = __fmaf_rn(mI, __fmaf_rn(di, Ld, nl < -dnl ? 0.0f : dnl), eD);
        eS = __fmaf_rn(mI, __fmaf_rn(di, Ls, ls_e), eS);
        const float LdI = __fmul_rn(Ld, I), LsI = __fmul_rn(Ls, I);
        sD = __fadd_rn(sD, LdI);
        aD = __fadd_rn(aD, fabsf(LdI));
        aS = __fadd_rn(aS, fabsf(LsI));
        sR = __fmaf_rn(LsI, L.color[0], sR);
        sG = __fmaf_rn(LsI, L.color[1], sG);
        sB = __fmaf_rn(LsI, L.color[2], sB);
    }
    float ma = 0.0f;
    for (int e = 0; e < P.n_ambient; e++) ma = __fadd_rn(ma, fabsf(P.ambient[e]));
    // A magnitude that is not finite decides nothing (comparisons with NaN are false).
    if (!(eD < 1e30f && eS < 1e30f && aD < 1e30f && aS < 1e30f && ma < 1e30f)) return false;
    const float g = __fmul_rn(u, small_u2f(2u * (uint32_t)(P.n_lights + P.n_ambient) + 24u));
    const float k255 = 0.003921569f;
    uint32_t c = 0;
    bool ok = true;
    auto chan = [&](int k, float spec) {
        const float col = col_ch(tc, k), kd = __fmul_rn(small_u2f(mat->diffuse[k]), __fmul_rn(col, k255));
        const float ks = small_u2f(mat->specular[k]);  // the light's colour is at most 255
        float la = 0.0f;  // the reference's own ambient term
        for (int e = 0; e < P.n_ambient; e++) la = __fadd_rn(la, __fmul_rn(P.ambient[e], col));
        float v = __fmaf_rn(__fmul_rn(ks, k255), spec, __fmaf_rn(kd, sD, la));
        const float lit = __fmaf_rn(ks, aS, __fmul_rn(kd, aD)), de = __fmul_rn(1.001f, __fmaf_rn(kd, eD, __fmul_rn(ks, eS)));
        float d = __fmaf_rn(g, __fmaf_rn(ma, col, lit), de);
        if (__fadd_ru(lit, de) <= __fmul_rd(2e-8f, la)) {  // too little light to move the ambient term by half an ulp
            v = la;
            d = 0.0f;
        }
        // Round (half up for v >= 0) and Clamp of both ends of [v - d, v + d]
        const float lo = fminf(fmaxf(__fsub_rd(v, d), 0.0f), 255.0f), hi = fminf(fmaxf(__fadd_ru(v, d), 0.0f), 255.0f);
        const uint32_t q = __float_as_uint(__fadd_rz(__fadd_rd(lo, 0.5f), 8388608.0f));
        ok &= q == __float_as_uint(__fadd_rz(__fadd_ru(hi, 0.5f), 8388608.0f));
        c |= (q & 0xffu) << (8 * k);
    };
    chan(0, sR);
    chan(1, sG);
    chan(2, sB);
    *out = c;
    return ok;
}

// Returns true for a pixel that AO still has to finish (its pre-AO colour is
// in rgba; the caller lists it).
// kTex: the scene has image textures (P.mat_tex set); without them the
// texture code is compiled out and the kernel keeps its registers.
// kFast: no output asks for the fragment's own attributes (normal, world
// position, uv, vertex colour), so a lit pixel's colour may come from
// blinn_fast and its depth from the depth buffer.
template <bool kTex, bool kFast>
PR_DEV bool shade_one(const ShadeParams& P, int x, int r) {
    if (x >= P.W || r >= P.H) return false;
    const int W = P.W, H = P.H;
    const int y = H - 1 - r;
    const size_t i = (size_t)r * W + x;
    const uint32_t ridx = P.win[i];
    uint32_t c0, c1, c2, c3;
    bool ao_pending = false;
    if (ridx == kNone) {
        c0 = P.background[0]; c1 = P.background[1]; c2 = P.background[2]; c3 = P.background[3];
        if (P.tri_id) P.tri_id[i] = kNone;
        if (P.depth) P.depth[i] = 0.0f;
        if (P.gmat) P.gmat[i] = -1;
        if (!kFast) {
            if (P.gnor) P.gnor[i] = make_float4(0, 0, 0, 0);
            if (P.gfnor) P.gfnor[i] = make_float4(0, 0, 0, 0);
            if (P.gwpos) P.gwpos[i] = make_float4(0, 0, 0, 0);
            if (P.guvd) P.guvd[i] = make_float4(0, 0, 0, 0);
            if (P.gvcol) P.gvcol[i] = make_uchar4(0, 0, 0, 0);
            if (P.dgb) {
                float4* D = P.dgb + 4 * i;
                D[0] = make_float4(__uint_as_float(kNone), __int_as_float(-1), 0.0f, 1.0f);
                D[1] = make_float4(0.0f, 0.0f, 0.0f, small_u2f(c3));
                D[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                D[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
    } else {
        RasterRec R;
        {
            const float4* rp = reinterpret_cast<const float4*>(P.rrec + ridx);
            const float4 q0 = rp[0], q1 = rp[1], q2 = rp[2], q3 = rp[3];
            R.v[0] = q0.x; R.v[1] = q0.y; R.v[2] = q0.z; R.v[3] = q0.w;
            R.v[4] = q1.x; R.v[5] = q1.y; R.v[6] = q1.z; R.v[7] = q1.w;
            R.v[8] = q2.x; R.sabc = q2.y;
            R.seq = __float_as_uint(q3.x);
            R.recipw[0] = q3.y; R.recipw[1] = q3.z; R.recipw[2] = q3.w;
        }
        const AttrRec& A = P.arec[ridx];
        const float fx = __fadd_rn(small_u2f((uint32_t)x), 0.5f), fy = __fadd_rn(small_u2f((uint32_t)y), 0.5f);
        const int matid = A.matid;
        const pr_material* mat = material_of(P, matid);
        const int tix = (kTex && mat) ? P.mat_tex[matid] : -1;  // the material's image texture, if any
        // the depth the raster kept (a zero may have lost its sign, a NaN its payload)
        float z = kFast ? P.depth_ao[i] : 0.0f;
        const bool exact_bc = !kFast || !mat || tix >= 0 || z == 0.0f || isnan(z);
        float bc[3] = {0.0f, 0.0f, 0.0f};
        if (exact_bc) {
            rec_bary(R, fx, fy, bc);
            z = __fadd_rn(__fadd_rn(__fmul_rn(bc[0], R.v[2]), __fmul_rn(bc[1], R.v[5])), __fmul_rn(bc[2], R.v[8]));
        }
        if (P.tri_id) P.tri_id[i] = R.seq >> 3;
        if (P.depth) P.depth[i] = z;
        if (P.gmat) P.gmat[i] = matid;
        float4 uv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        // the UV derivatives feed that G-buffer and a mipmapped texture's lod
        if (tix >= 0 || (!kFast && P.guvd))
            uv = frag_uv(P, R, A, fx, fy, bc, matid >= 0 && ((!kFast && P.guvd) || (tix >= 0 && P.tex[tix].use_mipmap)));
        V4 n = {0, 0, 0, 0}, wp = {0, 0, 0, 0}, fn = {0, 0, 0, 0};
        uint32_t vc = 0;
        if (!kFast) {
            n = frag_normal(A, bc);
            wp = frag_world(A, bc);
            fn = V4{A.fn[0], A.fn[1], A.fn[2], A.fn[3]};
            if (P.gnor) P.gnor[i] = make_float4(n.x, n.y, n.z, n.w);
            if (P.gfnor) P.gfnor[i] = make_float4(fn.x, fn.y, fn.z, fn.w);
            if (P.gwpos) P.gwpos[i] = make_float4(wp.x, wp.y, wp.z, wp.w);
            if (P.guvd) P.guvd[i] = uv;
        }
        if (!mat || (!kFast && P.gvcol)) vc = frag_col(P, R, A, bc);
        if (!kFast && P.gvcol) P.gvcol[i] = make_uchar4(vc & 0xffu, (vc >> 8) & 0xffu, (vc >> 16) & 0xffu, vc >> 24);
        uint32_t c = vc;
        float shadow_w = 1.0f;
        if (mat) {
            // FragmentShader (shader/blinn_cpu.go:24-106): the texture colour
            // Query(lod, U, 1-V); a uniform texture gives its texel at any lod
            uint32_t tc = (uint32_t)mat->texture[0] | (uint32_t)mat->texture[1] << 8 | (uint32_t)mat->texture[2] << 16 |
                          (uint32_t)mat->texture[3] << 24;
            if (tix >= 0) tc = texture_colour(P.tex + tix, P.texels, uv.z, uv.w, uv.x, __fsub_rn(1.0f, uv.y));
            c = tc;
            if (P.n_lights != 0) {
                if (kFast) {
                    uint32_t rgb;
                    if (!blinn_fast(P, R, A, mat, tc, fx, fy, &rgb)) rgb = blinn_exact_px(P, ridx, mat, tc, fx, fy);
                    c = rgb | (tc & 0xff000000u);
                } else {
                    c = blinn_exact(P, mat, tc, (mat->flags & PR_MAT_FLAT_SHADING) ? fn : n, wp) | (tc & 0xff000000u);
                }
            }
        }
        c0 = c & 0xffu;
        c1 = (c >> 8) & 0xffu;
        c2 = (c >> 16) & 0xffu;
        c3 = c >> 24;
        if (mat) {
            // Shadows (render/raster.go:339-352, render/shadow.go:230-283)
            if ((P.flags & PR_FRAME_SHADOWMAP) && (mat->flags & PR_MAT_RECEIVE_SHADOW)) {
                const float w = pow_half(shadow_count(P, x, y, z));
                shadow_w = w;
                c0 = go_f2u8(__fmul_rn(small_u2f(c0), w));
                c1 = go_f2u8(__fmul_rn(small_u2f(c1), w));
                c2 = go_f2u8(__fmul_rn(small_u2f(c2), w));
            }
            // AmbientOcclusionShade (material/ao.go:20-73) runs in ao_kernel
            // on a compacted list of these pixels.
            ao_pending = (mat->flags & PR_MAT_AO) && P.rgba && P.ao_list;
        }
        if (!kFast && P.dgb) diff_gbuffer_pixel(P, i, R.seq, matid, mat, shadow_w, c3, wp, fn, fx, fy);
    }
    if (ao_pending) {
        P.rgba[i] = make_uchar4(c0, c1, c2, c3);  // pre-AO, pre-gamma colour
        return true;
    }
    if (P.flags & PR_FRAME_GAMMA) {
        c0 = P.gamma[c0];
        c1 = P.gamma[c1];
        c2 = P.gamma[c2];
    }
    if (P.rgba) P.rgba[i] = make_uchar4(c0, c1, c2, c3);
    return false;
}

// Block-wide append of the AO pixels of a 32 x 8 tile (every thread of the
// 256-thread block calls): one atomic per tile, so the list runs tile by
// tile and an AO block marches a compact patch whose taps overlap.
PR_DEV void ao_append_tile(const ShadeParams& P, bool pending, uint32_t i) {
    __shared__ uint32_t s_cnt[8];
    __shared__ uint32_t s_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned m = __ballot_sync(0xffffffffu, pending);
    if (lane == 0) s_cnt[warp] = (uint32_t)__popc(m);
    __syncthreads();
    if (tid == 0) {
        uint32_t tot = 0;
        for (int w = 0; w < 8; w++) tot += s_cnt[w];
        s_base = tot ? atomicAdd(&P.cnt_w->n_ao, tot) : 0u;
    }
    __syncthreads();
    if (pending) {
        uint32_t o = s_base + (uint32_t)__popc(m & ((1u << lane) - 1u));
        for (int w = 0; w < warp; w++) o += s_cnt[w];
        P.ao_list[o] = i;
    }
}
template <bool kTex, bool kFast>
// 4 blocks per SM (64 registers, a few spilled): 32 warps to hide the
// record, attribute and shadow-map loads measured faster than 80 registers at 3.
__global__ void __launch_bounds__(256, 4) shade_kernel(const __grid_constant__ ShadeParams P) {
    after_previous();
    release_next();
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) P.cnt_w->stamp[2] = device_clock();
    const int x = (int)(blockIdx.x * 32 + tile_x(threadIdx.x)), r = (int)(blockIdx.y * 8 + tile_y(threadIdx.x));
    const bool pending = shade_one<kTex, kFast>(P, x, r);
    if (P.ao_list && !P.ao_listed) ao_append_tile(P, pending, (uint32_t)r * (uint32_t)P.W + (uint32_t)x);
}

// ---------------------------------------------------------------- AO

// The 8 march directions (material/ao.go:28): cos/sin of the float32 angle.
__constant__ float c_ao_dir[2][8];

constexpr int kAoTaps = 100;     // t = 0 .. 99 (material/ao.go:44)
constexpr int kAoTable = 100;    // tap offsets for t = 2 .. 101 (t >= 100: padding)
constexpr float kAoSkip = 1.0f - 0x1p-20f;
constexpr int kAoThreads = 256;
constexpr int kAoGroups = kAoTable / 4;  // groups of four taps: 2 .. 5, 6 .. 9, ...
constexpr int kNearGroups = 2;           // groups always looked at tap by tap
constexpr int kAoWin = 24;               // line windows, one per later group (the last entry is neutral)
static_assert(kAoGroups - kNearGroups <= kAoWin && kAoWin % 4 == 0, "one window per group, four at a time");

// A block's tap tables in shared memory: per (direction, tap) the byte
// offset and bounds on 1/dist, and the same per (direction, line window).
struct __align__(16) AoTables {
    int off[8][kAoTable];
    float rlo[8][kAoTable], rhi[8][kAoTable];
    int woff[8][kAoWin];
    float wlo[8][kAoWin], whi[8][kAoWin];
};

// Bounds on 1/dist of a tap at p + (ax, ay). Along an axis (ax or ay an
// integer t, the other below 2^-16) dist is t itself: p + t is exact, and the
// other's square, at most 2^-30, is lost in t^2. Else
// |dist - |(ax, ay)|| <= sqrt(2) (h + 2^-18) + 2.5e-7 |(ax, ay)|: h bounds the rounding of
// cur = RN(p + a), 2^-18 that of p - cur, the rest the float32 steps of both distances
PR_DEV void ao_inv_dist(const AoParams& P, float ax, float ay, float* rlo, float* rhi) {
    const float t = fmaxf(fabsf(ax), fabsf(ay));
    if (fminf(fabsf(ax), fabsf(ay)) < 0x1p-16f && t == floorf(t)) {
        *rlo = __frcp_rd(t);
        *rhi = __frcp_ru(t);
        return;
    }
    const float d0 = __fsqrt_rn(__fmaf_rn(ax, ax, __fmul_rn(ay, ay)));
    const float dl = __fadd_ru(__fmul_ru(1.5f, __fadd_ru(P.ao_half_ulp, 4e-6f)), __fmul_ru(d0, 4e-7f));
    *rlo = __frcp_rd(__fadd_ru(d0, dl));
    *rhi = __frcp_ru(__fsub_rd(d0, dl));
}

// distance of material/ao.go:52, p.Sub(cur).Len() with z = w = 0
PR_DEV float ao_distance(float pxf, float pyf, float cx, float cy) {
    const float ddx = __fsub_rn(pxf, cx), ddy = __fsub_rn(pyf, cy);
    return __fsqrt_rn(fma64f(ddx, ddx, __fmul_rn(ddy, ddy)));
}

// The exact ratio elevation/distance of tap t >= 2 (distance >= 1.998).
__device__ __noinline__ float ao_exact_ratio(int t, float el, float pxf, float pyf, float dX, float dY) {
    const float tf = small_u2f((uint32_t)t);
    const float cx = __fadd_rn(pxf, __fmul_rn(dX, tf)), cy = __fadd_rn(pyf, __fmul_rn(dY, tf));
    return __fdiv_rn(el, ao_distance(pxf, pyf, cx, cy));
}

// One tap evaluated from its float coordinates, as the reference does:
// cur = p + dir*t, int(cur) (in [0, W) for the taps the caller passes), the
// distance check and the ratio. A tap that cannot raise best past the lower
// bound lb (elev <= lb (1 - 2^-20) (t - 0.0101), using dist >= t - 0.002)
// needs neither its distance nor its division. Returns false for a NaN
// elevation at dist >= 1.
PR_DEV bool ao_tap_exact(int t, float pxf, float pyf, float dX, float dY, int W, int H, const float* depth,
                         float z, float lb, float& best) {
    const float tf = small_u2f((uint32_t)t);
    const float cx = __fadd_rn(pxf, __fmul_rn(dX, tf)), cy = __fadd_rn(pyf, __fmul_rn(dY, tf));
    const uint32_t ix = __float_as_uint(__fadd_rz(fmaxf(cx, 0.0f), 8388608.0f)) - 0x4B000000u;
    const uint32_t iy = __float_as_uint(__fadd_rz(fmaxf(cy, 0.0f), 8388608.0f)) - 0x4B000000u;
    const float el = __fsub_rn(__ldg(depth + ((size_t)(H - 1 - (int)iy) * W + ix)), z);
    if (el <= __fmul_rn(__fmul_rd(lb, kAoSkip), __fsub_rd(tf, 0.0101f))) return true;
    const float d = ao_distance(pxf, pyf, cx, cy);
    if (d < 1.0f) return true;
    if (isnan(el)) return false;
    best = fmaxf(best, __fdiv_rn(el, d));
    return true;
}

// p[0] moved by a signed number of bytes; base at an unsigned one (32-bit sums: one add per load)
PR_DEV float ld_at(const float* p, int bytes) { return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + bytes)); }
PR_DEV float ld_at_u(const float* base, uint32_t bytes) { return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(base) + bytes)); }

// The elevation of fast-path tap t again (settling a pending tap reloads it
// instead of carrying it).
PR_DEV float ao_tap_elev(const int (*s_off)[kAoTable], int k, int t, const float* p0, const float* pA, int tstar, float z,
                         bool tiny) {
    const float* q = (tiny && t < tstar) ? pA : p0;
    return __fsub_rn(ld_at(q, s_off[k][t - 2]), z);
}

// maxElevationAngle's march for taps 2 .. 101 in groups of four, from shared
// tables of index offsets and of bounds on 1/dist (see ao_kernel): the exact
// ratio RN(elev/dist) of a tap lies in [RD(elev rlo), RU(elev rhi)]. A tap
// whose upper bound does not exceed lb cannot raise the maximum; the others
// are candidates, of which one is held pending by its interval. Exact ratios
// are computed only when a new candidate's interval overlaps the pending one
// and, once, for the final pending tap. best is exact throughout and lb <= the
// largest exact ratio seen so far.
template <bool TINY>
PR_DEV bool ao_fast_groups(int n_groups, const int (*s_off)[kAoTable], const float (*s_rlo)[kAoTable],
                           const float (*s_rhi)[kAoTable], int k, const float* p0, const float* pA, int tstar, float z,
                           float pxf, float pyf, float dX, float dY, float& best) {
    float lb = best;
    int pt = 0;
    float phi = 0.0f;
    bool nan_seen = false;
#pragma unroll 2
    for (int g = 0; g < n_groups; g++) {
        const int t0 = 4 * g + 2;
        const int4 o = *reinterpret_cast<const int4*>(&s_off[k][4 * g]);
        const float4 rh = *reinterpret_cast<const float4*>(&s_rhi[k][4 * g]);
        const float* q0 = (TINY && t0 < tstar) ? pA : p0;
        const float* q1 = (TINY && t0 + 1 < tstar) ? pA : p0;
        const float* q2 = (TINY && t0 + 2 < tstar) ? pA : p0;
        const float* q3 = (TINY && t0 + 3 < tstar) ? pA : p0;
        float el[4], hi[4];
        el[0] = __fsub_rn(ld_at(q0, o.x), z);
        el[1] = __fsub_rn(ld_at(q1, o.y), z);
        el[2] = __fsub_rn(ld_at(q2, o.z), z);
        el[3] = __fsub_rn(ld_at(q3, o.w), z);
        if (g == kAoGroups - 1) el[2] = el[3] = 0.0f;  // padding taps
        hi[0] = __fmul_ru(el[0], rh.x);
        hi[1] = __fmul_ru(el[1], rh.y);
        hi[2] = __fmul_ru(el[2], rh.z);
        hi[3] = __fmul_ru(el[3], rh.w);
        const bool c0 = !(hi[0] <= lb), c1 = !(hi[1] <= lb), c2 = !(hi[2] <= lb), c3 = !(hi[3] <= lb);
        if (c0 | c1 | c2 | c3) {
            const float4 rl = *reinterpret_cast<const float4*>(&s_rlo[k][4 * g]);
            const float lo[4] = {rl.x, rl.y, rl.z, rl.w};
            const bool cu[4] = {c0, c1, c2, c3};
            // Branch-free: each candidate becomes the pending tap; a pending
            // tap it overlaps is recorded and settled after the group (rare).
            int st[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                nan_seen |= isnan(el[u]);
                const bool take = cu[u] & !isnan(el[u]);
                const float rlo = __fmul_rd(el[u], lo[u]);
                const bool ov = take & (pt != 0) & !(rlo >= phi);
                st[u] = ov ? pt : 0;
                pt = take ? t0 + u : pt;
                phi = take ? hi[u] : phi;
                lb = take ? fmaxf(lb, rlo) : lb;
            }
            if (nan_seen) return false;
            if ((st[0] | st[1] | st[2] | st[3]) != 0) {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (st[u]) best = fmaxf(best, ao_exact_ratio(st[u], ao_tap_elev(s_off, k, st[u], p0, pA, tstar, z,
                                                                                     TINY),
                                                               pxf, pyf, dX, dY));
                lb = fmaxf(lb, best);
            }
        }
    }
    if (pt != 0) best = fmaxf(best, ao_exact_ratio(pt, ao_tap_elev(s_off, k, pt, p0, pA, tstar, z, TINY), pxf, pyf, dX, dY));
    return true;
}

// The exact ratios of the taps of group g (taps 4g+2 .. 4g+5) whose upper
// bound exceeds lb; returns their maximum (0 if none). Each lane loops over
// its own such taps only.
template <bool TINY>
__device__ __noinline__ float ao_settle_group(const int (*s_off)[kAoTable], const float (*s_rhi)[kAoTable], int k, int g,
                                              const float* p0, const float* pA, int tstar, float z, float pxf, float pyf,
                                              float dX, float dY, float lb) {
    const int t0 = 4 * g + 2;
    float el[4];
    unsigned m = 0;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        el[u] = ao_tap_elev(s_off, k, t0 + u, p0, pA, tstar, z, TINY);
        if (__fmul_ru(el[u], s_rhi[k][4 * g + u]) > lb) m |= 1u << u;
    }
    float r = 0.0f;
    while (m) {
        const int u = __ffs(m) - 1;
        m &= m - 1u;
        const float e = u == 0 ? el[0] : (u == 1 ? el[1] : (u == 2 ? el[2] : el[3]));
        r = fmaxf(r, ao_exact_ratio(t0 + u, e, pxf, pyf, dX, dY));
    }
    return r;
}

// A direction's term of the total, RN(HalfPi - float32(Atan(x))), for its
// largest ratio x >= 0. Up to 2.4e-4, x^3/3 is below a quarter of the gap to
// the float32 below x, and atan_f32 is x itself.
PR_DEV float ao_term(float x) {
    return __fsub_rn(1.57079632679489661923f, x <= 2.4e-4f ? x : atan_f32(x));
}
// The largest ratio known to give the same term r = ao_term(lb) as lb: for
// lb <= x <= cut, Atan(lb) <= Atan(x) <= x, and HalfPi - x lies less than half
// an ulp of r (2^-24, r in (1, 2)) below r.
PR_DEV float ao_cut(float lb, float r) {
    return r > 1.0f ? fmaxf(lb, __fadd_rd(__fsub_rn(1.57079632679489661923f, r), 5.96e-8f)) : lb;
}

// The march of ao_fast_groups for frames without NaN depths: the term of one
// direction, whose taps outside the groups have the exact maximum best. All
// 32 lanes call, each with a pixel of its own.
// A term has 2^-23 steps and most ratios are below 1e-3, so bounds on the
// largest ratio usually fix it: lb <= ratio <= ub, and every tap that cannot
// exceed cut (ao_cut(lb)) is left out. The nearest two groups are looked at
// tap by tap; each group after them first as a whole, by its line maximum
// (ao_linemax_tile): the largest elevation among the window's four cells
// times the bounds on 1/dist of its nearest and its farthest tap bounds the
// window's largest ratio from both sides. A group that some lane's ratio may
// exceed the cut in is then looked at tap by tap, by all lanes at once (their
// pixels are neighbours, a group costs a third of a divergent lane's). Where
// the terms of lb and ub differ, the lane's open groups are evaluated exactly.
// GEN: lanes may have fewer groups than all, or a tiny component that crosses
// among their taps (b0 from tap tstar on, bA before); else every lane has
// all groups at b0.
// b0, bA: byte offsets of the pixel in depth and lm (frames hold at most 2^28
// pixels), moved by a column or row for a tiny component; either may wrap
// below 0, and offset sums wrap back. pix: the pixel's own.
template <bool GEN>
PR_DEV float ao_march(int n_groups, const AoTables& S, int k, const float* depth, uint32_t pix, uint32_t b0, uint32_t bA,
                      int tstar, float z, const float* lm, float pxf, float pyf, float dX, float dY, float best) {
    float lb = best, ub = best, cut = ao_cut(lb, ao_term(lb));
    unsigned open = 0;  // groups with a tap that may exceed the cut
    auto look = [&](int g) {
        const int t0 = 4 * g + 2;
        const int4 o = *reinterpret_cast<const int4*>(&S.off[k][4 * g]);
        const float4 rh = *reinterpret_cast<const float4*>(&S.rhi[k][4 * g]);
        uint32_t q[4] = {b0 + (uint32_t)o.x, b0 + (uint32_t)o.y, b0 + (uint32_t)o.z, b0 + (uint32_t)o.w};
        if (GEN) {
            const uint32_t d = bA - b0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (t0 + u < tstar) q[u] += d;
                if (g >= n_groups) q[u] = pix;  // elevation 0
            }
        }
        float e[4];
#pragma unroll
        for (int u = 0; u < 4; u++) e[u] = __fsub_rn(ld_at_u(depth, q[u]), z);
        const float gh = fmaxf(fmaxf(__fmul_ru(e[0], rh.x), __fmul_ru(e[1], rh.y)),
                               fmaxf(__fmul_ru(e[2], rh.z), __fmul_ru(e[3], rh.w)));
        if (gh > cut) {
            const float4 rl = *reinterpret_cast<const float4*>(&S.rlo[k][4 * g]);
            const float gl = fmaxf(fmaxf(__fmul_rd(e[0], rl.x), __fmul_rd(e[1], rl.y)),
                                   fmaxf(__fmul_rd(e[2], rl.z), __fmul_rd(e[3], rl.w)));
            lb = fmaxf(lb, gl);
            ub = fmaxf(ub, gh);
            cut = fmaxf(cut, lb);
            open |= 1u << g;
        }
    };
#pragma unroll
    for (int g = 0; g < kNearGroups; g++) look(g);
    unsigned todo = 0;  // groups (less kNearGroups) to be looked at tap by tap
#pragma unroll 2
    for (int w4 = 0; w4 < kAoWin; w4 += 4) {
        const int4 o = *reinterpret_cast<const int4*>(&S.woff[k][w4]);
        const float4 rh = *reinterpret_cast<const float4*>(&S.whi[k][w4]);
        const float4 rl = *reinterpret_cast<const float4*>(&S.wlo[k][w4]);
        const int oo[4] = {o.x, o.y, o.z, o.w};
        const float hh[4] = {rh.x, rh.y, rh.z, rh.w}, ll[4] = {rl.x, rl.y, rl.z, rl.w};
        float e[4];
        bool split[4], out[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int t1 = 4 * (w4 + u + kNearGroups) + 5;  // the group's last tap; a window reaches back to t1 - 5
            uint32_t q = b0 + (uint32_t)oo[u];
            split[u] = out[u] = false;
            if (GEN) {
                out[u] = w4 + u + kNearGroups >= n_groups;
                split[u] = tstar <= t1 && tstar > t1 - 6;  // the crossing tap lies inside the window
                if (t1 < tstar) q += bA - b0;
                if (out[u] || split[u]) q = pix;
            }
            e[u] = __fsub_rn(ld_at_u(lm, q), z);
        }
        float l = lb;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (!out[u] && (split[u] || __fmul_ru(e[u], hh[u]) > cut)) todo |= 1u << (w4 + u);
            if (!out[u] && !split[u]) l = fmaxf(l, __fmul_rd(e[u], ll[u]));
        }
        lb = l;
        cut = fmaxf(cut, l);
    }
    todo = __reduce_or_sync(0xffffffffu, todo & ((1u << (kAoGroups - kNearGroups)) - 1u));
    cut = fmaxf(cut, ao_cut(lb, ao_term(lb)));
    for (; todo; todo &= todo - 1u) look(__ffs(todo) - 1 + kNearGroups);
    const float r = ao_term(lb);
    if (ub <= ao_cut(lb, r) || ao_term(ub) == r) return r;
    while (open) {
        const int g = __ffs(open) - 1;
        open &= open - 1u;
        best = fmaxf(best, ao_settle_group<GEN>(S.off, S.rhi, k, g, depth + ((int)b0 >> 2), depth + ((int)bA >> 2), tstar, z,
                                                pxf, pyf, dX, dY, lb));
        lb = fmaxf(lb, best);
    }
    return ao_term(lb);  // a tap left out lies between an earlier lb and its cut, where the term is the same
}

// AmbientOcclusionShade (material/ao.go:20-73) for the pixels the shade
// kernel listed, one thread per pixel. Per direction, maxangle is the Max
// over taps of float32(Atan(elev/dist)); Atan and the rounding to float32 are
// monotone, so it is float32(Atan(best)) with best the largest ratio, and
// only positive ratios can exceed the initial 0. A NaN ratio (at a tap not
// skipped for dist < 1) makes the direction, and so the pixel, NaN.
//
// Tap positions. cur = p + float32(dir*t) (dir.Scale(t,t,1,1) then Add) and
// Go's int(cur) is in [0, W) exactly when -1 < cur < W; cur moves
// monotonically in t, so the first tap outside the buffer (where the
// reference returns) bounds the march, and is found by binary search unless
// tap 99 is inside. For x >= 0 and a = float32(dX t):
//  * a "regular" component (a an integer, or at least 2^-10 below the next
//    integer for every t <= 99, which holds for all 8 directions) has
//    int(RN(x + a)) = x + floor(a) for coordinates below 16384, since
//    RN(x + a) cannot round up to the next integer;
//  * a tiny negative component (-1 < a < 0: the cos of float32(Pi/2) and the
//    sin of float32(Pi)) has int(RN(x - |a|)) = x while |a| is at most half
//    the gap below x, else x - 1; |a| grows with t, so the switch happens at
//    one tap t*, found by binary search.
// So while cur >= 0, the depth index of tap t is the pixel's index plus a
// per-(direction, t) offset from a table, plus a correction before t* for a
// tiny component. Taps with cur < 0 (int truncates toward zero there) and
// the last taps that do not fill a group of four take the float path.
// Tap 1 always takes it: its distance may fall below 1 (diagonals).

// The tap tables of a W x H frame (every thread of the block calls).
PR_DEV void ao_tables(const AoParams& P, AoTables& S) {
    const int W = P.W;
    for (int e = threadIdx.x; e < 8 * kAoTable; e += blockDim.x) {
        const int k = e / kAoTable, q = e - k * kAoTable, t = q + 2;
        int o = 0;
        float rlo = 0.0f, rhi = 0.0f;
        if (k < P.n_dirs) {
            // the padding taps 100, 101 read the last tap's cell, with bounds 0
            const float tf = small_u2f((uint32_t)min(t, kAoTaps - 1));
            const float ax = __fmul_rn(c_ao_dir[0][k], tf), ay = __fmul_rn(c_ao_dir[1][k], tf);
            o = (int)floorf(ax) - (int)floorf(ay) * W;
            if (t < kAoTaps) ao_inv_dist(P, ax, ay, &rlo, &rhi);
        }
        S.off[k][q] = 4 * o;
        S.rlo[k][q] = rlo;
        S.rhi[k][q] = rhi;
    }
    // the line window of each group after the nearest: the four cells that end at the cell of its last tap t1
    for (int e = threadIdx.x; e < 8 * kAoWin; e += blockDim.x) {
        // the neutral last entry reads the window before it, with bounds 0
        const int k = e / kAoWin, w = e - k * kAoWin, g = min(w + kNearGroups, kAoGroups - 1);
        int o = 0;
        float lo = 0.0f, hi = 0.0f;
        if (k < P.n_dirs) {
            const float cx = c_ao_dir[0][k], cy = c_ao_dir[1][k];
            const int t1 = min(4 * g + 5, kAoTaps - 1);
            auto cell_x = [&](int t) { return (int)floorf(__fmul_rn(cx, small_u2f((uint32_t)t))); };
            auto cell_y = [&](int t) { return (int)floorf(__fmul_rn(cy, small_u2f((uint32_t)t))); };
            auto reach = [&](int t) { return max(abs(cell_x(t1) - cell_x(t)), abs(cell_y(t1) - cell_y(t))); };
            int t0 = t1;  // the window's nearest tap
            while (t0 > 2 && reach(t0 - 1) <= kLineReach) t0--;
            const int near = cell_x(t0) - cell_y(t0) * W, far = cell_x(t1) - cell_y(t1) * W;
            o = min(near, far);
            float a, b;
            ao_inv_dist(P, __fmul_rn(cx, small_u2f((uint32_t)t0)), __fmul_rn(cy, small_u2f((uint32_t)t0)), &a, &hi);
            ao_inv_dist(P, __fmul_rn(cx, small_u2f((uint32_t)t1)), __fmul_rn(cy, small_u2f((uint32_t)t1)), &lo, &b);
            if (w + kNearGroups >= kAoGroups) lo = hi = 0.0f;
        }
        S.woff[k][w] = 4 * o;
        S.wlo[k][w] = lo;
        S.whi[k][w] = hi;
    }
}

PR_DEV void ao_finish(const AoParams& P, uint32_t i, float T);

// A pixel's march along direction k: the first tap outside the frame and the
// first with cur < 0 (kAoTaps: none), by binary search.
PR_DEV void ao_reach(const AoParams& P, float pxf, float pyf, float dX, float dY, int* t_end, int* t_fast) {
    const float fW = (float)P.W, fH = (float)P.H;
    const float cx = __fadd_rn(pxf, __fmul_rn(dX, 99.0f)), cy = __fadd_rn(pyf, __fmul_rn(dY, 99.0f));
    *t_end = *t_fast = kAoTaps;
    if (cx >= 0.0f && cx < fW && cy >= 0.0f && cy < fH) return;
    int lo = 1, hi = kAoTaps;  // first tap outside (-1, W) x (-1, H), then first tap with cur < 0
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const float tf = small_u2f((uint32_t)mid);
        const float mx = __fadd_rn(pxf, __fmul_rn(dX, tf)), my = __fadd_rn(pyf, __fmul_rn(dY, tf));
        if (mx > -1.0f && mx < fW && my > -1.0f && my < fH)
            lo = mid + 1;
        else
            hi = mid;
    }
    *t_end = lo;
    hi = lo;
    lo = 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const float tf = small_u2f((uint32_t)mid);
        const float mx = __fadd_rn(pxf, __fmul_rn(dX, tf)), my = __fadd_rn(pyf, __fmul_rn(dY, tf));
        if (mx >= 0.0f && my >= 0.0f)
            lo = mid + 1;
        else
            hi = mid;
    }
    *t_fast = lo;
}

// The tap t* of a tiny component c at coordinate p: the first with |c t| above half the gap below p.
PR_DEV int ao_tiny_cross(float c, float p) {
    const float cf = fabsf(c);
    const uint32_t vb = __float_as_uint(p);
    const float h = __uint_as_float(((vb >> 23) - ((vb & 0x7fffffu) ? 24u : 25u)) << 23);
    if (!(__fmul_rn(cf, 99.0f) > h)) return kAoTaps;
    int lo = 1, hi = kAoTaps - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__fmul_rn(cf, small_u2f((uint32_t)mid)) > h)
            hi = mid;
        else
            lo = mid + 1;
    }
    return lo;
}

// Pixel i's total T in a frame with NaN depths (NaN: a direction met one), or
// without line maxima (no memory for them): every tap by itself.
__device__ __noinline__ float ao_total_taps(const AoParams& P, uint32_t i, const AoTables& S) {
    const int W = P.W, H = P.H, r = (int)(i / (uint32_t)W), x = (int)i - r * W, y = H - 1 - r;
    const float* p0 = P.depth + i;
    const float z = *p0;
    const float pxf = small_u2f((uint32_t)x), pyf = small_u2f((uint32_t)y);
    float total = 0.0f;
    for (int k = 0; k < P.n_dirs; k++) {
        const float dX = c_ao_dir[0][k], dY = c_ao_dir[1][k];
        int t_end, t_fast;
        ao_reach(P, pxf, pyf, dX, dY, &t_end, &t_fast);
        // the tables' bounds (0 for the padding taps 100, 101) need finite elevations of a finite depth
        if (!P.dir_fast[k] || !isfinite(z)) t_fast = 1;
        float best = 0.0f;
        bool ok = true;
        if (t_end > 1) ok = ao_tap_exact(1, pxf, pyf, dX, dY, W, H, P.depth, z, 0.0f, best);
        int t = 2;
        if (ok && t_fast > 2) {
            const int n_groups = t_fast == kAoTaps ? kAoGroups : (t_fast - 2) >> 2;
            const int tiny = P.dir_tiny[k];
            if (tiny)
                ok = ao_fast_groups<true>(n_groups, S.off, S.rlo, S.rhi, k, p0, p0 + (tiny == 1 ? 1 : -W),
                                          ao_tiny_cross(tiny == 1 ? dX : dY, tiny == 1 ? pxf : pyf), z, pxf, pyf, dX, dY, best);
            else
                ok = ao_fast_groups<false>(n_groups, S.off, S.rlo, S.rhi, k, p0, p0, 0, z, pxf, pyf, dX, dY, best);
            t = 2 + 4 * n_groups;
        }
        for (; ok && t < t_end; t++) ok = ao_tap_exact(t, pxf, pyf, dX, dY, W, H, P.depth, z, best, best);
        if (!ok) return __uint_as_float(0x7fc00000u);
        total = __fadd_rn(total, ao_term(best));
    }
    return __fdiv_rn(total, 12.5663706143591729539f);
}

// Pixel j of the AO list's n (every lane of a warp calls, those past the end
// with the last pixel and nothing to write): its total T, then (kApply) the
// colour scaling, or (!kApply) T stored for ao_apply_kernel.
// kLines: the frame has line maxima.
template <bool kApply, bool kLines>
PR_DEV void ao_one(const AoParams& P, uint32_t j, uint32_t n, const AoTables& S) {
    const bool mine = j < n;
    const uint32_t i = P.list[min(j, n - 1u)];
    float T;
    if (!kLines || P.cnt->nan_flag != 0u) {  // some NaN-depth fragment reached this frame (the raster flags every one)
        T = ao_total_taps(P, i, S);
    } else {
        const int W = P.W, H = P.H, r = (int)(i / (uint32_t)W), x = (int)i - r * W, y = H - 1 - r;
        const float z = P.depth[i];
        const float pxf = small_u2f((uint32_t)x), pyf = small_u2f((uint32_t)y);
        const bool inner = x >= 100 && x < W - 100 && y >= 100 && y < H - 100 && isfinite(z);  // every tap inside the frame
        const bool all_inner = __all_sync(0xffffffffu, inner);
        float total = 0.0f, shut = 0.0f;  // shut: the sum of the angles
        for (int k = 0; k < P.n_dirs; k++) {
            const float dX = c_ao_dir[0][k], dY = c_ao_dir[1][k];
            int t_end = kAoTaps, t_fast = kAoTaps;
            if (!all_inner) ao_reach(P, pxf, pyf, dX, dY, &t_end, &t_fast);
            if (!P.dir_fast[k] || !isfinite(z)) t_fast = 1;
            const int n_groups = t_fast == kAoTaps ? kAoGroups : max(t_fast - 2, 0) >> 2;
            float best = 0.0f;
            bool ok = true;  // false: a NaN elevation (z infinite)
            if (all_inner && fminf(fabsf(dX), fabsf(dY)) < 0x1p-16f)  // along an axis the first tap's dist is 1 (ao_inv_dist)
                best = fmaxf(0.0f, __fsub_rn(P.depth[i + (fabsf(dX) > 0.5f ? (dX > 0.0f ? 1 : -1) : (dY > 0.0f ? -W : W))], z));
            else if (t_end > 1)
                ok = ao_tap_exact(1, pxf, pyf, dX, dY, W, H, P.depth, z, 0.0f, best);
            // the taps past the last whole group, exactly
            for (int t = n_groups == kAoGroups ? kAoTaps : 2 + 4 * n_groups; ok && t < t_end; t++)
                ok = ao_tap_exact(t, pxf, pyf, dX, dY, W, H, P.depth, z, best, best);
            const int tiny = P.dir_tiny[k];
            int tstar = 0;
            const uint32_t pix = 4u * i;
            uint32_t b0 = pix, bA = pix;
            if (tiny) {
                tstar = ao_tiny_cross(tiny == 1 ? dX : dY, tiny == 1 ? pxf : pyf);
                bA = pix + (uint32_t)(tiny == 1 ? 4 : -4 * W);
                if (tstar >= kAoTaps) b0 = bA;  // the whole march stays in the pixel's column (or row)
                if (tstar <= 2 || tstar >= kAoTaps) tstar = 0;
            }
            // the line the direction runs along: x, rows, diagonal (x and row grow together), antidiagonal
            const int line = fabsf(dY) < 0.5f ? 0 : (fabsf(dX) < 0.5f ? 1 : ((dX > 0.0f) != (dY > 0.0f) ? 2 : 3));
            const float* lm = P.linemax + (size_t)line * ((size_t)W * H);
            const float term =
                __all_sync(0xffffffffu, n_groups == kAoGroups && tstar == 0)
                    ? ao_march<false>(kAoGroups, S, k, P.depth, pix, b0, b0, 0, z, lm, pxf, pyf, dX, dY, best)
                    : ao_march<true>(n_groups, S, k, P.depth, pix, b0, bA, tstar, z, lm, pxf, pyf, dX, dY, best);
            total = ok ? __fadd_rn(total, term) : __uint_as_float(0x7fc00000u);
            // Each term left is at most HalfPi: with the angles so far above 7.6e-3, T <= 1 - 6e-4 whatever they are
            // (the float32 sum and quotient err by less than 1e-5 of the 5.9e-5 to spare), and ao_scale gives 0,
            // as it does for NaN.
            shut = __fadd_rn(shut, __fsub_rn(1.57079632679489661923f, term));
            if (!P.exact_T && __all_sync(0xffffffffu, shut > 7.6e-3f || !ok)) break;
        }
        T = !P.exact_T && shut > 7.6e-3f ? 0.0f : __fdiv_rn(total, 12.5663706143591729539f);
    }
    if (!mine) return;
    if (kApply)
        ao_finish(P, i, T);
    else
        P.T[j] = T;
}

// material/ao.go:34-37 for pixel i with total T: the colour the shade kernel
// left (pre-AO, pre-gamma) times float32(Pow(T, 10000)), then gamma.
PR_DEV void ao_finish(const AoParams& P, uint32_t i, float T) {
    const uchar4 c = P.rgba[i];
    if (P.dgb) {
        // float32(Pow(T, 10000)) as a fixed factor of the differentiable radiance (0 for NaN, as the
        // reference's uint8(NaN) darkens the pixel)
        const float fa = isnan(T) ? 0.0f : (T == 1.0f ? 1.0f : powf(T, 10000.0f));
        P.dgb[4 * i].w *= fa;
    }
    uint3 o = ao_scale(T, c.x, c.y, c.z);
    if (P.gamma_on) {
        o.x = P.gamma[o.x];
        o.y = P.gamma[o.y];
        o.z = P.gamma[o.z];
    }
    P.rgba[i] = make_uchar4(o.x, o.y, o.z, c.w);
}

// 4 blocks per SM (64 registers). The tap tables come from the context
// (ao_tables_kernel): building them cost each block of 256 pixels 7% of its
// instructions. Bound by issue (71% active): 713k pixels at 1920x1080 take
// 206 us and 160 M warp instructions; every tap compared by itself, eight to
// a unit, took 286 us and 227 M.
template <bool kLines>
__global__ void __launch_bounds__(kAoThreads, 4) ao_kernel(const __grid_constant__ AoParams P) {
    __shared__ AoTables S;
    const uint32_t n = P.cnt->n_ao;
    if (blockIdx.x * blockDim.x >= n) return;  // whole block: no pixel of the list
    static_assert(sizeof(AoTables) % 16 == 0, "copied in 16-byte words");
    for (uint32_t e = threadIdx.x; e < sizeof(AoTables) / 16; e += blockDim.x)
        reinterpret_cast<uint4*>(&S)[e] = reinterpret_cast<const uint4*>(P.tables)[e];
    __syncthreads();
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x)
        ao_one<false, kLines>(P, base + threadIdx.x, n, S);
}
// The tap tables of a frame size, once per context and size.
__global__ void __launch_bounds__(kAoThreads) ao_tables_kernel(const __grid_constant__ AoParams P, void* out) {
    __shared__ AoTables S;
    ao_tables(P, S);
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < sizeof(AoTables) / 16; e += blockDim.x)
        reinterpret_cast<uint4*>(out)[e] = reinterpret_cast<const uint4*>(&S)[e];
}

// The colour scaling of every listed pixel from its stored total.
__global__ void ao_apply_kernel(const __grid_constant__ AoParams P) {
    after_previous();
    release_next();
    const uint32_t n = P.cnt->n_ao;
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        ao_finish(P, P.list[j], P.T[j]);
}

// Triangle.IsValid (geometry/primitive/triangle.go:63-80) of every input
// triangle, once per scene upload: it depends on model-space positions only.
__global__ void tri_flags_kernel(const float4* pos, uint32_t n, uint8_t* flags, const int32_t* mat,
                                 const uint32_t* obj_first, const uint32_t* blk_obj, const int32_t* obj_matbase,
                                 uint32_t n_objects, const pr_material* mats, uint32_t n_mats) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    uint8_t f = tri_is_valid(ld4(pos[3 * t]), ld4(pos[3 * t + 1]), ld4(pos[3 * t + 2])) ? kTriValid : 0;
    // the flat material of the triangle's fragments (MaterialID plus its geometry's base) has AO
    int m = mat[t];
    if (m >= 0) {
        uint32_t o = blk_obj[t >> 7];
        while (o + 1 < n_objects && obj_first[o + 1] <= t) o++;
        m += obj_matbase[o];
        if (m >= 0 && (uint32_t)m < n_mats && (mats[m].flags & PR_MAT_AO)) f |= kTriAO;
    }
    flags[t] = f;
}

// ---------------------------------------------------------------- batches

// The job owning launch block (or item) b: the largest j with start[j] <= b.
PR_DEV int job_of(const uint32_t* start, int n_jobs, uint32_t b) {
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (start[mid] <= b)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(128) setup_shadow_batch_kernel(const SetupParams* jobs, const uint32_t* blk, int n_jobs) {
    __shared__ ObjCache C;
    const int j = job_of(blk, n_jobs, blockIdx.x);
    const uint32_t t0 = (blockIdx.x - blk[j]) * blockDim.x;
    __shared__ ReserveSm S;
    obj_cache_fill(jobs[j], t0, C);
    setup_shadow_one(jobs[j], &C, t0 + threadIdx.x, S);
}
__global__ void __launch_bounds__(128) setup_main_batch_kernel(const SetupParams* jobs, const uint32_t* blk, int n_jobs) {
    __shared__ ObjCache C;
    const int j = job_of(blk, n_jobs, blockIdx.x);
    const uint32_t t0 = (blockIdx.x - blk[j]) * blockDim.x;
    __shared__ ReserveSm S;
    obj_cache_fill(jobs[j], t0, C);
    setup_main_one(jobs[j], &C, t0 + threadIdx.x, jobs[j].clip_list, S);
}
__global__ void __launch_bounds__(128) clip_batch_kernel(const SetupParams* jobs, const uint32_t* blk, int n_jobs) {
    const int j = job_of(blk, n_jobs, blockIdx.x);
    const SetupParams& P = jobs[j];
    const uint32_t n = P.cnt->n_clipped, b0 = blockIdx.x - blk[j], nb = blk[j + 1] - blk[j];
    constexpr uint32_t kPerBlock = 128 / kClipLanes;
    __shared__ ClipGroupSm s_g[kPerBlock];
    // the job's blocks stride over its list (uniform per block, as in clip_kernel)
    for (uint32_t b = b0 * kPerBlock; b < n; b += nb * kPerBlock) {
        clip_one_group(P, P.clip_list, b + threadIdx.x / kClipLanes, n, threadIdx.x % kClipLanes,
                       s_g[threadIdx.x / kClipLanes]);
        __syncwarp();
    }
}

// items[j] = work items (block tasks, then warp batches of 32 tasks) before pass j (one block; a chained scan in
// chunks of its 1024 threads).
__global__ void __launch_bounds__(1024) batch_scan_kernel(const RasterParams* jobs, int n_jobs, uint32_t* items,
                                                          uint32_t* queue, int fixup) {
    __shared__ uint32_t s[1024];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) {
        carry = 0;
        *queue = 0;
    }
    __syncthreads();
    for (int base = 0; base < n_jobs; base += blockDim.x) {
        const int j = base + threadIdx.x;
        uint32_t v = 0;
        if (j < n_jobs) {
            const Counters* c = jobs[j].cnt;
            const bool run = !c->overflow && (!fixup || c->nan_flag);
            v = run ? ((c->n_tasks + 31u) >> 5) + c->n_big : 0u;
        }
        s[threadIdx.x] = v;
        __syncthreads();
        for (int d = 1; d < (int)blockDim.x; d <<= 1) {
            const uint32_t t = threadIdx.x >= (unsigned)d ? s[threadIdx.x - d] : 0u;
            __syncthreads();
            s[threadIdx.x] += t;
            __syncthreads();
        }
        if (j < n_jobs) items[j] = carry + s[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry += s[threadIdx.x];
        __syncthreads();
    }
    if (threadIdx.x == 0) items[n_jobs] = carry;
}

// Persistent raster over every pass of a batch: each warp takes the next
// (pass, warp batch) item from the global queue.
__global__ void __launch_bounds__(kRasterWarps * 32, 6) raster_batch_kernel(const RasterParams* jobs, const uint32_t* items,
                                                                         int n_jobs, uint32_t* queue) {
    __shared__ RasterWarpSm s_w[kRasterWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t total = items[n_jobs];
    for (;;) {
        uint32_t it = 0;
        if (lane == 0) it = atomicAdd(queue, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= total) break;
        const int j = job_of(items, n_jobs, it);
        const RasterParams& P = jobs[j];
        const uint32_t k = it - items[j], n_big = P.cnt->n_big;
        if (k < n_big)
            raster_block(P, P.big[k], 0u, 1u, s_w[warp], true);
        else
            raster_warp(P, P.tasks, (k - n_big) * 32u, P.cnt->n_tasks, s_w[warp], true);
    }
}

__global__ void resolve_batch_kernel(const ResolveParams* jobs, const uint32_t* blk, int n_jobs) {
    const int j = job_of(blk, n_jobs, blockIdx.x);
    const ResolveParams& R = jobs[j];
    const size_t i = (size_t)(blockIdx.x - blk[j]) * blockDim.x + threadIdx.x;
    uint32_t ridx;
    if (i < (size_t)R.W * R.H)
        resolve_one(R.keys, R.nanseq, R.beaten, R.cnt, R.first_rec, R.win, R.depth_ao, i, &ridx);
}

// 256-thread blocks as 32 x 8 pixel tiles, row-major over each view's tiles.
template <bool kFast>
__global__ void __launch_bounds__(256) shade_batch_kernel(const ShadeParams* views, const uint32_t* blk, int n_views) {
    const int v = job_of(blk, n_views, blockIdx.x);
    const ShadeParams& P = views[v];
    const uint32_t b = blockIdx.x - blk[v], tiles_x = (uint32_t)(P.W + 31) / 32u;
    const uint32_t ty = b / tiles_x, tx = b - ty * tiles_x;
    const int x = (int)(tx * 32u + tile_x(threadIdx.x)), r = (int)(ty * 8u + tile_y(threadIdx.x));
    const bool pending = shade_one<false, kFast>(P, x, r);  // batches carry no image textures
    if (P.ao_list) ao_append_tile(P, pending, (uint32_t)r * (uint32_t)P.W + (uint32_t)x);
}

// The line maxima of every view with AO pixels, on shade_batch_kernel's tiles.
__global__ void __launch_bounds__(256) ao_linemax_batch_kernel(const AoParams* views, const uint32_t* blk, int n_views) {
    const int v = job_of(blk, n_views, blockIdx.x);
    const AoParams& P = views[v];
    if (P.cnt->nan_flag || P.cnt->n_ao == 0) return;
    const uint32_t b = blockIdx.x - blk[v], tiles_x = (uint32_t)(P.W + 31) / 32u;
    const uint32_t ty = b / tiles_x;
    ao_linemax_tile(P.W, P.H, (int)((b - ty * tiles_x) * 32u), (int)(ty * 8u), P.linemax,
                    [&](int x, int r) { return P.depth[(size_t)r * P.W + x]; });
}

// Persistent AO over every view's list, in chunks of one block taken from
// per-view counters; tap tables rebuilt when the frame size changes.
// kLines: the batch has line maxima.
template <bool kLines>
__global__ void __launch_bounds__(kAoThreads) ao_batch_kernel(const AoParams* views, int n_views,
                                                                uint32_t* chunk_ctr) {
    __shared__ AoTables S;
    __shared__ uint32_t s_chunk;
    int tab_w = -1, tab_dirs = -1;
    float tab_h = -1.0f;
    for (int v = 0; v < n_views; v++) {
        const AoParams& P = views[v];
        const uint32_t n = P.cnt->n_ao;
        if (n == 0) continue;
        if (P.W != tab_w || P.ao_half_ulp != tab_h || P.n_dirs != tab_dirs) {
            __syncthreads();
            ao_tables(P, S);
            __syncthreads();
            tab_w = P.W;
            tab_h = P.ao_half_ulp;
            tab_dirs = P.n_dirs;
        }
        for (;;) {
            if (threadIdx.x == 0) s_chunk = atomicAdd(&chunk_ctr[v], 1u);
            __syncthreads();
            const uint32_t c = s_chunk;
            __syncthreads();
            if (c * blockDim.x >= n) break;
            ao_one<true, kLines>(P, c * blockDim.x + threadIdx.x, n, S);
        }
    }
}

__global__ void pow_probe_kernel(const float* x, const float* y, float* fast, float* ref, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    fast[i] = go_pow_f32(x[i], y[i]);
    ref[i] = __double2float_rn(go_pow((double)x[i], (double)y[i]));
}

__global__ void ao_probe_kernel(const float* x, float* atan_fast, float* atan_ref, const float* T, const uchar4* col,
                                uchar4* o_fast, uchar4* o_ref, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    atan_fast[i] = atan_f32(x[i]);
    atan_ref[i] = __double2float_rn(go_atan((double)x[i]));
    const uchar4 c = col[i];
    const uint3 a = ao_scale(T[i], c.x, c.y, c.z);
    o_fast[i] = make_uchar4(a.x, a.y, a.z, c.w);
    const float P = __double2float_rn(go_pow((double)T[i], 10000.0));
    o_ref[i] = make_uchar4(go_f2u8(__fmul_rn(P, small_u2f(c.x))), go_f2u8(__fmul_rn(P, small_u2f(c.y))),
                           go_f2u8(__fmul_rn(P, small_u2f(c.z))), c.w);
}

__global__ void fma_probe_kernel(const float* a, const float* b, const float* c, float* out, float* out_ref, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = fma64f(a[i], b[i], c[i]);
    out_ref[i] = fma64f_slow(a[i], b[i], c[i]);
}

int check(cudaError_t e) { return e == cudaSuccess ? 0 : (int)e; }

// k on the stream; with `overlap` as a programmatic launch behind the kernel
// before it there (k begins with after_previous).
template <class... K, class... A>
int launch(bool overlap, void (*k)(K...), dim3 grid, dim3 block, void* stream, const A&... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.stream = (cudaStream_t)stream;
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = overlap ? 1 : 0;
    return check(cudaLaunchKernelEx(&c, k, K(args)...));
}

}  // namespace

int launch_setup_main_only(const SetupParams& p, uint32_t* clip_list, void* stream) {
    // a clearing block per 2048 keys
    const unsigned nb = (p.n_tris + 127) / 128 + (unsigned)((p.n_clear + 2047) / 2048);
    if (nb == 0) return 0;
    return launch(true, setup_main_kernel, nb, 128, stream, p, clip_list);
}
int launch_resolve(int W, int H, const unsigned long long* keys, uint32_t* nanseq, uint32_t* beaten, Counters* cnt,
                   uint32_t* win, float* depth_ao, const uint32_t* first_rec, uint8_t* attr_state,
                   const uint8_t* tri_flags, uint32_t* ao_list, float* linemax, void* stream) {
    if (W <= 0 || H <= 0) return 0;
    const dim3 grd((unsigned)((W + 31) / 32), (unsigned)((H + 7) / 8));
    return launch(true, resolve_kernel, grd, 256, stream, W, H, keys, nanseq, beaten, cnt, win, depth_ao, first_rec,
                  attr_state, tri_flags, ao_list, linemax);
}
int launch_attr(const SetupParams& p, bool overlap, void* stream) {
    return launch(overlap, attr_kernel, (unsigned)sm_count() * 8u, 128, stream, p);
}
int launch_pass_init(const PassMats& pm, int n_pass, const float* obj_model, uint32_t n_objects, float* out,
                     Counters* cnt, uint32_t rows, void* stream) {
    static_assert(kNumCounters <= 32, "a bit per counter row");
    const size_t n = (size_t)n_pass * n_objects * 16;
    return launch(false, pass_init_kernel, (unsigned)std::max<size_t>((n + 255) / 256, 1), 256, stream, pm, n_pass,
                  obj_model, n_objects, out, cnt, rows);
}
int launch_clip(const SetupParams& p, const uint32_t* clip_list, void* stream) {
    // the list's length is known only on the device: a few blocks per SM stride over it
    const unsigned nb = std::min((p.n_tris + 15) / 16, (unsigned)sm_count() * 4u);
    return launch(true, clip_kernel, std::max(nb, 1u), 128, stream, p, clip_list);
}
int launch_setup_shadow(const SetupParams& p, void* stream) {
    if (p.n_tris == 0) return 0;
    return launch(true, setup_shadow_kernel, (p.n_tris + 127) / 128, 128, stream, p);
}
int launch_raster(const RasterParams& p, int n_blocks, void* stream) {
    return launch(true, raster_kernel, (unsigned)n_blocks, kRasterWarps * 32, stream, p);
}
int launch_shadow_fixup_reset(int W, int H, const uint32_t* lastnan, uint32_t* smap, const Counters* cnt,
                              void* stream) {
    size_t n = (size_t)W * H;
    const unsigned nb = (unsigned)std::min<size_t>((n + 255) / 256, (size_t)sm_count() * 8);
    return launch(true, shadow_fixup_reset_kernel, std::max(nb, 1u), 256, stream, n, lastnan, smap, cnt);
}
int launch_nan_cleanup(size_t n, uint32_t* a, uint32_t va, uint32_t* b, uint32_t vb, const Counters* cnt,
                       void* stream) {
    const unsigned nb = (unsigned)std::min<size_t>((n + 255) / 256, (size_t)sm_count() * 8);
    return launch(true, nan_cleanup_kernel, std::max(nb, 1u), 256, stream, n, a, va, b, vb, cnt);
}
// No output asks for the fragment's own attributes.
bool shade_is_fast(const ShadeParams& p) { return !p.gnor && !p.gfnor && !p.gwpos && !p.guvd && !p.gvcol && !p.dgb; }
int launch_shade(const ShadeParams& p, bool overlap, void* stream) {
    const dim3 grd((p.W + 31) / 32, (p.H + 7) / 8);
    const bool fast = shade_is_fast(p);
    return launch(overlap,
                  p.mat_tex ? (fast ? shade_kernel<true, true> : shade_kernel<true, false>)
                            : (fast ? shade_kernel<false, true> : shade_kernel<false, false>),
                  grd, 256, stream, p);
}
int launch_tri_flags(const float4* pos, uint32_t n, uint8_t* flags, const int32_t* mat, const uint32_t* obj_first,
                     const uint32_t* blk_obj, const int32_t* obj_matbase, uint32_t n_objects, const pr_material* mats,
                     uint32_t n_mats, void* stream) {
    if (n == 0) return 0;
    tri_flags_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(pos, n, flags, mat, obj_first, blk_obj,
                                                                          obj_matbase, n_objects, mats, n_mats);
    return check(cudaGetLastError());
}
int launch_setup_shadow_batch(const SetupParams* jobs, const uint32_t* blk, int n_jobs, uint32_t n_blocks, void* stream) {
    if (n_blocks == 0) return 0;
    setup_shadow_batch_kernel<<<n_blocks, 128, 0, (cudaStream_t)stream>>>(jobs, blk, n_jobs);
    return check(cudaGetLastError());
}
int launch_setup_main_batch(const SetupParams* jobs, const uint32_t* blk, int n_jobs, uint32_t n_blocks, void* stream) {
    if (n_blocks == 0) return 0;
    setup_main_batch_kernel<<<n_blocks, 128, 0, (cudaStream_t)stream>>>(jobs, blk, n_jobs);
    return check(cudaGetLastError());
}
int launch_clip_batch(const SetupParams* jobs, const uint32_t* blk, int n_jobs, uint32_t n_blocks, void* stream) {
    if (n_blocks == 0) return 0;
    clip_batch_kernel<<<n_blocks, 128, 0, (cudaStream_t)stream>>>(jobs, blk, n_jobs);
    return check(cudaGetLastError());
}
int launch_batch_scan(const RasterParams* jobs, int n_jobs, uint32_t* items, uint32_t* queue, int fixup, void* stream) {
    batch_scan_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(jobs, n_jobs, items, queue, fixup);
    return check(cudaGetLastError());
}
int launch_raster_batch(const RasterParams* jobs, const uint32_t* items, int n_jobs, uint32_t* queue, int n_blocks,
                        void* stream) {
    raster_batch_kernel<<<n_blocks, kRasterWarps * 32, 0, (cudaStream_t)stream>>>(jobs, items, n_jobs, queue);
    return check(cudaGetLastError());
}
int launch_resolve_batch(const ResolveParams* jobs, const uint32_t* blk, int n_jobs, uint32_t n_blocks, void* stream) {
    if (n_blocks == 0) return 0;
    resolve_batch_kernel<<<n_blocks, 256, 0, (cudaStream_t)stream>>>(jobs, blk, n_jobs);
    return check(cudaGetLastError());
}
int launch_shade_batch(const ShadeParams* views, const uint32_t* blk, int n_views, uint32_t n_blocks, bool fast, void* stream) {
    if (n_blocks == 0) return 0;
    if (fast)
        shade_batch_kernel<true><<<n_blocks, 256, 0, (cudaStream_t)stream>>>(views, blk, n_views);
    else
        shade_batch_kernel<false><<<n_blocks, 256, 0, (cudaStream_t)stream>>>(views, blk, n_views);
    return check(cudaGetLastError());
}
int launch_ao_batch(const AoParams* views, int n_views, uint32_t* chunk_ctr, int n_blocks, bool lines, void* stream) {
    return launch(false, lines ? ao_batch_kernel<true> : ao_batch_kernel<false>, (unsigned)n_blocks, kAoThreads, stream, views,
                  n_views, chunk_ctr);
}
// ---------------------------------------------------------------- MSAA resize

constexpr int kMaxMsaa = 16;

// createWeights8 (internal/imageutil/resize.go:161-181) for output index y:
// the linear kernel's taps as int16 (x256, truncated) and the first input
// index, in the reference's float32 order. len <= 2 * kMaxMsaa.
PR_DEV int resize_taps(int y, float scale, float factor, int len, int16_t* coeff) {
    float interp = __fsub_rn(__fmul_rn(scale, __fadd_rn((float)y, 0.5f)), 0.5f);
    const int start = (int)interp - len / 2 + 1;  // int(interpX) truncates
    interp = __fsub_rn(interp, (float)start);
    for (int i = 0; i < len; i++) {
        const float in = fabsf(__fmul_rn(__fsub_rn(interp, (float)i), factor));
        const float k = in <= 1.0f ? __fsub_rn(1.0f, in) : 0.0f;  // linear()
        coeff[i] = (int16_t)(int)__fmul_rn(k, 256.0f);
    }
    return start;
}

// resizeRGBA's edge rule (resize.go:98-105): inside [0, max) as is, at or
// past max -> max, negative -> 0.
PR_DEV int resize_clamp(int i, int max) { return (unsigned)i < (unsigned)max ? i : (i >= max ? max : 0); }

// floor(acc / sum), 0 for sum == 0: taps are >= 0, so the quotient of a
// weighted sum of bytes by the weights' sum is a byte. rcp: 1 / sum; with
// acc < 2^21 the rounded product is off by less than one, which the remainder corrects.
PR_DEV uint32_t resize_div(uint32_t acc, uint32_t sum, float rcp) {
    if (sum == 0u) return 0u;
    const int q = (int)((float)acc * rcp), r = (int)acc - q * (int)sum;
    return (uint32_t)(q + (r >= (int)sum ? 1 : 0) - (r < 0 ? 1 : 0));
}

// imageutil.Resize's two passes for a block of 32 x 8 output pixels: the taps
// of its columns and rows once, the horizontal pass (into the reference's
// uint8 temporary) for every input row its vertical taps reach, then the
// vertical pass over those values. Rows that several outputs share are done
// once; a thread per output with both passes and its own taps took 82 us for
// 3840x2160 -> 1920x1080, this 44 us (6 us of memory traffic; bound by issue).
constexpr int kResizeW = 32, kResizeH = 8;
constexpr int kResizeRows = (kResizeH - 1) * kMaxMsaa + 2 * kMaxMsaa + 2;  // starts step by at most scale + 1 rounding
__global__ void __launch_bounds__(kResizeW* kResizeH) msaa_resize_kernel(const uchar4* in, int in_w, int in_h, uchar4* out,
                                                                        int w, int h) {
    __shared__ int16_t s_cx[kResizeW][2 * kMaxMsaa + 2], s_cy[kResizeH][2 * kMaxMsaa];
    __shared__ int s_x0[kResizeW], s_y0[kResizeH];
    __shared__ uchar4 s_t[kResizeRows][kResizeW];
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kResizeW + tx;
    const int bx = blockIdx.x * kResizeW, by = blockIdx.y * kResizeH;
    // calcFactors, then createWeights8's filterLength and filterFactor
    const float sx = __fdiv_rn((float)in_w, (float)w), sy = __fdiv_rn((float)in_h, (float)h);
    const int lx = min(2 * max((int)ceilf(sx), 1), 2 * kMaxMsaa), ly = min(2 * max((int)ceilf(sy), 1), 2 * kMaxMsaa);
    const float fx = fminf(__fdiv_rn(1.0f, sx), 1.0f), fy = fminf(__fdiv_rn(1.0f, sy), 1.0f);
    if (tid < kResizeW)
        s_x0[tid] = resize_taps(min(bx + tid, w - 1), sx, fx, lx, s_cx[tid]);
    else if (tid < kResizeW + kResizeH)
        s_y0[tid - kResizeW] = resize_taps(min(by + tid - kResizeW, h - 1), sy, fy, ly, s_cy[tid - kResizeW]);
    after_previous();
    __syncthreads();
    const int16_t *cx = s_cx[tx], *cy = s_cy[ty];
    const int x0 = s_x0[tx], first = s_y0[0], rows = min(s_y0[kResizeH - 1] + ly - first, kResizeRows);
    uint32_t sum = 0;
    for (int i = 0; i < lx; i++) sum += (uint32_t)cx[i];
    float rcp = __frcp_rn((float)sum);
    for (int r = ty; r < rows; r += kResizeH) {
        const uchar4* row = in + (size_t)resize_clamp(first + r, in_h - 1) * in_w;
        uint32_t t[4] = {0, 0, 0, 0};
        for (int i = 0; i < lx; i++) {
            const uint32_t c = (uint32_t)cx[i];
            const uchar4 p = row[resize_clamp(x0 + i, in_w - 1)];
            t[0] += c * p.x;
            t[1] += c * p.y;
            t[2] += c * p.z;
            t[3] += c * p.w;
        }
        s_t[r][tx] = make_uchar4(resize_div(t[0], sum, rcp), resize_div(t[1], sum, rcp), resize_div(t[2], sum, rcp),
                                 resize_div(t[3], sum, rcp));
    }
    __syncthreads();
    const int x = bx + tx, y = by + ty;
    if (x >= w || y >= h) return;
    uint32_t acc[4] = {0, 0, 0, 0};
    sum = 0;
    for (int j = 0; j < ly; j++) {
        const uint32_t c = (uint32_t)cy[j];
        const uchar4 p = s_t[s_y0[ty] - first + j][tx];
        acc[0] += c * p.x;
        acc[1] += c * p.y;
        acc[2] += c * p.z;
        acc[3] += c * p.w;
        sum += c;
    }
    rcp = __frcp_rn((float)sum);
    out[(size_t)y * w + x] = make_uchar4(resize_div(acc[0], sum, rcp), resize_div(acc[1], sum, rcp),
                                         resize_div(acc[2], sum, rcp), resize_div(acc[3], sum, rcp));
}

int launch_msaa_resize(const uchar4* in, int in_w, int in_h, uchar4* out, int w, int h, void* stream) {
    if (w <= 0 || h <= 0 || in_w < w || in_h < h || in_w > w * kMaxMsaa || in_h > h * kMaxMsaa) return -1;
    const dim3 block(kResizeW, kResizeH), grid((unsigned)((w + kResizeW - 1) / kResizeW), (unsigned)((h + kResizeH - 1) / kResizeH));
    return launch(true, msaa_resize_kernel, grid, block, stream, in, in_w, in_h, out, w, h);
}

size_t ao_tables_bytes() { return sizeof(AoTables); }
int launch_ao_tables(const AoParams& p, void* out, void* stream) {
    ao_tables_kernel<<<1, kAoThreads, 0, (cudaStream_t)stream>>>(p, out);
    return check(cudaGetLastError());
}
int launch_ao_linemax_batch(const AoParams* views, const uint32_t* blk, int n_views, uint32_t n_blocks, void* stream) {
    if (n_blocks == 0) return 0;
    ao_linemax_batch_kernel<<<n_blocks, 256, 0, (cudaStream_t)stream>>>(views, blk, n_views);
    return check(cudaGetLastError());
}
int launch_ao_T(const AoParams& p, void* stream) {
    // One pixel per thread for the largest possible list (every pixel): the
    // block scheduler balances the uneven per-pixel work; blocks past the
    // list's length exit at once.
    const size_t n = (size_t)p.W * p.H;
    if (n == 0) return 0;
    const unsigned nb = (unsigned)((n + kAoThreads - 1) / kAoThreads);
    return launch(false, p.linemax ? ao_kernel<true> : ao_kernel<false>, nb, kAoThreads, stream, p);
}
int launch_ao_apply(const AoParams& p, int n_blocks, void* stream) {
    return launch(false, ao_apply_kernel, (unsigned)n_blocks, 256, stream, p);
}
int set_ao_tables(const float* cosv, const float* sinv, int n, void* stream) {
    float d[2][8] = {};
    for (int k = 0; k < n && k < 8; k++) {
        d[0][k] = cosv[k];
        d[1][k] = sinv[k];
    }
    cudaError_t e = cudaMemcpyToSymbolAsync(c_ao_dir, d, sizeof(d), 0, cudaMemcpyHostToDevice, (cudaStream_t)stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
    return check(e);
}
int launch_decode_shadow(const uint32_t* smap, float* out, size_t n, void* stream) {
    if (n == 0) return 0;
    decode_shadow_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(smap, out, n);
    return check(cudaGetLastError());
}
int launch_pow_probe(const float* x, const float* y, float* fast, float* ref, int n, void* stream) {
    if (n <= 0) return 0;
    pow_probe_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(x, y, fast, ref, n);
    return check(cudaGetLastError());
}
int launch_ao_probe(const float* x, float* atan_fast, float* atan_ref, const float* T, const void* col, void* o_fast,
                    void* o_ref, int n, void* stream) {
    if (n <= 0) return 0;
    ao_probe_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(x, atan_fast, atan_ref, T, (const uchar4*)col,
                                                                        (uchar4*)o_fast, (uchar4*)o_ref, n);
    return check(cudaGetLastError());
}
int launch_fma_probe(const float* a, const float* b, const float* c, float* out, float* out_ref, int n, void* stream) {
    if (n <= 0) return 0;
    fma_probe_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(a, b, c, out, out_ref, n);
    return check(cudaGetLastError());
}
int sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

}  // namespace prk

namespace prk {

// ===========================================================================
// Allocation-free depth-map raster (pr_depth_map_noalloc).
//
// For callers that must not allocate device memory themselves: a host whose
// device memory is entirely owned by another allocator (a framework's fixed
// caching pool), or a frame loop that cannot afford cudaMalloc/cudaFree
// (cudaFree synchronises the whole device). It runs the shadow-map raster
// (setup_shadow_kernel + raster_kernel, the drawDepth pass) with every byte
// of scratch carved from the fixed array below, which each GPU that loads the
// library keeps until the process exits.
//
// Calls share the array: two calls whose work overlaps on the GPU (different
// streams, or different host threads) race on it and corrupt each other's
// results. Each call clears the parts that must start at zero.
// ===========================================================================

namespace {

constexpr uint32_t kNoAllocMaxTris = 65536;
constexpr uint32_t kNoAllocMaxObjects = 256;
constexpr uint32_t kNoAllocMaxTexels = 1u << 20;  // e.g. 1024 x 1024
constexpr uint32_t kNoAllocMaxTasks = 4u * kNoAllocMaxTris;
constexpr uint32_t kNoAllocTaskShift = 10;  // 1024-pixel tasks: the fixed task table covers large triangles
// The longest side that setup_shadow_kernel and raster_kernel take: corners are
// 16 bits, and rec_pixel's quotient of an index below bw + 2^10 is exact while
// (bw + 2^10) bw < 2^32. Longer maps go through the kernels below.
constexpr int kNoAllocMaxSide = 65000;

constexpr size_t kNaCounters = 0;                                   // Counters
constexpr size_t kNaObjFirst = 256;                                 // u32 [max_objects + 1]
constexpr size_t kNaObjModel = kNaObjFirst + 4096;                  // f32 [max_objects][16]
constexpr size_t kNaRecords = kNaObjModel + kNoAllocMaxObjects * 64; // RasterRec [max_tris]
constexpr size_t kNaTasks = kNaRecords + (size_t)kNoAllocMaxTris * sizeof(RasterRec);
constexpr size_t kNaKeys = kNaTasks + (size_t)kNoAllocMaxTasks * sizeof(uint2);
constexpr size_t kNaLastNan = kNaKeys + (size_t)kNoAllocMaxTexels * 4;
constexpr size_t kNaObjTrans = kNaLastNan + (size_t)kNoAllocMaxTexels * 4;  // f32 [kNaParamObjects][16]
constexpr uint32_t kNaParamObjects = 32;                                   // objects passed as kernel parameters
constexpr size_t kNaBlkObj = kNaObjTrans + kNaParamObjects * 64;           // u32 [max_tris / 128]
constexpr size_t kNaBytes = kNaBlkObj + kNoAllocMaxTris / 128 * 4;
static_assert(kNaBytes <= (16u << 20), "scratch layout exceeds 16 MiB");

static __device__ __align__(256) unsigned char g_noalloc_scratch[16u << 20];

// The objects of a call with few of them, and Proj·View, by value.
struct NaObjects {
    uint32_t n;  // 0: the tables come by copies
    uint32_t first[kNaParamObjects + 1];
    float model[kNaParamObjects][16];
    float pv[16];
};

// Everything a call needs before its setup, in one launch: the keys of the
// caller's map, the NaN bookkeeping and counters at rest, and (O.n) the object
// tables: first triangles, Proj·View·Model (as pass_init_kernel) and the object
// of each 128-triangle block.
__global__ void __launch_bounds__(256) noalloc_init_kernel(const float* depth, uint32_t* keys, uint32_t* lastnan, size_t n,
                                                           Counters* cnt, uint32_t* obj_first, float* obj_trans,
                                                           uint32_t* blk_obj, uint32_t n_tris,
                                                           const __grid_constant__ NaObjects O) {
    release_next();  // launched in full order itself
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float d = depth[i];
        keys[i] = isnan(d) ? 0u : fkey(d);  // key 0 stands for NaN (below every value)
        lastnan[i] = 0u;
    }
    if (blockIdx.x != 0) return;
    for (uint32_t e = threadIdx.x; e < sizeof(Counters) / 4; e += blockDim.x) reinterpret_cast<uint32_t*>(cnt)[e] = 0u;
    if (O.n == 0) return;
    for (uint32_t e = threadIdx.x; e <= O.n; e += blockDim.x) obj_first[e] = O.first[e];
    for (uint32_t e = threadIdx.x; e < O.n * 16u; e += blockDim.x) {
        const uint32_t r = (e >> 2) & 3u, c = e & 3u;
        const float* m = O.pv + r * 4;
        const float* q = O.model[e >> 4];
        obj_trans[e] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], q[c]), __fmul_rn(m[1], q[4 + c])), __fmul_rn(m[2], q[8 + c])),
                                 __fmul_rn(m[3], q[12 + c]));
    }
    for (uint32_t e = threadIdx.x; e * 128u < n_tris; e += blockDim.x) blk_obj[e] = find_object(O.first, O.n, e * 128u);
}

// Back into the caller's map: a texel whose key the raster changed takes the
// decoded key; the others keep their bits, so a -0 or a NaN payload that no
// fragment replaced stays as it was, as in the reference's map.
// After a task overflow the map stays as it was.
__global__ void decode_changed_kernel(const uint32_t* keys, float* depth, size_t n, const Counters* cnt) {
    after_previous();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || cnt->overflow) return;
    const float d = depth[i];
    const uint32_t k0 = isnan(d) ? 0u : fkey(d), k = keys[i];
    if (k != k0) depth[i] = fkey_decode(k);
}

// Maps with a side above kNoAllocMaxSide (so at most 16 texels across):
// records whose box is four whole words, and a warp per record. Every texel of
// a box takes the exact test; the tasks the other path would have made are
// counted, for the same limit.
__global__ void __launch_bounds__(128) long_map_setup_kernel(const __grid_constant__ SetupParams P) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= P.n_tris) return;
    SubVtx v[3];
    float sabc = 0.0f;
    ScrBox box = {};
    long long x0 = 1, x1 = 0, y0 = 0, y1 = -1;
    RasterRec& R = P.rrec[t];
    if (shadow_geom(P, nullptr, t, v, &sabc, &box) && pixel_range(v[0].pos, v[1].pos, v[2].pos, sabc, P.W, P.H, x0, x1, y0, y1)) {
        for (int k = 0; k < 3; k++) {
            R.v[3 * k] = v[k].pos.x;
            R.v[3 * k + 1] = v[k].pos.y;
            R.v[3 * k + 2] = v[k].pos.z;
        }
        R.sabc = sabc;
        atomicAdd(&P.cnt->n_tasks, n_tasks_of((uint32_t)((x1 - x0 + 1) * (y1 - y0 + 1)), P.task_shift));
    } else {
        x0 = 1, x1 = 0;
    }
    R.bx = (uint32_t)x0;
    R.by = (uint32_t)x1;
    R.recipw[0] = __uint_as_float((uint32_t)y0);
    R.recipw[1] = __uint_as_float((uint32_t)y1);
}
__global__ void __launch_bounds__(256) long_map_raster_kernel(const __grid_constant__ RasterParams P, uint32_t n) {
    if (P.cnt->n_tasks > kNoAllocMaxTasks) {
        atomicOr(&P.cnt_w->overflow, 2u);
        return;
    }
    if (P.mode == kShadowFixup && P.cnt_w->nan_flag == 0) return;
    const uint32_t lane = threadIdx.x & 31u, nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < n; t += nw) {
        const RasterRec& R = P.rrec[t];
        const int x0 = (int)R.bx, x1 = (int)R.by, y0 = __float_as_int(R.recipw[0]), y1 = __float_as_int(R.recipw[1]);
        if (x0 > x1) continue;
        SmRec r;
        r.ab = make_float4(R.v[0], R.v[1], R.v[3], R.v[4]);
        r.e0 = make_float4(__fsub_rn(R.v[3], R.v[0]), __fsub_rn(R.v[4], R.v[1]), __fsub_rn(R.v[6], R.v[0]), __fsub_rn(R.v[7], R.v[1]));
        r.e1 = make_float4(__fsub_rn(R.v[6], R.v[3]), __fsub_rn(R.v[7], R.v[4]), 0.0f, R.sabc);
        r.zs = make_float4(R.v[2], R.v[5], R.v[8], 0.0f);
        const uint32_t bw = (uint32_t)(x1 - x0 + 1), area = bw * (uint32_t)(y1 - y0 + 1);  // at most 2^20
        for (uint32_t k = lane; k < area; k += 32u) {
            const uint32_t row = k / bw;
            const int px = x0 + (int)(k - row * bw), py = y0 + (int)row;
            float z;
            if (pixel_depth(r, px, py, &z)) put_fragment(P, px, py, z, t);
        }
    }
}

std::mutex g_noalloc_mu;
void* g_noalloc_addr[64] = {};

}  // namespace

}  // namespace prk

extern "C" int pr_depth_map_noalloc(const pr_depth_map_desc* d) {
    using namespace prk;
    auto err = [](int code, const char* msg) { return set_last_error(code, msg); };
    if (!d) return err(PR_ERR_INVALID_ARG, "pr_depth_map_noalloc: desc is NULL");
    if (d->size < sizeof(pr_depth_map_desc)) return err(PR_ERR_INVALID_ARG, "pr_depth_map_noalloc: desc->size too small");
    if (d->n_tris > kNoAllocMaxTris)
        return err(PR_ERR_INVALID_ARG, "pr_depth_map_noalloc: n_tris exceeds PR_NOALLOC_MAX_TRIS (65536)");
    if (d->n_objects > kNoAllocMaxObjects)
        return err(PR_ERR_INVALID_ARG, "pr_depth_map_noalloc: n_objects exceeds PR_NOALLOC_MAX_OBJECTS (256)");
    if (d->width <= 0 || d->height <= 0 || (uint64_t)d->width * (uint64_t)d->height > kNoAllocMaxTexels)
        return err(PR_ERR_INVALID_ARG, "pr_depth_map_noalloc: width*height must be in 1..PR_NOALLOC_MAX_TEXELS (1048576)");
    if (!d->depth || (d->n_tris > 0 && (!d->pos || d->n_objects == 0)) || (d->n_objects > 0 && !d->objects))
        return err(PR_ERR_INVALID_ARG, "pr_depth_map_noalloc: NULL input or output pointer");
    uint64_t expect = 0;
    for (uint32_t o = 0; o < d->n_objects; o++) {
        if (d->objects[o].first_tri != expect)
            return err(PR_ERR_INVALID_ARG, "pr_depth_map_noalloc: objects must tile the triangles in order");
        expect += d->objects[o].n_tris;
        if (expect > d->n_tris)
            return err(PR_ERR_INVALID_ARG, "pr_depth_map_noalloc: objects do not cover n_tris");
    }
    if (expect != d->n_tris) return err(PR_ERR_INVALID_ARG, "pr_depth_map_noalloc: objects do not cover n_tris");

    // Once per device, with that device current: the device address of the
    // scratch array (its host-side name is not a device address).
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
        return err(PR_ERR_NO_DEVICE, "pr_depth_map_noalloc: no current CUDA device");
    unsigned char* base = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_addr[dev]) {
            void* p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess || !p) return err(PR_ERR_CUDA, "pr_depth_map_noalloc: cudaGetSymbolAddress failed");
            g_noalloc_addr[dev] = p;
        }
        base = (unsigned char*)g_noalloc_addr[dev];
    }
    cudaStream_t st = (cudaStream_t)d->stream;
    (void)cudaGetLastError();  // a failure of an earlier runtime call is not this call's
    Counters* cnt = (Counters*)(base + kNaCounters);
    uint32_t* obj_first = (uint32_t*)(base + kNaObjFirst);
    float* obj_model = (float*)(base + kNaObjModel);
    RasterRec* rrec = (RasterRec*)(base + kNaRecords);
    uint2* tasks = (uint2*)(base + kNaTasks);
    uint32_t* keys = (uint32_t*)(base + kNaKeys);
    uint32_t* lastnan = (uint32_t*)(base + kNaLastNan);
    const size_t n = (size_t)d->width * d->height;

    prh::M4 pv = prh::mulm(prh::M4{{d->proj[0], d->proj[1], d->proj[2], d->proj[3], d->proj[4], d->proj[5], d->proj[6],
                                     d->proj[7], d->proj[8], d->proj[9], d->proj[10], d->proj[11], d->proj[12],
                                     d->proj[13], d->proj[14], d->proj[15]}},
                           prh::M4{{d->view[0], d->view[1], d->view[2], d->view[3], d->view[4], d->view[5], d->view[6],
                                     d->view[7], d->view[8], d->view[9], d->view[10], d->view[11], d->view[12],
                                     d->view[13], d->view[14], d->view[15]}});
    // object tables: a few as kernel parameters, more by copies (host -> the scratch array)
    const bool by_param = d->n_objects > 0 && d->n_objects <= kNaParamObjects;
    NaObjects O;
    O.n = by_param ? d->n_objects : 0u;
    cudaError_t e = cudaSuccess;
    uint32_t first[kNoAllocMaxObjects + 1];
    float model[kNoAllocMaxObjects * 16];
    if (by_param) {
        for (uint32_t o = 0; o < d->n_objects; o++) {
            O.first[o] = d->objects[o].first_tri;
            std::memcpy(O.model[o], d->objects[o].model, 64);
        }
        O.first[d->n_objects] = d->n_tris;
        std::memcpy(O.pv, pv.m, 64);
    } else if (d->n_objects > 0) {
        for (uint32_t o = 0; o < d->n_objects; o++) {
            first[o] = d->objects[o].first_tri;
            std::memcpy(model + o * 16, d->objects[o].model, 64);
        }
        first[d->n_objects] = d->n_tris;
        e = cudaMemcpyAsync(obj_first, first, (d->n_objects + 1) * 4, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(obj_model, model, d->n_objects * 64, cudaMemcpyHostToDevice, st);
    }
    if (e != cudaSuccess) return err(PR_ERR_CUDA, "pr_depth_map_noalloc: scratch initialisation failed");
    float* obj_trans = (float*)(base + kNaObjTrans);
    uint32_t* blk_obj = (uint32_t*)(base + kNaBlkObj);
    int rc = launch(false, noalloc_init_kernel, (unsigned)((n + 255) / 256), 256, st, d->depth, keys, lastnan, n, cnt, obj_first,
                    obj_trans, blk_obj, d->n_tris, O);
    if (rc) return err(PR_ERR_CUDA, "pr_depth_map_noalloc: scratch initialisation failed");

    SetupParams sp{};
    sp.pos = (const float4*)d->pos;
    sp.obj_first = obj_first;
    sp.obj_model = obj_model;
    sp.n_tris = d->n_tris;
    sp.n_objects = d->n_objects;
    sp.W = d->width;
    sp.H = d->height;
    sp.perspective = 0;
    if (by_param) {
        sp.obj_trans = obj_trans;
        sp.blk_obj = blk_obj;
    }
    prh::M4 vp = prh::viewport((float)d->width, (float)d->height);
    std::memcpy(sp.pv, pv.m, 64);
    std::memcpy(sp.viewport, vp.m, 64);
    sp.vp_std = 1;  // prh::viewport's pattern
    sp.rrec = rrec;
    sp.cap_rec = kNoAllocMaxTris;
    sp.tasks = tasks;
    sp.cap_tasks = kNoAllocMaxTasks;
    sp.cnt = cnt;
    sp.task_shift = kNoAllocTaskShift;
    const bool long_map = d->width > kNoAllocMaxSide || d->height > kNoAllocMaxSide;
    RasterParams rp{};
    rp.task_shift = kNoAllocTaskShift;
    rp.rrec = rrec;
    rp.tasks = tasks;
    rp.cnt = cnt;
    rp.cnt_w = cnt;
    rp.W = d->width;
    rp.H = d->height;
    rp.smap = keys;
    rp.lastnan = lastnan;
    auto raster = [&](RasterMode mode, uint32_t* take) {
        rp.mode = mode;
        rp.take = take;
        return long_map ? launch(false, long_map_raster_kernel, (unsigned)sm_count() * 8u, 256, st, rp, d->n_tris)
                        : launch_raster(rp, sm_count() * 8, st);
    };
    rc = !long_map ? launch_setup_shadow(sp, st)
                   : d->n_tris ? launch(false, long_map_setup_kernel, (d->n_tris + 127u) / 128u, 128, st, sp) : 0;
    if (!rc) rc = raster(kShadow, &cnt->take[0]);
    if (!rc) rc = launch_shadow_fixup_reset(d->width, d->height, lastnan, keys, cnt, st);
    if (!rc) rc = raster(kShadowFixup, &cnt->take[1]);
    if (rc) return err(PR_ERR_CUDA, "pr_depth_map_noalloc: kernel launch failed");
    rc = launch(true, decode_changed_kernel, (unsigned)((n + 255) / 256), 256, st, keys, d->depth, n, cnt);
    if (rc) return err(PR_ERR_CUDA, "pr_depth_map_noalloc: kernel launch failed");
    Counters h{};
    e = cudaMemcpyAsync(&h, cnt, sizeof(Counters), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return err(PR_ERR_CUDA, "pr_depth_map_noalloc: execution failed");
    if (h.overflow)
        return err(PR_ERR_OVERFLOW, "pr_depth_map_noalloc: more raster tasks than PR_NOALLOC_MAX_TASKS (262144); "
                                    "the depth map was left unchanged");
    return PR_OK;
}
