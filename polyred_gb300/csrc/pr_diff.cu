// Differentiable deferred shading: the float radiance of the shade pass and
// its adjoint, with visibility held fixed by the differentiation G-buffer the
// forward frame writes (shade_kernel / ao_kernel).
//
// The radiance follows shade + FragmentShader (render/raster.go:320-356,
// shader/blinn_cpu.go:24-106) before Round and the uint8 conversions:
//   material pixel, channel c:
//     La_c = sum_e Ie col_c                       (col: the 1x1 texture's texel)
//     per light: point    D = lp - x, L = D/|D|, I = Il/|D|
//                directional  L = -dir, I = Il
//       V = unit(cam - x), H = unit(L + V)
//       Ld = clamp(n.L, 0, 1), Ls = clamp(n.H, 0, 1)^s
//     pre_c = La_c + kd_c sum_l Ld col_c I + ks_c sum_l Ls lcol_c I
//     R_c = fac clamp(pre_c, 0, 255),   n = unit(sum_k b_k N_k) (or the face normal)
//   material-less pixel: R_c = 255 sum_k p_k C_k,c
//   background: the background colour.
// The backward pass recomputes every term above from the G-buffer and the
// parameters (nothing per light is stored) and accumulates: per-vertex colour
// and normal gradients by float atomics (one 16-byte atomic per vertex where
// the caller's arrays allow it), per-light and ambient gradients by warp sums
// kept in registers, per-material ones by a warp sum per material of the warp,
// both then block sums in shared memory and double atomics.
#include <cuda_runtime.h>

#include <algorithm>

#include "pr_devmath.cuh"
#include "pr_kernels.cuh"

namespace prk {
namespace {

using namespace prd;

constexpr int kDiffThreads = 256;

struct F3 { float x, y, z; };
__device__ __forceinline__ F3 f3(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ F3 operator+(F3 a, F3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ F3 operator-(F3 a, F3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F3 operator*(float s, F3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ float dot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float norm3(F3 a) { return sqrtf(dot(a, a)); }

__device__ __forceinline__ uint32_t find_obj(const uint32_t* first, uint32_t n_obj, uint32_t t) {
    uint32_t lo = 0, hi = n_obj - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (first[mid] <= t)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

PR_DEV float warp_sum(float v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

// Add (x, y, z) to a vertex's float4. vec: the array is 16-byte aligned.
PR_DEV void add_vertex(float4* p, float x, float y, float z, bool vec) {
    if (vec) {
        atomicAdd(p, make_float4(x, y, z, 0.0f));
    } else {
        float* q = reinterpret_cast<float*>(p);
        atomicAdd(q + 0, x);
        atomicAdd(q + 1, y);
        atomicAdd(q + 2, z);
    }
}

// A warp's pixels are consecutive; every lane runs every step (a lane past
// the image, or whose pixel is not lit, with nothing to add), so that the
// shared gradients are summed by shuffles: one atomic per lane on the same
// few shared words serialised the backward pass (1920x1080, two lights: 281 us).
constexpr int kAccSlots = (kMaxLights * 4 + kMaxAmbient + 31) / 32;  // light and ambient sums per lane
// Steps of kDiffThreads pixels a backward block takes at most: a material's
// sums then add 8 x 16 warp sums in float32, fewer than the 256 pixels that a
// block of one step added one by one, and a light's 16 per lane and 8 of those.
constexpr unsigned kDiffSteps = 16;
template <bool BACKWARD>
__global__ void __launch_bounds__(kDiffThreads) diff_kernel(const __grid_constant__ DiffParamsK P) {
    // block sums: [mat*7 + {kd0..2, ks0..2, shin}] [light*4 + {pos0..2, I}] [ambient]
    __shared__ float s_acc[kDiffMaxMats * 7 + kMaxLights * 4 + kMaxAmbient];
    const int n_acc = P.n_mats * 7 + P.n_lights * 4 + P.n_ambient;
    const int lane = threadIdx.x & 31;
    float acc[kAccSlots];  // this lane's light and ambient sums: value v is lane v % 32's, slot v / 32
    if (BACKWARD) {
        for (int k = threadIdx.x; k < n_acc; k += blockDim.x) s_acc[k] = 0.0f;
#pragma unroll
        for (int k = 0; k < kAccSlots; k++) acc[k] = 0.0f;
        __syncthreads();
    }
    auto keep = [&](int v, float total) {
#pragma unroll
        for (int k = 0; k < kAccSlots; k++)
            if (v == k * 32 + lane) acc[k] += total;
    };
    const size_t npx = (size_t)P.W * P.H;
    for (size_t first = (size_t)blockIdx.x * blockDim.x; first < npx; first += (size_t)gridDim.x * blockDim.x) {
        const size_t i = first + threadIdx.x;
        const bool in = i < npx;
        const float4 none = make_float4(__uint_as_float(0xFFFFFFFFu), 0.0f, 0.0f, 0.0f), zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float4 d0 = in ? P.dgb[4 * i] : none, d1 = in ? P.dgb[4 * i + 1] : zero, d2 = in ? P.dgb[4 * i + 2] : zero,
                     d3 = in ? P.dgb[4 * i + 3] : zero;
        const uint32_t t = __float_as_uint(d0.x);
        const int m = __float_as_int(d0.y);
        const uint32_t fl = __float_as_uint(d0.z);
        const float fac = d0.w;
        float R[3] = {0.0f, 0.0f, 0.0f};
        float g[3] = {0.0f, 0.0f, 0.0f};
        if (BACKWARD && in) {
            const float4 gr = P.grad[i];
            g[0] = gr.x;
            g[1] = gr.y;
            g[2] = gr.z;
        }
        const float alpha = d1.w;
        bool lit = false;
        if (t == 0xFFFFFFFFu) {
            R[0] = P.bg[0];
            R[1] = P.bg[1];
            R[2] = P.bg[2];
        } else if (fl & kDgbUnlit) {
            const float p[3] = {d1.x, d1.y, d1.z};
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float4 C = P.vcol[3 * (size_t)t + k];
                R[0] += 255.0f * p[k] * C.x;
                R[1] += 255.0f * p[k] * C.y;
                R[2] += 255.0f * p[k] * C.z;
                if (BACKWARD && P.g_vcol)
                    add_vertex(P.g_vcol + 3 * (size_t)t + k, g[0] * 255.0f * p[k], g[1] * 255.0f * p[k], g[2] * 255.0f * p[k],
                               P.vec_vcol);
            }
        } else if ((fl & (kDgbLit | kDgbConst)) && m >= 0 && m < P.n_mats) {
            if (fl & kDgbConst) {
                const pr_material& mat = P.mats[m];
                R[0] = fac * (float)mat.texture[0];
                R[1] = fac * (float)mat.texture[1];
                R[2] = fac * (float)mat.texture[2];
            } else {
                lit = true;
            }
        }
        if (__any_sync(0xffffffffu, lit)) {
            float col[3] = {0, 0, 0}, kd[3] = {0, 0, 0}, ks[3] = {0, 0, 0}, s = 1.0f;
            const F3 x = f3(d2.x, d2.y, d2.z);
            bool flat = false;
            const float* M = nullptr;
            F3 n = f3(0, 0, 0);
            float mlen = 1.0f;
            if (lit) {
                const pr_material& mat = P.mats[m];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    col[c] = (float)mat.texture[c];
                    kd[c] = P.kd[3 * m + c];
                    ks[c] = P.ks[3 * m + c];
                }
                s = P.shin[m];
                // normal
                flat = (fl & kDgbFlat) != 0;
                if (flat) {
                    n = f3(d3.x, d3.y, d3.z);
                } else {
                    M = P.obj_normal + 16 * (size_t)find_obj(P.obj_first, P.n_objects, t);
                    const float b[3] = {d1.x, d1.y, d1.z};
                    F3 mv = f3(0, 0, 0);
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const float4 v = P.vnor[3 * (size_t)t + k];
                        const F3 N = f3(M[0] * v.x + M[1] * v.y + M[2] * v.z + M[3] * v.w,
                                        M[4] * v.x + M[5] * v.y + M[6] * v.z + M[7] * v.w,
                                        M[8] * v.x + M[9] * v.y + M[10] * v.z + M[11] * v.w);
                        mv = mv + b[k] * N;
                    }
                    mlen = norm3(mv);
                    n = (1.0f / mlen) * mv;
                }
            }
            float La[3] = {0, 0, 0}, Ld[3] = {0, 0, 0}, Ls[3] = {0, 0, 0};
            const F3 Vd = f3(P.cam[0], P.cam[1], P.cam[2]) - x;
            const F3 V = (1.0f / norm3(Vd)) * Vd;
            // per-light terms, recomputed in the backward pass
            auto light_terms = [&](int l, F3& L, float& I, float& dist, F3& H, float& hlen, float& nd, float& nh, float& ld,
                                   float& ls) {
                const LightK& Lk = P.lights[l];
                if (Lk.type == PR_LIGHT_POINT) {
                    const F3 D = f3(Lk.pos[0], Lk.pos[1], Lk.pos[2]) - x;
                    dist = norm3(D);
                    L = (1.0f / dist) * D;
                    I = Lk.intensity / dist;
                } else {
                    L = f3(-Lk.dir[0], -Lk.dir[1], -Lk.dir[2]);
                    dist = 1.0f;
                    I = Lk.intensity;
                }
                const F3 Hv = L + V;
                hlen = norm3(Hv);
                H = (1.0f / hlen) * Hv;
                nd = dot(n, L);
                nh = dot(n, H);
                ld = fminf(fmaxf(nd, 0.0f), 1.0f);
                const float nhc = fminf(fmaxf(nh, 0.0f), 1.0f);
                ls = nhc > 0.0f ? powf(nhc, s) : 0.0f;
            };
            float pre[3] = {0, 0, 0};
            if (lit) {
                for (int e = 0; e < P.n_ambient; e++) {
                    La[0] += P.ambient[e] * col[0];
                    La[1] += P.ambient[e] * col[1];
                    La[2] += P.ambient[e] * col[2];
                }
                for (int l = 0; l < P.n_lights; l++) {
                    F3 L, H;
                    float I, dist, hlen, nd, nh, ld, ls;
                    light_terms(l, L, I, dist, H, hlen, nd, nh, ld, ls);
                    const LightK& Lk = P.lights[l];
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        Ld[c] += ld * col[c] * I;
                        Ls[c] += ls * Lk.color[c] * I;
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    pre[c] = La[c] + kd[c] * Ld[c] + ks[c] * Ls[c];
                    R[c] = fac * fminf(fmaxf(pre[c], 0.0f), 255.0f);
                }
            }
            if (BACKWARD) {
                float gg[3];
#pragma unroll
                for (int c = 0; c < 3; c++) gg[c] = (lit && pre[c] > 0.0f && pre[c] < 255.0f) ? g[c] * fac : 0.0f;
                F3 gn = f3(0, 0, 0);
                float gshin = 0.0f;
                const float Aw = gg[0] * kd[0] * col[0] + gg[1] * kd[1] * col[1] + gg[2] * kd[2] * col[2];
                for (int l = 0; l < P.n_lights; l++) {
                    const LightK& Lk = P.lights[l];
                    // loss contribution A ld I + B ls I
                    const float Bw = gg[0] * ks[0] * Lk.color[0] + gg[1] * ks[1] * Lk.color[1] + gg[2] * ks[2] * Lk.color[2];
                    float dI = 0.0f;
                    F3 gD = f3(0, 0, 0);
                    if (lit && !(Aw == 0.0f && Bw == 0.0f)) {
                        F3 L, H;
                        float I, dist, hlen, nd, nh, ld, ls;
                        light_terms(l, L, I, dist, H, hlen, nd, nh, ld, ls);
                        dI = (Aw * ld + Bw * ls) * (Lk.type == PR_LIGHT_POINT ? 1.0f / dist : 1.0f);
                        const float nhc = fminf(fmaxf(nh, 0.0f), 1.0f);
                        if (ls > 0.0f && nhc < 1.0f) gshin += Bw * I * ls * logf(nhc);
                        const float gnd = (nd > 0.0f && nd < 1.0f) ? Aw * I : 0.0f;
                        const float gnh = (nh > 0.0f && nh < 1.0f) ? Bw * I * s * powf(nhc, s - 1.0f) : 0.0f;
                        gn = gn + gnd * L + gnh * H;
                        if (Lk.type == PR_LIGHT_POINT) {
                            // L(D) through n.L and through H = unit(L + V); I = Il/|D|
                            const F3 gL = gnd * n + (gnh / hlen) * (n - nh * H);
                            gD = (1.0f / dist) * (gL - dot(L, gL) * L) + (-(Aw * ld + Bw * ls) * I / dist) * L;
                        }
                    }
                    keep(4 * l + 3, warp_sum(dI));
                    if (Lk.type == PR_LIGHT_POINT) {  // uniform
                        keep(4 * l + 0, warp_sum(gD.x));
                        keep(4 * l + 1, warp_sum(gD.y));
                        keep(4 * l + 2, warp_sum(gD.z));
                    }
                }
                if (P.n_ambient) {
                    const float gcol = warp_sum(gg[0] * col[0] + gg[1] * col[1] + gg[2] * col[2]);
                    for (int e = 0; e < P.n_ambient; e++) keep(4 * P.n_lights + e, gcol);
                }
                // the materials of the warp's lit pixels, one at a time (usually one or two)
                const float mv[7] = {gg[0] * Ld[0], gg[1] * Ld[1], gg[2] * Ld[2], gg[0] * Ls[0], gg[1] * Ls[1], gg[2] * Ls[2], gshin};
                unsigned todo = __ballot_sync(0xffffffffu, lit);
                while (todo) {
                    const int mm = __shfl_sync(0xffffffffu, m, __ffs(todo) - 1);
                    const bool same = lit && m == mm;
                    float mine = 0.0f;
#pragma unroll
                    for (int c = 0; c < 7; c++) {
                        // a channel without gradient adds nothing, whatever its sums are
                        const bool on = same && (c == 6 || gg[c < 3 ? c : c - 3] != 0.0f);
                        const float total = warp_sum(on ? mv[c] : 0.0f);
                        if (lane == c) mine = total;
                    }
                    if (lane < 7 && mine != 0.0f) atomicAdd(s_acc + 7 * mm + lane, mine);
                    todo &= ~__ballot_sync(0xffffffffu, same);
                }
                if (lit && !flat && P.g_vnor) {
                    const F3 gm = (1.0f / mlen) * (gn - dot(n, gn) * n);
                    const float b[3] = {d1.x, d1.y, d1.z};
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const F3 gN = b[k] * gm;
                        const float vx = M[0] * gN.x + M[4] * gN.y + M[8] * gN.z, vy = M[1] * gN.x + M[5] * gN.y + M[9] * gN.z,
                                    vz = M[2] * gN.x + M[6] * gN.y + M[10] * gN.z;
                        if (vx != 0.0f || vy != 0.0f || vz != 0.0f)
                            add_vertex(P.g_vnor + 3 * (size_t)t + k, vx, vy, vz, P.vec_vnor);
                    }
                }
            }
        }
        if (!BACKWARD && in) P.radiance[i] = make_float4(R[0], R[1], R[2], alpha);
    }
    if (BACKWARD) {
        const int n_la = P.n_lights * 4 + P.n_ambient;
#pragma unroll
        for (int k = 0; k < kAccSlots; k++)
            if (k * 32 + lane < n_la && acc[k] != 0.0f) atomicAdd(s_acc + 7 * P.n_mats + k * 32 + lane, acc[k]);
        __syncthreads();
        for (int k = threadIdx.x; k < n_acc; k += blockDim.x) {
            const float v = s_acc[k];
            if (v != 0.0f) atomicAdd(P.g_acc + k, (double)v);
        }
    }
}

__global__ void col_to_float_kernel(const uchar4* col, float4* out, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const uchar4 c = col[i];
        out[i] = make_float4(c.x / 255.0f, c.y / 255.0f, c.z / 255.0f, c.w / 255.0f);
    }
}

int check(cudaError_t e) { return e == cudaSuccess ? 0 : (int)e; }

}  // namespace

namespace {
__global__ void fill_u32_kernel(uint32_t* p, uint32_t v, size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}
}  // namespace

int launch_fill_u32(uint32_t* p, uint32_t v, size_t n, void* stream) {
    if (n == 0) return 0;
    const size_t nb = std::min<size_t>((n + 255) / 256, 4096);
    fill_u32_kernel<<<(unsigned)nb, 256, 0, (cudaStream_t)stream>>>(p, v, n);
    return check(cudaGetLastError());
}

int launch_col_to_float(const uchar4* col, float4* out, size_t n, void* stream) {
    if (n == 0) return 0;
    col_to_float_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(col, out, n);
    return check(cudaGetLastError());
}

int launch_diff(const DiffParamsK& p, bool backward, void* stream) {
    const size_t npx = (size_t)p.W * p.H;
    if (npx == 0) return 0;
    const unsigned nb = (unsigned)((npx + kDiffThreads - 1) / kDiffThreads);
    // Backward: blocks of several steps, so that a warp's register sums cover
    // many pixels: one wave of them, but at most kDiffSteps steps each. A block's
    // sums are float32 until it ends; without that bound their number of terms
    // (and their rounding) grew with the image: 54,000 pixels a block at 7680x4320
    // (the whole call 1920x1080 168 us either way, 3840x2160 599 -> 538 us).
    const unsigned nbw = std::max(std::min(nb, (unsigned)sm_count() * 4u), (nb + kDiffSteps - 1) / kDiffSteps);
    if (backward)
        diff_kernel<true><<<nbw, kDiffThreads, 0, (cudaStream_t)stream>>>(p);
    else
        diff_kernel<false><<<nb, kDiffThreads, 0, (cudaStream_t)stream>>>(p);
    return check(cudaGetLastError());
}

}  // namespace prk
