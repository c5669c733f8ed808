// Gradients of LayerNorm and training BatchNorm (with the ReLU that follows it) as the kernels read them, instead of the
// op-by-op graph of the reverse rules: that graph is nine row or column reduces and a dozen full-size passes per layer
// (LayerNorm [5000,1001] float32: 7 launches, 106 us; BatchNorm + ReLU [64,128,28,28] bfloat16: 23 launches, 190 us). Both are
// bound by memory: x and dy are read once (LayerNorm, BatchNorm of layers that shared memory holds) or twice, dx is written
// once, and everything per channel or column is folded in a fixed order.
//
//   LayerNorm   xh = (x - mean) * rstd, g = dy * gamma:  dx = rstd * (g - mean(g) - xh * mean(g * xh)),
//               dgamma = sum over rows of dy * xh, dbeta = sum of dy
//   BatchNorm   d = dy where the activation is positive:  S0 = sum d, S1 = sum d * xh per channel,
//               dx = gamma * rstd * (d - (S0 + xh * S1) / count), dgamma = S1, dbeta = S0
// A clamped variance (max(E[x^2] - E[x]^2, 0) at 0) passes no gradient, as in the graph.
#include "common.cuh"

#include <algorithm>
#include <cooperative_groups.h>
#include <type_traits>

namespace b200jt {
namespace nbwd {

template <typename T, int N> struct Vec;
template <> struct Vec<float, 1> {
    static __device__ __forceinline__ void ld(const float* p, float* o) { o[0] = *p; }
    static __device__ __forceinline__ void st(float* p, const float* o) { *p = o[0]; }
};
template <> struct Vec<__nv_bfloat16, 1> {
    static __device__ __forceinline__ void ld(const __nv_bfloat16* p, float* o) { o[0] = __bfloat162float(*p); }
    static __device__ __forceinline__ void st(__nv_bfloat16* p, const float* o) { *p = __float2bfloat16(o[0]); }
};
template <> struct Vec<float, 4> {
    static __device__ __forceinline__ void ld(const float* p, float* o) { const float4 v = *(const float4*)p; o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
    static __device__ __forceinline__ void st(float* p, const float* o) { *(float4*)p = make_float4(o[0], o[1], o[2], o[3]); }
};
template <> struct Vec<float, 8> {
    static __device__ __forceinline__ void ld(const float* p, float* o) { Vec<float, 4>::ld(p, o); Vec<float, 4>::ld(p + 4, o + 4); }
    static __device__ __forceinline__ void st(float* p, const float* o) { Vec<float, 4>::st(p, o); Vec<float, 4>::st(p + 4, o + 4); }
};
template <> struct Vec<__nv_bfloat16, 8> {
    static __device__ __forceinline__ void ld(const __nv_bfloat16* p, float* o) {
        const uint4 v = *(const uint4*)p;
        const __nv_bfloat162* h = (const __nv_bfloat162*)&v;
#pragma unroll
        for (int i = 0; i < 4; i++) { const float2 f = __bfloat1622float2(h[i]); o[2 * i] = f.x; o[2 * i + 1] = f.y; }
    }
    static __device__ __forceinline__ void st(__nv_bfloat16* p, const float* o) {
        uint4 v;
        __nv_bfloat162* h = (__nv_bfloat162*)&v;
#pragma unroll
        for (int i = 0; i < 4; i++) h[i] = __floats2bfloat162_rn(o[2 * i], o[2 * i + 1]);
        *(uint4*)p = v;
    }
};

template <typename T, int N> struct alignas(N * sizeof(T) < 16 ? N * sizeof(T) : 16) Raw { T v[N]; };      // a vector as it lies in memory

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}
// Sums of NV values over the GROUP threads of a row (a warp, or a CTA of up to 256).
constexpr int cta_of(int group) { return group == 32 ? 256 : group; }
template <int GROUP, int NV>
__device__ __forceinline__ void row_sum(float (&v)[NV], float* sm) {
#pragma unroll
    for (int i = 0; i < NV; i++) v[i] = warp_sum(v[i]);
    if constexpr (GROUP > 32) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        __syncthreads();
        if (lane == 0)
#pragma unroll
            for (int i = 0; i < NV; i++) sm[i * 8 + warp] = v[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NV; i++) {
            float t = 0.f;
#pragma unroll
            for (int w = 0; w < GROUP / 32; w++) t += sm[i * 8 + w];
            v[i] = t;
        }
    }
}

// GROUP threads hold a row of x and of dy in registers (E elements each, in vectors of N) and keep their columns' sums for
// dgamma / dbeta across the rows they visit; a CTA writes one pair of partial rows at the end.
template <typename T, int N, int GROUP, int E, bool DX, bool PARAMS>
__global__ void __launch_bounds__(cta_of(GROUP))
layer_norm_bwd_kernel(const T* __restrict__ x, const T* __restrict__ dy, const float* __restrict__ gamma, T* __restrict__ dx,
                      float* __restrict__ partial, int64_t rows, int cols, float eps) {
    constexpr int VPT = E / N, RPC = cta_of(GROUP) / GROUP;
    __shared__ float sm[32];
    extern __shared__ float fold[];                             // GROUP == 32 and PARAMS: [2][cols]
    const int g = threadIdx.x / GROUP, t = threadIdx.x % GROUP;
    const int nvec = cols / N;
    const float rc = 1.f / (float)cols;
    float ag[PARAMS ? VPT : 1][N] = {}, ab[PARAMS ? VPT : 1][N] = {};
    // The next row is on its way through this one's reductions where the registers for it cost no resident CTA: [43690, 768] float32
    // 114 -> 89 us, [8192, 4096] bfloat16 91 -> 70; elsewhere it cost more than it gave ([120000, 128] float32 48 and, with it, 76).
    constexpr bool AHEAD = DX && PARAMS && N > 1 && (sizeof(T) == 4 ? GROUP == 128 : GROUP == 256 && E == 16);
    Raw<T, N> na[AHEAD ? VPT : 1], nb[AHEAD ? VPT : 1];
    // columns beyond the row read its last vector and count as zeros, rows beyond the last read that one: no branch between the loads
    auto fetch = [&](int64_t row) {
        row = row < rows ? row : rows - 1;
#pragma unroll
        for (int k = 0; k < VPT; k++) {
            const int64_t at = row * cols + (int64_t)min(t + k * GROUP, nvec - 1) * N;
            na[k] = *(const Raw<T, N>*)(x + at);
            nb[k] = *(const Raw<T, N>*)(dy + at);
        }
    };
    if constexpr (AHEAD) fetch((int64_t)blockIdx.x * RPC + g);
    for (int64_t row0 = (int64_t)blockIdx.x * RPC; row0 < rows; row0 += (int64_t)gridDim.x * RPC) {
        const int64_t row = row0 + g;
        if (GROUP == 32 && row >= rows) break;                  // warps leave on their own; a CTA per row leaves as one
        float a[VPT][N], b[VPT][N];
        float s[2] = {0.f, 0.f};
#pragma unroll
        for (int k = 0; k < VPT; k++) {
            if constexpr (AHEAD) {
                Vec<T, N>::ld(na[k].v, a[k]);
                Vec<T, N>::ld(nb[k].v, b[k]);
            } else {
                const int64_t at = row * cols + (int64_t)min(t + k * GROUP, nvec - 1) * N;
                Vec<T, N>::ld(x + at, a[k]);
                Vec<T, N>::ld(dy + at, b[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < VPT; k++)
#pragma unroll
            for (int e = 0; e < N; e++) {
                if (t + k * GROUP >= nvec) a[k][e] = b[k][e] = 0.f;
                s[0] += a[k][e]; s[1] += a[k][e] * a[k][e];
            }
        if constexpr (AHEAD) fetch(row + (int64_t)gridDim.x * RPC);
        row_sum<GROUP, 2>(s, sm);
        const float mean = s[0] * rc, var = fmaxf(s[1] * rc - mean * mean, 0.f), rstd = 1.f / sqrtf(var + eps);
        float c[2] = {0.f, 0.f};
        constexpr int BATCH = VPT < 8 ? VPT : 8;
#pragma unroll
        for (int k0 = 0; k0 < VPT; k0 += BATCH) {
            float gm[BATCH][N];
            if (DX) {
#pragma unroll
                for (int k = 0; k < BATCH; k++) {
                    const int vi = min(t + (k0 + k) * GROUP, nvec - 1);
                    if (gamma) {
                        if constexpr (N == 1) gm[k][0] = gamma[vi];
                        else Vec<float, N>::ld(gamma + (int64_t)vi * N, gm[k]);
                    } else {
#pragma unroll
                        for (int e = 0; e < N; e++) gm[k][e] = 1.f;
                    }
                }
            }
#pragma unroll
            for (int k = k0; k < k0 + BATCH; k++)
#pragma unroll
                for (int e = 0; e < N; e++) {
                    const float xh = (a[k][e] - mean) * rstd;
                    if constexpr (PARAMS) { ag[k][e] += b[k][e] * xh; ab[k][e] += b[k][e]; }
                    if (DX) {
                        const float gy = b[k][e] * gm[k - k0][e];
                        c[0] += gy; c[1] += gy * xh;
                        a[k][e] = xh; b[k][e] = gy;
                    }
                }
        }
        if constexpr (DX) {
            row_sum<GROUP, 2>(c, sm + 16);
            const float c0 = c[0] * rc, c1 = var > 0.f ? c[1] * rc : 0.f;
#pragma unroll
            for (int k = 0; k < VPT; k++) {
                const int vi = t + k * GROUP;
                if (vi >= nvec) continue;
                float o[N];
#pragma unroll
                for (int e = 0; e < N; e++) o[e] = rstd * (b[k][e] - c0 - a[k][e] * c1);
                Vec<T, N>::st(dx + row * cols + (int64_t)vi * N, o);
            }
        }
    }
    if constexpr (PARAMS) {
        float* out = partial + (int64_t)blockIdx.x * 2 * cols;
        if constexpr (GROUP > 32) {
#pragma unroll
            for (int k = 0; k < VPT; k++) {
                const int vi = t + k * GROUP;
                if (vi >= nvec) continue;
#pragma unroll
                for (int e = 0; e < N; e++) { out[vi * N + e] = ag[k][e]; out[cols + vi * N + e] = ab[k][e]; }
            }
        } else {                                                // the warps add their sums one after the other
            for (int w = 0; w < 8; w++) {
                if (g == w)
#pragma unroll
                    for (int k = 0; k < VPT; k++) {
                        const int vi = t + k * GROUP;
                        if (vi >= nvec) continue;
#pragma unroll
                        for (int e = 0; e < N; e++) {
                            const int i = vi * N + e;
                            fold[i] = w ? fold[i] + ag[k][e] : ag[k][e];
                            fold[cols + i] = w ? fold[cols + i] + ab[k][e] : ab[k][e];
                        }
                    }
                __syncthreads();
            }
            for (int i = threadIdx.x; i < 2 * cols; i += 256) out[i] = fold[i];
        }
    }
}

// out[i] = sum over p < parts of partial[p * n + i], in order of p within 32 interleaved chains. (Eight of them were bound by their
// length: 592 rows of 2002 sums 6.5 us.)
__global__ void __launch_bounds__(1024) fold_rows_kernel(const float* __restrict__ partial, float* __restrict__ out, int n, int parts) {
    __shared__ float sm[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (i < n)
#pragma unroll 4
        for (int p = w; p < parts; p += 32) s += partial[(int64_t)p * n + i];
    sm[w][lane] = s;
    __syncthreads();
    const float t = warp_sum(sm[lane][w]);                     // warp w adds the chains of column w
    if (lane == 0 && blockIdx.x * 32 + w < n) out[blockIdx.x * 32 + w] = t;
}

// ---- BatchNorm ---------------------------------------------------------------------------------------------------------
// Two sets of formulas. float32 x: the closed form above in float32. bfloat16 x: the meta-op graph rounds every node to its
// dtype, the statistics included, and what it makes of the small terms of dx (they vanish below a rounding of the large one)
// and of signs near zero is several per cent of a weight gradient further on, so the same steps are rounded at the same
// places here, in registers: `round` 1 rounds what the graph keeps in bfloat16 when the activation is float32, 2 every node
// (a bfloat16 activation).
struct BnArgs {
    const float *stats, *gamma, *beta;
    float rcount, eps;
    int relu, round, N_, C;
    int64_t HW;
};
__device__ __forceinline__ float bf(float v) { return __bfloat162float(__float2bfloat16(v)); }
struct BnChannel { float mean, rstd, sd, w, b; bool live; };
// square: E[x * x] with the products rounded as in the graph (only looked at when round > 0)
__device__ __forceinline__ BnChannel bn_channel(const BnArgs& g, int c, float square) {
    BnChannel k;
    const float gamma = g.gamma ? g.gamma[c] : 1.f, beta = g.beta ? g.beta[c] : 0.f;
    k.mean = g.stats[c] * g.rcount;
    if (g.round == 0) {
        const float var = fmaxf(g.stats[g.C + c] * g.rcount - k.mean * k.mean, 0.f);
        k.live = var > 0.f;
        k.sd = sqrtf(var + g.eps);
        k.w = gamma / k.sd;
        k.b = beta - k.mean * k.w;
    } else {
        k.mean = bf(k.mean);
        const float var = fmaxf(bf(bf(square) - bf(k.mean * k.mean)), 0.f);
        k.live = var != 0.f;
        k.sd = bf(sqrtf(bf(var + g.eps)));
        k.w = gamma / k.sd;
        if (g.round == 2) k.w = bf(k.w);
        const float mw = __fmul_rn(k.mean, k.w);
        k.b = g.round == 2 ? bf(beta - bf(mw)) : __fsub_rn(beta, mw);
    }
    k.rstd = 1.f / k.sd;
    return k;
}
// Whether the gradient of the ReLU passes (x: an element of the normalised tensor's input).
__device__ __forceinline__ bool passes(const BnArgs& g, const BnChannel& k, float x) {
    if (!g.relu) return true;
    if (g.round == 0) return x * k.w + k.b > 0.f;
    const float p = __fmul_rn(x, k.w);
    return (g.round == 2 ? bf(p) : p) + k.b > 0.f;
}

// What the sums of a channel become (in place), and the gradient of w in the rounded forms.
__device__ __forceinline__ float bn_gradients(const BnArgs& g, const BnChannel& k, float& s0, float& s1) {
    float dw = 0.f;
    if (g.round == 2) {
        s0 = bf(s0);
        dw = bf(bf(s1) + bf(k.mean * -s0));
        s1 = bf(dw / k.sd);
    } else if (g.round == 1) {
        dw = __fadd_rn(s1, __fmul_rn(k.mean, -s0));
        s1 = dw / k.sd;
    }
    return dw;
}
// dx of one element, closed form w * d + p * x + q, rounded form ((w * d + x * p) + x * p) + q, each step to bfloat16
struct BnDx { float p, q; };
__device__ __forceinline__ BnDx bn_dx(const BnArgs& g, const BnChannel& k, int c, float s0, float s1, float dw) {
    BnDx r;
    if (g.round == 0) {
        r.p = k.live ? -k.w * k.rstd * s1 * g.rcount : 0.f;
        r.q = -k.w * s0 * g.rcount - r.p * k.mean;
    } else {
        const float gamma = g.gamma ? g.gamma[c] : 1.f;
        float num = __fmul_rn(-dw, gamma), wd = __fmul_rn(k.w, -s0);
        if (g.round == 2) num = bf(num);
        const float dvar = k.live ? bf(bf(num / bf(k.sd * k.sd)) / bf(k.sd * 2.f)) : 0.f;
        const float t = bf(k.mean * -dvar);
        r.p = bf(dvar * g.rcount);
        r.q = bf(bf(bf(bf(wd) + t) + t) * g.rcount);
    }
    return r;
}
__device__ __forceinline__ float bn_dx_of(const BnArgs& g, const BnChannel& k, const BnDx& r, float x, float dy) {
    const float u = passes(g, k, x) ? dy : 0.f;
    if (g.round == 0) return k.w * u + (r.p * x + r.q);
    const float t = bf(x * r.p);
    return bf(bf(bf(k.w * u) + t) + t) + r.q;                   // the store rounds the last sum
}

// One vector's part of the three passes over a layer: the sum of bfloat16(x * x), the two sums, dx.
template <typename TX, typename TD, int N, bool HALF> struct BnPass {
    static __device__ __forceinline__ void square(const TX* x, float& s) {
        float a[N];
        Vec<TX, N>::ld(x, a);
#pragma unroll
        for (int e = 0; e < N; e++) s += bf(a[e] * a[e]);
    }
    static __device__ __forceinline__ void sums(const BnArgs& g, const BnChannel& k, const TX* x, const TD* dy, float (&s)[2]) {
        float a[N], d[N];
        Vec<TX, N>::ld(x, a);
        Vec<TD, N>::ld(dy, d);
#pragma unroll
        for (int e = 0; e < N; e++) {
            const float v = passes(g, k, a[e]) ? d[e] : 0.f;
            s[0] += v;
            s[1] += g.round == 0 ? v * ((a[e] - k.mean) * k.rstd) : g.round == 2 ? bf(a[e] * v) : a[e] * v;
        }
    }
    static __device__ __forceinline__ void grad(const BnArgs& g, const BnChannel& k, const BnDx& r, const TX* x, const TD* dy, TX* dx) {
        float a[N], d[N];
        Vec<TX, N>::ld(x, a);
        Vec<TD, N>::ld(dy, d);
#pragma unroll
        for (int e = 0; e < N; e++) a[e] = bn_dx_of(g, k, r, a[e], d[e]);
        Vec<TX, N>::st(dx, a);
    }
};
// Every step in bfloat16 (g.round == 2, x and dy bfloat16): the passes are bound by their conversions, a dozen an element when each
// rounds alone (64 x 128 x 28 x 28 in one launch: 24.6 us, in pairs 18.3; in two 29.2 and 25). The products' factors are all bfloat16, so that one packed multiplication rounds two of them as float32 and a
// conversion would; sums stay float32 and are converted in pairs. x * w + b > 0 is x * w > -b: a float32 sum is 0 only if it is.
struct Pair { float x, y; };
__device__ __forceinline__ Pair floats(__nv_bfloat162 v) { const float2 f = __bfloat1622float2(v); return {f.x, f.y}; }
__device__ __forceinline__ __nv_bfloat162 masked(const BnArgs& g, const BnChannel& k, __nv_bfloat162 a, __nv_bfloat162 d) {
    if (!g.relu) return d;
    const Pair p = floats(__hmul2_rn(a, __float2bfloat162_rn(k.w)));
    unsigned v;
    memcpy(&v, &d, 4);
    v &= (p.x > -k.b ? 0xffffu : 0u) | (p.y > -k.b ? 0xffff0000u : 0u);
    memcpy(&d, &v, 4);
    return d;
}
template <> struct BnPass<__nv_bfloat16, __nv_bfloat16, 8, true> {
    using B = __nv_bfloat16;
    struct alignas(16) Pack { __nv_bfloat162 h[4]; };
    static __device__ __forceinline__ void square(const B* x, float& s) {
        const Pack a = *(const Pack*)x;
#pragma unroll
        for (int e = 0; e < 4; e++) { const Pair q = floats(__hmul2_rn(a.h[e], a.h[e])); s += q.x; s += q.y; }
    }
    static __device__ __forceinline__ void sums(const BnArgs& g, const BnChannel& k, const B* x, const B* dy, float (&s)[2]) {
        const Pack a = *(const Pack*)x, d = *(const Pack*)dy;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const __nv_bfloat162 v = masked(g, k, a.h[e], d.h[e]);
            const Pair f = floats(v), q = floats(__hmul2_rn(a.h[e], v));
            s[0] += f.x; s[0] += f.y;
            s[1] += q.x; s[1] += q.y;
        }
    }
    static __device__ __forceinline__ void grad(const BnArgs& g, const BnChannel& k, const BnDx& r, const B* x, const B* dy, B* dx) {
        const Pack a = *(const Pack*)x, d = *(const Pack*)dy;
        Pack o;
        const __nv_bfloat162 w = __float2bfloat162_rn(k.w), p = __float2bfloat162_rn(r.p);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const Pair u = floats(__hmul2_rn(w, masked(g, k, a.h[e], d.h[e]))), t = floats(__hmul2_rn(a.h[e], p));
            const Pair y = floats(__floats2bfloat162_rn(u.x + t.x, u.y + t.y)), z = floats(__floats2bfloat162_rn(y.x + t.x, y.y + t.y));
            o.h[e] = __floats2bfloat162_rn(z.x + r.q, z.y + r.q);
        }
        *(Pack*)dx = o;
    }
};

// A cluster of up to 8 CTAs per channel: CTA j takes the planes n = j, j + cluster size, ..., as one run of N-element vectors over
// all its threads (a plane at a time left 158 of 256 threads idle at 28 x 28: 64 x 128 x 28 x 28 29 us, 15.5 us this way),
// and the CTAs' sums meet through distributed shared memory in rank order. With the graph's rounding a first sweep forms
// E[bfloat16(x * x)] (the second sweep reads x from L2). sums: [4][C] = dbeta, dgamma, that mean square, the gradient of w.
template <typename TX, typename TD, int N, bool HALF>
__global__ void __launch_bounds__(256)
bn_bwd_sums_kernel(const TX* __restrict__ x, const TD* __restrict__ dy, float* __restrict__ sums, const BnArgs g) {
    using Pass = BnPass<TX, TD, N, HALF>;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int c = blockIdx.y;
    const int rank = (int)cluster.block_rank(), size = (int)cluster.num_blocks();
    // a plane has fewer than 2^31 elements, a channel's planes together may have more
    const unsigned hv = (unsigned)g.HW / N, dj = 256 / hv, di = 256 - dj * hv, j0 = threadIdx.x / hv, i0 = threadIdx.x - j0 * hv;
    const int64_t total = (int64_t)((g.N_ - rank + size - 1) / size) * hv;
    __shared__ float sm[32], mine[4];
    auto planes = [&](auto&& f) {
        unsigned j = j0, i = i0;
#pragma unroll 4
        for (int64_t v = threadIdx.x; v < total; v += 256) {
            f(((int64_t)(rank + j * size) * g.C + c) * g.HW + i * N);
            j += dj; i += di;
            if (i >= hv) { i -= hv; j++; }
        }
    };
    float square = 0.f;
    if (g.round > 0) {
        float s[1] = {0.f};
        planes([&](int64_t i) { Pass::square(x + i, s[0]); });
        row_sum<256, 1>(s, sm);
        if (threadIdx.x == 0) mine[0] = s[0];
        cluster.sync();
        for (int r = 0; r < size; r++) square += cluster.map_shared_rank(mine, r)[0];
        square *= g.rcount;
    }
    const BnChannel k = bn_channel(g, c, square);
    float s[2] = {0.f, 0.f};
    planes([&](int64_t i) { Pass::sums(g, k, x + i, dy + i, s); });
    row_sum<256, 2>(s, sm);
    if (threadIdx.x == 0) { mine[1] = s[0]; mine[2] = s[1]; }
    cluster.sync();
    if (rank == 0 && threadIdx.x == 0) {
        float s0 = 0.f, s1 = 0.f;
        for (int r = 0; r < size; r++) { s0 += cluster.map_shared_rank(mine, r)[1]; s1 += cluster.map_shared_rank(mine, r)[2]; }
        const float dw = bn_gradients(g, k, s0, s1);
        sums[c] = s0; sums[g.C + c] = s1; sums[2 * g.C + c] = square; sums[3 * g.C + c] = dw;
    }
    cluster.sync();                                             // no CTA leaves while its sums are read
}

// dx over the tensor as one stream of N-element vectors; the channels' coefficients are derived once per CTA.
template <typename TX, typename TD, int N, bool HALF>
__global__ void __launch_bounds__(256)
bn_bwd_dx_kernel(const TX* __restrict__ x, const TD* __restrict__ dy, const float* __restrict__ sums, TX* __restrict__ dx, const BnArgs g) {
    extern __shared__ float co[];                               // per channel: w, b, p, q
    for (int c = threadIdx.x; c < g.C; c += 256) {
        const BnChannel k = bn_channel(g, c, sums[2 * g.C + c]);
        const BnDx r = bn_dx(g, k, c, sums[c], sums[g.C + c], sums[3 * g.C + c]);
        co[c] = k.w; co[g.C + c] = k.b; co[2 * g.C + c] = r.p; co[3 * g.C + c] = r.q;
    }
    __syncthreads();
    const int64_t vpp = g.HW / N, nvec = (int64_t)g.N_ * g.C * vpp;
    for (int64_t v = blockIdx.x * 256ll + threadIdx.x; v < nvec; v += (int64_t)gridDim.x * 256) {
        const int c = nvec < 0x7fffffff ? ((unsigned)v / (unsigned)vpp) % (unsigned)g.C : (int)((v / vpp) % g.C);
        BnChannel k;
        k.w = co[c]; k.b = co[g.C + c];
        const BnDx r = {co[2 * g.C + c], co[3 * g.C + c]};
        BnPass<TX, TD, N, HALF>::grad(g, k, r, x + v * N, dy + v * N, dx + v * N);
    }
}

// Both of the above in one launch, for layers that shared memory holds: the CTAs of a channel's cluster keep their planes of x and dy
// in it, so that these are read once, and nothing but the sums meets between the two parts. Each thread copies, and later reads,
// its own vectors: the copies need no barrier. 64 x 128 x 28 x 28 bfloat16: 18.3 us, the two kernels 15.7 + 13.5 and a launch
// between them; from cold caches 64 x 1024 x 14 x 14 82 and 138, float32 45 and 69.
template <int BYTES>
__device__ __forceinline__ void hold(void* to, const void* from) {
    if constexpr (BYTES >= 16) {
#pragma unroll
        for (int b = 0; b < BYTES; b += 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(to) + b), "l"((const char*)from + b) : "memory");
    } else if constexpr (BYTES == 4) *(float*)to = *(const float*)from;
    else *(unsigned short*)to = *(const unsigned short*)from;
}
template <typename TX, typename TD, int N, bool HALF>
__global__ void __launch_bounds__(256)
bn_bwd_held_kernel(const TX* __restrict__ x, const TD* __restrict__ dy, float* __restrict__ sums, TX* __restrict__ dx, const BnArgs g) {
    using Pass = BnPass<TX, TD, N, HALF>;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char held[];
    __shared__ float sm[32], mine[4];
    const int c = blockIdx.y;
    const int rank = (int)cluster.block_rank(), size = (int)cluster.num_blocks();
    const unsigned hv = (unsigned)g.HW / N, dj = 256 / hv, di = 256 - dj * hv, j0 = threadIdx.x / hv, i0 = threadIdx.x - j0 * hv;
    const int total = (int)((g.N_ - rank + size - 1) / size * hv), most = (int)((g.N_ + size - 1) / size * hv);
    TX* hx = (TX*)held;
    TD* hd = (TD*)(held + ((size_t)most * N * sizeof(TX) + 15) / 16 * 16);
    auto planes = [&](auto&& f) {
        unsigned j = j0, i = i0;
#pragma unroll 4
        for (int v = threadIdx.x; v < total; v += 256) {
            f(v * N, ((int64_t)(rank + j * size) * g.C + c) * g.HW + i * N);
            j += dj; i += di;
            if (i >= hv) { i -= hv; j++; }
        }
    };
    planes([&](int v, int64_t at) { hold<N * sizeof(TX)>(hx + v, x + at); });
    asm volatile("cp.async.commit_group;" ::: "memory");
    planes([&](int v, int64_t at) { hold<N * sizeof(TD)>(hd + v, dy + at); });
    asm volatile("cp.async.commit_group;" ::: "memory");
    float square = 0.f;
    if (g.round > 0) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        float s[1] = {0.f};
#pragma unroll 4
        for (int v = threadIdx.x; v < total; v += 256) Pass::square(hx + v * N, s[0]);
        row_sum<256, 1>(s, sm);
        if (threadIdx.x == 0) mine[0] = s[0];
        cluster.sync();
        for (int r = 0; r < size; r++) square += cluster.map_shared_rank(mine, r)[0];
        square *= g.rcount;
    }
    const BnChannel k = bn_channel(g, c, square);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    float s[2] = {0.f, 0.f};
#pragma unroll 4
    for (int v = threadIdx.x; v < total; v += 256) Pass::sums(g, k, hx + v * N, hd + v * N, s);
    row_sum<256, 2>(s, sm);
    if (threadIdx.x == 0) { mine[1] = s[0]; mine[2] = s[1]; }
    cluster.sync();
    float s0 = 0.f, s1 = 0.f;
    for (int r = 0; r < size; r++) { s0 += cluster.map_shared_rank(mine, r)[1]; s1 += cluster.map_shared_rank(mine, r)[2]; }
    cluster.barrier_arrive();                                   // its sums are read; waited for at the end: no CTA leaves before
    const float dw = bn_gradients(g, k, s0, s1);
    if (rank == 0 && threadIdx.x == 0) { sums[c] = s0; sums[g.C + c] = s1; sums[2 * g.C + c] = square; sums[3 * g.C + c] = dw; }
    const BnDx r = bn_dx(g, k, c, s0, s1, dw);
    planes([&](int v, int64_t at) { Pass::grad(g, k, r, hx + v, hd + v, dx + at); });
    cluster.barrier_wait();
}

// Rows stay in registers up to 8192 columns (32 elements a thread); the host keeps the op-by-op graph for longer ones.
constexpr int kMaxCols = 8192;
// Persistent CTAs: enough rows in flight to cover the latency of a row's reductions, few enough partial rows to fold: no more than
// are resident (two per SM with 16 elements a thread), and beyond one per SM at least four rows for each. [640, 4096] bfloat16 33 ->
// 19 us, [5000, 4096] 67 -> 42, float32 67 -> 59, [16384, 512] 33 -> 23.5.
constexpr int kMostCtas = 8;                                   // per SM, of the forms for up to 1024 columns; four of those beyond
inline int ln_ctas(int64_t rows, int rpc, int per_sm, bool params) {
    const int64_t sms = kNumSMs - sm_reserve();
    int64_t need = (rows + rpc - 1) / rpc;
    if (params) need = std::min(need, std::max(sms, rows / 4));
    return (int)std::max<int64_t>(1, std::min<int64_t>(need, sms * per_sm));
}

template <typename T, int N, int GROUP, int E>
int launch_ln(const T* x, const T* dy, const float* gamma, T* dx, float* params, float* partial, int64_t rows, int cols, float eps, int ctas, cudaStream_t st) {
    const size_t smem = params && GROUP == 32 ? sizeof(float) * 2 * cols : 0;
    if (dx && params) layer_norm_bwd_kernel<T, N, GROUP, E, true, true><<<ctas, cta_of(GROUP), smem, st>>>(x, dy, gamma, dx, partial, rows, cols, eps);
    else if (dx) layer_norm_bwd_kernel<T, N, GROUP, E, true, false><<<ctas, cta_of(GROUP), 0, st>>>(x, dy, gamma, dx, partial, rows, cols, eps);
    else layer_norm_bwd_kernel<T, N, GROUP, E, false, true><<<ctas, cta_of(GROUP), smem, st>>>(x, dy, gamma, dx, partial, rows, cols, eps);
    B200JT_LAUNCH_CHECK();
    if (params) {
        fold_rows_kernel<<<(2 * cols + 31) / 32, 1024, 0, st>>>(partial, params, 2 * cols, ctas);
        B200JT_LAUNCH_CHECK();
    }
    return 0;
}

// A warp to a row of up to 512 columns (256 one by one), a CTA beyond; 16-byte vectors where columns and pointers allow, else one
// element. CTAs as small as the rows: [50000, 768] bfloat16 165 us with 256 threads to the row, 81 with 128, float32 175 and 125;
// [3000, 301] 9.7 and 4.9 with 64. Ragged rows: [60000, 301] 173 us with 256 threads, 65 with a warp, whose parameter sums a CTA adds
// one warp after the other (10 us: worth it from some 8000 rows on); [100000, 1001] 350 with 256 threads, 369 with 128.
template <typename T, int V>
int run_ln(const T* x, const T* dy, const float* gamma, T* dx, float* params, float* partial, int64_t rows, int cols, float eps, cudaStream_t st) {
    const bool vec = cols % V == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)dy % 16 == 0 && (uintptr_t)dx % 16 == 0 && (uintptr_t)gamma % 16 == 0;
#define B200JT_LN(GROUP, E)                                                                                                      \
    do { const int ctas = ln_ctas(rows, cta_of(GROUP) / GROUP, E > (params ? 8 : 16) ? 2 : 4, params);                           \
         return vec ? launch_ln<T, V, GROUP, E>(x, dy, gamma, dx, params, partial, rows, cols, eps, ctas, st)                    \
                    : launch_ln<T, 1, GROUP, E>(x, dy, gamma, dx, params, partial, rows, cols, eps, ctas, st); } while (0)
    if (cols <= 256) B200JT_LN(32, 8);
    if (cols <= 512 && (vec || rows >= 8192)) B200JT_LN(32, 16);
    if (cols <= 512) return launch_ln<T, 1, 64, 8>(x, dy, gamma, dx, params, partial, rows, cols, eps, ln_ctas(rows, 1, kMostCtas, params), st);
    if (cols <= 1024 && vec) return launch_ln<T, V, 128, 8>(x, dy, gamma, dx, params, partial, rows, cols, eps, ln_ctas(rows, 1, kMostCtas, params), st);
    if (cols <= 1024) return launch_ln<T, 1, 256, 4>(x, dy, gamma, dx, params, partial, rows, cols, eps, ln_ctas(rows, 1, 4, params), st);
    if (cols <= 2048) B200JT_LN(256, 8);
    if (cols <= 4096) B200JT_LN(256, 16);
    B200JT_LN(256, 32);
#undef B200JT_LN
}

// As many CTAs as run at once, four per SM; at most a cluster of 8, a plane for each and a vector for each thread.
inline int bn_cluster(const BnArgs& g, int n) {
    int size = 1;
    while (size < 8 && size * 2 * g.C <= 4 * (kNumSMs - sm_reserve()) && size * 2 <= g.N_ && g.N_ / (size * 2) * (g.HW / n) >= 256) size *= 2;
    return size;
}
inline void cluster_launch(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int size, int C, cudaStream_t st) {
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = (unsigned)size; at->val.clusterDim.y = 1; at->val.clusterDim.z = 1;
    cfg->gridDim = dim3(size, C);
    cfg->blockDim = dim3(256);
    cfg->stream = st;
    cfg->attrs = at;
    cfg->numAttrs = 1;
}
template <typename TX, typename TD, int N> constexpr bool can_half = std::is_same<TX, __nv_bfloat16>::value && std::is_same<TD, __nv_bfloat16>::value && N == 8;
template <typename TX, typename TD, int N> inline bool half_steps(const BnArgs& g) { return can_half<TX, TD, N> && g.round == 2; }
// A layer is held with four CTAs to an SM where a cluster of 8 allows it, and with two at the least (bfloat16 256 x 256 x 28 x 28,
// 98 KB each: 135 us, 149 in two kernels; float32 128 x 128 x 28 x 28: 55 and 63); one alone would load, add and store in turn.
constexpr int64_t kHeldWanted = 55 << 10, kHeldMost = 112 << 10;

template <typename TX, typename TD, int N>
int launch_bn_sums(const b200jt_tensor* x, const b200jt_tensor* dy, float* sums, const BnArgs& g, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    cluster_launch(&cfg, &at, bn_cluster(g, N), g.C, st);
    B200JT_CUDA(cudaLaunchKernelEx(&cfg, half_steps<TX, TD, N>(g) ? bn_bwd_sums_kernel<TX, TD, N, can_half<TX, TD, N>> : bn_bwd_sums_kernel<TX, TD, N, false>, (const TX*)x->ptr, (const TD*)dy->ptr, sums, g));
    return 0;
}

template <typename TX, typename TD, int V>
int run_bn_sums(const b200jt_tensor* x, const b200jt_tensor* dy, float* sums, const BnArgs& g, cudaStream_t st) {
    const bool vec = g.HW % V == 0 && (uintptr_t)x->ptr % 16 == 0 && (uintptr_t)dy->ptr % 16 == 0;
    return vec ? launch_bn_sums<TX, TD, V>(x, dy, sums, g, st) : launch_bn_sums<TX, TD, 1>(x, dy, sums, g, st);
}

template <typename TX, typename TD, int V>
int run_bn_dx(const b200jt_tensor* x, const b200jt_tensor* dy, const float* sums, const b200jt_tensor* dx, const BnArgs& g, cudaStream_t st) {
    const bool vec = g.HW % V == 0 && (uintptr_t)x->ptr % 16 == 0 && (uintptr_t)dy->ptr % 16 == 0 && (uintptr_t)dx->ptr % 16 == 0;
    const int64_t n = (int64_t)g.N_ * g.C * g.HW / (vec ? V : 1);
    const unsigned grid = grid_for(n, 256, 6);
    const size_t smem = sizeof(float) * 4 * g.C;
    if (vec && half_steps<TX, TD, V>(g)) bn_bwd_dx_kernel<TX, TD, V, can_half<TX, TD, V>><<<grid, 256, smem, st>>>((const TX*)x->ptr, (const TD*)dy->ptr, sums, (TX*)dx->ptr, g);
    else if (vec) bn_bwd_dx_kernel<TX, TD, V, false><<<grid, 256, smem, st>>>((const TX*)x->ptr, (const TD*)dy->ptr, sums, (TX*)dx->ptr, g);
    else bn_bwd_dx_kernel<TX, TD, 1, false><<<grid, 256, smem, st>>>((const TX*)x->ptr, (const TD*)dy->ptr, sums, (TX*)dx->ptr, g);
    B200JT_LAUNCH_CHECK();
    return 0;
}

// `held`: whether shared memory holds the layer; if not, nothing was launched (the return value is 0 or a CUDA error, which may be 1)
template <typename TX, typename TD, int N>
int launch_bn_held(const b200jt_tensor* x, const b200jt_tensor* dy, float* sums, const b200jt_tensor* dx, const BnArgs& g, cudaStream_t st, bool* held) {
    const int64_t plane = g.HW * (int64_t)(sizeof(TX) + sizeof(TD));
    int size = bn_cluster(g, N);
    while (size < 8 && size * 2 <= g.N_ && (g.N_ + size - 1) / size * plane > kHeldWanted) size *= 2;
    const int64_t smem = (g.N_ + size - 1) / size * plane + 16;
    *held = smem <= kHeldMost;
    if (!*held) return 0;
    const auto kernel = half_steps<TX, TD, N>(g) ? bn_bwd_held_kernel<TX, TD, N, can_half<TX, TD, N>> : bn_bwd_held_kernel<TX, TD, N, false>;
    static const cudaError_t attr = [] {
        const cudaError_t e = cudaFuncSetAttribute(bn_bwd_held_kernel<TX, TD, N, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kHeldMost);
        return e != cudaSuccess ? e : cudaFuncSetAttribute(bn_bwd_held_kernel<TX, TD, N, can_half<TX, TD, N>>, cudaFuncAttributeMaxDynamicSharedMemorySize, kHeldMost);
    }();
    B200JT_CUDA(attr);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    cluster_launch(&cfg, &at, size, g.C, st);
    cfg.dynamicSmemBytes = (size_t)smem;
    B200JT_CUDA(cudaLaunchKernelEx(&cfg, kernel, (const TX*)x->ptr, (const TD*)dy->ptr, sums, (TX*)dx->ptr, g));
    return 0;
}

template <typename TX, typename TD, int V>
int run_bn(const b200jt_tensor* x, const b200jt_tensor* dy, float* sums, const b200jt_tensor* dx, const BnArgs& g, cudaStream_t st) {
    const bool vec = g.HW % V == 0 && ((uintptr_t)x->ptr | (uintptr_t)dy->ptr | (uintptr_t)dx->ptr) % 16 == 0;
    bool held;
    int rc = vec ? launch_bn_held<TX, TD, V>(x, dy, sums, dx, g, st, &held) : launch_bn_held<TX, TD, 1>(x, dy, sums, dx, g, st, &held);
    if (rc || held) return rc;
    rc = run_bn_sums<TX, TD, V>(x, dy, sums, g, st);
    return rc ? rc : run_bn_dx<TX, TD, V>(x, dy, sums, dx, g, st);
}

inline bool f32_or_bf16(int dt) { return dt == B200JT_FLOAT32 || dt == B200JT_BFLOAT16; }

int bn_args(const b200jt_tensor* x, const b200jt_tensor* dy, const float* stats, double count, const float* gamma, const float* beta,
            double eps, int relu, BnArgs* g) {
    B200JT_CHECK_ARG(valid_tensor(x) && valid_tensor(dy) && x->ndim >= 2, "x and dy must be [N, C, ...]");
    B200JT_CHECK_ARG(f32_or_bf16(x->dtype) && f32_or_bf16(dy->dtype) && numel(x) == numel(dy), "x and dy must be float32 or bfloat16 and of one size");
    B200JT_CHECK_ARG(stats && count > 0 && relu >= 0 && relu <= 5, "stats is NULL, count <= 0 or relu not in 0..5");
    *g = BnArgs{stats, gamma, beta, (float)(1.0 / count), (float)eps, relu & 1, relu >> 1, (int)x->shape[0], (int)x->shape[1], 1};
    for (int d = 2; d < x->ndim; d++) g->HW *= x->shape[d];
    B200JT_CHECK_ARG(g->C <= 2048 && g->HW < 0x7fffffff, "at most 2048 channels of 2^31 elements each");
    return 0;
}

}  // namespace nbwd
}  // namespace b200jt

using namespace b200jt;
using namespace b200jt::nbwd;

extern "C" size_t b200jt_layer_norm_backward_workspace(const b200jt_tensor* x, int want_params) {
    if (!valid_tensor(x) || !want_params) return 0;
    const int64_t cols = x->shape[x->ndim - 1], rows = cols ? numel(x) / cols : 0;
    if (cols < 1 || cols > kMaxCols || rows < 1) return 0;
    return sizeof(float) * 2 * cols * (size_t)ln_ctas(rows, 1, cols <= 1024 ? kMostCtas : 4, true);
}

extern "C" int b200jt_layer_norm_backward(const b200jt_tensor* x, const b200jt_tensor* gamma, const b200jt_tensor* dy, const b200jt_tensor* dx,
                                          float* params, double eps, void* workspace, size_t workspace_bytes, void* stream) {
    B200JT_CHECK_ARG(valid_tensor(x) && valid_tensor(dy) && f32_or_bf16(x->dtype) && dy->dtype == x->dtype && numel(dy) == numel(x),
                     "x and dy must both be float32 or bfloat16 and of one size");
    B200JT_CHECK_ARG(dx || params, "neither dx nor the parameter gradients are wanted");
    B200JT_CHECK_ARG(!dx || (valid_tensor(dx) && dx->dtype == x->dtype && numel(dx) == numel(x)), "dx must have x's dtype and size");
    const int64_t cols = x->shape[x->ndim - 1], rows = cols ? numel(x) / cols : 0;
    B200JT_CHECK_ARG(cols >= 1 && cols <= kMaxCols && rows >= 1, "1 to 8192 columns");
    B200JT_CHECK_ARG(!gamma || (valid_tensor(gamma) && gamma->dtype == B200JT_FLOAT32 && numel(gamma) == cols), "gamma must be float32 [cols]");
    const size_t need = b200jt_layer_norm_backward_workspace(x, params != nullptr);
    B200JT_CHECK_ARG(workspace_bytes >= need && (need == 0 || workspace), "workspace too small: need " + std::to_string(need) + " bytes");
    const float* gp = gamma ? (const float*)gamma->ptr : nullptr;
    void* dxp = dx ? dx->ptr : nullptr;
    cudaStream_t st = (cudaStream_t)stream;
    if (x->dtype == B200JT_FLOAT32)
        return run_ln<float, 4>((const float*)x->ptr, (const float*)dy->ptr, gp, (float*)dxp, params, (float*)workspace, rows, (int)cols, (float)eps, st);
    using B = __nv_bfloat16;
    return run_ln<B, 8>((const B*)x->ptr, (const B*)dy->ptr, gp, (B*)dxp, params, (float*)workspace, rows, (int)cols, (float)eps, st);
}

extern "C" int b200jt_bn_backward_sums(const b200jt_tensor* x, const b200jt_tensor* dy, const float* stats, double count, const float* gamma,
                                       const float* beta, double eps, int relu, float* sums, void* stream) {
    BnArgs g;
    int rc = bn_args(x, dy, stats, count, gamma, beta, eps, relu, &g);
    if (rc) return rc;
    B200JT_CHECK_ARG(sums && numel(x) > 0, "sums is NULL or x is empty");
    cudaStream_t st = (cudaStream_t)stream;
    using B = __nv_bfloat16;
    if (x->dtype == B200JT_FLOAT32) return dy->dtype == B200JT_FLOAT32 ? run_bn_sums<float, float, 4>(x, dy, sums, g, st) : run_bn_sums<float, B, 8>(x, dy, sums, g, st);
    return dy->dtype == B200JT_FLOAT32 ? run_bn_sums<B, float, 8>(x, dy, sums, g, st) : run_bn_sums<B, B, 8>(x, dy, sums, g, st);
}

extern "C" int b200jt_bn_backward_dx(const b200jt_tensor* x, const b200jt_tensor* dy, const float* stats, double count, const float* gamma,
                                     const float* beta, double eps, int relu, const float* sums, const b200jt_tensor* dx, void* stream) {
    BnArgs g;
    int rc = bn_args(x, dy, stats, count, gamma, beta, eps, relu, &g);
    if (rc) return rc;
    B200JT_CHECK_ARG(sums && numel(x) > 0 && valid_tensor(dx) && dx->dtype == x->dtype && numel(dx) == numel(x), "dx must have x's dtype and size");
    cudaStream_t st = (cudaStream_t)stream;
    using B = __nv_bfloat16;
    if (x->dtype == B200JT_FLOAT32) return dy->dtype == B200JT_FLOAT32 ? run_bn_dx<float, float, 4>(x, dy, sums, dx, g, st) : run_bn_dx<float, B, 8>(x, dy, sums, dx, g, st);
    return dy->dtype == B200JT_FLOAT32 ? run_bn_dx<B, float, 8>(x, dy, sums, dx, g, st) : run_bn_dx<B, B, 8>(x, dy, sums, dx, g, st);
}

extern "C" int b200jt_bn_backward(const b200jt_tensor* x, const b200jt_tensor* dy, const float* stats, double count, const float* gamma,
                                  const float* beta, double eps, int relu, float* sums, const b200jt_tensor* dx, void* stream) {
    BnArgs g;
    int rc = bn_args(x, dy, stats, count, gamma, beta, eps, relu, &g);
    if (rc) return rc;
    B200JT_CHECK_ARG(sums && numel(x) > 0 && valid_tensor(dx) && dx->dtype == x->dtype && numel(dx) == numel(x), "sums is NULL, x is empty or dx has not x's dtype and size");
    cudaStream_t st = (cudaStream_t)stream;
    using B = __nv_bfloat16;
    if (x->dtype == B200JT_FLOAT32) return dy->dtype == B200JT_FLOAT32 ? run_bn<float, float, 4>(x, dy, sums, dx, g, st) : run_bn<float, B, 8>(x, dy, sums, dx, g, st);
    return dy->dtype == B200JT_FLOAT32 ? run_bn<B, float, 8>(x, dy, sums, dx, g, st) : run_bn<B, B, 8>(x, dy, sums, dx, g, st);
}
