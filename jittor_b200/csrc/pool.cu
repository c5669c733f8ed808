// 2-D pooling, forward and backward: the kernels `Pool.execute` builds with jt.code in the reference
// (python/jittor/pool.py:54-95 forward body, :96-118 backward body) as fixed sm_100a kernels.
//
// Window of output (oh, ow): rows [oh*sh - ph, oh*sh - ph + kh) x columns [ow*sw - pw, ow*sw - pw + kw), clipped to the
// input (padding is never read). maximum / minimum fold the clipped window starting from the op's init value; mean
// divides the clipped sum by kh*kw (count_include_pad) or by the clipped area.
// Backward: the reference scatters with atomicAdd, one thread per window; for maximum / minimum only the FIRST element
// of the window (row-major scan) that equals the pooled value receives the gradient. Here every INPUT element gathers
// from the windows that contain it instead (at most ceil(kh/sh) * ceil(kw/sw) of them), re-deriving "am I the first
// match" by scanning the part of the window that precedes it: no atomics, no zero fill, deterministic.
#include "atomic_ops.cuh"

#include <algorithm>
#include <type_traits>

namespace b200jt {
namespace pool {

struct Geo {
    int N, C, H, W, OH, OW, kh, kw, sh, sw, ph, pw;
    int count_include_pad;
};

template <typename T> struct AccOf { using type = float; };
template <> struct AccOf<double> { using type = double; };

template <typename T> __device__ __forceinline__ typename AccOf<T>::type ld(const T* p) { return (typename AccOf<T>::type)(*p); }
template <> __device__ __forceinline__ float ld<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <> __device__ __forceinline__ float ld<__half>(const __half* p) { return __half2float(*p); }
template <typename T, typename A> __device__ __forceinline__ T cvt(A v) { return (T)v; }
template <> __device__ __forceinline__ __nv_bfloat16 cvt<__nv_bfloat16, float>(float v) { return __float2bfloat16(v); }
template <> __device__ __forceinline__ __half cvt<__half, float>(float v) { return __float2half(v); }

// OP: 0 maximum, 1 minimum, 2 mean. KS: 0 = window and stride read from the geometry record, else a compile-time
// (kernel, stride) pair code so that the window arithmetic folds to constants for the common layers:
// 1: 2x2 stride 2, 2: 3x3 stride 2, 3: 3x3 stride 1.
template <int KS> struct Win {
    __device__ __forceinline__ static int kh(const Geo& g) { return KS == 1 ? 2 : KS >= 2 ? 3 : g.kh; }
    __device__ __forceinline__ static int kw(const Geo& g) { return KS == 1 ? 2 : KS >= 2 ? 3 : g.kw; }
    __device__ __forceinline__ static int sh(const Geo& g) { return KS == 1 || KS == 2 ? 2 : KS == 3 ? 1 : g.sh; }
    __device__ __forceinline__ static int sw(const Geo& g) { return KS == 1 || KS == 2 ? 2 : KS == 3 ? 1 : g.sw; }
};

// Thread layout of both kernels: blockDim (32, 8) covers 32 columns x 8 rows of one image plane, blockIdx.z walks the
// N*C planes (grid-stride), so no division is needed to find a thread's coordinates.
template <typename T, int OP, int KS>
__global__ void __launch_bounds__(256) pool_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, int32_t* __restrict__ indices,
                                                       uint8_t* __restrict__ taps, Geo g, T init) {
    using A = typename AccOf<T>::type;
    using Wn = Win<KS>;
    const int ow = blockIdx.x * 32 + threadIdx.x, oh = blockIdx.y * 8 + threadIdx.y;
    if (ow >= g.OW || oh >= g.OH) return;
    int p0 = oh * Wn::sh(g) - g.ph, q0 = ow * Wn::sw(g) - g.pw;
    const int p1 = min(p0 + Wn::kh(g), g.H), q1 = min(q0 + Wn::kw(g), g.W);
    p0 = max(p0, 0); q0 = max(q0, 0);
    const int64_t planes = (int64_t)g.N * g.C;
    for (int64_t nc = blockIdx.z; nc < planes; nc += gridDim.z) {
        const T* xp = x + nc * (int64_t)g.H * g.W;
        const int64_t o = (nc * g.OH + oh) * g.OW + ow;
        if (KS != 0) {
            // compile-time window: all loads of PL planes are issued before the first use (a rolled loop would wait
            // for every element in turn; one plane alone leaves too few bytes in flight), out-of-range taps predicated
            constexpr int KH = KS == 1 ? 2 : 3, KW = KH, PL = 4;
            const int pb = oh * Wn::sh(g) - g.ph, qb = ow * Wn::sw(g) - g.pw;
            A vals[PL][KH * KW];
            bool ok[KH * KW];
#pragma unroll
            for (int a = 0; a < KH; a++)
#pragma unroll
                for (int b = 0; b < KW; b++)
                    ok[a * KW + b] = (unsigned)(pb + a) < (unsigned)g.H && (unsigned)(qb + b) < (unsigned)g.W;
#pragma unroll
            for (int u = 0; u < PL; u++) {
                const int64_t pl = nc + (int64_t)u * gridDim.z;
                const T* xu = x + pl * (int64_t)g.H * g.W;
#pragma unroll
                for (int t = 0; t < KH * KW; t++)
                    vals[u][t] = (ok[t] && pl < planes) ? ld<T>(xu + (int64_t)(pb + t / KW) * g.W + qb + t % KW) : (A)0;
            }
#pragma unroll
            for (int u = 0; u < PL; u++) {
                const int64_t pl = nc + (int64_t)u * gridDim.z;
                if (pl >= planes) break;
                const int64_t ou = (pl * g.OH + oh) * g.OW + ow;
                if (OP == 2) {
                    A acc = 0;
#pragma unroll
                    for (int t = 0; t < KH * KW; t++) acc += vals[u][t];
                    const int count = g.count_include_pad ? KH * KW : (p1 - p0) * (q1 - q0);
                    y[ou] = cvt<T, A>(acc / (A)count);
                } else {
                    A best = ld<T>(&init);
                    int tap = -1;
#pragma unroll
                    for (int t = 0; t < KH * KW; t++)
                        if (ok[t] && (OP == 0 ? best < vals[u][t] : vals[u][t] < best)) { best = vals[u][t]; tap = t; }
                    y[ou] = cvt<T, A>(best);
                    if (indices) indices[ou] = tap < 0 ? -1 : (pb + tap / KW) * g.W + qb + tap % KW;
                    if (taps) taps[ou] = tap < 0 ? 255 : (uint8_t)tap;
                }
            }
            nc += (int64_t)(PL - 1) * gridDim.z;
            continue;
        }
        if (OP == 2) {
            A acc = 0;
            for (int p = p0; p < p1; p++)
                for (int q = q0; q < q1; q++) acc += ld<T>(xp + (int64_t)p * g.W + q);
            const int count = g.count_include_pad ? Wn::kh(g) * Wn::kw(g) : (p1 - p0) * (q1 - q0);
            y[o] = cvt<T, A>(acc / (A)count);
        } else {
            A best = ld<T>(&init);
            int where = -1, tap = 255;
            for (int p = p0; p < p1; p++)
                for (int q = q0; q < q1; q++) {
                    const A v = ld<T>(xp + (int64_t)p * g.W + q);
                    // a strict comparison keeps the first extreme element, as the reference's index variant does
                    if (OP == 0 ? best < v : v < best) { best = v; where = p * g.W + q; tap = (p - oh * g.sh + g.ph) * g.kw + q - ow * g.sw + g.pw; }
                }
            y[o] = cvt<T, A>(best);
            if (indices) indices[o] = where;
            if (taps) taps[o] = (uint8_t)tap;
        }
    }
}

template <typename T, int OP, int KS>
__global__ void __launch_bounds__(256) pool_bwd_kernel(const T* __restrict__ x, const T* __restrict__ y, const T* __restrict__ dy,
                                                       T* __restrict__ dx, Geo g) {
    using A = typename AccOf<T>::type;
    using Wn = Win<KS>;
    const int q = blockIdx.x * 32 + threadIdx.x, p = blockIdx.y * 8 + threadIdx.y;
    if (q >= g.W || p >= g.H) return;
    const int kh = Wn::kh(g), kw = Wn::kw(g), sh = Wn::sh(g), sw = Wn::sw(g);
    // windows containing row p: oh*sh - ph <= p < oh*sh - ph + kh
    const int oh_lo = max(0, (p + g.ph - kh + sh) / sh), oh_hi = min(g.OH - 1, (p + g.ph) / sh);
    const int ow_lo = max(0, (q + g.pw - kw + sw) / sw), ow_hi = min(g.OW - 1, (q + g.pw) / sw);
    const int64_t planes = (int64_t)g.N * g.C;
    for (int64_t nc = blockIdx.z; nc < planes; nc += gridDim.z) {
        const T* xp = x + nc * (int64_t)g.H * g.W;
        const T* yp = y + nc * (int64_t)g.OH * g.OW;
        const T* dp = dy + nc * (int64_t)g.OH * g.OW;
        const A mine = ld<T>(xp + (int64_t)p * g.W + q);
        A acc = 0;
        if (KS != 0) {
            // at most NW x NW windows contain this element; their pooled values and gradients are fetched up front
            constexpr int NW = KS == 1 ? 1 : KS == 2 ? 2 : 3;
            A yv[NW * NW], dv[NW * NW];
            bool in[NW * NW];
#pragma unroll
            for (int a = 0; a < NW; a++)
#pragma unroll
                for (int b = 0; b < NW; b++) {
                    const int oh = oh_lo + a, ow = ow_lo + b;
                    in[a * NW + b] = oh <= oh_hi && ow <= ow_hi;
                    const int64_t o = (int64_t)oh * g.OW + ow;
                    yv[a * NW + b] = in[a * NW + b] && OP != 2 ? ld<T>(yp + o) : (A)0;
                    dv[a * NW + b] = in[a * NW + b] ? ld<T>(dp + o) : (A)0;
                }
#pragma unroll
            for (int a = 0; a < NW; a++)
#pragma unroll
                for (int b = 0; b < NW; b++) {
                    if (!in[a * NW + b]) continue;
                    const int oh = oh_lo + a, ow = ow_lo + b;
                    int p0 = oh * sh - g.ph, q0 = ow * sw - g.pw;
                    const int p1 = min(p0 + kh, g.H), q1 = min(q0 + kw, g.W);
                    p0 = max(p0, 0); q0 = max(q0, 0);
                    if (OP == 2) {
                        const int count = g.count_include_pad ? kh * kw : (p1 - p0) * (q1 - q0);
                        acc += dv[a * NW + b] / (A)count;
                    } else {
                        if (!(mine == yv[a * NW + b])) continue;
                        bool first = true;
                        for (int pp = p0; pp <= p && first; pp++) {
                            const int qe = pp == p ? q : q1;
                            for (int qq = q0; qq < qe; qq++)
                                if (ld<T>(xp + (int64_t)pp * g.W + qq) == mine) { first = false; break; }
                        }
                        if (first) acc += dv[a * NW + b];
                    }
                }
            dx[(nc * g.H + p) * (int64_t)g.W + q] = cvt<T, A>(acc);
            continue;
        }
        for (int oh = oh_lo; oh <= oh_hi; oh++) {
            int p0 = oh * sh - g.ph;
            const int p1 = min(p0 + kh, g.H);
            p0 = max(p0, 0);
            if (p < p0 || p >= p1) continue;
            for (int ow = ow_lo; ow <= ow_hi; ow++) {
                int q0 = ow * sw - g.pw;
                const int q1 = min(q0 + kw, g.W);
                q0 = max(q0, 0);
                if (q < q0 || q >= q1) continue;
                if (OP == 2) {
                    const int count = g.count_include_pad ? kh * kw : (p1 - p0) * (q1 - q0);
                    acc += ld<T>(dp + (int64_t)oh * g.OW + ow) / (A)count;
                } else {
                    const A v = ld<T>(yp + (int64_t)oh * g.OW + ow);
                    if (!(mine == v)) continue;
                    bool first = true;
                    for (int pp = p0; pp <= p && first; pp++) {
                        const int qe = pp == p ? q : q1;
                        for (int qq = q0; qq < qe; qq++)
                            if (ld<T>(xp + (int64_t)pp * g.W + qq) == v) { first = false; break; }
                    }
                    if (first) acc += ld<T>(dp + (int64_t)oh * g.OW + ow);
                }
            }
        }
        dx[(nc * g.H + p) * (int64_t)g.W + q] = cvt<T, A>(acc);
    }
}

// Backward of maximum / minimum from the forward's index map: input element (p, q) receives dy of every window whose
// recorded first extreme element it is. No comparison of values, no scan, and x is not read at all. I: int32_t, an index into
// the plane, or uint8_t, a place in the window.
template <typename T, typename I, int KS>
__global__ void __launch_bounds__(256) pool_bwd_indices_kernel(const I* __restrict__ idx, const T* __restrict__ dy,
                                                               T* __restrict__ dx, Geo g) {
    using A = typename AccOf<T>::type;
    using Wn = Win<KS>;
    const int q = blockIdx.x * 32 + threadIdx.x, p = blockIdx.y * 8 + threadIdx.y;
    if (q >= g.W || p >= g.H) return;
    const int kh = Wn::kh(g), kw = Wn::kw(g), sh = Wn::sh(g), sw = Wn::sw(g);
    const int oh_lo = max(0, (p + g.ph - kh + sh) / sh), oh_hi = min(g.OH - 1, (p + g.ph) / sh);
    const int ow_lo = max(0, (q + g.pw - kw + sw) / sw), ow_hi = min(g.OW - 1, (q + g.pw) / sw);
    constexpr bool TAP = sizeof(I) == 1;
    auto me = [&](int oh, int ow) { return TAP ? (p - oh * sh + g.ph) * kw + q - ow * sw + g.pw : p * g.W + q; };
    const int64_t planes = (int64_t)g.N * g.C;
    constexpr int PL = 4;
    for (int64_t nc = blockIdx.z; nc < planes; nc += (int64_t)PL * gridDim.z) {
        A acc[PL];
#pragma unroll
        for (int u = 0; u < PL; u++) acc[u] = 0;
        if (KS != 0) {
            constexpr int NW = KS == 1 ? 1 : KS == 2 ? 2 : 3;
            int iv[PL][NW * NW];
            A dv[PL][NW * NW];
#pragma unroll
            for (int u = 0; u < PL; u++) {
                const int64_t pl = nc + (int64_t)u * gridDim.z;
#pragma unroll
                for (int a = 0; a < NW; a++)
#pragma unroll
                    for (int b = 0; b < NW; b++) {
                        const int oh = oh_lo + a, ow = ow_lo + b;
                        const bool in = oh <= oh_hi && ow <= ow_hi && pl < planes;
                        const int64_t o = (pl * g.OH + oh) * g.OW + ow;
                        iv[u][a * NW + b] = in ? idx[o] : -2;
                        dv[u][a * NW + b] = in ? ld<T>(dy + o) : (A)0;
                    }
            }
#pragma unroll
            for (int u = 0; u < PL; u++)
#pragma unroll
                for (int t = 0; t < NW * NW; t++) if (iv[u][t] == me(oh_lo + t / NW, ow_lo + t % NW)) acc[u] += dv[u][t];
        } else {
            for (int u = 0; u < PL; u++) {
                const int64_t pl = nc + (int64_t)u * gridDim.z;
                if (pl >= planes) break;
                for (int oh = oh_lo; oh <= oh_hi; oh++)
                    for (int ow = ow_lo; ow <= ow_hi; ow++) {
                        const int64_t o = (pl * g.OH + oh) * g.OW + ow;
                        if (idx[o] == me(oh, ow)) acc[u] += ld<T>(dy + o);
                    }
            }
        }
#pragma unroll
        for (int u = 0; u < PL; u++) {
            const int64_t pl = nc + (int64_t)u * gridDim.z;
            if (pl < planes) dx[(pl * g.H + p) * (int64_t)g.W + q] = cvt<T, A>(acc[u]);
        }
    }
}

static int window_code(const Geo& g) {
    if (g.kh == 2 && g.kw == 2 && g.sh == 2 && g.sw == 2) return 1;
    if (g.kh == 3 && g.kw == 3 && g.sh == 2 && g.sw == 2) return 2;
    if (g.kh == 3 && g.kw == 3 && g.sh == 1 && g.sw == 1) return 3;
    return 0;
}

// ---- tiles: 2x2 stride 2, 3x3 stride 2 and 3x3 stride 1 windows, padding 0 or 1 ---------------------------------------
// A thread makes a tile of RU x VO outputs (forward) or the RU*S x VO*S inputs under it (backward) of one plane. Both are
// bound by memory if the arithmetic stays out of the way, so: neighbouring lanes read and write neighbouring 16-byte vectors
// where the rows' length and the pointers allow (VO outputs = S * VO inputs = 16 bytes, halved until it divides the rows; two
// vectors a lane were 10 % slower, single elements two apart a third of the speed), an input row is folded once and its result
// shared by the windows above and below, the place of a maximum comes from comparisons with the 3-input maximum, and the
// position of the first extreme element is kept as ONE byte (its place in the window) instead of a 4-byte index -- the map
// is written forward and read backward, 103 MB each way for [64,128,112,112] with int32. 3x3 s2 p1 on that shape, float32:
// forward 0.142 -> 0.091 ms, backward 0.161 -> 0.086 ms (0.96 of HBM).
template <typename T, int N> __device__ __forceinline__ void load_n(const T* p, float* o) {
    if constexpr (N == 1) o[0] = ld<T>(p);
    else if constexpr (sizeof(T) * N > 16) { load_n<T, N / 2>(p, o); load_n<T, N / 2>(p + N / 2, o + N / 2); }
    else {
        struct alignas(sizeof(T) * N) Pack { T v[N]; };
        const Pack k = *reinterpret_cast<const Pack*>(p);
#pragma unroll
        for (int i = 0; i < N; i++) o[i] = ld<T>(&k.v[i]);
    }
}
template <typename T, int N> __device__ __forceinline__ void store_n(T* p, const float* o) {
    if constexpr (N == 1) *p = cvt<T, float>(o[0]);
    else if constexpr (sizeof(T) * N > 16) { store_n<T, N / 2>(p, o); store_n<T, N / 2>(p + N / 2, o + N / 2); }
    else {
        struct alignas(sizeof(T) * N) Pack { T v[N]; } k;
#pragma unroll
        for (int i = 0; i < N; i++) k.v[i] = cvt<T, float>(o[i]);
        *reinterpret_cast<Pack*>(p) = k;
    }
}
// N elements of a row from column c, of which the columns outside [0, w) read as `pad`; A: elements per access
template <typename T, int N, int A> __device__ __forceinline__ void load_row(const T* row, int c, int w, bool live, float pad, float* o) {
#pragma unroll
    for (int i = 0; i < N; i += A) {
        if (live && c + i < w) load_n<T, A>(row + c + i, o + i);
        else {
#pragma unroll
            for (int e = 0; e < A; e++) o[i + e] = pad;
        }
    }
}

// output rows of a tile: enough loads in flight without running out of registers. Forward, float32 3x3 s2 p1 on [64,128,112,112]: 102 us
// with 4 rows and 88 registers, 91 with 2 and 48; single outputs a thread (57 x 57) 43 with 4 and 47 with 2.
constexpr int rows_up(int vo) { return vo >= 4 ? 2 : 4; }
constexpr int rows_up_fwd(int vo) { return vo >= 2 ? 2 : 4; }
struct TileMap {                                // flat thread index -> (plane, tile row, tile column)
    int cols, rows;
    int64_t threads;
    __device__ __forceinline__ bool at(int64_t i, int64_t& plane, int& r, int& c) const {
        if (i >= threads) return false;
        if (threads < 0x7fffffff) {
            const unsigned u = (unsigned)i, t = u / (unsigned)cols, p = t / (unsigned)rows;
            c = (int)(u - t * (unsigned)cols);
            r = (int)(t - p * (unsigned)rows);
            plane = p;
        } else {
            const int64_t t = i / cols;
            c = (int)(i - t * cols);
            plane = t / rows;
            r = (int)(t - plane * rows);
        }
        return true;
    }
};

// MEAN divides by K * K; else maximum, or minimum as the maximum of the negated values (sign = -1). VO: outputs a lane makes in
// a row and per access of y and the map; AX: elements per access of x.
template <typename T, bool MEAN, int K, int S, int PAD, int VO, int AX>
__global__ void __launch_bounds__(256) pool_fwd_tile_kernel(const T* __restrict__ x, T* __restrict__ y, int32_t* __restrict__ indices,
                                                            uint8_t* __restrict__ taps, const Geo g, const TileMap map, float init, float sign) {
    constexpr int RU = rows_up_fwd(VO), ROWS = (RU - 1) * S + K, SPAN = (VO - 1) * S + K;
    constexpr int RIGHT = SPAN - PAD - VO * S > 0 ? SPAN - PAD - VO * S : 0;
    int64_t plane;
    int r, c;
    if (!map.at(blockIdx.x * 256ll + threadIdx.x, plane, r, c)) return;
    const int oh0 = r * RU, ow0 = c * VO, p0 = oh0 * S - PAD, q0 = ow0 * S;
    const T* xp = x + plane * (int64_t)g.H * g.W;
    const float pad = MEAN ? 0.f : init * sign;           // as it stands in x
    float h[ROWS][VO];
    int ht[ROWS][VO];
#pragma unroll
    for (int a = 0; a < ROWS; a++) {
        const int p = p0 + a;
        const bool live = (unsigned)p < (unsigned)g.H;
        const T* row = xp + (int64_t)p * g.W;
        float v[PAD + VO * S + RIGHT];
        if (PAD) v[0] = live && q0 > 0 ? ld<T>(row + q0 - 1) : pad;
        load_row<T, VO * S, AX>(row, q0, g.W, live, pad, v + PAD);
#pragma unroll
        for (int e = 0; e < RIGHT; e++) v[PAD + VO * S + e] = live && q0 + VO * S + e < g.W ? ld<T>(row + q0 + VO * S + e) : pad;
        if (!MEAN && sign < 0.f)
#pragma unroll
            for (int e = 0; e < PAD + VO * S + RIGHT; e++) v[e] = -v[e];
#pragma unroll
        for (int j = 0; j < VO; j++) {
            if (MEAN) {
                float s = v[j * S];
#pragma unroll
                for (int b = 1; b < K; b++) s += v[j * S + b];
                h[a][j] = s;
            } else {
                float m = v[j * S];
#pragma unroll
                for (int b = 1; b < K; b++) m = fmaxf(m, v[j * S + b]);
                int tap = K - 1;                // the first element that equals the row's maximum
#pragma unroll
                for (int b = K - 2; b >= 0; b--) tap = v[j * S + b] == m ? b : tap;
                h[a][j] = m; ht[a][j] = tap;
            }
        }
    }
#pragma unroll
    for (int u = 0; u < RU; u++) {
        const int oh = oh0 + u;
        if (oh >= g.OH) break;
        float o[VO];
        int t[VO];
#pragma unroll
        for (int j = 0; j < VO; j++) {
            o[j] = h[u * S][j];
#pragma unroll
            for (int a = 1; a < K; a++) {
                if (MEAN) o[j] += h[u * S + a][j];
                else o[j] = fmaxf(o[j], h[u * S + a][j]);
            }
            if (MEAN) o[j] /= (float)(K * K);
            else {
                int tap = (K - 1) * K + ht[u * S + K - 1][j];
#pragma unroll
                for (int a = K - 2; a >= 0; a--) tap = h[u * S + a][j] == o[j] ? a * K + ht[u * S + a][j] : tap;
                const bool found = o[j] > init;                 // fmaxf passes NaN by, as the strict comparisons of the per-element kernel do
                t[j] = found ? tap : 255;
                o[j] = (found ? o[j] : init) * sign;
            }
        }
        const int64_t at = (plane * g.OH + oh) * g.OW + ow0;
        if (ow0 >= g.OW) break;                 // VO divides the row
        store_n<T, VO>(y + at, o);
        if (!MEAN && taps) {
            struct alignas(VO) Bytes { uint8_t v[VO]; } k;
#pragma unroll
            for (int e = 0; e < VO; e++) k.v[e] = (uint8_t)t[e];
            *reinterpret_cast<Bytes*>(taps + at) = k;
        }
        if (!MEAN && indices)
#pragma unroll
            for (int e = 0; e < VO; e++)
                indices[at + e] = t[e] == 255 ? -1 : (oh * S - PAD + t[e] / K) * g.W + (ow0 + e) * S - PAD + t[e] % K;
    }
}

// Inputs under the tile from the windows that reach them: a window's gradient goes to the element its byte names (mean: to
// all of them). Windows are taken in ascending order, so a sum has the bits of the per-element kernels.
template <typename T, bool MEAN, int K, int S, int PAD, int VO, int AX>
__global__ void __launch_bounds__(256) pool_bwd_tile_kernel(const uint8_t* __restrict__ taps, const T* __restrict__ dy, T* __restrict__ dx,
                                                            const Geo g, const TileMap map) {
    constexpr int RU = rows_up(VO), LO = (K - 1 - PAD) / S, HR = (S * RU - 1 + PAD) / S, HC = (S * VO - 1 + PAD) / S;
    int64_t plane;
    int r, c;
    if (!map.at(blockIdx.x * 256ll + threadIdx.x, plane, r, c)) return;
    const int oh0 = r * RU, ow0 = c * VO;
    const int64_t ob = plane * (int64_t)g.OH * g.OW;
    float acc[S * RU][S * VO] = {};
#pragma unroll
    for (int i = -LO; i <= HR; i++) {
        const int oh = oh0 + i;
        const bool live = (unsigned)oh < (unsigned)g.OH;
        const int64_t at = ob + (int64_t)oh * g.OW;
        float d[LO + HC + 1];
        int t[LO + HC + 1];
#pragma unroll
        for (int j = -LO; j <= HC; j++) {
            if (j >= 0 && j < VO) continue;
            const bool in = live && (unsigned)(ow0 + j) < (unsigned)g.OW;
            d[LO + j] = in ? ld<T>(dy + at + ow0 + j) : 0.f;
            if (!MEAN) t[LO + j] = in ? taps[at + ow0 + j] : 255;
        }
        struct alignas(VO) Bytes { uint8_t v[VO]; } k;
#pragma unroll
        for (int e = 0; e < VO; e++) { k.v[e] = 255; d[LO + e] = 0.f; }
        if (live && ow0 < g.OW) {
            load_n<T, VO>(dy + at + ow0, d + LO);
            if (!MEAN) k = *reinterpret_cast<const Bytes*>(taps + at + ow0);
        }
#pragma unroll
        for (int e = 0; e < VO; e++) t[LO + e] = k.v[e];
#pragma unroll
        for (int j = -LO; j <= HC; j++)
#pragma unroll
            for (int a = 0; a < K; a++)
#pragma unroll
                for (int b = 0; b < K; b++) {
                    const int p = i * S + a - PAD, q = j * S + b - PAD;
                    if (p < 0 || p >= S * RU || q < 0 || q >= S * VO) continue;
                    if (MEAN) acc[p][q] += d[LO + j];
                    else if (t[LO + j] == a * K + b) acc[p][q] += d[LO + j];
                }
    }
    T* out = dx + plane * (int64_t)g.H * g.W;
#pragma unroll
    for (int p = 0; p < S * RU; p++) {
        if (oh0 * S + p >= g.H) break;
        if (MEAN)
#pragma unroll
            for (int q = 0; q < S * VO; q++) acc[p][q] /= (float)(K * K);
#pragma unroll
        for (int q = 0; q < S * VO; q += AX)
            if (ow0 * S + q < g.W) store_n<T, AX>(out + (int64_t)(oh0 * S + p) * g.W + ow0 * S + q, acc[p] + q);
    }
}

// a mean over K * K elements everywhere: padding counts, or no window leaves the input
inline bool whole_mean(const Geo& g) {
    return g.count_include_pad || (g.ph == 0 && g.pw == 0 && (g.OH - 1) * g.sh + g.kh <= g.H && (g.OW - 1) * g.sw + g.kw <= g.W);
}
// Whether the tile kernels take a layer; rows and columns beyond what the outputs cover still get their zero gradient.
template <typename T> bool tiled(const Geo& g) {
    return (int64_t)g.N * g.C * g.H * g.W < (1LL << 38) && sizeof(T) <= 4 && window_code(g) != 0 && g.ph == g.pw && g.ph <= 1 &&
           (window_code(g) != 1 || g.ph == 0);
}

static dim3 plane_grid(int w, int h, int64_t planes) {
    const unsigned gx = (unsigned)((w + 31) / 32), gy = (unsigned)((h + 7) / 8);
    // enough plane slices to fill the machine a few times over, each block then strides over the remaining planes
    const int64_t want = ((int64_t)kNumSMs * 16 + (int64_t)gx * gy - 1) / ((int64_t)gx * gy);
    const unsigned gz = (unsigned)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(planes, 65535), want));
    return dim3(gx, gy, gz);
}

static int parse(const b200jt_tensor* x, const b200jt_tensor* y, const char* op, int kh, int kw, int sh, int sw, int ph, int pw,
                 int count_include_pad, Geo* g, int* opc) {
    B200JT_CHECK_ARG(valid_tensor(x) && valid_tensor(y) && x->ndim == 4 && y->ndim == 4, "pool2d takes NCHW tensors");
    B200JT_CHECK_ARG(x->dtype == y->dtype, "x and y must have the same dtype");
    B200JT_CHECK_ARG(kh > 0 && kw > 0, "kernel_size must be greater than zero");
    B200JT_CHECK_ARG(sh > 0 && sw > 0, "stride must be greater than zero");
    B200JT_CHECK_ARG(ph >= 0 && pw >= 0, "padding must be non-negative");
    B200JT_CHECK_ARG(x->shape[0] == y->shape[0] && x->shape[1] == y->shape[1], "batch / channel mismatch between x and y");
    B200JT_CHECK_ARG(op != nullptr, "op is null");
    *opc = !strcmp(op, "maximum") ? 0 : !strcmp(op, "minimum") ? 1 : !strcmp(op, "mean") ? 2 : -1;
    B200JT_CHECK_ARG(*opc >= 0, std::string("pool2d op must be maximum, minimum or mean, got '") + op + "'");
    for (int d = 0; d < 4; d++)
        B200JT_CHECK_ARG(x->shape[d] < (1LL << 31) && y->shape[d] < (1LL << 31), "dimension too large");
    g->N = (int)x->shape[0]; g->C = (int)x->shape[1]; g->H = (int)x->shape[2]; g->W = (int)x->shape[3];
    g->OH = (int)y->shape[2]; g->OW = (int)y->shape[3];
    g->kh = kh; g->kw = kw; g->sh = sh; g->sw = sw; g->ph = ph; g->pw = pw; g->count_include_pad = count_include_pad;
    return 0;
}

// f(integral constants K, S, PAD, VO, AX) for the layer's window and the widest accesses its rows allow: x / y stand for the
// pointers rows of W and of OW elements are read or written at, m for the map of one byte per output.
template <typename T, typename F> void dispatch_tile(const Geo& g, const void* x, const void* y, const void* m, F&& f) {
    const int s = window_code(g) == 3 ? 1 : 2;
    int vo = 16 / (s * (int)sizeof(T));
    while (vo > 1 && (g.W % (s * vo) || g.OW % vo || (uintptr_t)x % (s * vo * sizeof(T)) || (uintptr_t)y % (vo * sizeof(T)) || (uintptr_t)m % vo)) vo /= 2;
    const bool pair = s == 1 || (g.W % 2 == 0 && (uintptr_t)x % (2 * sizeof(T)) == 0);
#define B200JT_POOL(K, S, P, VO, AX) return f(std::integral_constant<int, K>(), std::integral_constant<int, S>(), std::integral_constant<int, P>(), std::integral_constant<int, VO>(), std::integral_constant<int, AX>())
#define B200JT_POOL2(K, P)                                                                                             \
    do { if constexpr (sizeof(T) == 2) if (vo == 4) B200JT_POOL(K, 2, P, 4, 8);                                        \
         if (vo == 2) B200JT_POOL(K, 2, P, 2, 4);                                                                      \
         if (pair) B200JT_POOL(K, 2, P, 1, 2);                                                                         \
         B200JT_POOL(K, 2, P, 1, 1); } while (0)
#define B200JT_POOL1(P)                                                                                                \
    do { if constexpr (sizeof(T) == 2) if (vo == 8) B200JT_POOL(3, 1, P, 8, 8);                                        \
         if (vo == 4) B200JT_POOL(3, 1, P, 4, 4);                                                                      \
         if (vo == 2) B200JT_POOL(3, 1, P, 2, 2);                                                                      \
         B200JT_POOL(3, 1, P, 1, 1); } while (0)
    switch (window_code(g)) {
        case 1: B200JT_POOL2(2, 0);
        case 2: if (g.ph) B200JT_POOL2(3, 1); B200JT_POOL2(3, 0);
        default: if (g.ph) B200JT_POOL1(1); B200JT_POOL1(0);
    }
#undef B200JT_POOL1
#undef B200JT_POOL2
#undef B200JT_POOL
}
static TileMap tile_map(const Geo& g, int h, int w, int th, int tw) {
    TileMap m;
    m.rows = (h + th - 1) / th; m.cols = (w + tw - 1) / tw;
    m.threads = (int64_t)g.N * g.C * m.rows * m.cols;
    return m;
}

template <typename T, int OP>
static void launch_fwd(const T* xp, T* yp, int32_t* indices, uint8_t* taps, const Geo& g, T init, cudaStream_t st) {
    if constexpr (sizeof(T) <= 4) {
        if (tiled<T>(g) && (OP != 2 || whole_mean(g))) {
            float init_f;
            if constexpr (std::is_same_v<T, float>) init_f = init;
            else if constexpr (std::is_same_v<T, __half>) init_f = __half2float(init);
            else init_f = __bfloat162float(init);
            const float sign = OP == 1 ? -1.f : 1.f;
            dispatch_tile<T>(g, xp, yp, taps, [&](auto k, auto s, auto p, auto vo, auto ax) {
                const TileMap m = tile_map(g, g.OH, g.OW, rows_up_fwd(vo()), vo());
                pool_fwd_tile_kernel<T, OP == 2, k(), s(), p(), vo(), ax()><<<(unsigned)((m.threads + 255) / 256), 256, 0, st>>>(
                    xp, yp, indices, taps, g, m, init_f * sign, sign);
            });
            return;
        }
    }
    const dim3 grid = plane_grid(g.OW, g.OH, (int64_t)g.N * g.C), block(32, 8);
    switch (window_code(g)) {
        case 1: pool_fwd_kernel<T, OP, 1><<<grid, block, 0, st>>>(xp, yp, indices, taps, g, init); break;
        case 2: pool_fwd_kernel<T, OP, 2><<<grid, block, 0, st>>>(xp, yp, indices, taps, g, init); break;
        case 3: pool_fwd_kernel<T, OP, 3><<<grid, block, 0, st>>>(xp, yp, indices, taps, g, init); break;
        default: pool_fwd_kernel<T, OP, 0><<<grid, block, 0, st>>>(xp, yp, indices, taps, g, init);
    }
}

template <typename T, bool MEAN>
static bool launch_bwd_tile(const uint8_t* taps, const T* dp, T* op, const Geo& g, cudaStream_t st) {
    if constexpr (sizeof(T) <= 4) {
        if (!tiled<T>(g)) return false;
        dispatch_tile<T>(g, op, dp, taps, [&](auto k, auto s, auto p, auto vo, auto ax) {
            const TileMap m = tile_map(g, g.H, g.W, rows_up(vo()) * s(), vo() * s());
            pool_bwd_tile_kernel<T, MEAN, k(), s(), p(), vo(), ax()><<<(unsigned)((m.threads + 255) / 256), 256, 0, st>>>(taps, dp, op, g, m);
        });
        return true;
    }
    return false;
}

template <typename T, int OP>
static void launch_bwd(const T* xp, const T* yp, const T* dp, T* op, const Geo& g, cudaStream_t st) {
    if constexpr (OP == 2)
        if (whole_mean(g) && launch_bwd_tile<T, true>(nullptr, dp, op, g, st)) return;
    const dim3 grid = plane_grid(g.W, g.H, (int64_t)g.N * g.C), block(32, 8);
    switch (window_code(g)) {
        case 1: pool_bwd_kernel<T, OP, 1><<<grid, block, 0, st>>>(xp, yp, dp, op, g); break;
        case 2: pool_bwd_kernel<T, OP, 2><<<grid, block, 0, st>>>(xp, yp, dp, op, g); break;
        case 3: pool_bwd_kernel<T, OP, 3><<<grid, block, 0, st>>>(xp, yp, dp, op, g); break;
        default: pool_bwd_kernel<T, OP, 0><<<grid, block, 0, st>>>(xp, yp, dp, op, g);
    }
}

template <typename T, typename I>
static int run_bwd_indices(const I* idx, const b200jt_tensor* dy, const b200jt_tensor* dx, const Geo& g, cudaStream_t st) {
    if (numel(dx) == 0) return 0;
    const int64_t planes = (int64_t)g.N * g.C;
    const T* dp = (const T*)dy->ptr; T* op = (T*)dx->ptr;
    if constexpr (sizeof(I) == 1)
        if (launch_bwd_tile<T, false>(idx, dp, op, g, st)) { B200JT_LAUNCH_CHECK(); return 0; }
    const dim3 grid = plane_grid(g.W, g.H, (planes + 3) / 4), block(32, 8);
    switch (window_code(g)) {
        case 1: pool_bwd_indices_kernel<T, I, 1><<<grid, block, 0, st>>>(idx, dp, op, g); break;
        case 2: pool_bwd_indices_kernel<T, I, 2><<<grid, block, 0, st>>>(idx, dp, op, g); break;
        case 3: pool_bwd_indices_kernel<T, I, 3><<<grid, block, 0, st>>>(idx, dp, op, g); break;
        default: pool_bwd_indices_kernel<T, I, 0><<<grid, block, 0, st>>>(idx, dp, op, g);
    }
    B200JT_LAUNCH_CHECK();
    return 0;
}

template <typename T>
static int run_fwd(const b200jt_tensor* x, const b200jt_tensor* y, int32_t* indices, uint8_t* taps, const Geo& g, int opc, cudaStream_t st) {
    if (numel(y) == 0) return 0;
    const T* xp = (const T*)x->ptr; T* yp = (T*)y->ptr;
    if (opc == 0) launch_fwd<T, 0>(xp, yp, indices, taps, g, init_value<T>(OP_MAX), st);
    else if (opc == 1) launch_fwd<T, 1>(xp, yp, indices, taps, g, init_value<T>(OP_MIN), st);
    else launch_fwd<T, 2>(xp, yp, indices, taps, g, init_value<T>(OP_ADD), st);
    B200JT_LAUNCH_CHECK();
    return 0;
}

template <typename T>
static int run_bwd(const b200jt_tensor* x, const b200jt_tensor* y, const b200jt_tensor* dy, const b200jt_tensor* dx,
                   const Geo& g, int opc, cudaStream_t st) {
    if (numel(x) == 0) return 0;
    const T *xp = (const T*)x->ptr, *yp = (const T*)y->ptr, *dp = (const T*)dy->ptr; T* op = (T*)dx->ptr;
    if (opc == 0) launch_bwd<T, 0>(xp, yp, dp, op, g, st);
    else if (opc == 1) launch_bwd<T, 1>(xp, yp, dp, op, g, st);
    else launch_bwd<T, 2>(xp, yp, dp, op, g, st);
    B200JT_LAUNCH_CHECK();
    return 0;
}

}  // namespace pool
}  // namespace b200jt

using namespace b200jt;

static int pool2d(const b200jt_tensor* x, const b200jt_tensor* y, int32_t* indices, uint8_t* taps, const char* op,
                  int kh, int kw, int sh, int sw, int ph, int pw, int count_include_pad, void* stream) {
    pool::Geo g; int opc;
    if (int rc = pool::parse(x, y, op, kh, kw, sh, sw, ph, pw, count_include_pad, &g, &opc)) return rc;
    B200JT_CHECK_ARG(!(indices || taps) || opc != 2, "indices are only produced for maximum and minimum");
    B200JT_CHECK_ARG(!taps || (int64_t)kh * kw <= 255, "windows of at most 255 elements");
    cudaStream_t st = (cudaStream_t)stream;
    switch (x->dtype) {
        case B200JT_FLOAT32: return pool::run_fwd<float>(x, y, indices, taps, g, opc, st);
        case B200JT_FLOAT64: return pool::run_fwd<double>(x, y, indices, taps, g, opc, st);
        case B200JT_BFLOAT16: return pool::run_fwd<__nv_bfloat16>(x, y, indices, taps, g, opc, st);
        case B200JT_FLOAT16: return pool::run_fwd<__half>(x, y, indices, taps, g, opc, st);
    }
    return fail(-1, "b200jt_pool2d: dtype must be float32, float64, float16 or bfloat16");
}

extern "C" int b200jt_pool2d(const b200jt_tensor* x, const b200jt_tensor* y, int32_t* indices, const char* op,
                             int kh, int kw, int sh, int sw, int ph, int pw, int count_include_pad, void* stream) {
    return pool2d(x, y, indices, nullptr, op, kh, kw, sh, sw, ph, pw, count_include_pad, stream);
}

extern "C" int b200jt_pool2d_taps(const b200jt_tensor* x, const b200jt_tensor* y, uint8_t* taps, const char* op,
                                  int kh, int kw, int sh, int sw, int ph, int pw, void* stream) {
    B200JT_CHECK_ARG(taps != nullptr, "taps is null");
    return pool2d(x, y, nullptr, taps, op, kh, kw, sh, sw, ph, pw, 1, stream);
}

extern "C" int b200jt_pool2d_backward(const b200jt_tensor* x, const b200jt_tensor* y, const b200jt_tensor* dy,
                                      const b200jt_tensor* dx, const char* op,
                                      int kh, int kw, int sh, int sw, int ph, int pw, int count_include_pad, void* stream) {
    pool::Geo g; int opc;
    if (int rc = pool::parse(x, y, op, kh, kw, sh, sw, ph, pw, count_include_pad, &g, &opc)) return rc;
    B200JT_CHECK_ARG(valid_tensor(dy) && valid_tensor(dx) && dy->ndim == 4 && dx->ndim == 4 &&
                     dy->dtype == x->dtype && dx->dtype == x->dtype, "dy, dx must be NCHW tensors of x's dtype");
    for (int d = 0; d < 4; d++)
        B200JT_CHECK_ARG(dy->shape[d] == y->shape[d] && dx->shape[d] == x->shape[d], "dy must have y's shape and dx x's shape");
    cudaStream_t st = (cudaStream_t)stream;
    switch (x->dtype) {
        case B200JT_FLOAT32: return pool::run_bwd<float>(x, y, dy, dx, g, opc, st);
        case B200JT_FLOAT64: return pool::run_bwd<double>(x, y, dy, dx, g, opc, st);
        case B200JT_BFLOAT16: return pool::run_bwd<__nv_bfloat16>(x, y, dy, dx, g, opc, st);
        case B200JT_FLOAT16: return pool::run_bwd<__half>(x, y, dy, dx, g, opc, st);
    }
    return fail(-1, "b200jt_pool2d_backward: dtype must be float32, float64, float16 or bfloat16");
}

extern "C" int b200jt_pool2d_backward_indices(const b200jt_tensor* x, const b200jt_tensor* y, const int32_t* indices,
                                              const b200jt_tensor* dy, const b200jt_tensor* dx,
                                              int kh, int kw, int sh, int sw, int ph, int pw, void* stream) {
    pool::Geo g; int opc;
    if (int rc = pool::parse(x, y, "maximum", kh, kw, sh, sw, ph, pw, 1, &g, &opc)) return rc;
    B200JT_CHECK_ARG(indices != nullptr, "indices is null");
    B200JT_CHECK_ARG(valid_tensor(dy) && valid_tensor(dx) && dy->ndim == 4 && dx->ndim == 4 &&
                     dy->dtype == x->dtype && dx->dtype == x->dtype, "dy, dx must be NCHW tensors of x's dtype");
    for (int d = 0; d < 4; d++)
        B200JT_CHECK_ARG(dy->shape[d] == y->shape[d] && dx->shape[d] == x->shape[d], "dy must have y's shape and dx x's shape");
    B200JT_CHECK_ARG((int64_t)g.H * g.W < (1LL << 31), "plane too large for int32 indices");
    cudaStream_t st = (cudaStream_t)stream;
    switch (x->dtype) {
        case B200JT_FLOAT32: return pool::run_bwd_indices<float>(indices, dy, dx, g, st);
        case B200JT_FLOAT64: return pool::run_bwd_indices<double>(indices, dy, dx, g, st);
        case B200JT_BFLOAT16: return pool::run_bwd_indices<__nv_bfloat16>(indices, dy, dx, g, st);
        case B200JT_FLOAT16: return pool::run_bwd_indices<__half>(indices, dy, dx, g, st);
    }
    return fail(-1, "b200jt_pool2d_backward_indices: dtype must be float32, float64, float16 or bfloat16");
}

extern "C" int b200jt_pool2d_backward_taps(const uint8_t* taps, const b200jt_tensor* dy, const b200jt_tensor* dx,
                                           int kh, int kw, int sh, int sw, int ph, int pw, void* stream) {
    pool::Geo g; int opc;
    if (int rc = pool::parse(dx, dy, "maximum", kh, kw, sh, sw, ph, pw, 1, &g, &opc)) return rc;
    B200JT_CHECK_ARG(taps != nullptr && (int64_t)kh * kw <= 255, "taps is null, or the window has more than 255 elements");
    cudaStream_t st = (cudaStream_t)stream;
    switch (dx->dtype) {
        case B200JT_FLOAT32: return pool::run_bwd_indices<float>(taps, dy, dx, g, st);
        case B200JT_FLOAT64: return pool::run_bwd_indices<double>(taps, dy, dx, g, st);
        case B200JT_BFLOAT16: return pool::run_bwd_indices<__nv_bfloat16>(taps, dy, dx, g, st);
        case B200JT_FLOAT16: return pool::run_bwd_indices<__half>(taps, dy, dx, g, st);
    }
    return fail(-1, "b200jt_pool2d_backward_taps: dtype must be float32, float64, float16 or bfloat16");
}
