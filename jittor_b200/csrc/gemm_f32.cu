// float32 contractions on CUDA cores: matmul and the convolution as an implicit GEMM -- forward, transposed / data gradient
// and weight gradient -- in one kernel, C[m, n] = sum over k of A(m, k) * B(k, n) with fp32 fused multiply-adds.
//
// What bounds it: the FMA pipe when the tiles fill the GPU, latency otherwise (a layer of a small network is a few MFLOP). The
// kernels this replaces (one 4 x 4 or 2 x 2 block per thread, index arithmetic and a trip to memory per staged element, no
// split of k) ran config 0's convolution at 8.6 TFLOP/s and a 16-image weight gradient, whose 1 or 2 tiles sat on one SM
// each, at 0.004 TFLOP/s. Here:
//   * 8 x 8 or 8 x 4 outputs per thread and packed fma.rn.f32x2: two FMAs per issue slot, the products of a pair of rows with
//     a pair of columns straight and swapped, so that no operand has to be duplicated in registers;
//   * operands reach shared memory by cp.async in a three-stage ring, zero-filled at the edges (a 4-byte copy takes any
//     alignment, so ragged shapes take the same path);
//   * the part of a gather's address that depends on k only is tabulated per CTA, 256 entries at a time; the part that depends
//     on the column only sits in registers or shared memory, so a staged element costs two additions and two range checks;
//   * k is split over a cluster of up to 8 CTAs that fold their partial tiles through distributed shared memory in rank order
//     (one launch, no scratch, the same bits every run), and beyond that over slices folded by a second kernel.
#include "gemm_simt.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace cg = cooperative_groups;

namespace b200jt {
namespace f32 {

typedef unsigned long long u64;
constexpr int BK = 16, STAGES = 3, TAB = 256;

__device__ __forceinline__ void fma2(u64& c, u64 a, u64 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ u64 swap2(u64 v) {
    u64 r;
    asm("{ .reg .b32 lo, hi; mov.b64 {lo, hi}, %1; mov.b64 %0, {hi, lo}; }" : "=l"(r) : "l"(v));
    return r;
}
__device__ __forceinline__ float lo2(u64 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(u64 v) { return __uint_as_float((unsigned)(v >> 32)); }

__device__ __forceinline__ void copy4(float* dst, const float* src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 4 : 0));
}
__device__ __forceinline__ void copy16(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes));
}

// n / d for 0 <= n < 2^31 and a d fixed at launch: one multiply-high and a shift, the method of Granlund and Montgomery (Division
// by invariant integers using multiplication, 1994); d = 1: shift 0, multiplier 0 stands for n.
struct FastDiv {
    unsigned d = 1, mul = 0, shift = 0;
    FastDiv() = default;
    explicit FastDiv(int div) {
        d = (unsigned)div;
        if (d > 1) {
            while ((1u << shift) < d && shift < 31) shift++;            // 2^(shift-1) < d <= 2^shift
            shift--;
            mul = (unsigned)(((1ull << (32 + shift)) + d - 1) / d);     // ceil(2^(32+shift) / d) fits 32 bits
        }
    }
    __device__ __forceinline__ int div(int n) const { return mul ? (int)(__umulhi((unsigned)n, mul) >> shift) : n; }
};

// ---- what the operands are -------------------------------------------------------------------------------------------
// MATMUL: A and B are strided matrices. Otherwise A is the dense side (weights, or the output gradient) and B the gathered
// side (pixels of x through the window, or of the output gradient for the transposed form); the output is contiguous along n.
enum Mode { MATMUL, FWD, TRANSPOSED, WGRAD };

// One residue class of a transposed convolution's output rows (or columns) modulo the stride: the taps that reach it and how
// many output rows it has. Every pair of classes is a stride-1 gather with its own taps, so no product with a hole is formed.
struct ResidueClass { int first, step, count, extent; FastDiv by_count, by_extent; };
constexpr int kMaxStride = 8;

struct Args {
    const float *a, *b;
    float* c;
    int M, N, K;
    // MATMUL
    int64_t a_sm, a_sk, b_sk, b_sn, a_bs, b_bs, c_bs;
    // convolutions: the forward layer's shape; TRANSPOSED: C/H/W of its input (the forward's output), Co/OH/OW of its output
    ConvShape s;
    FastDiv by_kw, by_kh, by_ow, by_oh, by_pix;
    ResidueClass rh[kMaxStride], rw[kMaxStride];
    int outer;                   // slices folded by the second kernel (1: the result goes to c)
    int64_t c_numel;
};

struct KEntry { int goff, doff; short dih, diw; int pad; };      // gather offset, dense offset, window displacement
struct Col { int base; short ih, iw; };                           // of a gathered column

template <Mode MODE>
__device__ __forceinline__ KEntry kentry(const Args& g, int ry, int rx, int k) {
    const ConvShape& s = g.s;
    KEntry e;
    e.pad = 0;
    if (MODE == FWD) {
        const int t = g.by_kw.div(k), kw = k - t * s.KW, c = g.by_kh.div(t), kh = t - c * s.KH;
        e.dih = (short)(kh * s.dh); e.diw = (short)(kw * s.dw);
        e.goff = c * s.H * s.W + e.dih * s.W + e.diw; e.doff = k;
    } else if (MODE == TRANSPOSED) {
        const ResidueClass &p = g.rh[ry], &q = g.rw[rx];
        const int t = q.by_count.div(k), b = k - t * q.count, c = p.by_count.div(t), a = t - c * p.count;
        const int kh = p.first + a * p.step, kw = q.first + b * q.step;
        e.dih = (short)((ry + s.ph - kh * s.dh) / s.sh); e.diw = (short)((rx + s.pw - kw * s.dw) / s.sw);
        e.goff = c * s.H * s.W + e.dih * s.W + e.diw; e.doff = c * s.Co * s.KH * s.KW + kh * s.KW + kw;
    } else {
        const int P = s.OH * s.OW, img = g.by_pix.div(k), pix = k - img * P, oh = g.by_ow.div(pix), ow = pix - oh * s.OW;
        e.dih = (short)(oh * s.sh - s.ph); e.diw = (short)(ow * s.sw - s.pw);
        e.goff = img * s.C * s.H * s.W + e.dih * s.W + e.diw; e.doff = img * s.Co * P + pix;
    }
    return e;
}

// Column n of the gathered side, and where it goes in the output.
template <Mode MODE>
__device__ __forceinline__ Col column(const Args& g, int ry, int rx, int n, int& coff) {
    const ConvShape& s = g.s;
    Col c;
    if (MODE == WGRAD) {
        const int t = g.by_kw.div(n), kw = n - t * s.KW, ch = g.by_kh.div(t), kh = t - ch * s.KH;
        c.ih = (short)(kh * s.dh); c.iw = (short)(kw * s.dw);
        c.base = ch * s.H * s.W + c.ih * s.W + c.iw;
        coff = n;
    } else {
        const int QH = MODE == FWD ? s.OH : g.rh[ry].extent, QW = MODE == FWD ? s.OW : g.rw[rx].extent;
        const int t = (MODE == FWD ? g.by_ow : g.rw[rx].by_extent).div(n), ow = n - t * QW;
        const int img = (MODE == FWD ? g.by_oh : g.rh[ry].by_extent).div(t), oh = t - img * QH;
        if (MODE == FWD) {
            c.ih = (short)(oh * s.sh - s.ph); c.iw = (short)(ow * s.sw - s.pw);
            coff = img * s.Co * s.OH * s.OW + oh * s.OW + ow;
        } else {
            c.ih = (short)oh; c.iw = (short)ow;
            coff = img * s.Co * s.OH * s.OW + (oh * s.sh + ry) * s.OW + ow * s.sw + rx;
        }
        c.base = img * s.C * s.H * s.W + c.ih * s.W + c.iw;
    }
    return c;
}

template <int BM, int BN> constexpr int ring_floats() { return STAGES * BK * (BM + 4 + BN + 4); }
template <Mode MODE, int BM, int BN> constexpr int smem_bytes() {
    constexpr int ring = ring_floats<BM, BN>() * 4, fold = BM * BN * 4;
    constexpr int tables = MODE == MATMUL ? 0 : 2 * TAB * (int)sizeof(KEntry) + BN * ((int)sizeof(Col) + 4);
    return (ring > fold ? ring : fold) + tables;
}

// AK / BKF: the operand is contiguous along k (threads walk k when they stage it), else along m / n.
template <Mode MODE, bool AK, bool BKF, int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), BM * BN >= 128 * 128 ? 2 : TM * TN == 16 && BM == 64 ? 3 : 4)
contract_kernel(const __grid_constant__ Args g) {
    constexpr int T = (BM / TM) * (BN / TN), GM = TM / 4, GN = TN / 4, PA = BM + 4, PB = BN + 4;
    extern __shared__ __align__(16) float smem[];
    float* As = smem;                                  // [STAGES][BK][PA]
    float* Bs = smem + STAGES * BK * PA;               // [STAGES][BK][PB]
    constexpr int ring = ring_floats<BM, BN>(), fold_n = BM * BN;
    [[maybe_unused]] KEntry* ktab = (KEntry*)(smem + (ring > fold_n ? ring : fold_n));      // [2][TAB]
    [[maybe_unused]] Col* cols = (Col*)(ktab + 2 * TAB);
    [[maybe_unused]] int* coffs = (int*)(cols + BN);

    cg::cluster_group cluster = cg::this_cluster();
    const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int slices = S * g.outer;
    const int zi = blockIdx.z / slices, slice = blockIdx.z - zi * slices;
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    // a warp covers 4 x 8 thread tiles: 64 bytes of A and 128 of B per shared load
    const int tx = lane % 8 + 8 * (warp % (BN / TN / 8)), ty = lane / 8 + 4 * (warp / (BN / TN / 8));
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int M = g.M;
    int N = g.N, K = g.K;
    [[maybe_unused]] int ry = 0, rx = 0;
    const float *a = g.a, *b = g.b;
    float* c = g.c;
    if constexpr (MODE == MATMUL) { a += zi * g.a_bs; b += zi * g.b_bs; c += g.outer > 1 ? 0 : zi * g.c_bs; }
    if constexpr (MODE == TRANSPOSED) {
        ry = zi / g.s.sw; rx = zi - ry * g.s.sw;
        N = g.s.N * g.rh[ry].extent * g.rw[rx].extent; K = g.s.C * g.rh[ry].count * g.rw[rx].count;
        if (n0 >= N) return;                           // the whole cluster shares n0 and the class
    }
    const int tiles_k = (K + BK - 1) / BK, per = (tiles_k + slices - 1) / slices;
    const int kt0 = slice * per, nt = max(0, min(per, tiles_k - kt0));
    const int kbeg = kt0 * BK;
    [[maybe_unused]] const int kend = min(K, kbeg + nt * BK);

    if constexpr (MODE != MATMUL) {
        for (int i = tid; i < BN; i += T) {
            int coff = -1;
            Col col{0, -30000, -30000};
            if (n0 + i < N) col = column<MODE>(g, ry, rx, n0 + i, coff);
            cols[i] = col; coffs[i] = coff;
        }
        for (int i = tid; i < TAB; i += T) if (kbeg + i < kend) ktab[i] = kentry<MODE>(g, ry, rx, kbeg + i);
        __syncthreads();
    }
    [[maybe_unused]] Col my_col{};
    if constexpr (MODE == FWD || MODE == TRANSPOSED) my_col = cols[tid % BN];
    const bool vec_a = MODE == MATMUL && !AK && (g.a_sk & 3) == 0 && ((uintptr_t)a & 15) == 0;
    const bool vec_b = MODE == MATMUL && !BKF && (g.b_sk & 3) == 0 && ((uintptr_t)b & 15) == 0;

    // half 0 copies A's tile, half 1 B's: issued apart so that the copies do not queue up in front of the FMAs' shared loads
    auto issue = [&](int t, int stage, int half) {
        const int k0 = kbeg + t * BK;
        float* as = As + stage * BK * PA;
        float* bs = Bs + stage * BK * PB;
        [[maybe_unused]] const KEntry* tab = ktab + (((t / (TAB / BK)) & 1) * TAB + (t % (TAB / BK)) * BK);
        if (half == 0) {
        if constexpr (MODE == MATMUL && !AK) {
            if (vec_a) {
#pragma unroll
                for (int i = 0; i < (BM * BK / 4 + T - 1) / T; i++) {
                    const int q = tid + i * T;
                    if ((BM * BK / 4) % T != 0 && q >= BM * BK / 4) break;
                    const int mm = (q % (BM / 4)) * 4, kk = q / (BM / 4);
                    const int left = k0 + kk < K ? M - (m0 + mm) : 0;
                    copy16(as + kk * PA + mm, left > 0 ? a + (int64_t)(k0 + kk) * g.a_sk + m0 + mm : a, left >= 4 ? 16 : left > 0 ? left * 4 : 0);
                }
            } else {
#pragma unroll 4
                for (int q = tid; q < BM * BK; q += T) {
                    const int mm = q % BM, kk = q / BM;
                    const bool ok = m0 + mm < M && k0 + kk < K;
                    copy4(as + kk * PA + mm, ok ? a + (int64_t)(k0 + kk) * g.a_sk + m0 + mm : a, ok);
                }
            }
        } else {
            const int kk = tid % BK;
            const bool kok = k0 + kk < K;
            const float* src;
            int64_t sm;
            if constexpr (MODE == MATMUL || MODE == FWD) { src = a + k0 + kk; sm = MODE == FWD ? (int64_t)K : g.a_sm; }
            else { src = a + (kok ? tab[kk].doff : 0); sm = MODE == WGRAD ? g.s.OH * g.s.OW : g.s.KH * g.s.KW; }
            src += (m0 + tid / BK) * sm;
#pragma unroll
            for (int i = 0; i < BM * BK / T; i++) {
                const int mm = tid / BK + i * (T / BK);
                const bool ok = kok && m0 + mm < M;
                copy4(as + kk * PA + mm, ok ? src + (int64_t)(i * (T / BK)) * sm : a, ok);
            }
        }
        return;
        }
        if constexpr (MODE == MATMUL) {
            if constexpr (BKF) {
                const int kk = tid % BK;
                const bool kok = k0 + kk < K;
                const float* src = b + k0 + kk + (int64_t)(n0 + tid / BK) * g.b_sn;
#pragma unroll
                for (int i = 0; i < BN * BK / T; i++) {
                    const int nn = tid / BK + i * (T / BK);
                    const bool ok = kok && n0 + nn < N;
                    copy4(bs + kk * PB + nn, ok ? src + (int64_t)(i * (T / BK)) * g.b_sn : b, ok);
                }
            } else if (vec_b) {
#pragma unroll
                for (int i = 0; i < (BN * BK / 4 + T - 1) / T; i++) {
                    const int q = tid + i * T;
                    if ((BN * BK / 4) % T != 0 && q >= BN * BK / 4) break;
                    const int nn = (q % (BN / 4)) * 4, kk = q / (BN / 4);
                    const int left = k0 + kk < K ? N - (n0 + nn) : 0;
                    copy16(bs + kk * PB + nn, left > 0 ? b + (int64_t)(k0 + kk) * g.b_sk + n0 + nn : b, left >= 4 ? 16 : left > 0 ? left * 4 : 0);
                }
            } else {
#pragma unroll 4
                for (int q = tid; q < BN * BK; q += T) {
                    const int nn = q % BN, kk = q / BN;
                    const bool ok = n0 + nn < N && k0 + kk < K;
                    copy4(bs + kk * PB + nn, ok ? b + (int64_t)(k0 + kk) * g.b_sk + n0 + nn : b, ok);
                }
            }
        } else if constexpr (MODE == WGRAD) {
            const int kk = tid % BK;
            KEntry e{0, 0, -30000, 0, 0};
            if (k0 + kk < K) e = tab[kk];
#pragma unroll
            for (int i = 0; i < BN * BK / T; i++) {
                const int nn = tid / BK + i * (T / BK);
                const Col col = cols[nn];
                const bool ok = (unsigned)(col.ih + e.dih) < (unsigned)g.s.H && (unsigned)(col.iw + e.diw) < (unsigned)g.s.W;
                copy4(bs + kk * PB + nn, ok ? b + (col.base + e.goff) : b, ok);
            }
        } else {
#pragma unroll
            for (int i = 0; i < BN * BK / T; i++) {
                const int kk = tid / BN + i * (T / BN);
                const KEntry e = tab[kk];
                const bool ok = k0 + kk < K && (unsigned)(my_col.ih + e.dih) < (unsigned)g.s.H && (unsigned)(my_col.iw + e.diw) < (unsigned)g.s.W;
                copy4(bs + kk * PB + tid % BN, ok ? b + (my_col.base + e.goff) : b, ok);
            }
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;"); };

    u64 D[TM / 2][TN / 2], X[TM / 2][TN / 2];          // (row 2i, col 2j | row 2i+1, col 2j+1) and (row 2i, col 2j+1 | row 2i+1, col 2j)
#pragma unroll
    for (int i = 0; i < TM / 2; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) D[i][j] = X[i][j] = 0;

#pragma unroll
    for (int t = 0; t < STAGES - 1; t++) {
        if (t < nt) { issue(t, t, 0); issue(t, t, 1); }
        commit();
    }
    // A tile's copies are issued in two halves between the FMAs: with one CTA per SM a 64 x 64 x 16 step is 1400 cycles of
    // FMAs and shared loads and 900 of address arithmetic.
    int stage = 0;
    for (int t = 0; t < nt; t++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2));
        __syncthreads();
        const int j = t + STAGES - 1;
        if constexpr (MODE != MATMUL) {
            if ((j + 1) % (TAB / BK) == 0 && j + 1 < nt) {
                KEntry* next = ktab + (((j + 1) / (TAB / BK)) & 1) * TAB;
                const int k0 = kbeg + (j + 1) * BK;
                for (int i = tid; i < TAB; i += T) if (k0 + i < kend) next[i] = kentry<MODE>(g, ry, rx, k0 + i);
            }
        }
        const int into = stage == 0 ? STAGES - 1 : stage - 1;
        const float* as = As + stage * BK * PA + ty * 4;
        const float* bs = Bs + stage * BK * PB + tx * 4;
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            if (kk % (BK / 2) == 1 && j < nt) issue(j, into, kk / (BK / 2));
            {
                u64 av[TM / 2], bv[TN / 2], bx[TN / 2];
#pragma unroll
                for (int q = 0; q < GM; q++) {
                    const ulonglong2 v = *(const ulonglong2*)(as + kk * PA + q * (BM / GM));
                    av[2 * q] = v.x; av[2 * q + 1] = v.y;
                }
#pragma unroll
                for (int q = 0; q < GN; q++) {
                    const ulonglong2 v = *(const ulonglong2*)(bs + kk * PB + q * (BN / GN));
                    bv[2 * q] = v.x; bv[2 * q + 1] = v.y;
                    bx[2 * q] = swap2(v.x); bx[2 * q + 1] = swap2(v.y);
                }
#pragma unroll
                for (int i = 0; i < TM / 2; i++)
#pragma unroll
                    for (int jj = 0; jj < TN / 2; jj++) { fma2(D[i][jj], av[i], bv[jj]); fma2(X[i][jj], av[i], bx[jj]); }
            }
        }
        commit();
        stage = stage == STAGES - 1 ? 0 : stage + 1;
    }

    // ---- results: straight to c, or through the cluster fold
    const int64_t c_sm = MODE == MATMUL ? (int64_t)N : MODE == WGRAD ? (int64_t)g.N : (int64_t)g.s.OH * g.s.OW;
    if (g.outer > 1) c += (int64_t)(slice / S) * g.c_numel + (MODE == MATMUL ? zi * g.c_bs : 0);
    const bool vec_c = (c_sm & 3) == 0 && ((uintptr_t)c & 15) == 0;
    auto store4 = [&](int m, int nn, float4 v) {       // columns n0 + nn .. + 3 of row m
        if (m >= M) return;
        float* row = c + m * c_sm;
        if constexpr (MODE == MATMUL) {
            if (vec_c && n0 + nn + 3 < N) { *(float4*)(row + n0 + nn) = v; return; }
            const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++) if (n0 + nn + i < N) row[n0 + nn + i] = e[i];
        } else {
            const int o = coffs[nn];
            if (vec_c && o >= 0 && (o & 3) == 0 && coffs[nn + 3] == o + 3) { *(float4*)(row + o) = v; return; }
            const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++) if (coffs[nn + i] >= 0) row[coffs[nn + i]] = e[i];
        }
    };
    auto each4 = [&](auto&& put) {
#pragma unroll
        for (int i = 0; i < TM / 2; i++) {
            const int r = ty * 4 + (i / 2) * (BM / GM) + (i % 2) * 2;
#pragma unroll
            for (int q = 0; q < GN; q++) {
                const int nn = tx * 4 + q * (BN / GN);
                put(r, nn, make_float4(lo2(D[i][2 * q]), lo2(X[i][2 * q]), lo2(D[i][2 * q + 1]), lo2(X[i][2 * q + 1])));
                put(r + 1, nn, make_float4(hi2(X[i][2 * q]), hi2(D[i][2 * q]), hi2(X[i][2 * q + 1]), hi2(D[i][2 * q + 1])));
            }
        }
    };
    if (S == 1) {
        each4([&](int r, int nn, float4 v) { store4(m0 + r, nn, v); });
        return;
    }
    asm volatile("cp.async.wait_all;");
    __syncthreads();
    each4([&](int r, int nn, float4 v) { *(float4*)(smem + r * BN + nn) = v; });
    cluster.sync();
    const int rows = BM / S;
    for (int e = tid; e < rows * (BN / 4); e += T) {
        const int r = rank * rows + e / (BN / 4), nn = (e % (BN / 4)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int p = 0; p < S; p++) {
            const float4 u = *(const float4*)(cluster.map_shared_rank(smem, p) + r * BN + nn);
            v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
        store4(m0 + r, nn, v);
    }
    // no CTA leaves while others read its tile; every value read has been used, so the barrier needs no fence
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(256) fold_kernel(const float* __restrict__ part, float* __restrict__ c, int64_t n, int slices) {
    for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        float v = 0.f;
        for (int s = 0; s < slices; s++) v += part[(int64_t)s * n + i];
        c[i] = v;
    }
}

// ---- tile and split ----------------------------------------------------------------------------------------------------
struct Tile { int bm, bn, occ; double alone, more, most, gather; };
// Share of the FMA rate one resident CTA reaches alone, what each further one adds, what a full SM reaches, and the factor
// for gathered operands (their address arithmetic competes for issue slots). Fitted to sweeps of tile x cluster x slices
// over square, flat and k-long products and convolution layers from 0.3 to 4000 us: the rule's choice is within a few
// per cent of the sweep's best.
// The 8 x 8 tile is the most efficient; 4 x 4 spreads a small tile over 8 warps, which covers latencies with one CTA per SM;
// the two flat ones are for few rows (output channels of small layers, input channels of a first layer's data gradient).
constexpr Tile kTiles[] = {{128, 128, 2, 0.64, 0.05, 0.70, 0.94}, {64, 64, 4, 0.26, 0.12, 0.57, 0.90}, {32, 128, 4, 0.26, 0.12, 0.57, 0.82},
                           {64, 64, 3, 0.35, 0.12, 0.54, 0.90}, {16, 128, 4, 0.20, 0.09, 0.42, 0.85}};
constexpr int kNumTiles = 5;
struct Split { int tile = 1, cluster = 1, outer = 1; double cycles = 1e300; };

// Cycles of the slowest SM: CTAs per SM x the tile's FMAs at the rate that many resident CTAs reach, plus what a split costs.
// Every combination of tile, cluster size and slice count is tried: 0.2 to 1.5 us of host time a call.
inline Split plan(int64_t M, int64_t N, int64_t K, int64_t copies, bool may_fold, bool gather) {
    Split best;
    const int64_t kt = std::max<int64_t>(1, (K + BK - 1) / BK);
    for (int t = 0; t < kNumTiles; t++) {
        const Tile& T = kTiles[t];
        const int64_t tiles = ((M + T.bm - 1) / T.bm) * ((N + T.bn - 1) / T.bn) * copies;
        for (int o = 1; o <= (may_fold ? 64 : 1); o *= 2)
            for (int s = 1; s <= 8; s *= 2) {
                const int64_t n = (int64_t)s * o;
                if (n > kt || (n > 1 && (kt + n - 1) / n < 3) || copies * n > 60000) break;
                const double per_k = (double)T.bm * T.bn * BK / 128.0;                      // cycles of one BK step at the full rate
                const double work = (double)((kt + n - 1) / n) * per_k + 400;
                const int64_t r = (tiles * n + kNumSMs - 1) / kNumSMs;
                const double eff = std::min(T.most, T.alone + (std::min<int64_t>(r, T.occ) - 1) * T.more) * (gather ? T.gather : 1.0);
                const double c = (double)r * (work / eff + 600) + (s > 1 ? 1500.0 + (double)r * T.bm * T.bn / 8 : 0) + (o > 1 ? 4000.0 + (double)M * N * copies * o / 800 : 0);
                if (c < best.cycles) best = {t, s, o, c};
            }
    }
    return best;
}

template <Mode MODE, bool AK, bool BKF, int BM, int BN, int TM, int TN>
int launch_tile(const Args& g, int64_t n_cols, int copies, int cluster, cudaStream_t st) {
    auto kernel = contract_kernel<MODE, AK, BKF, BM, BN, TM, TN>;
    constexpr int smem = smem_bytes<MODE, BM, BN>();
    static const cudaError_t attr = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    B200JT_CUDA(attr);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)((n_cols + BN - 1) / BN), (unsigned)((g.M + BM - 1) / BM), (unsigned)(copies * cluster * g.outer));
    cfg.blockDim = dim3((BM / TM) * (BN / TN));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1; at.val.clusterDim.y = 1; at.val.clusterDim.z = (unsigned)cluster;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    B200JT_CUDA(cudaLaunchKernelEx(&cfg, kernel, g));
    return 0;
}

template <Mode MODE, bool AK, bool BKF>
int launch(Args& g, int64_t n_cols, int copies, const Split& p, void* workspace, cudaStream_t st) {
    float* c = g.c;
    g.outer = p.outer;
    if (p.outer > 1) g.c = (float*)workspace;
    int rc;
    if (p.tile == 0) rc = launch_tile<MODE, AK, BKF, 128, 128, 8, 8>(g, n_cols, copies, p.cluster, st);
    else if (p.tile == 1) rc = launch_tile<MODE, AK, BKF, 64, 64, 8, 4>(g, n_cols, copies, p.cluster, st);
    else if (p.tile == 2) rc = launch_tile<MODE, AK, BKF, 32, 128, 8, 4>(g, n_cols, copies, p.cluster, st);
    else if (p.tile == 3) rc = launch_tile<MODE, AK, BKF, 64, 64, 4, 4>(g, n_cols, copies, p.cluster, st);
    else rc = launch_tile<MODE, AK, BKF, 16, 128, 4, 4>(g, n_cols, copies, p.cluster, st);
    if (rc) return rc;
    if (p.outer > 1) {
        fold_kernel<<<grid_for(g.c_numel, 256), 256, 0, st>>>((const float*)workspace, c, g.c_numel, p.outer);
        B200JT_LAUNCH_CHECK();
    }
    return 0;
}

}  // namespace f32

using namespace f32;

static constexpr int64_t kMaxElems = 0x7fffffff;

bool matmul_f32_supported(int64_t batch, int64_t M, int64_t N, int64_t K) {
    return M > 0 && N > 0 && K > 0 && M <= 65535 * 32ll && N < kMaxElems - 128 && K < kMaxElems - 64 && batch <= 60000;
}
double matmul_f32_ns(int64_t M, int64_t N, int64_t K) { return plan(M, N, K, 1, true, false).cycles / 1.9; }
size_t matmul_f32_workspace(int64_t M, int64_t N, int64_t K) {
    if (!matmul_f32_supported(1, M, N, K)) return 0;
    const Split p = plan(M, N, K, 1, true, false);
    return p.outer > 1 ? (size_t)(M * N * p.outer) * 4 : 0;
}
int matmul_f32(const void* a, const void* b, void* c, int64_t batch, int64_t a_batch, int64_t b_batch, int64_t M, int64_t N, int64_t K,
               bool trans_a, bool trans_b, void* workspace, size_t workspace_bytes, cudaStream_t st) {
    Args g{};
    g.a = (const float*)a; g.b = (const float*)b; g.c = (float*)c;
    g.M = (int)M; g.N = (int)N; g.K = (int)K;
    g.a_sm = trans_a ? 1 : K; g.a_sk = trans_a ? M : 1;
    g.b_sk = trans_b ? 1 : N; g.b_sn = trans_b ? K : 1;
    g.a_bs = a_batch > 1 ? M * K : 0; g.b_bs = b_batch > 1 ? K * N : 0; g.c_bs = M * N;
    g.c_numel = M * N * batch;
    Split p = plan(M, N, K, batch, batch == 1, false);
    if (p.outer > 1 && workspace_bytes < (size_t)g.c_numel * p.outer * 4) p = plan(M, N, K, batch, false, false);
    if (trans_a) return trans_b ? launch<MATMUL, false, true>(g, N, (int)batch, p, workspace, st) : launch<MATMUL, false, false>(g, N, (int)batch, p, workspace, st);
    return trans_b ? launch<MATMUL, true, true>(g, N, (int)batch, p, workspace, st) : launch<MATMUL, true, false>(g, N, (int)batch, p, workspace, st);
}

// Offsets are 32-bit, window coordinates 16-bit.
static bool conv_fits(const ConvShape& s) {
    const int64_t x = (int64_t)s.N * s.C * s.H * s.W, y = (int64_t)s.N * s.Co * s.OH * s.OW, w = (int64_t)s.C * s.Co * s.KH * s.KW;
    const auto small = [](int64_t v) { return v < 14000; };
    return s.groups <= 1 && x > 0 && y > 0 && w > 0 && x < kMaxElems - 4096 && y < kMaxElems - 4096 && w < kMaxElems - 4096 && small(s.H) && small(s.W) &&
           small(s.OH) && small(s.OW) && small(s.ph) && small(s.pw) && small((int64_t)s.KH * s.dh) && small((int64_t)s.KW * s.dw) &&
           small((int64_t)s.OH * s.sh) && small((int64_t)s.OW * s.sw) && s.Co <= 65535 * 32;
}
bool conv2d_f32_supported(const ConvShape& s) { return conv_fits(s); }
static void set_divisors(Args& g) {
    const ConvShape& s = g.s;
    g.by_kw = FastDiv(s.KW); g.by_kh = FastDiv(s.KH); g.by_ow = FastDiv(s.OW); g.by_oh = FastDiv(s.OH); g.by_pix = FastDiv(s.OH * s.OW);
}
int conv2d_f32(const void* x, const void* w, void* y, const ConvShape& s, cudaStream_t st) {
    Args g{};
    g.a = (const float*)w; g.b = (const float*)x; g.c = (float*)y; g.s = s;
    g.M = s.Co; g.N = s.N * s.OH * s.OW; g.K = s.C * s.KH * s.KW;
    set_divisors(g);
    return launch<FWD, true, false>(g, g.N, 1, plan(g.M, g.N, g.K, 1, false, true), nullptr, st);
}
bool conv2d_transpose_f32_supported(const ConvShape& s) { return conv_fits(s) && s.sh <= kMaxStride && s.sw <= kMaxStride; }
int conv2d_transpose_f32(const void* x, const void* w, void* y, const ConvShape& s, cudaStream_t st) {
    Args g{};
    g.a = (const float*)w; g.b = (const float*)x; g.c = (float*)y; g.s = s;
    const int classes = s.sh * s.sw;
    const auto residues = [](ResidueClass* out, int stride, int pad, int dil, int taps, int extent) {
        for (int r = 0; r < stride; r++) {
            ResidueClass c{0, 1, 0, (extent - r + stride - 1) / stride, FastDiv(1), FastDiv(1)};
            int prev = 0;
            for (int k = 0; k < taps; k++)
                if ((r + pad - k * dil) % stride == 0) {
                    if (c.count == 0) c.first = k; else if (c.count == 1) c.step = k - prev;
                    prev = k; c.count++;
                }
            c.by_count = FastDiv(std::max(1, c.count)); c.by_extent = FastDiv(std::max(1, c.extent));
            out[r] = c;
        }
    };
    residues(g.rh, s.sh, s.ph, s.dh, s.KH, s.OH);
    residues(g.rw, s.sw, s.pw, s.dw, s.KW, s.OW);
    g.M = s.Co; g.N = s.N * ((s.OH + s.sh - 1) / s.sh) * ((s.OW + s.sw - 1) / s.sw); g.K = s.C * ((s.KH + s.sh - 1) / s.sh) * ((s.KW + s.sw - 1) / s.sw);
    return launch<TRANSPOSED, true, false>(g, g.N, classes, plan(g.M, g.N, g.K, classes, false, true), nullptr, st);
}
static Args wgrad_args(const ConvShape& s) {
    Args g{};
    g.s = s;
    g.M = s.Co; g.N = s.C * s.KH * s.KW; g.K = s.N * s.OH * s.OW;
    g.c_numel = (int64_t)g.M * g.N;
    set_divisors(g);
    return g;
}
size_t conv2d_wgrad_f32_workspace(const ConvShape& s) {
    if (!conv_fits(s)) return 0;
    const Args g = wgrad_args(s);
    const Split p = plan(g.M, g.N, g.K, 1, true, true);
    return p.outer > 1 ? (size_t)(g.c_numel * p.outer) * 4 : 0;
}
int conv2d_wgrad_f32(const void* x, const void* dy, void* dw, const ConvShape& s, void* workspace, size_t workspace_bytes, cudaStream_t st) {
    Args g = wgrad_args(s);
    g.a = (const float*)dy; g.b = (const float*)x; g.c = (float*)dw;
    Split p = plan(g.M, g.N, g.K, 1, true, true);
    if (p.outer > 1 && workspace_bytes < (size_t)g.c_numel * p.outer * 4) p = plan(g.M, g.N, g.K, 1, false, true);
    return launch<WGRAD, true, true>(g, g.N, 1, p, workspace, st);
}

}  // namespace b200jt
