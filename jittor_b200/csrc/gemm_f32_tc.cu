// float32 matmul on the 5th-generation tensor cores: every operand is split into three bfloat16 parts that add up to it
// (x = x0 + x1 + x2, each part the rest rounded to nearest), and C is the sum of the six largest of the nine products of parts:
// x0 y0 + x0 y1 + x1 y0 + x1 y1 + x0 y2 + x2 y0. The other three are 2^-24 of a product together at most, and leave an error of 2^-27.4
// (2-norm, normal operands) by themselves. The products of bfloat16 parts are exact in float32.
//
//   split pass   both operands -> three planes of bfloat16 rows at a pitch TMA takes, one launch;
//   main kernel  the warp-specialised ring of the bfloat16 GEMM with stages of 32 of K that hold all planes of both operands
//                (48 KB: 24 KB of A, 24 KB of B, each in one or two TMA boxes), 12 MMAs a stage. The tensor core adds with
//                truncation, so nothing is summed there for long: the MMAs of two stages run from the smallest products to
//                the largest into a fresh accumulator, and the epilogue's warps add it to float32 registers while the next
//                two stages fill the other one. (After every stage, the way of the accumulators out of TMEM is what bounds a
//                pair: 456 instead of 349 us for 4096 x 2048 x 4096.)
//   error        relative to a 64-bit product (2-norm): normal operands 0.8e-7 to 1.3e-7 for K = 64 to 4096, where the kernel
//                on the FMA pipe, whose chains are longer, has 1.3e-7 to 8.1e-7. Operands of one sign (|normal|): 0.8e-7 to 1.3e-7,
//                of which 0.84e-7 is the truncation, always towards zero; the FMA kernel 0.5e-7 (500 x 4096 x 1000, K in short
//                chains over many CTAs) to 1.9e-7 (1024 x 777 x 1024). Collecting after every stage where CTAs work alone: one sign
//                0.66e-7 to 0.9e-7, but both signs up to 1.6e-7 and up to 4 % more time.
//   few tiles    K is split over a cluster of up to 8 CTAs that fold their tiles through distributed shared memory in rank
//                order; large products use CTA pairs (tcgen05 cta_group::2, 256 x 256 tiles).
//
// The operands are scaled by 2^24 on their way and the result by 2^-48: the tensor core takes subnormal parts for zero, and that way
// every part of every float32, subnormal ones among them, is a normal bfloat16.
// Infinities (they meet the zeros of the other operand's smaller parts), values from 2^104 and sums from 2^80 on leave the scaled range:
// there an element that came out infinite or NaN is computed again by float32 FMAs. The split pass notes each operand's largest
// magnitude, so that a NaN that stems from a NaN in an operand is left as it is. A CTA does this for its own tiles when its pipeline
// has run empty (a part of K each where a cluster shares a tile): no wait of the ring depends on it.
#include "gemm_simt.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <cooperative_groups.h>
#include <mutex>

namespace cg = cooperative_groups;

namespace b200jt {
namespace tcf32 {

using namespace tc;

constexpr int BM = 128, BK = 32, PLANES = 3;
constexpr int OP_BYTES = PLANES * BM * BK * 2;      // one operand's part of a stage: three planes of 128 x 32
constexpr int BOX_BYTES = PLANES * 64 * BK * 2;     // MN-major box: 64 of the operand's own axis x 32 of K, three planes
constexpr int STAGE_BYTES = 2 * OP_BYTES, STAGES = 4;
constexpr int GROUP = 2;                            // stages that are summed in one accumulator before it is collected
constexpr float SCALE = 16777216.f, UNSCALE = 1.f / SCALE / SCALE;
constexpr int THREADS = 320;                        // producer, MMA and 8 epilogue warps
constexpr int TURN_PITCH = 33;                      // floats per row of the square a warp turns around for its stores
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256 + 8 * 32 * TURN_PITCH * 4;
constexpr int MAX_SPLIT = 8;

struct Args {
    const float *a, *b;            // for elements that are computed again, their steps along M, K and N below
    int64_t a_sm, a_sk, b_sk, b_sn;
    int M, N, K, tiles_m, tiles_n, bn, k_blocks, units, group, splits;
    const float* peaks;            // largest magnitude that each block of the split pass met, a's blocks first
    int peaks_a, peaks_b;
};

// rows of 64 bytes, 64-byte swizzle: 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t desc_k64(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}

__device__ __forceinline__ bool finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

// Whether anything but a NaN of an operand can have made an element infinite or NaN: by the operands' largest magnitudes, infinities
// among them and NaN not. All threads of the CTA; `sm` holds two words for each warp.
__device__ __noinline__ bool left_range(const Args& A, float* sm) {
    float a = 0.f, b = 0.f;
    for (int i = threadIdx.x; i < A.peaks_a; i += THREADS) a = fmaxf(a, A.peaks[i]);
    for (int i = threadIdx.x; i < A.peaks_b; i += THREADS) b = fmaxf(b, A.peaks[A.peaks_a + i]);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) { a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, d)); b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, d)); }
    if ((threadIdx.x & 31) == 0) { sm[threadIdx.x >> 5] = a; sm[THREADS / 32 + (threadIdx.x >> 5)] = b; }
    __syncthreads();
    for (int w = 0; w < THREADS / 32; w++) { a = fmaxf(a, sm[w]); b = fmaxf(b, sm[THREADS / 32 + w]); }
    __syncthreads();
    return a >= 0x1p103f || b >= 0x1p103f || (double)a * b * A.K >= 0x1p79;
}

// 128 x 64 elements of the product from row m0 and column n0 on over k0 <= k < k1, as float32 FMAs, to `out` (rows x cols of them, or
// only those that are infinite or NaN there). 16 of K at a time go through shared memory, the next ones on their way meanwhile; 256
// threads hold 8 x 4 elements each and add 256 of K to a sum at a time. All threads of the CTA; bound by the latency of two computing
// warps a scheduler (FMA pipe 0.4 busy). 4096 x 2048 x 4096 with every element infinite: 4.1 ms, the FMA kernel 1.5; one infinity 1.4.
constexpr int AGAIN_K = 16, AGAIN_PA = BM + 4, AGAIN_PB = 64 + 4;
__device__ __noinline__ void fma_again(const Args& A, int m0, int n0, int k0, int k1, float* stage, float* out, int64_t pitch, int rows, int cols, bool only_odd) {
    constexpr int NA = (BM * AGAIN_K + THREADS - 1) / THREADS, NB = (64 * AGAIN_K + THREADS - 1) / THREADS, SIZE = AGAIN_K * (AGAIN_PA + AGAIN_PB);
    const bool ak = A.a_sk == 1, bk = A.b_sk == 1;              // neighbouring threads read along the axis that lies in memory
    // element e of an operand's 16 x `extent` part: where it goes among the 16 of K and along the operand's own axis
    const auto k_of = [](int e, int extent, bool kc) { return kc ? e % AGAIN_K : e / extent; };
    const auto own_of = [](int e, int extent, bool kc) { return kc ? e / AGAIN_K : e % extent; };
    const float *pa[NA], *pb[NB];                               // null where nothing is read
    float va[NA], vb[NB];
#pragma unroll
    for (int i = 0; i < NA; i++) {
        const int e = threadIdx.x + i * THREADS, r = m0 + own_of(e, BM, ak);
        pa[i] = e < BM * AGAIN_K && r < A.M ? A.a + r * A.a_sm + (k0 + k_of(e, BM, ak)) * A.a_sk : nullptr;
    }
#pragma unroll
    for (int i = 0; i < NB; i++) {
        const int e = threadIdx.x + i * THREADS, r = n0 + own_of(e, 64, bk);
        pb[i] = e < 64 * AGAIN_K && r < A.N ? A.b + r * A.b_sn + (k0 + k_of(e, 64, bk)) * A.b_sk : nullptr;
    }
    auto fetch = [&](int k) {
#pragma unroll
        for (int i = 0; i < NA; i++) {
            va[i] = pa[i] && k + k_of(threadIdx.x + i * THREADS, BM, ak) < k1 ? *pa[i] : 0.f;
            if (pa[i]) pa[i] += AGAIN_K * A.a_sk;
        }
#pragma unroll
        for (int i = 0; i < NB; i++) {
            vb[i] = pb[i] && k + k_of(threadIdx.x + i * THREADS, 64, bk) < k1 ? *pb[i] : 0.f;
            if (pb[i]) pb[i] += AGAIN_K * A.b_sk;
        }
    };
    auto put = [&](float* s) {
#pragma unroll
        for (int i = 0; i < NA; i++) {
            const int e = threadIdx.x + i * THREADS;
            if (e < BM * AGAIN_K) s[k_of(e, BM, ak) * AGAIN_PA + own_of(e, BM, ak)] = va[i];
        }
#pragma unroll
        for (int i = 0; i < NB; i++) {
            const int e = threadIdx.x + i * THREADS;
            if (e < 64 * AGAIN_K) s[AGAIN_K * AGAIN_PA + k_of(e, 64, bk) * AGAIN_PB + own_of(e, 64, bk)] = vb[i];
        }
    };
    const int ty = threadIdx.x / 16 * 8, tx = threadIdx.x % 16 * 4;
    unsigned long long sum[8][2] = {}, acc[8][2] = {};         // pairs of columns
    fetch(k0);
    put(stage);
    __syncthreads();
    for (int k = k0, it = 0; k < k1; k += AGAIN_K, it++) {
        const float* s = stage + (it & 1) * SIZE;
        if (k + AGAIN_K < k1) fetch(k + AGAIN_K);
        if (threadIdx.x < 256) {
#pragma unroll
            for (int q = 0; q < AGAIN_K; q++) {
                const float4 lo = *(const float4*)(s + q * AGAIN_PA + ty), hi = *(const float4*)(s + q * AGAIN_PA + ty + 4);
                const ulonglong2 y = *(const ulonglong2*)(s + AGAIN_K * AGAIN_PA + q * AGAIN_PB + tx);
                const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    unsigned long long xx;
                    asm("mov.b64 %0, {%1, %1};" : "=l"(xx) : "f"(x[i]));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][0]) : "l"(xx), "l"(y.x));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][1]) : "l"(xx), "l"(y.y));
                }
            }
            if (it % (256 / AGAIN_K) == 256 / AGAIN_K - 1)
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 2; j++) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum[i][j]) : "l"(acc[i][j])); acc[i][j] = 0; }
        }
        if (k + AGAIN_K < k1) put(stage + (~it & 1) * SIZE);
        __syncthreads();
    }
    if (threadIdx.x < 256)
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (ty + i < rows && tx + j < cols) {
                    const auto half = [&](unsigned long long v) { return __uint_as_float((uint32_t)(j & 1 ? v >> 32 : v)); };
                    float* at = out + (ty + i) * pitch + tx + j;
                    if (!only_odd || !finite(*at)) *at = half(sum[i][j / 2]) + half(acc[i][j / 2]);
                }
    __syncthreads();
}
__device__ __forceinline__ void tile_at(const Args& A, int u, int& tm, int& tn) {      // groups of tile-rows are walked together: B tiles stay in L2
    const int per_group = A.group * A.tiles_n, g = u / per_group, r = u - g * per_group;
    const int rows = min(A.group, A.tiles_m - g * A.group);
    tm = g * A.group + r % rows; tn = r / rows;
}

// The cluster's parts of a tile, each in its CTA's `mine`, are added up in rank order; a CTA stores 1 / splits of the rows. Returns
// whether one of this thread's elements came out infinite or NaN. AGAIN: only those that did are stored, by the thread that met them.
template <bool AGAIN>
__device__ __forceinline__ bool fold_parts(const Args& A, float* c, float* mine, int m0, int n0, int rank) {
    cg::cluster_group cluster = cg::this_cluster();
    const int splits = A.splits, rows = BM / splits, quads = A.bn / 4, pitch = A.bn + 4;
    const bool vec = (A.N & 3) == 0 && ((uintptr_t)c & 15) == 0;
    bool odd = false;
    cluster.sync();
    for (int e = threadIdx.x; e < rows * quads; e += THREADS) {
        const int r = rank * rows + e / quads, q = (e % quads) * 4;
        const int m = m0 + r, n = n0 + q;
        if (m >= A.M || n >= A.N) continue;
        float4 w[MAX_SPLIT], v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int p = 0; p < MAX_SPLIT; p++) if (p < splits) w[p] = *(const float4*)(cluster.map_shared_rank(mine, p) + r * pitch + q);
#pragma unroll
        for (int p = 0; p < MAX_SPLIT; p++) if (p < splits) { v.x += w[p].x; v.y += w[p].y; v.z += w[p].z; v.w += w[p].w; }
        const float scale = AGAIN ? 1.f : UNSCALE, o[4] = {v.x * scale, v.y * scale, v.z * scale, v.w * scale};
        float* out = c + (int64_t)m * A.N + n;
        if constexpr (AGAIN) {
#pragma unroll
            for (int i = 0; i < 4; i++) if (n + i < A.N && !finite(out[i])) out[i] = o[i];
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) odd |= !finite(o[i]);
            if (vec) *(float4*)out = make_float4(o[0], o[1], o[2], o[3]);
            else
#pragma unroll
                for (int i = 0; i < 4; i++) if (n + i < A.N) out[i] = o[i];
        }
    }
    return odd;
}

// What a CTA (or the cluster of one tile) does when an element of its tiles came out infinite or NaN.
template <bool PAIR>
__device__ __noinline__ void compute_again(const Args& A, float* c, unsigned char* smem, float* sm) {
    constexpr int CTAS = PAIR ? 2 : 1;
    const int splits = PAIR ? 1 : A.splits, rank = PAIR || splits > 1 ? (int)cluster_rank() : 0;
    const int first = blockIdx.x / (CTAS * splits), step = gridDim.x / (CTAS * splits);
    if (!left_range(A, sm)) return;
    int tm, tn;
    if (!PAIR && splits > 1) {
        const int pitch = A.bn + 4;
        float* mine = (float*)smem;
        tile_at(A, first, tm, tn);
        for (int n = 0; n < A.bn; n += 64)
            fma_again(A, tm * BM, tn * A.bn + n, A.k_blocks * rank / splits * BK, min(A.K, A.k_blocks * (rank + 1) / splits * BK), mine + BM * pitch, mine + n, pitch,
                      BM, min(64, A.bn - n), false);
        fold_parts<true>(A, c, mine, tm * BM, tn * A.bn, rank);
        cg::this_cluster().sync();     // no CTA leaves while its tile is read
        return;
    }
    for (int u = first; u < A.units; u += step) {
        tile_at(A, u, tm, tn);
        const int m0 = (tm * CTAS + (PAIR ? rank : 0)) * BM, rows = min(BM, A.M - m0), end = min(A.N, (tn + 1) * A.bn);
        for (int n0 = tn * A.bn; n0 < end; n0 += 64) {
            const int cols = min(64, end - n0);
            float* out = c + (int64_t)m0 * A.N + n0;
            bool odd = false;
            for (int e = threadIdx.x; e < rows * 64; e += THREADS) odd |= e % 64 < cols && !finite(out[(int64_t)(e / 64) * A.N + e % 64]);
            if (__syncthreads_or(odd)) fma_again(A, m0, n0, 0, A.K, (float*)smem, out, A.N, rows, cols, true);
        }
    }
}

// PAIR: two CTAs share one tile of 256 rows, each with its own rows of A and half of the columns of B.
// AMN / BMN: the operand's own axis (M / N) is the contiguous one in memory.
template <bool PAIR, bool AMN, bool BMN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, float* __restrict__ c,
                const __grid_constant__ Args A) {
    constexpr int CTAS = PAIR ? 2 : 1, CHUNKS = PAIR ? 4 : 2;           // 32-column chunks of an epilogue warp
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + STAGES * STAGE_BYTES);
    uint64_t* full = bars;
    uint64_t* empty = bars + STAGES;
    uint64_t* acc_full = bars + 2 * STAGES;
    uint64_t* acc_empty = bars + 2 * STAGES + 2;
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 4);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    volatile int* odd_flag = abort_flag + 1;                           // an element of this CTA's (or of its cluster's) came out infinite or NaN
    float* turn = (float*)(smem + STAGES * STAGE_BYTES + 256);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int splits = PAIR ? 1 : A.splits;                            // CTAs of a cluster that share a tile's K
    const int rank = PAIR || splits > 1 ? (int)cluster_rank() : 0;
    const int side = PAIR ? rank : 0, split = PAIR ? 0 : rank;
    const int first = blockIdx.x / (CTAS * splits), step = gridDim.x / (CTAS * splits);
    const int kb0 = A.k_blocks * split / splits, kb1 = A.k_blocks * (split + 1) / splits;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int b = 0; b < 2; b++) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, 8 * CTAS); }
        *abort_flag = *odd_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc<CTAS>(tmem_slot);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    // everything above runs while the split pass drains; its planes, and c, are touched below only
    asm volatile("griddepcontrol.wait;" ::: "memory");

    if (warp == 0) {
        if (lane == 0) {
            const int half = A.bn / CTAS, boxes = (half + 63) / 64;
            const uint32_t bytes = CTAS * (uint32_t)(OP_BYTES + (BMN ? boxes * BOX_BYTES : PLANES * half * BK * 2));
            int stage = 0; uint32_t phase = 0;
            bool ok = true;
            for (int u = first; u < A.units && ok; u += step) {
                int tm, tn;
                tile_at(A, u, tm, tn);
                const int row0 = (tm * CTAS + side) * BM, col0 = tn * A.bn + side * half;
                for (int kb = kb0; kb < kb1; kb++) {
                    if (!(ok = mbar_wait(empty + stage, phase ^ 1, abort_flag, 31))) break;
                    unsigned char* sa = smem + stage * STAGE_BYTES;
                    unsigned char* sb = sa + OP_BYTES;
                    if (side == 0) mbar_expect_tx(full + stage, bytes);
                    const uint32_t bar = PAIR ? leader_addr(full + stage) : smem_u32(full + stage);
                    if (AMN) {
                        tma_load_tile<CTAS>(sa, &map_a, bar, row0, kb * BK, 0);
                        tma_load_tile<CTAS>(sa + BOX_BYTES, &map_a, bar, row0 + 64, kb * BK, 0);
                    } else tma_load_tile<CTAS>(sa, &map_a, bar, kb * BK, row0, 0);
                    if (BMN) {
                        for (int q = 0; q < boxes; q++) tma_load_tile<CTAS>(sb + q * BOX_BYTES, &map_b, bar, col0 + q * 64, kb * BK, 0);
                    } else tma_load_tile<CTAS>(sb, &map_b, bar, kb * BK, col0, 0);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
            if (!ok) {
                for (int s = 0; s < STAGES; s++)
                    for (uint32_t i = 0; i < 4096 && !mbar_try(full + s, 0) && !mbar_try(full + s, 1); i++) __nanosleep(64);
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && side == 0) {
            const uint32_t idesc = make_idesc(BM * CTAS, A.bn, BMN) | ((AMN ? 1u : 0u) << 15);
            // 16 of K further: 32 bytes inside a swizzled row, or 16 rows of 128 bytes. Planes: in units of 16 bytes
            constexpr int A_KSTEP = AMN ? 128 : 2, B_KSTEP = BMN ? 128 : 2, A_PLANE = (AMN ? 64 : BM) * BK * 2 / 16;
            const int b_plane = (BMN ? 64 : A.bn / CTAS) * BK * 2 / 16;
            int stage = 0; uint32_t phase = 0;
            int it = 0;
            bool ok = true;
            for (int u = first; u < A.units && ok; u += step) {
                for (int kb = kb0; kb < kb1; kb += GROUP, it++) {
                    const int buf = it & 1, n = min(GROUP, kb1 - kb);
                    if (!(ok = mbar_wait<PAIR>(acc_empty + buf, ((it >> 1) & 1) ^ 1, abort_flag, 32))) break;
                    const uint32_t d = tmem_base + buf * 256;
                    uint64_t da[GROUP], db[GROUP];
#pragma unroll
                    for (int i = 0; i < GROUP; i++) {
                        if (i >= n) break;
                        const int at = stage + i < STAGES ? stage + i : stage + i - STAGES;
                        if (!(ok = mbar_wait(full + at, phase ^ (uint32_t)(stage + i >= STAGES), abort_flag, 33))) break;
                        const uint32_t sa = smem_u32(smem + at * STAGE_BYTES), sb = sa + OP_BYTES;
                        da[i] = AMN ? make_smem_desc_mn(sa, BOX_BYTES, 1024) : desc_k64(sa);
                        db[i] = BMN ? make_smem_desc_mn(sb, BOX_BYTES, 1024) : desc_k64(sb);
                    }
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int p = 0; p < 6; p++) {
                        constexpr int PA[6] = {1, 0, 2, 0, 1, 0}, PB[6] = {1, 2, 0, 1, 0, 0};
#pragma unroll
                        for (int i = 0; i < GROUP; i++) {
                            if (i >= n) break;
#pragma unroll
                            for (int k = 0; k < BK / UMMA_K; k++)
                                umma_f16<CTAS>(d, da[i] + PA[p] * A_PLANE + k * A_KSTEP, db[i] + (uint64_t)(PB[p] * b_plane) + k * B_KSTEP, idesc, (p | i | k) != 0);
                        }
                    }
                    for (int i = 0; i < n; i++) {
                        umma_commit<CTAS>(empty + stage);
                        if (++stage == STAGES) { stage = 0; phase ^= 1; }
                    }
                    umma_commit<CTAS>(acc_full + buf);
                }
            }
        }
    } else {
        const int quad = warp & 3, grp = (warp - 2) >> 2;
        float* square = turn + (warp - 2) * 32 * TURN_PITCH;
        int it = 0;
        bool ok = true;
        for (int u = first; u < A.units && ok; u += step) {
            int tm, tn;
            tile_at(A, u, tm, tn);
            float acc[CHUNKS][32];
#pragma unroll
            for (int i = 0; i < CHUNKS; i++)
#pragma unroll
                for (int e = 0; e < 32; e++) acc[i][e] = 0.f;
            for (int kb = kb0; kb < kb1; kb += GROUP, it++) {
                const int buf = it & 1;
                ok = mbar_wait(acc_full + buf, (it >> 1) & 1, abort_flag, 34);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + buf * 256 + grp * 32;
#pragma unroll
                for (int i = 0; i < CHUNKS; i++) {
                    if (grp * 32 + i * 64 >= A.bn) break;
                    uint32_t r[32];
                    tmem_ld32(taddr + i * 64, r);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int e = 0; e < 32; e++) acc[i][e] += __uint_as_float(r[e]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) { if (PAIR) mbar_arrive_leader(acc_empty + buf); else mbar_arrive(acc_empty + buf); }
            }
            if (!ok) break;
            const int row0 = (tm * CTAS + side) * BM + quad * 32;
            if (splits > 1) {                                // this CTA's part of the tile, where the ring was: all its loads have been used
                float* mine = (float*)smem + (quad * 32 + lane) * (A.bn + 4) + grp * 32;
#pragma unroll
                for (int i = 0; i < CHUNKS; i++) {
                    if (grp * 32 + i * 64 >= A.bn) break;
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        *(float4*)(mine + i * 64 + q * 4) = make_float4(acc[i][q * 4], acc[i][q * 4 + 1], acc[i][q * 4 + 2], acc[i][q * 4 + 3]);
                }
                continue;
            }
#pragma unroll
            for (int i = 0; i < CHUNKS; i++) {
                const int ch = grp * 32 + i * 64, col0 = tn * A.bn + ch;
                if (ch >= A.bn || row0 >= A.M || col0 >= A.N) break;     // uniform over the warp
                bool odd = false;
#pragma unroll
                for (int e = 0; e < 32; e++) odd |= !finite(acc[i][e]);
                if (odd) *odd_flag = 1;
                __syncwarp();
#pragma unroll
                for (int e = 0; e < 32; e++) square[lane * TURN_PITCH + e] = acc[i][e];
                __syncwarp();
                float* out = c + (int64_t)row0 * A.N + col0 + lane;
                const int rows = min(32, A.M - row0);
                if (col0 + lane < A.N)
#pragma unroll 8
                    for (int r = 0; r < rows; r++) out[(int64_t)r * A.N] = square[r * TURN_PITCH + lane] * UNSCALE;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync();          // neither CTA leaves while the other may still signal it or read its tiles
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_dealloc<CTAS>(tmem_base);
    }
    bool odd = *odd_flag;
    if (!PAIR && splits > 1) {
        int tm, tn;
        tile_at(A, first, tm, tn);     // one tile to a cluster
        cg::cluster_group cluster = cg::this_cluster();
        if (fold_parts<false>(A, c, (float*)smem, tm * BM, tn * A.bn, rank))
            for (int p = 0; p < splits; p++) *cluster.map_shared_rank((int*)odd_flag, p) = 1;
        cluster.sync();                // no CTA leaves while its tile is read
        odd = *odd_flag;
    }
    if (odd) compute_again<PAIR>(A, c, smem, turn);
}

// rows of float32 -> three planes of bfloat16 rows (pitch a multiple of 8; what lies past a row's end is never loaded), eight
// elements a thread. Two jobs in one launch: the first `blocks_a` blocks are a's.
struct SplitJob { const float* in; __nv_bfloat16* out; int64_t rows, chunks, plane; int cols, vec; };
__device__ __forceinline__ void split_pair(float x, float y, uint32_t* p) {
    x *= SCALE; y *= SCALE;
#pragma unroll
    for (int i = 0; i < PLANES; i++) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
        p[i] = *reinterpret_cast<const uint32_t*>(&h);
        const float2 f = __bfloat1622float2(h);
        x -= f.x; y -= f.y;
    }
}
__global__ void __launch_bounds__(256)
split_rows_kernel(const __grid_constant__ SplitJob a, const __grid_constant__ SplitJob b, int blocks_a, float* __restrict__ peaks) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ unsigned most[8];
    float peak = 0.f;
    const bool second = (int)blockIdx.x >= blocks_a;
    const SplitJob& job = second ? b : a;
    const int64_t n = job.rows * job.chunks, stride = (int64_t)(second ? gridDim.x - blocks_a : blocks_a) * 256;
    for (int64_t i = (int64_t)(blockIdx.x - (second ? blocks_a : 0)) * 256 + threadIdx.x; i < n; i += stride) {
        const int64_t row = i / job.chunks;
        const int c0 = (int)(i - row * job.chunks) * 8;
        const float* p = job.in + row * job.cols + c0;
        float v[8];
        if (job.vec && c0 + 8 <= job.cols) {
            const float4 lo = *(const float4*)p, hi = *(const float4*)(p + 4);
            v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
        } else {
#pragma unroll
            for (int e = 0; e < 8; e++) v[e] = c0 + e < job.cols ? p[e] : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 8; e++) peak = fmaxf(peak, fabsf(v[e]));         // of a number and NaN the number
        uint32_t q[4][PLANES];
#pragma unroll
        for (int e = 0; e < 4; e++) split_pair(v[2 * e], v[2 * e + 1], q[e]);
#pragma unroll
        for (int s = 0; s < PLANES; s++)
            *reinterpret_cast<uint4*>(job.out + s * job.plane + i * 8) = make_uint4(q[0][s], q[1][s], q[2][s], q[3][s]);
    }
    const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(peak));         // of floats from 0 up, as of their bits
    if ((threadIdx.x & 31) == 0) most[threadIdx.x >> 5] = top;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int w = 0; w < 8; w++) t = max(t, most[w]);
        peaks[blockIdx.x] = __uint_as_float(t);
    }
}

// [3 planes][rows][pitch] bfloat16; boxes of three planes x box_rows rows x box_cols columns
static bool make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t pitch, int box_cols, int box_rows) {
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, PLANES};
    cuuint64_t strides[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)(rows * pitch) * 2};
    cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, PLANES};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool PAIR>
static const void* kernel_of(bool amn, bool bmn) {
    return amn ? (bmn ? (const void*)gemm_f32_kernel<PAIR, true, true> : (const void*)gemm_f32_kernel<PAIR, true, false>)
               : (bmn ? (const void*)gemm_f32_kernel<PAIR, false, true> : (const void*)gemm_f32_kernel<PAIR, false, false>);
}
static const void* kernel_of(bool pair, bool amn, bool bmn) { return pair ? kernel_of<true>(amn, bmn) : kernel_of<false>(amn, bmn); }

// How many tiles run at once with 1, 2, 4 or 8 CTAs to a tile's K, or with a pair to a tile; zeros on error.
struct Slots { int pair = 0, by_split[4] = {}; };
static const Slots& slots() {
    static std::once_flag once;
    static Slots s;
    std::call_once(once, [] {
        for (int f = 0; f < 8; f++)
            if (cudaFuncSetAttribute(kernel_of(f & 4, f & 1, f & 2), cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) return;
        const auto clusters = [](const void* kernel, int size) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = size; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(kNumSMs / size * size); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = SMEM_BYTES; cfg.attrs = at; cfg.numAttrs = 1;
            int n = 0;
            return cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess ? std::min(n, kNumSMs / size) : 0;
        };
        Slots r;
        r.pair = clusters(kernel_of(true, false, false), 2);
        for (int i = 0; i < 4; i++) r.by_split[i] = i ? clusters(kernel_of(false, false, false), 1 << i) : kNumSMs;
        s = r;
    });
    return s;
}

struct Plan { bool tc, pair; int bn, splits; };

// Tile, cluster and path by estimated time. A stage of 32 of K measured 0.84 us with 128 columns on a CTA (its 48 KB in and the
// 96 KB that the MMAs read share the SM's 128 bytes a cycle) and 1.18 us with 256 on a pair; the split pass reads 4 bytes an
// element and writes 6. The FMA kernel stays where that pass costs more than it gives -- few rows by a large matrix (16 x 4096 x
// 4096: 32 and 61 us), small products (300 x 300 x 300: 10 and 14), short K by a wide result (9472 x 39 x 1024: 26.3 and 26.6) --
// and the estimates are within a fifth of the times measured for 28 shapes; 500 x 777 x 1000: 29 and 18 us, 1024 x 1024 x 1024: 61
// and 28, 4096 x 2048 x 4096: 1410 and 349. 3 us in hand: of 54 products drawn from 16 to 9472 a side none was then slower than
// the FMA kernel by more than the timer shows (with 1 us in hand, and half of what the stores take: 4588 x 72 x 3272, 64 and 69).
// `force`: B200JT_F32TC, with which tests force each path in turn; the switches of its tiles count only beside it.
static Plan estimate(int64_t M, int64_t N, int64_t K, const char* force) {
    Plan best{false, false, 128, 1};
    double best_ns = 1e30;
    const auto set = [&](const char* name) { return force ? getenv(name) : nullptr; };
    const char* fp = set("B200JT_F32TC_PAIR"); const char* fb = set("B200JT_F32TC_BN"); const char* fs = set("B200JT_F32TC_SPLITS");
    const int64_t kb = (K + BK - 1) / BK;
    for (int pair = 0; pair < 2; pair++) {
        if ((fp && atoi(fp) != pair) || (pair && !slots().pair)) continue;
        const int tile_m = BM * (1 + pair);
        for (int bn = pair ? 128 : 32; bn <= (pair ? 256 : 128); bn += pair ? 64 : 32) {
            if (fb ? atoi(fb) != bn : bn > 32 && bn - 32 >= N) continue;
            const double stage = pair ? 600 + 2.27 * bn : 500 + 2.65 * bn;
            const int64_t tiles = (M + tile_m - 1) / tile_m * ((N + bn - 1) / bn);
            for (int i = 0; i <= (pair ? 0 : 3); i++) {
                const int s = 1 << i, at_once = pair ? slots().pair : slots().by_split[i];
                if (fs && !pair ? atoi(fs) != s : s > 1 && (tiles > at_once || kb / s < 2)) continue;
                if (s > kb || !at_once) continue;
                const double ns = 4500 + 10.0 * (M * K + K * N) / 4000 + (double)((tiles + at_once - 1) / at_once) * ((double)((kb + s - 1) / s) * stage + bn * 16.0) + (s > 1 ? 1500 : 0);
                if (ns < best_ns) { best_ns = ns; best = {true, pair != 0, bn, s}; }
            }
        }
    }
    best.tc = best_ns < 1e30 && (force ? atoi(force) != 0 : best_ns + 3000 < matmul_f32_ns(M, N, K));
    return best;
}

// Some 400 candidates of both paths, a few us: each thread keeps its last 64 plans.
static Plan plan_for(int64_t M, int64_t N, int64_t K) {
    if (const char* force = getenv("B200JT_F32TC")) return estimate(M, N, K, force);
    struct Entry { int64_t M = -1, N = 0, K = 0; Plan p; };
    static thread_local Entry kept[64];
    uint64_t h = 0;
    for (int64_t k : {M, N, K}) h = (h ^ (uint64_t)k) * 0x9E3779B97F4A7C15ull;
    Entry& e = kept[h >> 58];
    if (e.M != M || e.N != N || e.K != K) e = {M, N, K, estimate(M, N, K, nullptr)};
    return e.p;
}

inline int64_t pitch8(int64_t n) { return (n + 7) / 8 * 8; }
inline size_t plane_elems(int64_t rows, int64_t cols) { return (size_t)rows * pitch8(cols); }
constexpr size_t PEAK_BYTES = 2 * 8 * kNumSMs * sizeof(float);          // a word for every block of the split pass
inline size_t planes_bytes(int64_t rows, int64_t cols) { return (plane_elems(rows, cols) * PLANES * 2 + 255) & ~(size_t)255; }

}  // namespace tcf32

bool matmul_f32_tc_wanted(int64_t M, int64_t N, int64_t K) {
    return matmul_f32_supported(1, M, N, K) && K >= 32 && M < (1LL << 30) && N < (1LL << 30) && K < (1LL << 30) && tc::encode_fn() != nullptr &&
           tcf32::plan_for(M, N, K).tc;
}
size_t matmul_f32_tc_workspace(int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b) {
    using namespace tcf32;
    return (trans_a ? planes_bytes(K, M) : planes_bytes(M, K)) + (trans_b ? planes_bytes(N, K) : planes_bytes(K, N)) + PEAK_BYTES + 256;
}
int matmul_f32_tc(const void* a, const void* b, void* c, int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b, void* workspace, cudaStream_t st) {
    using namespace tcf32;
    const Plan p = plan_for(M, N, K);
    const bool amn = trans_a, bmn = !trans_b;
    __nv_bfloat16* pa = (__nv_bfloat16*)(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    const int64_t ra = amn ? K : M, ca = amn ? M : K, rb = bmn ? K : N, cb = bmn ? N : K;
    __nv_bfloat16* pb = (__nv_bfloat16*)((unsigned char*)pa + planes_bytes(ra, ca));
    float* peaks = (float*)((unsigned char*)pb + planes_bytes(rb, cb));
    unsigned ga, gb;
    {
        const auto job = [](const void* in, __nv_bfloat16* out, int64_t rows, int64_t cols) {
            return SplitJob{(const float*)in, out, rows, pitch8(cols) / 8, (int64_t)plane_elems(rows, cols), (int)cols, cols % 4 == 0 && (uintptr_t)in % 16 == 0};
        };
        const SplitJob ja = job(a, pa, ra, ca), jb = job(b, pb, rb, cb);
        ga = grid_for(ja.rows * ja.chunks, 256); gb = grid_for(jb.rows * jb.chunks, 256);
        split_rows_kernel<<<ga + gb, 256, 0, st>>>(ja, jb, (int)ga, peaks);
        B200JT_LAUNCH_CHECK();
    }
    const int ctas = p.pair ? 2 : 1;
    CUtensorMap ma, mb;
    if (!(amn ? make_map(&ma, pa, K, M, pitch8(M), 64, BK) : make_map(&ma, pa, M, K, pitch8(K), BK, BM)) ||
        !(bmn ? make_map(&mb, pb, K, N, pitch8(N), 64, BK) : make_map(&mb, pb, N, K, pitch8(K), BK, p.bn / ctas)))
        return fail(-4, "matmul: cuTensorMapEncodeTiled failed");
    Args A;
    A.a = (const float*)a; A.b = (const float*)b;
    A.a_sm = trans_a ? 1 : K; A.a_sk = trans_a ? M : 1; A.b_sk = trans_b ? 1 : N; A.b_sn = trans_b ? K : 1;
    A.M = (int)M; A.N = (int)N; A.K = (int)K; A.bn = p.bn; A.k_blocks = (int)((K + BK - 1) / BK); A.splits = p.splits;
    A.tiles_m = (int)((M + BM * ctas - 1) / (BM * ctas)); A.tiles_n = (int)((N + p.bn - 1) / p.bn);
    A.group = std::max(1, 1024 / (BM * ctas));
    A.peaks = peaks; A.peaks_a = (int)ga; A.peaks_b = (int)gb;
    const int64_t units = (int64_t)A.tiles_m * A.tiles_n;
    if (units * p.splits >= (1LL << 30)) return fail(-1, "matmul: too many tiles");
    A.units = (int)units;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = ctas * p.splits; at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(p.splits > 1 ? units * p.splits : std::min<int64_t>(units, p.pair ? slots().pair : kNumSMs) * ctas));
    cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = SMEM_BYTES; cfg.stream = st; cfg.attrs = at;
    cfg.numAttrs = ctas * p.splits > 1 ? 2 : 1;
    void* args[] = {&ma, &mb, &c, &A};
    B200JT_CUDA(cudaLaunchKernelExC(&cfg, kernel_of(p.pair, amn, bmn), args));
    return 0;
}

int tcf32_status_fetch_and_clear() { return tc::status_fetch_and_clear(); }

}  // namespace b200jt
