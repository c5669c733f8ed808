// bf16 GEMM on the 5th-generation tensor cores: C[M,N] = A[M,K] . Bt[N,K]^T, fp32 accumulation in TMEM.
//
// The broadcast-multiply-sum matmul of the reference (python/jittor/nn.py:157-159) is a dense contraction; its
// relay is cublasGemmEx (python/jittor/extern/cuda/cublas/ops/cublas_matmul_op.cc:117-123). Here it is one
// persistent, warp-specialised kernel:
//   warp 0     TMA producer: cp.async.bulk.tensor loads of 64-deep bf16 tiles, 128-byte swizzle, into a 192 KB
//              shared-memory ring, completion on mbarriers;
//   warp 1     MMA issuer: one lane issues tcgen05.mma.kind::f16 (M = 128 per CTA, N <= 256, K = 16) on shared-memory
//              descriptors, for one CTA or for a pair of CTAs; accumulators live in TMEM; tcgen05.commit releases ring
//              slots / publishes accumulators;
//   warps 2-9  epilogue: tcgen05.ld (32 lanes x 32 columns), fp32 -> bf16, 16-byte global stores.
// Work items are scheduled statically in groups of tile-rows for L2 reuse; one CTA per SM. Ragged M/N/K edges rely on TMA
// zero fill and masked stores. No load is multicast.
// Every mbarrier wait is bounded: on expiry the CTA records a status word, stops issuing, drains and frees TMEM.
#include "gemm_simt.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <cstring>
#include <mutex>

namespace b200jt {

namespace tc {

constexpr int BM = 128, BK = 64;                    // rows of one CTA's MMA tile; BK * 2 B = 128 B = swizzle width
constexpr int MAX_BN = 256;
constexpr int A_BYTES = BM * BK * 2;
constexpr int BOX_BYTES = 64 * BK * 2;              // one MN-major box: 64 elements of the operand's own axis x 64 of K
constexpr int THREADS = 320;                        // producer, MMA and 8 epilogue warps
constexpr int EPI_PITCH = 40;                       // bf16 per staged row: 16-byte aligned, eight rows on different banks

// What bounds a large product is the tensor pipe as long as the operands' way from L2 into shared memory stays below it: a
// 128 x 256 tile per SM takes 48 KB per 4.2 MFLOP, a 256 x 256 tile per CTA pair 32 KB per SM, a 512 x 256 tile per pair 48 KB
// per 8.4 MFLOP. 16384 x 4096 x 4096: 375, 342 and 356 us (1467, 1607 and 1542 TFLOP/s; 256 x 256 per single CTA was 465);
// 4096 x 4096 x 16384 with both operands MN-major: 550, 429 and 390 us (and 560 with A transposed by a pass of its own).
//   PAIR  two CTAs of a cluster share one accumulator of 256 rows (tcgen05 cta_group::2): each loads its 128 rows of A and
//         HALF of the Bt tile, the leader's MMA reads both. No load is multicast.
//   MT    accumulators per CTA: 2 re-uses each Bt stage for two MMAs and takes all 512 TMEM columns; with 1 there are two
//         accumulator sets and the epilogue of a tile overlaps the next tile's MMAs.
template <bool PAIR, int MT> struct Cfg {
    static constexpr int CTAS = PAIR ? 2 : 1;
    static constexpr int B_BYTES = MAX_BN / CTAS * BK * 2;
    static constexpr int STAGE_BYTES = MT * A_BYTES + B_BYTES;
    static constexpr int STAGES = (192 * 1024) / STAGE_BYTES;
    static constexpr int EPI_BYTES = 8 * 32 * EPI_PITCH * 2;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/ + EPI_BYTES;
    static constexpr int NBUF = 2 / MT;             // accumulator sets in the 512 TMEM columns
    static constexpr int TILE_M = CTAS * MT * BM;
};

struct GemmArgs {
    int M, N, K;
    int tiles_m, tiles_n, bn, k_blocks;
    int units;                     // work items: batch x tiles, or `whole` tiles and then splits x the others
    int batch, splits, group;      // group: tile-rows that are walked together (L2 reuse of the Bt tiles)
    int whole;                     // tiles that are not split (splits > 1)
    int a_batched, b_batched;      // an operand whose batch extent is 1 is shared by all products
};

struct Unit { int batch, tm, tn, kb0, kb1, part; };      // part: place among the partial tiles, -1: the product itself
__device__ __forceinline__ void tile_at(const GemmArgs& A, int t, int& tm, int& tn) {
    const int per_group = A.group * A.tiles_n, g = t / per_group, r = t - g * per_group;
    const int rows = min(A.group, A.tiles_m - g * A.group);
    tm = g * A.group + r % rows; tn = r / rows;
}
__device__ __forceinline__ Unit unit_at(const GemmArgs& A, int u) {
    Unit w;
    const int tiles = A.tiles_m * A.tiles_n;
    w.batch = 0; w.kb0 = 0; w.kb1 = A.k_blocks; w.part = -1;
    if (A.splits == 1) { w.batch = u / tiles; u -= w.batch * tiles; }
    else if (u >= A.whole) {
        w.part = u - A.whole;
        const int others = tiles - A.whole, split = w.part / others;
        u -= split * others;
        w.kb0 = (int)((int64_t)A.k_blocks * split / A.splits);
        w.kb1 = (int)((int64_t)A.k_blocks * (split + 1) / A.splits);
    }
    tile_at(A, u, w.tm, w.tn);
    return w;
}

// AMN / BMN: the operand's own axis (M / N) is the contiguous one in memory; it is then loaded in 64 x 64 boxes and used
// as an MN-major operand, so no operand is ever transposed by a pass of its own.
// Accumulators leave as bf16 in c, or -- where K is split -- as fp32 partial tiles in part[split][split tile][TILE_M][bn], which
// fold_kernel adds in split order. The tensor maps are 3-D ([batch][rows][cols]).
template <bool PAIR, int MT, bool AMN, bool BMN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 __nv_bfloat16* __restrict__ c, float* __restrict__ part, const __grid_constant__ GemmArgs A) {
    using F = Cfg<PAIR, MT>;
    constexpr int STAGES = F::STAGES, STAGE_BYTES = F::STAGE_BYTES, NBUF = F::NBUF, CTAS = F::CTAS;
    extern __shared__ unsigned char smem_raw[];
    // operand tiles need 1024-byte alignment for the 128-byte swizzle
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + STAGES * STAGE_BYTES);
    uint64_t* full = bars;                       // [STAGES] TMA -> MMA (a pair uses the leader's)
    uint64_t* empty = bars + STAGES;             // [STAGES] MMA -> TMA
    uint64_t* acc_full = bars + 2 * STAGES;      // [2] MMA -> epilogue
    uint64_t* acc_empty = bars + 2 * STAGES + 2; // [2] epilogue -> MMA (a pair uses the leader's)
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 4);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    unsigned char* epi = smem + STAGES * STAGE_BYTES + 256;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = PAIR ? (int)cluster_rank() : 0;
    const int first = blockIdx.x / CTAS, step = gridDim.x / CTAS;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int b = 0; b < NBUF; b++) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, 8 * CTAS); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc<CTAS>(tmem_slot);             // all 512 columns
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync();                               // the peer's barriers exist before anything signals them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            const int half = A.bn / CTAS;                   // this CTA's columns of the Bt tile
            const int boxes = (half + 63) / 64;
            const uint32_t bytes = CTAS * (uint32_t)(MT * A_BYTES + (BMN ? boxes * BOX_BYTES : half * BK * 2));
            int stage = 0; uint32_t phase = 0;
            bool ok = true;
            for (int u = first; u < A.units && ok; u += step) {
                const Unit w = unit_at(A, u);
                const int ba = A.a_batched ? w.batch : 0, bb = A.b_batched ? w.batch : 0;
                const int col0 = w.tn * A.bn + rank * half;
                for (int kb = w.kb0; kb < w.kb1; kb++) {
                    if (!(ok = mbar_wait(empty + stage, phase ^ 1, abort_flag, 1))) break;
                    unsigned char* sa = smem + stage * STAGE_BYTES;
                    if (rank == 0) mbar_expect_tx(full + stage, bytes);      // both CTAs' bytes
                    const uint32_t bar = PAIR ? leader_addr(full + stage) : smem_u32(full + stage);
#pragma unroll
                    for (int j = 0; j < MT; j++) {
                        const int row0 = w.tm * F::TILE_M + (j * CTAS + rank) * BM;
                        if (AMN) {
                            tma_load_tile<CTAS>(sa + j * A_BYTES, &map_a, bar, row0, kb * BK, ba);
                            tma_load_tile<CTAS>(sa + j * A_BYTES + BOX_BYTES, &map_a, bar, row0 + 64, kb * BK, ba);
                        } else tma_load_tile<CTAS>(sa + j * A_BYTES, &map_a, bar, kb * BK, row0, ba);
                    }
                    unsigned char* sb = sa + MT * A_BYTES;
                    if (BMN) {
                        for (int q = 0; q < boxes; q++) tma_load_tile<CTAS>(sb + q * BOX_BYTES, &map_b, bar, col0 + q * 64, kb * BK, bb);
                    } else tma_load_tile<CTAS>(sb, &map_b, bar, kb * BK, col0, bb);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
            if (!ok) {
                // give copies that are already in flight a bounded chance to land before the CTA goes away
                for (int s = 0; s < STAGES; s++)
                    for (uint32_t i = 0; i < 4096 && !mbar_try(full + s, 0) && !mbar_try(full + s, 1); i++) __nanosleep(64);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (of a pair: the leader's) ----------------
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = make_idesc(BM * CTAS, A.bn, BMN) | ((AMN ? 1u : 0u) << 15);
            // advancing K by 16: K-major +32 B inside the swizzled row (+2 units of 16 B); MN-major 16 rows of 128 B
            constexpr int A_KSTEP = AMN ? (UMMA_K * 128) / 16 : 2, B_KSTEP = BMN ? (UMMA_K * 128) / 16 : 2;
            int stage = 0; uint32_t phase = 0;
            int it = 0;
            bool ok = true;
            for (int u = first; u < A.units && ok; u += step, it++) {
                const Unit w = unit_at(A, u);
                const int buf = it % NBUF;
                const uint32_t acc_phase = (it / NBUF) & 1;
                if (!(ok = mbar_wait<PAIR>(acc_empty + buf, acc_phase ^ 1, abort_flag, 2))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tmem_d = tmem_base + buf * (MT * MAX_BN);
                for (int kb = w.kb0; kb < w.kb1; kb++) {
                    if (!(ok = mbar_wait(full + stage, phase, abort_flag, 3))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
                    const uint64_t db = BMN ? make_smem_desc_mn(sa + MT * A_BYTES, BOX_BYTES, 1024) : make_smem_desc(sa + MT * A_BYTES);
#pragma unroll
                    for (int j = 0; j < MT; j++) {
                        const uint64_t da = AMN ? make_smem_desc_mn(sa + j * A_BYTES, BOX_BYTES, 1024) : make_smem_desc(sa + j * A_BYTES);
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; k++)
                            umma_f16<CTAS>(tmem_d + j * MAX_BN, da + A_KSTEP * k, db + B_KSTEP * k, idesc, kb > w.kb0 || k != 0);
                    }
                    umma_commit<CTAS>(empty + stage);            // slot reusable (in both CTAs) once these MMAs have read it
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
                if (ok) umma_commit<CTAS>(acc_full + buf);       // accumulator complete
            }
        }
    } else {
        // ---------------- epilogue: two warps per TMEM lane quadrant (warp % 4), each with every other 32 columns ----------------
        // Products with a short K are all epilogue: with one warp per quadrant and a
        // lane to a row 15416 x 962 x 128 took 52 us, 8000 x 1001 x 256 34 us; 40 and 28 us this way.
        const int quad = warp & 3, grp = (warp - 2) >> 2;
        int it = 0;
        bool ok = true;
        const bool vec_ok = (A.N % 8 == 0) && (((uintptr_t)c & 15) == 0);
        __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(epi) + (warp - 2) * (32 * EPI_PITCH);
        for (int u = first; u < A.units && ok; u += step, it++) {
            const Unit w = unit_at(A, u);
            const int buf = it % NBUF;
            const uint32_t acc_phase = (it / NBUF) & 1;
            ok = mbar_wait(acc_full + buf, acc_phase, abort_flag, 4);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int j = 0; j < MT; j++) {
                const int row0 = w.tm * F::TILE_M + (j * CTAS + rank) * BM + quad * 32, row = row0 + lane;
                const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + buf * (MT * MAX_BN) + j * MAX_BN;
#pragma unroll 1
                for (int ch = grp * 32; ch < A.bn; ch += 64) {
                    const int col0 = w.tn * A.bn + ch;
                    if (row0 >= A.M || col0 >= A.N) break;       // uniform over the warp
                    uint32_t r[32];
                    tmem_ld32(taddr + ch, r);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (w.part >= 0) {
                        float* prow = part + ((int64_t)w.part * F::TILE_M + row - w.tm * F::TILE_M) * A.bn + ch;
                        if (row < A.M) {
#pragma unroll
                            for (int q = 0; q < 8; q++)
                                *reinterpret_cast<uint4*>(prow + q * 4) = make_uint4(r[q * 4], r[q * 4 + 1], r[q * 4 + 2], r[q * 4 + 3]);
                        }
                        continue;
                    }
                    __align__(16) __nv_bfloat162 h[16];
#pragma unroll
                    for (int e = 0; e < 16; e++) h[e] = __floats2bfloat162_rn(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]));
                    // turned around in shared memory: a warp then writes 64 bytes of a row at a time
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 4; q++) reinterpret_cast<uint4*>(rows + lane * EPI_PITCH)[q] = reinterpret_cast<const uint4*>(h)[q];
                    __syncwarp();
                    __nv_bfloat16* c0 = c + ((int64_t)w.batch * A.M + row0) * A.N + col0;
                    if (vec_ok) {
                        const int at = (lane & 3) * 8;
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const int i = q * 8 + (lane >> 2);
                            if (row0 + i < A.M && col0 + at < A.N)
                                *reinterpret_cast<uint4*>(c0 + (int64_t)i * A.N + at) = *reinterpret_cast<const uint4*>(rows + i * EPI_PITCH + at);
                        }
                    } else if (col0 + lane < A.N) {               // rows start at any multiple of 2 bytes
#pragma unroll 8
                        for (int i = 0; i < 32; i++)
                            if (row0 + i < A.M) c0[(int64_t)i * A.N + lane] = rows[i * EPI_PITCH + lane];
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) { if (PAIR) mbar_arrive_leader(acc_empty + buf); else mbar_arrive(acc_empty + buf); }
        }
    }
    // ---------------- teardown ----------------
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync();          // neither CTA leaves while the other may still signal it or read its tiles
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_dealloc<CTAS>(tmem_base);
    }
}

// The split tiles' elements: sums over splits (ascending) of the partial tiles, rounded to bf16 once; four columns per thread.
__global__ void __launch_bounds__(256)
fold_kernel(const float* __restrict__ part, __nv_bfloat16* __restrict__ c, const __grid_constant__ GemmArgs A, int tile_m) {
    const int quads = A.bn / 4, others = A.tiles_m * A.tiles_n - A.whole;
    const int64_t per_tile = (int64_t)tile_m * quads, n = others * per_tile;
    const bool vec = A.N % 4 == 0 && ((uintptr_t)c & 7) == 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int t = (int)(i / per_tile), q = (int)(i - t * per_tile), r = q / quads;
        int tm, tn;
        tile_at(A, A.whole + t, tm, tn);
        const int m = tm * tile_m + r, col = tn * A.bn + (q - r * quads) * 4;
        if (m >= A.M || col >= A.N) continue;
        float4 acc = __ldcs(reinterpret_cast<const float4*>(part) + i);
        for (int s = 1; s < A.splits; s++) {
            const float4 v = __ldcs(reinterpret_cast<const float4*>(part) + s * n + i);
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        __nv_bfloat16* out = c + (int64_t)m * A.N + col;
        const __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x, acc.y), hi = __floats2bfloat162_rn(acc.z, acc.w);
        if (vec) {
            uint2 v; *reinterpret_cast<__nv_bfloat162*>(&v.x) = lo; *reinterpret_cast<__nv_bfloat162*>(&v.y) = hi;
            *reinterpret_cast<uint2*>(out) = v;
        } else {
            out[0] = lo.x;
            if (col + 1 < A.N) out[1] = lo.y;
            if (col + 2 < A.N) out[2] = hi.x;
            if (col + 3 < A.N) out[3] = hi.y;
        }
    }
}

// TMA wants rows at multiples of 16 bytes: [rows, cols] -> [rows, pitch] with pitch a multiple of 8, for an operand whose
// contiguous extent is not one. Columns past cols are outside the tensor map and are not written.
__global__ void __launch_bounds__(256)
pad_rows_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out, int64_t rows, int cols, int pitch) {
    const int chunks = pitch / 8;
    const int64_t n = rows * chunks;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / chunks; const int c0 = (int)(i - r * chunks) * 8;
        const __nv_bfloat16* p = in + r * cols + c0;
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = c0 + e < cols ? p[e] : __float2bfloat16(0.f);
        *reinterpret_cast<uint4*>(out + i * 8) = *reinterpret_cast<const uint4*>(v);
    }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    });
    return fn;
}

PFN_cuTensorMapEncodeIm2col_v12000 encode_im2col_fn() {
    static PFN_cuTensorMapEncodeIm2col_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeIm2col_v12000)p;
    });
    return fn;
}

// bf16 [batch][rows][cols] with row pitch `pitch`, a {BK, box_rows, 1} box and 128-byte swizzle
static bool make_map(CUtensorMap* map, const void* base, int64_t batch, int64_t rows, int64_t cols, int64_t pitch, int box_rows) {
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)batch};
    cuuint64_t strides[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)rows * pitch * 2};
    cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

template <bool PAIR, int MT>
static const void* kernel_of(bool amn, bool bmn) {
    return amn ? (bmn ? (const void*)gemm_bf16_kernel<PAIR, MT, true, true> : (const void*)gemm_bf16_kernel<PAIR, MT, true, false>)
               : (bmn ? (const void*)gemm_bf16_kernel<PAIR, MT, false, true> : (const void*)gemm_bf16_kernel<PAIR, MT, false, false>);
}
static const void* kernel_of(bool pair, int mt, bool amn, bool bmn) {
    return !pair ? kernel_of<false, 1>(amn, bmn) : mt == 1 ? kernel_of<true, 1>(amn, bmn) : kernel_of<true, 2>(amn, bmn);
}
static int smem_of(bool pair, int mt) {
    return !pair ? Cfg<false, 1>::SMEM_BYTES : mt == 1 ? Cfg<true, 1>::SMEM_BYTES : Cfg<true, 2>::SMEM_BYTES;
}

// How many CTA pairs run at once (a persistent grid must not exceed it); 0 on error.
static int pair_slots() {
    static std::once_flag once;
    static int slots = 0;
    std::call_once(once, [] {
        for (int pair = 0; pair < 2; pair++)
            for (int mt = 1; mt <= 1 + pair; mt++)
                for (int f = 0; f < 4; f++)
                    if (cudaFuncSetAttribute(kernel_of(pair, mt, f & 1, f & 2), cudaFuncAttributeMaxDynamicSharedMemorySize, smem_of(pair, mt)) != cudaSuccess) return;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(kNumSMs); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem_of(true, 1); cfg.attrs = at; cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel_of(true, 1, false, false), &cfg) != cudaSuccess || n < 1) return;
        slots = std::min(n, kNumSMs / 2);
    });
    return slots;
}

struct Plan { bool pair; int mt, bn, splits; int64_t whole; double ns; };

// Tile and split by estimated time. A k-block costs the larger of its MMAs (11 TFLOP/s per SM) and its operands' way from L2
// (about 110 B per ns and SM); a tile adds its epilogue where no second accumulator hides it; split K adds the way of the partial
// sums out and back and a second launch.
static Plan estimate(int64_t batch, int64_t M, int64_t N, int64_t K, bool bmn, bool may_split) {
    Plan best{false, 1, MAX_BN, 1, 0, 1e30};
    const int64_t kb = (K + BK - 1) / BK;
    const int pslots = pair_slots();
    const char* fp = getenv("B200JT_GEMM_PAIR"); const char* fm = getenv("B200JT_GEMM_MT");      // read on every call:
    const char* fb = getenv("B200JT_GEMM_BN"); const char* fs = getenv("B200JT_GEMM_SPLITS");    // tests force each variant in turn
    for (int pair = 0; pair < 2; pair++) {
        if ((fp && atoi(fp) != pair) || (pair && !pslots)) continue;
        for (int mt = 1; mt <= 1 + pair; mt++) {
            if (fm && atoi(fm) != mt && pair) continue;
            const int tile_m = BM * mt * (1 + pair), slots = pair ? pslots : kNumSMs;
            const int64_t tm = (M + tile_m - 1) / tile_m;
            for (int bn = 32; bn <= MAX_BN; bn += 32) {
                if (fb ? atoi(fb) != bn : bn > 32 && bn - 32 >= N) continue;
                const int half = bn / (1 + pair);
                const double feed = (mt * A_BYTES + (bmn ? (half + 63) / 64 * BOX_BYTES : half * BK * 2)) / 110.0;
                const double mma = mt * std::max(bn, 64) * 1.5;
                const double block = std::max(feed, mma) + 20;
                const int64_t tiles = tm * ((N + bn - 1) / bn) * batch;
                const double epi = mt * bn * 4.0;
                // K whole, or split where the tiles leave a round part empty: all of them when they do not fill one round, else those
                // of the last round. 4096 x 4096 x 16384 (256 tiles of 256 x 256 on 74 pairs): 3 rounds and a half one instead of 4.
                const int64_t last = tiles % slots, whole = tiles - last;
                int64_t tried = 0;
                for (int q = 0; q < 3; q++) {
                    int64_t s = q == 0 || last == 0 ? 1 : q == 1 ? slots / last : slots / last / 2;
                    s = std::min(s, kb / 4);
                    if (fs) s = std::min<int64_t>(atoi(fs), kb);
                    if (s < 1 || !may_split || last == 0) s = 1;
                    if (s == tried) continue;
                    tried = s;
                    const int64_t kept = s == 1 ? 0 : whole;
                    const double once = kb * block + (mt == 2 ? epi : 0);
                    double ns = 2500 + epi;
                    if (s == 1) ns += (double)((tiles + slots - 1) / slots) * once;
                    else {
                        const int64_t others = tiles - kept;
                        ns += (double)(kept / slots) * once + (double)((others * s + slots - 1) / slots) * ((kb + s - 1) / s * block + (mt == 2 ? epi : 0)) +
                              3000 + (double)s * others * tile_m * bn * 8 / 4000;
                    }
                    if (ns < best.ns) best = {pair != 0, mt, bn, (int)s, kept, ns};
                }
            }
        }
    }
    return best;
}

// The estimate runs over some 70 candidates (1.5 us): each thread keeps its last 64 plans.
static Plan plan_for(int64_t batch, int64_t M, int64_t N, int64_t K, bool bmn, bool may_split) {
    if (getenv("B200JT_GEMM_PAIR") || getenv("B200JT_GEMM_MT") || getenv("B200JT_GEMM_BN") || getenv("B200JT_GEMM_SPLITS"))
        return estimate(batch, M, N, K, bmn, may_split);
    struct Entry { int64_t key[5] = {-1, 0, 0, 0, 0}; Plan p; };
    static thread_local Entry kept[64];
    const int64_t key[5] = {batch, M, N, K, (int64_t)bmn * 2 + may_split};
    uint64_t h = 0;
    for (int64_t k : key) h = (h ^ (uint64_t)k) * 0x9E3779B97F4A7C15ull;
    Entry& e = kept[h >> 58];
    if (memcmp(e.key, key, sizeof(key)) != 0) { e.p = estimate(batch, M, N, K, bmn, may_split); memcpy(e.key, key, sizeof(key)); }
    return e.p;
}

static int launch(const Plan& p, const void* a, const void* b, void* c, float* part, int64_t batch, int64_t a_batch, int64_t b_batch,
                  int64_t M, int64_t N, int64_t K, int64_t pitch_a, int64_t pitch_b, bool amn, bool bmn, cudaStream_t st) {
    const int ctas = p.pair ? 2 : 1, tile_m = BM * p.mt * ctas;
    if (!pair_slots()) return fail(-4, "matmul: no room for the kernel's shared memory");
    CUtensorMap ma, mb;
    // K-major operands: boxes of 64 K-elements x rows; MN-major ones: boxes of 64 of their own elements x 64 K-rows
    if (!(amn ? make_map(&ma, a, a_batch, K, M, pitch_a, 64) : make_map(&ma, a, a_batch, M, K, pitch_a, BM)) ||
        !(bmn ? make_map(&mb, b, b_batch, K, N, pitch_b, 64) : make_map(&mb, b, b_batch, N, K, pitch_b, p.bn / ctas)))
        return fail(-4, "matmul: cuTensorMapEncodeTiled failed");
    GemmArgs A;
    A.M = (int)M; A.N = (int)N; A.K = (int)K; A.bn = p.bn; A.k_blocks = (int)((K + BK - 1) / BK);
    A.tiles_m = (int)((M + tile_m - 1) / tile_m); A.tiles_n = (int)((N + p.bn - 1) / p.bn);
    A.batch = (int)batch; A.splits = p.splits; A.group = std::max(1, 1024 / tile_m);
    A.a_batched = a_batch > 1; A.b_batched = b_batch > 1; A.whole = (int)p.whole;
    const int64_t tiles = (int64_t)A.tiles_m * A.tiles_n, units = p.splits > 1 ? p.whole + (tiles - p.whole) * p.splits : tiles * batch;
    if (units >= (1LL << 30)) return fail(-1, "matmul: too many tiles");
    A.units = (int)units;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = ctas; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(std::min<int64_t>(units, p.pair ? pair_slots() : kNumSMs) * ctas));
    cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem_of(p.pair, p.mt); cfg.stream = st; cfg.attrs = at; cfg.numAttrs = p.pair ? 1 : 0;
    void* args[] = {&ma, &mb, &c, &part, &A};
    B200JT_CUDA(cudaLaunchKernelExC(&cfg, kernel_of(p.pair, p.mt, amn, bmn), args));
    if (p.splits > 1) {
        fold_kernel<<<grid_for((tiles - p.whole) * tile_m * (p.bn / 4), 256), 256, 0, st>>>(part, (__nv_bfloat16*)c, A, tile_m);
        B200JT_LAUNCH_CHECK();
    }
    return 0;
}

inline int64_t pitch8(int64_t n) { return (n + 7) / 8 * 8; }
inline size_t round256(size_t n) { return (n + 255) & ~(size_t)255; }

}  // namespace tc

// Any extents (an operand whose contiguous extent is not a multiple of 8 is first copied to TMA's pitch) once the product is
// large enough to pay for a pipeline's fill and drain.
bool matmul_tc_supported(int64_t M, int64_t N, int64_t K, const void* a, const void* b, const void* c) {
    return K >= 32 && (double)M * N * K >= (double)(1 << 18) && M < (1LL << 30) && N < (1LL << 30) && K < (1LL << 30) &&
           ((uintptr_t)a % 16 == 0) && ((uintptr_t)b % 16 == 0) && ((uintptr_t)c % 2 == 0) && tc::encode_fn() != nullptr;
}

size_t matmul_tc_workspace(int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b, bool may_split) {
    using namespace tc;
    const int64_t ca = trans_a ? M : K, cb = trans_b ? K : N;
    size_t bytes = 0;
    if (ca % 8) bytes += round256((size_t)(trans_a ? K : M) * pitch8(ca) * 2);
    if (cb % 8) bytes += round256((size_t)(trans_b ? N : K) * pitch8(cb) * 2);
    if (!may_split) return bytes;
    const Plan p = plan_for(1, M, N, K, !trans_b, true);
    if (p.splits > 1) {
        const int64_t tile_m = BM * p.mt * (1 + p.pair);
        bytes += (size_t)p.splits * ((M + tile_m - 1) / tile_m * ((N + p.bn - 1) / p.bn) - p.whole) * tile_m * p.bn * 4;
    }
    return bytes;
}

int matmul_tc(const void* a, const void* b, void* c, int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b,
              void* workspace, bool may_split, cudaStream_t st) {
    using namespace tc;
    unsigned char* ws = (unsigned char*)workspace;
    const Plan p = plan_for(1, M, N, K, !trans_b, may_split);
    auto padded = [&](const void*& q, int64_t rows, int64_t cols) {
        if (cols % 8 == 0) return cols;
        const int64_t pitch = pitch8(cols);
        pad_rows_kernel<<<grid_for(rows * (pitch / 8), 256), 256, 0, st>>>((const __nv_bfloat16*)q, (__nv_bfloat16*)ws, rows, (int)cols, (int)pitch);
        q = ws; ws += round256((size_t)rows * pitch * 2);
        return pitch;
    };
    const int64_t pa = trans_a ? padded(a, K, M) : padded(a, M, K);
    const int64_t pb = trans_b ? padded(b, N, K) : padded(b, K, N);
    B200JT_LAUNCH_CHECK();
    return launch(p, a, b, c, (float*)ws, 1, 1, 1, M, N, K, pa, pb, trans_a, !trans_b, st);
}

// One launch for `batch` products c[i] = a[i or 0] . b[i or 0]: no scratch, so operands whose pitches suit TMA as they are.
bool batched_matmul_tc_supported(int64_t batch, int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b,
                                 const void* a, const void* b, const void* c) {
    if (K < 64 || M < 128 || N < 64 || !matmul_tc_supported(M, N, K, a, b, c) || batch >= (1LL << 31)) return false;
    if ((trans_a ? M : K) % 8 != 0 || (trans_b ? K : N) % 8 != 0) return false;
    return batch * ((M + 127) / 128) * ((N + 31) / 32) < (1LL << 30);
}

int batched_matmul_tc(const void* a, const void* b, void* c, int64_t batch, int64_t a_batch, int64_t b_batch,
                      int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b, cudaStream_t st) {
    using namespace tc;
    return launch(plan_for(batch, M, N, K, !trans_b, false), a, b, c, nullptr, batch, a_batch, b_batch, M, N, K,
                  trans_a ? M : K, trans_b ? K : N, trans_a, !trans_b, st);
}

int tc_status_fetch_and_clear() { return tc::status_fetch_and_clear(); }

}  // namespace b200jt
