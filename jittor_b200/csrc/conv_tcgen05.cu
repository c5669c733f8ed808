// Reindex-lowered conv2d (python/jittor/nn.py:1009-1017) as an implicit GEMM on tcgen05: bf16 in, fp32 accumulate in TMEM.
//
// The reference never materialises the 7-D window tensor; its relay is cudnnConvolutionForward
// (python/jittor/extern/cuda/cudnn/ops/cudnn_conv_op.cc:293). Here:
//   GEMM view   M = N*OH*OW output pixels, N = Cout, K = KH*KW*Cin, walked tap by tap in 64-channel blocks;
//   layout      x is first copied NCHW -> NHWC (channels innermost) and w OIHW -> [tap][Cout][Cin], so that both
//               operands are K-major and every TMA box starts at a channel offset that is a multiple of 64 (the
//               16-byte start rule); the spatial shift of a tap comes with the load, and what lies outside x is zero-filled,
//               which is exactly the reindex overflow value 0;
//   tile        128 consecutive output pixels (one im2col TMA load of 128 rows x 128 B per k-block: rows, images and
//               padding are the map's business) x up to 256 output channels, or twice the pixels for a pair of CTAs;
//   pipeline    same persistent warp-specialised ring as the GEMM (TMA warp, MMA warp, 8 epilogue warps, TMEM
//               double buffering); strides 1..4 through the traversal stride of the x tensor map;
//   epilogue    tcgen05.ld -> bf16 -> y in NCHW; optionally per-channel sum / sum of squares of the stored values
//               (the two reduce.mean of BatchNorm, python/jittor/nn.py:674-675) accumulated per CTA in shared memory
//               and flushed with one atomicAdd per channel.
#include "gemm_simt.cuh"
#include "tc_common.cuh"

#include <mutex>

namespace b200jt {
namespace tcconv {

using namespace tc;

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int A_BYTES = BM * BK * 2;
// PAIR: the two CTAs of a cluster work on one tile of 256 pixels (tcgen05 cta_group::2). Each loads its own 128 pixels and HALF
// of the weights, the leader's MMA reads both: 32 KB instead of 48 KB per stage and SM at 256 output channels. A tile alone on
// its SM waits for the latency of its loads, so a ring holds as many stages as fit.
template <int BN_T, bool PAIR> struct Ring {
    static constexpr int STAGE_BYTES = A_BYTES + BN_T * BK * 2 / (PAIR ? 2 : 1);
    static constexpr int STAGES = (192 * 1024) / STAGE_BYTES < 8 ? (192 * 1024) / STAGE_BYTES : 8;
};
constexpr int RING_BYTES = 192 * 1024;
constexpr int STATS_MAX_CO = 512;                   // widest layer whose statistics the epilogue can keep per CTA
constexpr int STATS_BYTES = 2 * STATS_MAX_CO * 4;
constexpr int OUT_STAGE_BYTES = 8 * 32 * 32 * 2;      // one 32 channel x 32 pixel square per epilogue warp
constexpr int SMEM_BYTES = RING_BYTES + 1024 + 256 + STATS_BYTES + OUT_STAGE_BYTES;
constexpr int THREADS = 320;                         // producer, MMA and 8 epilogue warps
// Channel pitch of the channels-last copies: TMA wants row pitches of 16 bytes. Channels past C are outside the tensor map and
// read as zero, so any channel count runs here.
inline int pitch8(int c) { return (c + 7) / 8 * 8; }

struct ConvArgs {
    int N, C, H, W, Co, KH, KW, OH, OW, sh, sw, ph, pw, dh, dw;
    int64_t pixels;                  // N * OH * OW
    int tiles_m, tiles_n;
    int vec;                         // pixels per store of y: 8 or 4 where OH * OW is a multiple (and y aligned), else 1
    int last_k;                      // MMA steps of 16 channels in a tap's last channel block
};

// A warp's square of 32 channels (rows of 64 bytes) x 32 pixels in shared memory, 16-byte chunks of a row at chunk ^ (row / 2 % 4): a
// pixel per lane going in, eight chunks of two rows or one chunk of eight rows coming out all touch every bank once.
__device__ __forceinline__ int square_chunk(int ch, int chunk) { return ch * 4 + (chunk ^ ((ch >> 1) & 3)); }
__device__ __forceinline__ __nv_bfloat16* square_at(__nv_bfloat16* square, int ch, int px) { return square + square_chunk(ch, px >> 3) * 8 + (px & 7); }

// Adds the square's channel sums and sums of squares to the CTA's: a lane reads its channel's 32 pixels and adds pairs of them with
// packed float32 arithmetic. (A halving exchange between the lanes was 62 shuffles and 280 instructions for a square, half of the
// epilogue of a 1 x 1 layer.)
__device__ __forceinline__ void add_square_sums(const __nv_bfloat16* square, int co0, int Co, float* sstat) {
    const int lane = threadIdx.x & 31;
    unsigned long long s[2] = {0, 0}, q[2] = {0, 0};
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const uint4 v = reinterpret_cast<const uint4*>(square)[square_chunk(lane, c)];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            unsigned long long two;
            asm("mov.b64 %0, {%1, %2};" : "=l"(two) : "r"(w[i] << 16), "r"(w[i] & 0xffff0000u));
            asm("add.rn.f32x2 %0, %0, %1;" : "+l"(s[i & 1]) : "l"(two));
            asm("fma.rn.f32x2 %0, %1, %1, %0;" : "+l"(q[i & 1]) : "l"(two));
        }
    }
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(s[0]) : "l"(s[1]));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(q[0]) : "l"(q[1]));
    if (co0 + lane < Co) {
        atomicAdd(sstat + co0 + lane, __uint_as_float((uint32_t)s[0]) + __uint_as_float((uint32_t)(s[0] >> 32)));
        atomicAdd(sstat + STATS_MAX_CO + co0 + lane, __uint_as_float((uint32_t)q[0]) + __uint_as_float((uint32_t)(q[0] >> 32)));
    }
}

// NCHW y: a warp turns its 32 pixels x 32 channels around in shared memory and stores rows of up to 8 pixels. (TMA box stores
// of [8][8] pixels move a row of 16 bytes in 1.7 ns, whatever there is to it: 6.8 us for a 128 x 256 tile.)
// NHWC ("acdb"): a lane stores the 32 consecutive channels of its pixel as four 16-byte vectors.
// BN_T: output channels per tile (256, or less where that fills the last wave of the persistent grid better).
// The epilogue's eight warps are two per TMEM lane quadrant, each with every other 32 channels: four warps took longer than the
// main loop of a 1 x 1 layer (64 x 64 x 56 x 56 -> 256 channels with statistics, layout pass included: 142 us with four warps and
// box stores, 87 us with eight and rows of pixels, 68 us since the sums come from the square).
// Every tile walks K from its first tap, so that an image gives the same bits wherever it stands in a batch. (Starts spread over
// the tiles, which keeps them from reading the same weights at the same time, were no faster: 814 and 806 us for 256 x 256 x 56 x 56,
// 50 and 50 us for 7 x 432 x 28 x 28 -> 320.)
template <bool NHWC, int BN_T, bool PAIR>
__global__ void __launch_bounds__(THREADS, 1)
conv_bf16_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                 __nv_bfloat16* __restrict__ y, float* __restrict__ stats, const __grid_constant__ ConvArgs A) {
    constexpr int CTAS = PAIR ? 2 : 1, STAGES = Ring<BN_T, PAIR>::STAGES, STAGE_BYTES = Ring<BN_T, PAIR>::STAGE_BYTES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + RING_BYTES);
    uint64_t* full = bars;                       // a pair uses the leader's
    uint64_t* empty = bars + STAGES;
    uint64_t* acc_full = bars + 2 * STAGES;      // acc_empty: a pair uses the leader's
    uint64_t* acc_empty = bars + 2 * STAGES + 2;
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 4);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    float* sstat = (float*)(smem + RING_BYTES + 256);      // [2][STATS_MAX_CO] per-CTA channel sums
    unsigned char* stage_out = smem + RING_BYTES + 256 + STATS_BYTES;   // [8 warps][32 ch][32 px] bf16

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = PAIR ? (int)cluster_rank() : 0;
    const int first = blockIdx.x / CTAS, step = gridDim.x / CTAS;
    const int total = A.tiles_m * A.tiles_n;
    const int cblocks = (A.C + BK - 1) / BK;
    const int k_blocks = A.KH * A.KW * cblocks;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        for (int b = 0; b < 2; b++) { mbar_init(acc_full + b, 1); mbar_init(acc_empty + b, 8 * CTAS); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < 2 * STATS_MAX_CO; i += blockDim.x) sstat[i] = 0.f;
    if (warp == 1) tmem_alloc<CTAS>(tmem_slot);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync();                 // the peer's barriers exist before anything signals them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    // Everything above runs while the layout pass drains; what that pass writes, and y, are touched below only. With the weight
    // gradient and its fold launched the same way, a training pass of 64 x 128 x 28 x 28 went from 147.5 to 139.4 us.
    asm volatile("griddepcontrol.wait;" ::: "memory");

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0; uint32_t phase = 0;
            bool ok = true;
            for (int t = first; t < total && ok; t += step) {
                const int tm = t / A.tiles_n, tn = t - tm * A.tiles_n;
                int64_t q = ((int64_t)tm * CTAS + rank) * BM;
                if (q >= A.pixels) q = 0;                       // a pair's second half past the last pixel: any pixels, none is stored
                const int n = (int)(q / (A.OH * A.OW)), in = (int)(q - (int64_t)n * (A.OH * A.OW));
                const int h = in / A.OW * A.sh - A.ph, w = in % A.OW * A.sw - A.pw;
                int tap = 0, cb = 0, kh = 0, kw = 0;
                for (int kb = 0; kb < k_blocks; kb++) {
                    if (!(ok = mbar_wait(empty + stage, phase ^ 1, abort_flag, 11))) break;
                    unsigned char* sa = smem + stage * STAGE_BYTES;
                    if (rank == 0) mbar_expect_tx(full + stage, CTAS * A_BYTES + BN_T * BK * 2);      // both CTAs' bytes
                    const uint32_t bar = PAIR ? leader_addr(full + stage) : smem_u32(full + stage);
                    tma_load_im2col<CTAS>(sa, &map_x, bar, cb * BK, w, h, n, kw * A.dw, kh * A.dh);
                    tma_load_tile<CTAS>(sa + A_BYTES, &map_w, bar, cb * BK, tap * A.Co + tn * BN_T + rank * (BN_T / CTAS));
                    if (++cb == cblocks) {
                        cb = 0; tap++;
                        if (++kw == A.KW) { kw = 0; kh++; }
                    }
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
            if (!ok) {
                for (int s = 0; s < STAGES; s++)
                    for (uint32_t i = 0; i < 4096 && !mbar_try(full + s, 0) && !mbar_try(full + s, 1); i++) __nanosleep(64);
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = make_idesc(BM * CTAS, BN_T);
            int stage = 0; uint32_t phase = 0;
            int it = 0;
            bool ok = true;
            for (int t = first; t < total && ok; t += step, it++) {
                const int buf = it & 1;
                const uint32_t acc_phase = (it >> 1) & 1;
                if (!(ok = mbar_wait<PAIR>(acc_empty + buf, acc_phase ^ 1, abort_flag, 12))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tmem_d = tmem_base + buf * BN;
                int cb = 0;
                for (int kb = 0; kb < k_blocks; kb++) {
                    if (!(ok = mbar_wait(full + stage, phase, abort_flag, 13))) break;
                    if (++cb == cblocks) cb = 0;
                    const int steps = cb == 0 ? A.last_k : BK / UMMA_K;          // no MMA on channels that do not exist
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
                    const uint64_t da = make_smem_desc(sa), db = make_smem_desc(sa + A_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; k++)
                        if (k < steps) umma_f16<CTAS>(tmem_d, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                    umma_commit<CTAS>(empty + stage);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
                if (ok) umma_commit<CTAS>(acc_full + buf);
            }
        }
    } else {
        const int quad = warp & 3, grp = (warp - 2) >> 2;
        int it = 0;
        bool ok = true;
        const int64_t plane = (int64_t)A.OH * A.OW;
        for (int t = first; t < total && ok; t += step, it++) {
            const int tm = t / A.tiles_n, tn = t - tm * A.tiles_n;
            const int buf = it & 1;
            const uint32_t acc_phase = (it >> 1) & 1;
            ok = mbar_wait(acc_full + buf, acc_phase, abort_flag, 14);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // this lane's pixel, and the 8 pixels it stores: the (lane % 4)th of the warp's four runs, channels lane / 4 + 8 i of a chunk
            const int64_t p0 = ((int64_t)tm * CTAS + rank) * BM + quad * 32, p = p0 + lane;
            const bool valid = p < A.pixels;
            auto plane_at = [&](int64_t q) { const int64_t n = q / plane; return y + n * (A.Co - 1) * plane + q; };
            __nv_bfloat16* yl = NHWC ? y + p * A.Co : plane_at(p);
            const int64_t run = p0 + (lane & 3) * 8;
            __nv_bfloat16* y0 = plane_at(run) + (lane >> 2) * plane;
            __nv_bfloat16* y1 = plane_at(run + 4) + (lane >> 2) * plane;
            __nv_bfloat16* square = reinterpret_cast<__nv_bfloat16*>(stage_out) + (warp - 2) * 1024;
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + buf * BN;
#pragma unroll 1
            for (int ch = grp; ch < BN_T / 32; ch += 2) {
                const int co0 = tn * BN_T + ch * 32;
                uint32_t v[32];
                tmem_ld32(taddr + ch * 32, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                __syncwarp();
                if (NHWC) {
                    // NHWC: this lane's pixel, channels co0 .. co0 + 31 are contiguous
                    __align__(16) __nv_bfloat16 row[32];
#pragma unroll
                    for (int e = 0; e < 32; e++) {
                        row[e] = __float2bfloat16(__uint_as_float(v[e]));
                        if (stats) *square_at(square, e, lane) = valid ? row[e] : __float2bfloat16(0.f);
                    }
                    if (valid) {
                        __nv_bfloat16* yq = yl + co0;
                        if (co0 + 32 <= A.Co && (A.Co & 7) == 0) {
#pragma unroll
                            for (int q = 0; q < 4; q++) reinterpret_cast<uint4*>(yq)[q] = reinterpret_cast<const uint4*>(row)[q];
                        } else {
#pragma unroll
                            for (int e = 0; e < 32; e++) if (co0 + e < A.Co) yq[e] = row[e];
                        }
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 32; e++) *square_at(square, e, lane) = __float2bfloat16(valid ? __uint_as_float(v[e]) : 0.f);
                    __syncwarp();
                    if (A.vec == 1) {           // planes start anywhere: a channel at a time, neighbouring lanes on neighbouring pixels
#pragma unroll
                        for (int e = 0; e < 32; e++)
                            if (valid && co0 + e < A.Co) yl[(int64_t)(co0 + e) * plane] = *square_at(square, e, lane);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            if (co0 + i * 8 + (lane >> 2) < A.Co) {
                                const uint4 px = reinterpret_cast<const uint4*>(square)[square_chunk(i * 8 + (lane >> 2), lane & 3)];
                                const int64_t d = (int64_t)(co0 + i * 8) * plane;
                                if (A.vec == 8) { if (run < A.pixels) *reinterpret_cast<uint4*>(y0 + d) = px; }
                                else {
                                    if (run < A.pixels) *reinterpret_cast<uint2*>(y0 + d) = make_uint2(px.x, px.y);
                                    if (run + 4 < A.pixels) *reinterpret_cast<uint2*>(y1 + d) = make_uint2(px.z, px.w);
                                }
                            }
                        }
                    }
                }
                if (stats) {                    // of the values as stored, zero where there is no pixel
                    if (NHWC) __syncwarp();
                    add_square_sums(square, co0, A.Co, sstat);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) { if (PAIR) mbar_arrive_leader(acc_empty + buf); else mbar_arrive(acc_empty + buf); }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (PAIR) cluster_sync();          // neither CTA leaves while the other may still signal it or read its tiles
    if (stats) {
        for (int i = threadIdx.x; i < A.Co; i += blockDim.x) {
            atomicAdd(stats + i, sstat[i]);
            atomicAdd(stats + A.Co + i, sstat[STATS_MAX_CO + i]);
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_dealloc<CTAS>(tmem_base);
    }
}

// ---- layout passes -----------------------------------------------------------------------------------------
// in[b][R][Cn] -> out[b][Cn][pitch] (bf16; pitch >= R is a multiple of 8, the elements past R are zero), tiles of TR rows x 64
// columns, 16-byte global accesses on both sides. HBM sets the time as long as whole runs are written: TR = 128 writes 256 bytes
// at a time (256 x 256 x 56 x 56: 126 us, 6.5 TB/s; 128 bytes at a time 169 us, 64 bytes 194 us). The tile is kept as 32-bit pairs,
// word w of row r at w ^ (r / 8) ^ (r % 4), which spreads both the rows of the first phase and the columns of the second over all banks.
// Block (0,0,0) also zeroes `zero[0..n_zero)`. The first wz slices (blockIdx.z < wz) of the same grid re-order the weights
// instead (w -> wt[taps][Co][wpitch]; w_mode 0: w[Co][C][taps], 1: w[Co][taps][C], 2: w[C][Co][taps] with the taps reversed, the
// filter of the input gradient), the next a.n slices are a's images and the rest b's: the layout passes of a convolution, of its
// input gradient and of its weight gradient are one launch each.
struct LayoutJob { const __nv_bfloat16* in = nullptr; __nv_bfloat16* out = nullptr; int R = 0, Cn = 0, pitch = 0, n = 0; };
template <int TR>
__global__ void __launch_bounds__(256)
transpose_bf16_batched_kernel(const __grid_constant__ LayoutJob a, const __grid_constant__ LayoutJob b, int wz, const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ wt, int Co, int C, int taps, int wpitch,
                              float* __restrict__ zero, int n_zero, int w_mode) {
    __shared__ uint32_t tile[TR][32];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (zero && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0)       // the statistics the conv epilogue adds into
        for (int i = threadIdx.x; i < n_zero; i += blockDim.x) zero[i] = 0.f;
    if ((int)blockIdx.z < wz) {
        const int64_t n = (int64_t)Co * C * taps;
        const int64_t nblk = (int64_t)gridDim.x * gridDim.y * wz;
        const int64_t blk = ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        for (int64_t i = blk * blockDim.x + threadIdx.x; i < n; i += nblk * blockDim.x) {
            const int c = (int)(i % C); const int64_t t2 = i / C;
            const int co = (int)(t2 % Co); const int tap = (int)(t2 / Co);
            wt[t2 * wpitch + c] = w[w_mode == 0 ? ((int64_t)co * C + c) * taps + tap : w_mode == 1 ? ((int64_t)co * taps + tap) * C + c
                                                : ((int64_t)c * Co + co) * taps + (taps - 1 - tap)];
        }
        return;
    }
    const int slice = (int)blockIdx.z - wz;
    const bool second = slice >= a.n;
    const LayoutJob& job = second ? b : a;
    const int64_t image = second ? slice - a.n : slice;
    const int R = job.R, Cn = job.Cn, pitch = job.pitch;
    const int r0 = blockIdx.y * TR, c0 = blockIdx.x * 64;
    if (r0 >= R || c0 >= Cn) return;
    const __nv_bfloat16* __restrict__ in = job.in;
    const int64_t boff = image * R * Cn;
    __nv_bfloat16* __restrict__ out = job.out + image * pitch * Cn;
    const int j = threadIdx.x & 7, i = threadIdx.x >> 3;          // 8 chunks of 8 elements x 32 rows
    const bool vec_in = Cn % 8 == 0 && ((uintptr_t)in & 15) == 0;
    uint4 v[TR / 32];
#pragma unroll
    for (int p = 0; p < TR / 32; p++) {
        const int r = r0 + i + p * 32, c = c0 + j * 8;
        v[p] = make_uint4(0, 0, 0, 0);
        if (r < R && vec_in && c + 8 <= Cn) v[p] = __ldcs(reinterpret_cast<const uint4*>(in + boff + (int64_t)r * Cn + c));
        else if (r < R) {
            __align__(16) __nv_bfloat16 one[8];
#pragma unroll
            for (int e = 0; e < 8; e++) one[e] = c + e < Cn ? in[boff + (int64_t)r * Cn + c + e] : __float2bfloat16(0.f);
            v[p] = *reinterpret_cast<const uint4*>(one);
        }
    }
#pragma unroll
    for (int p = 0; p < TR / 32; p++) {
        const int row = i + p * 32, x = (row >> 3) ^ (row & 3);
        tile[row][(j * 4) ^ x] = v[p].x; tile[row][(j * 4 + 1) ^ x] = v[p].y;
        tile[row][(j * 4 + 2) ^ x] = v[p].z; tile[row][(j * 4 + 3) ^ x] = v[p].w;
    }
    __syncthreads();
    constexpr int OCT = TR / 8;                                   // a warp writes whole runs of TR elements
    const int lane = threadIdx.x & 31, oct = lane % OCT, r = r0 + oct * 8;
    if (r >= pitch) return;
#pragma unroll
    for (int p = 0; p < OCT / 8; p++) {
        const int pair = lane / OCT * OCT + (threadIdx.x >> 5) + p * 8, c = c0 + 2 * pair;      // two output rows = input columns
        if (c >= Cn) continue;
        uint32_t u[8];
#pragma unroll
        for (int e = 0; e < 8; e++) u[e] = tile[oct * 8 + e][pair ^ oct ^ (e & 3)];
        uint4 lo, hi;
        lo.x = __byte_perm(u[0], u[1], 0x5410); lo.y = __byte_perm(u[2], u[3], 0x5410);
        lo.z = __byte_perm(u[4], u[5], 0x5410); lo.w = __byte_perm(u[6], u[7], 0x5410);
        hi.x = __byte_perm(u[0], u[1], 0x7632); hi.y = __byte_perm(u[2], u[3], 0x7632);
        hi.z = __byte_perm(u[4], u[5], 0x7632); hi.w = __byte_perm(u[6], u[7], 0x7632);
        __stcs(reinterpret_cast<uint4*>(out + (int64_t)c * pitch + r), lo);
        if (c + 1 < Cn) __stcs(reinterpret_cast<uint4*>(out + (int64_t)(c + 1) * pitch + r), hi);
    }
}

inline int layout_rows(int c) { return c > 64 ? 128 : 64; }       // tile rows of the pass for c channels

// Channels-last tensor [N][H][W][C] read as windows: `pixels` window origins x 64 channels per load. The bounding box holds the
// origins (the corners: padding before, and padding minus the filter's reach after), the traversal strides are the convolution's,
// the tap's shift comes with the load. Outside the tensor -- padding, channels past C, images past N -- reads as zero.
static bool make_map_im2col(CUtensorMap* map, const void* base, int N, int H, int W, int C, int sh, int sw, int ph, int pw, int reach_h, int reach_w, int pixels) {
    auto fn = encode_im2col_fn();
    if (!fn) return false;
    cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
    const cuuint64_t cp = (cuuint64_t)pitch8(C) * 2;
    cuuint64_t strides[3] = {cp, W * cp, (cuuint64_t)H * W * cp};
    int lower[2] = {-pw, -ph}, upper[2] = {pw - reach_w, ph - reach_h};
    cuuint32_t estr[4] = {1, (cuuint32_t)sw, (cuuint32_t)sh, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, lower, upper, BK, (cuuint32_t)pixels, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// The corners and shifts an im2col map of four axes can hold: corners of the bounding box from -128 to 127, shifts from 0 to 255.
// 3 x 3 filters dilated by up to 127 with the padding that keeps the size fit.
static bool im2col_fits(const ConvShape& s) {
    const auto fits = [](int64_t pad, int64_t reach) { return pad <= 128 && reach <= 255 && reach - pad <= 128 && pad - reach <= 127; };
    return fits(s.ph, (s.KH - 1) * (int64_t)s.dh) && fits(s.pw, (s.KW - 1) * (int64_t)s.dw);
}

static bool make_map_w(CUtensorMap* map, const void* base, const ConvShape& s, int bn) {
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)s.C, (cuuint64_t)s.Co * s.KH * s.KW};
    cuuint64_t strides[1] = {(cuuint64_t)pitch8(s.C) * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)bn};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool NHWC>
static const void* kernel_of(int bn, bool pair) {
    return pair ? (bn == 256 ? (const void*)conv_bf16_kernel<NHWC, 256, true> : bn == 128 ? (const void*)conv_bf16_kernel<NHWC, 128, true>
                                                                                       : (const void*)conv_bf16_kernel<NHWC, 64, true>)
                : (bn == 256 ? (const void*)conv_bf16_kernel<NHWC, 256, false> : bn == 128 ? (const void*)conv_bf16_kernel<NHWC, 128, false>
                                                                                        : (const void*)conv_bf16_kernel<NHWC, 64, false>);
}
static const void* kernel_of(bool nhwc, int bn, bool pair) { return nhwc ? kernel_of<true>(bn, pair) : kernel_of<false>(bn, pair); }

// How many CTA pairs run at once (a persistent grid must not exceed it); 0 on error.
static int pair_slots() {
    static std::once_flag once;
    static int slots = 0;
    std::call_once(once, [] {
        for (int out = 0; out < 2; out++)
            for (int bn = 64; bn <= 256; bn *= 2)
                for (int pair = 0; pair < 2; pair++)
                    if (cudaFuncSetAttribute(kernel_of(out, bn, pair), cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) return;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(kNumSMs); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = SMEM_BYTES; cfg.attrs = at; cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel_of(0, 256, true), &cfg) != cudaSuccess || n < 1) return;
        slots = std::min(n, kNumSMs / 2);
    });
    return slots;
}

}  // namespace tcconv

// Any channel counts (the channels-last copies are padded to TMA's pitch, missing channels read as zero) and any extents, down
// to the 8 channels that half of the smallest MMA step needs: below that the padding costs more than the CUDA-core kernel.
// 304 -> 48 channels of 56 x 56, 18 images: 1.98 ms on the CUDA cores; 40 -> 27 channels of 7 x 7, 218 images: 106 us.
bool conv2d_tc_supported(const ConvShape& s, const void* x, const void* w, const void* y) {
    const int64_t px = (int64_t)s.N * s.OH * s.OW;
    return s.sh >= 1 && s.sh <= 4 && s.sw >= 1 && s.sw <= 4 && px >= 16 && s.C >= 8 && tcconv::im2col_fits(s) && ((uintptr_t)x % 2 == 0) &&
           ((uintptr_t)w % 2 == 0) && ((uintptr_t)y % 2 == 0) && (int64_t)s.Co * s.KH * s.KW < (1LL << 31) && s.N <= 65000 &&
           (int64_t)s.OH * s.OW < (1LL << 31) && px / 128 * ((s.Co + 63) / 64) < (1LL << 30) && tc::encode_fn() != nullptr && tc::encode_im2col_fn() != nullptr;
}

// The channels-last layouts are read and written where they lie and keep the rules they are documented with.
bool conv2d_tc_layout_supported(const ConvShape& s) {
    return s.C % 8 == 0 && s.C >= 64 && s.Co >= 64 && s.H >= 8 && s.W >= 8 && (int64_t)s.N * s.OH * s.OW >= 1024;
}
bool conv2d_wgrad_tc_layout_supported(const ConvShape& s) {
    return s.C % 8 == 0 && s.Co % 8 == 0 && s.C >= 64 && s.Co >= 64 && s.H >= 8 * s.sh && s.W >= 8 * s.sw && s.OH >= 8 && s.OW >= 8 &&
           (int64_t)s.N * s.OH * s.OW >= 4096;
}

size_t conv2d_tc_workspace(const ConvShape& s) {
    const size_t cp = tcconv::pitch8(s.C);
    const size_t xb = ((size_t)s.N * s.H * s.W * cp * 2 + 1023) & ~(size_t)1023;
    const size_t wb = ((size_t)s.Co * cp * s.KH * s.KW * 2 + 1023) & ~(size_t)1023;
    return xb + wb + 1024;
}

int conv2d_tc(const void* x, const void* w, void* y, float* stats, const ConvShape& s, void* workspace, cudaStream_t st,
              const ConvLayout& lay, bool* stats_filled) {
    using namespace tcconv;
    unsigned char* ws = (unsigned char*)(((uintptr_t)workspace + 1023) & ~(uintptr_t)1023);
    // NHWC ("acdb") activations are what the kernel reads: no staging pass for x then
    __nv_bfloat16* xt = lay.x_nhwc ? (__nv_bfloat16*)const_cast<void*>(x) : (__nv_bfloat16*)ws;
    const int cp = pitch8(s.C);
    __nv_bfloat16* wt = (__nv_bfloat16*)(ws + (((size_t)s.N * s.H * s.W * cp * 2 + 1023) & ~(size_t)1023));
    const int HW = s.H * s.W;
    {   // x[N][C][HW] -> xt[N][HW][C], and the weights tap-major, in one launch
        const int64_t nw = (int64_t)s.Co * s.C * s.KH * s.KW;
        const LayoutJob job{(const __nv_bfloat16*)x, xt, s.C, HW, cp, lay.x_nhwc ? 0 : s.N};
        const unsigned gx = (unsigned)((HW + 63) / 64), gy = (unsigned)((s.C + layout_rows(s.C) - 1) / layout_rows(s.C));
        const int64_t per_slice = (int64_t)gx * gy * 256;
        const unsigned wz = (unsigned)std::min<int64_t>(32, std::max<int64_t>(1, (nw + per_slice - 1) / per_slice));
        dim3 g(gx, gy, (unsigned)job.n + wz);          // the first wz slices re-order the weights
        float* zero = (stats && s.Co <= STATS_MAX_CO) ? stats : nullptr;   // zeroed here instead of by a memset node
        const auto kernel = layout_rows(s.C) == 128 ? transpose_bf16_batched_kernel<128> : transpose_bf16_batched_kernel<64>;
        kernel<<<g, 256, 0, st>>>(job, LayoutJob(), (int)wz, (const __nv_bfloat16*)w, wt, s.Co, s.C, s.KH * s.KW, cp, zero, 2 * s.Co,
                                  lay.w_grad ? 2 : lay.w_ohwi ? 1 : 0);
        B200JT_LAUNCH_CHECK();
    }
    ConvArgs A;
    A.N = s.N; A.C = s.C; A.H = s.H; A.W = s.W; A.Co = s.Co; A.KH = s.KH; A.KW = s.KW; A.OH = s.OH; A.OW = s.OW;
    A.sh = s.sh; A.sw = s.sw; A.ph = s.ph; A.pw = s.pw; A.dh = s.dh; A.dw = s.dw;
    A.pixels = (int64_t)s.N * s.OH * s.OW;
    A.last_k = (s.C - (s.C + BK - 1) / BK * BK + BK + UMMA_K - 1) / UMMA_K;
    // Tile by estimated time: the grid is persistent with a static round-robin, so it takes ceil(tiles / slots) rounds, each of a
    // tile's main loop and the part of its epilogue that the next tile's main loop does not hide (about half). A k-block of 64 channels
    // measured 342, 354, 477 ns with 64, 128, 256 output channels and 347, 380, 445 ns on a pair: most of it is the feed of the
    // x boxes (their 128 rows of 128 bytes), so narrow tiles feed the MMAs worse but leave less of the last round idle. The epilogue costs
    // 12.5 ns a channel, with statistics too since they come from the square: over 24 layers with statistics, each forced through the six
    // variants, the choice is 0.9 % from the best on average and 5 % at most (with 23 ns, what the shuffles took, 1.4 and 10 %).
    const int slots = pair_slots();
    const char* bn_env = getenv("B200JT_CONV_BN");          // read on every call: tests force each variant in turn
    const char* pair_env = getenv("B200JT_CONV_PAIR");
    const int forced_bn = bn_env ? atoi(bn_env) : 0;
    const int k_blocks = s.KH * s.KW * ((s.C + BK - 1) / BK);
    bool pair = false; int bn = 256; double best = 1e30;
    for (int p = 0; p < 2; p++) {
        if ((pair_env && atoi(pair_env) != p) || (p && !slots)) continue;
        for (int b = 64; b <= 256; b *= 2) {
            if ((forced_bn == 64 || forced_bn == 128 || forced_bn == 256) && forced_bn != b) continue;
            const int64_t t = (A.pixels + BM * (p + 1) - 1) / (BM * (p + 1)) * ((s.Co + b - 1) / b);
            const double block = 300 + (p ? 0.57 : 0.69) * b;
            const double epilogue = 600 + b * 12.5;
            const int n = p ? slots : kNumSMs;
            const double ns = (double)((t + n - 1) / n) * (k_blocks * block + 0.5 * epilogue + 250 * p) + epilogue;
            if (ns < best) { best = ns; pair = p; bn = b; }
        }
    }
    const int ctas = pair ? 2 : 1;
    A.tiles_m = (int)((A.pixels + BM * ctas - 1) / (BM * ctas));
    A.tiles_n = (s.Co + bn - 1) / bn;
    CUtensorMap mx, mw;
    if (!make_map_im2col(&mx, xt, s.N, s.H, s.W, s.C, s.sh, s.sw, s.ph, s.pw, s.dh * (s.KH - 1), s.dw * (s.KW - 1), BM) || !make_map_w(&mw, wt, s, bn / ctas)) return fail(-4, "conv2d: cuTensorMapEncodeTiled failed");
    if (!slots) return fail(-4, "conv2d: no room for the kernel's shared memory");
    A.vec = 8;
    while (A.vec > 1 && ((int64_t)s.OH * s.OW % A.vec || (uintptr_t)y % (2 * A.vec))) A.vec /= 2;
    if (A.vec == 2) A.vec = 1;
    float* fused = (stats && s.Co <= STATS_MAX_CO) ? stats : nullptr;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = 2; at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(std::min(A.tiles_m * A.tiles_n, pair ? slots : kNumSMs) * ctas));
    cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = SMEM_BYTES; cfg.stream = st; cfg.attrs = at; cfg.numAttrs = pair ? 2 : 1;
    void* args[] = {&mx, &mw, &y, &fused, &A};
    B200JT_CUDA(cudaLaunchKernelExC(&cfg, kernel_of(lay.y_nhwc, bn, pair), args));
    *stats_filled = fused != nullptr;
    return 0;
}

// ---- weight gradient ---------------------------------------------------------------------------------------
// dw[o,c,kh,kw] = sum over (n,oh,ow) of dy[n,o,oh,ow] * x[n,c,oh*stride-pad+kh*dil, ow*stride-pad+kw*dil]: the reduce.add
// over (batch, rows, columns) of reindex(x) * broadcast(dy) that ConvTuner relays to cudnnConvolutionBackwardFilter
// (python/jittor/extern/cuda/cudnn/ops/cudnn_conv_backward_w_op.cc:292). As a GEMM per filter tap:
//   D[c, o] = sum over pixels of X_tap[pixel, c] * DY[pixel, o],     M = Cin (128 per CTA), N = Cout (256), K = N*OH*OW.
// x and dy are first copied to NHWC, so an im2col TMA load of 64 output pixels x 64 channels lands as 64 rows of 128 B with
// the channel axis contiguous: both operands are MN-major (their own axis contiguous, K = pixel strided), and the same box
// geometry as the forward kernel carries the tap's shift and the stride in its coordinates. One CTA owns one
// (tap, 128 input channels, 256 output channels) accumulator in TMEM and walks a contiguous range of 64-pixel blocks; the
// K axis is split over `splits` CTAs per accumulator to fill the GPU, each writing fp32 partial sums that a second kernel
// adds in split order (deterministic) and stores as bf16 in OIHW order.
namespace tcwgrad {

using namespace tc;

constexpr int BM = 128, PIX = 64, THREADS = 192;
constexpr int CHUNK_BYTES = PIX * 64 * 2;                    // one box: 64 pixels x 64 channels of bf16
// TAPS filter taps per CTA share the dy tile of a stage (their x tiles differ by the tap's shift): with two taps a stage is
// 2 * 16 KB of x + 32 KB of dy for twice the MMAs, i.e. two thirds of the operand bytes per FLOP -- the feed from L2 into
// shared memory is what bounds the one-tap form. Two accumulators fill the 512 TMEM columns; three 64 KB stages.
template <int TAPS> struct Ring {
    static constexpr int STAGES = TAPS == 2 ? 3 : 4;
    static constexpr int MAX_STAGE_BYTES = (TAPS * (BM / 64) + 256 / 64) * CHUNK_BYTES;
    static constexpr int SMEM_BYTES = STAGES * MAX_STAGE_BYTES + 1024 + 256;
};

struct WgradArgs {
    int N, C, H, W, Co, KH, KW, OH, OW, sh, sw, ph, pw, dh, dw;
    int64_t blocks;                  // the K axis in units of 64 consecutive output pixels
    int tiles_m, tiles_n, splits, groups;      // groups: ceil(taps / TAPS) tap groups
};

template <int BN_T, int TAPS>
__global__ void __launch_bounds__(THREADS, 1)
wgrad_bf16_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_dy,
                  float* __restrict__ part, const __grid_constant__ WgradArgs A) {
    constexpr int STAGES = Ring<TAPS>::STAGES, MAX_STAGE_BYTES = Ring<TAPS>::MAX_STAGE_BYTES;
    constexpr int XBOX = BM / 64, YBOX = BN_T / 64;           // boxes per tap of x, boxes of dy
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + STAGES * MAX_STAGE_BYTES);
    uint64_t* full = bars;
    uint64_t* empty = bars + STAGES;
    uint64_t* acc_full = bars + 2 * STAGES;
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int taps = A.KH * A.KW;
    const int base = A.groups * A.tiles_m * A.tiles_n;
    const int split = blockIdx.x / base;
    int tile = blockIdx.x - split * base;
    const int group = tile % A.groups; tile /= A.groups;
    const int tn = tile % A.tiles_n, tm = tile / A.tiles_n;
    const int tap0 = group * TAPS;
    const int ntap = min(TAPS, taps - tap0);                 // the last group of an odd tap count holds one tap
    const int64_t p0 = A.blocks * split / A.splits, p1 = A.blocks * (split + 1) / A.splits;
    const int k_blocks = (int)(p1 - p0);                     // >= 1: the host keeps splits <= blocks

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(TAPS * BN_T) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    asm volatile("griddepcontrol.wait;" ::: "memory");          // for the layout pass

    if (warp == 0) {
        // The whole warp walks the blocks; lane 0 waits for the slot and announces the bytes, then every lane that owns a box
        // issues it: chunk j of a stage belongs to lane j -- x chunks of tap 0, x chunks of tap 1, then the dy chunks.
        const bool is_x = lane < TAPS * XBOX;
        const int t = is_x ? lane / XBOX : 0;                 // which of this CTA's taps the lane's x box serves
        const int tap = min(tap0 + t, taps - 1);
        const int kh = tap / A.KW, kw = tap - kh * A.KW;
        const int plane = A.OH * A.OW;
        int n = (int)(p0 * PIX / plane), in = (int)(p0 * PIX - (int64_t)n * plane);
        const bool owns = is_x ? t < ntap : lane < TAPS * XBOX + YBOX;
        const CUtensorMap* map = is_x ? &map_x : &map_dy;
        const int c0 = is_x ? tm * BM + (lane - t * XBOX) * 64 : tn * BN_T + (lane - TAPS * XBOX) * 64;
        const int sw = is_x ? A.sw : 1, sh = is_x ? A.sh : 1, pw = is_x ? A.pw : 0, ph = is_x ? A.ph : 0;
        const int dw = is_x ? kw * A.dw : 0, dh = is_x ? kh * A.dh : 0;
        const uint32_t stage_bytes = (uint32_t)(ntap * XBOX + YBOX) * CHUNK_BYTES;
        int stage = 0; uint32_t phase = 0;
        bool ok = true;
        for (int kb = 0; kb < k_blocks; kb++) {
            if (lane == 0) {
                ok = mbar_wait(empty + stage, phase ^ 1, abort_flag, 21);
                if (ok) mbar_expect_tx(full + stage, stage_bytes);
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
            // pixels outside x or past the last image and channels past C / Co are zero-filled by TMA
            if (owns) {
                const int oh = in / A.OW, ow = in - oh * A.OW;
                tma_load_im2col<1>(smem + stage * MAX_STAGE_BYTES + lane * CHUNK_BYTES, map, smem_u32(full + stage), c0, ow * sw - pw, oh * sh - ph, n, dw, dh);
            }
            for (in += PIX; in >= plane; in -= plane) n++;
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok && lane == 0) {
            for (int s = 0; s < STAGES; s++)
                for (uint32_t i = 0; i < 4096 && !mbar_try(full + s, 0) && !mbar_try(full + s, 1); i++) __nanosleep(64);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = make_idesc(BM, BN_T, true) | (1u << 15);      // A and B both MN-major
            constexpr int KSTEP = (UMMA_K * 128) / 16;                                // 16 pixel rows of 128 B, in 16-byte units
            int stage = 0; uint32_t phase = 0;
            bool ok = true;
            for (int kb = 0; kb < k_blocks; kb++) {
                if (!(ok = mbar_wait(full + stage, phase, abort_flag, 22))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t sa = smem_u32(smem + stage * MAX_STAGE_BYTES);
                const uint64_t db = make_smem_desc_mn(sa + TAPS * XBOX * CHUNK_BYTES, CHUNK_BYTES, 1024);
#pragma unroll
                for (int t = 0; t < TAPS; t++) {
                    if (t < ntap) {
                        const uint64_t da = make_smem_desc_mn(sa + t * XBOX * CHUNK_BYTES, CHUNK_BYTES, 1024);
#pragma unroll
                        for (int k = 0; k < PIX / UMMA_K; k++)
                            umma_f16(tmem_base + t * BN_T, da + KSTEP * k, db + KSTEP * k, idesc, (kb | k) != 0);
                    }
                }
                umma_commit(empty + stage);
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
            if (ok) umma_commit(acc_full);
        }
    } else {
        const int quad = warp & 3;
        bool ok = mbar_wait(acc_full, 0, abort_flag, 23);
        ok = __all_sync(0xffffffffu, ok);
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");      // the fold's CTAs may take their places; they wait for this grid
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int c = tm * BM + quad * 32 + lane;                        // TMEM lane = input channel
            const bool vec = (A.Co & 3) == 0;
            for (int t = 0; t < ntap; t++) {
                const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + t * BN_T;
                float* prow = part + (((int64_t)split * taps + tap0 + t) * A.C + c) * A.Co;
#pragma unroll 1
                for (int ch = 0; ch < BN_T / 32; ch++) {
                    uint32_t v[32];
                    tmem_ld32(taddr + ch * 32, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    const int o0 = tn * BN_T + ch * 32;
                    if (c < A.C && o0 < A.Co) {
                        if (vec && o0 + 32 <= A.Co) {
#pragma unroll
                            for (int q = 0; q < 8; q++)
                                *reinterpret_cast<uint4*>(prow + o0 + q * 4) = make_uint4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
                        } else {
#pragma unroll
                            for (int e = 0; e < 32; e++) if (o0 + e < A.Co) prow[o0 + e] = __uint_as_float(v[e]);
                        }
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TAPS * BN_T) : "memory");
    }
}

// Bound by the latency of its reads from L2 (29 parts of 128 x 128 x 9 values: 17 MB), hence 16 of them under way per thread.
// dw[o][c][tap] (or [o][tap][c] for the "ohwi" layout) = sum over splits (ascending) of part[split][tap][c][o], rounded to bf16 once.
__global__ void __launch_bounds__(256)
wgrad_fold_kernel(const float* __restrict__ part, __nv_bfloat16* __restrict__ dw, int splits, int taps, int C, int Co, int ohwi) {
    const int64_t n = (int64_t)taps * C * Co;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int o = (int)(i % Co); const int64_t t = i / Co;
        const int c = (int)(t % C); const int tap = (int)(t / C);
        float acc = 0.f;
        int s = 0;
        for (; s + 16 <= splits; s += 16) {                      // 16 loads under way: the partial sums come from L2
            float v[16];
#pragma unroll
            for (int k = 0; k < 16; k++) v[k] = part[(int64_t)(s + k) * n + i];
#pragma unroll
            for (int k = 0; k < 16; k++) acc += v[k];
        }
#pragma unroll 8
        for (; s < splits; s++) acc += part[(int64_t)s * n + i];
        dw[ohwi ? ((int64_t)o * taps + tap) * C + c : ((int64_t)o * C + c) * taps + tap] = __float2bfloat16(acc);
    }
}

struct Plan { int bn, taps_per_cta, groups, tiles_m, tiles_n, splits; int64_t blocks; size_t xb, dyb, pb; };

static Plan plan_for(const ConvShape& s) {
    Plan p;
    const int taps = s.KH * s.KW;
    const char* env = getenv("B200JT_WGRAD_TAPS");           // 1 forces one tap per CTA (tests run both forms)
    p.bn = s.Co <= 128 ? 128 : 256;
    p.taps_per_cta = (taps >= 2 && !(env && atoi(env) == 1)) ? 2 : 1;
    p.groups = (taps + p.taps_per_cta - 1) / p.taps_per_cta;
    p.tiles_m = (s.C + BM - 1) / BM;
    p.tiles_n = (s.Co + p.bn - 1) / p.bn;
    p.blocks = ((int64_t)s.N * s.OH * s.OW + PIX - 1) / PIX;
    // fill the GPU once when the accumulators alone do not; every split keeps at least 8 blocks (512 pixels) of K
    auto splits_for = [&](int64_t groups) {
        const int64_t base = groups * p.tiles_m * p.tiles_n;
        return std::max<int64_t>(1, std::min<int64_t>(base >= kNumSMs ? 1 : kNumSMs / base, p.blocks / 8));
    };
    p.splits = (int)splits_for(p.groups);
    p.xb = ((size_t)s.N * s.H * s.W * tcconv::pitch8(s.C) * 2 + 1023) & ~(size_t)1023;
    p.dyb = ((size_t)s.N * s.OH * s.OW * tcconv::pitch8(s.Co) * 2 + 1023) & ~(size_t)1023;
    // the partial sums are sized for whichever form splits K more finely, so the workspace query does not depend on the switch
    const int64_t most = std::max(splits_for(taps), splits_for((taps + 1) / 2));
    p.pb = ((size_t)most * taps * s.C * s.Co * 4 + 1023) & ~(size_t)1023;
    return p;
}

}  // namespace tcwgrad

// Any channel counts and extents, as for the forward kernel: the sums over pixels were 8.4 ms on the CUDA cores for 304 -> 48
// channels of 56 x 56 (3 x 3 filter, 18 images).
bool conv2d_wgrad_tc_supported(const ConvShape& s, const void* x, const void* dy, const void* dw) {
    const int64_t taps = (int64_t)s.KH * s.KW;
    return s.groups == 1 && s.sh >= 1 && s.sh <= 4 && s.sw >= 1 && s.sw <= 4 && s.N <= 65000 && tcconv::im2col_fits(s) && (int64_t)s.OH * s.OW < (1LL << 31) &&
           taps * ((s.C + 127) / 128) * ((s.Co + 255) / 256) <= (1 << 20) &&
           ((uintptr_t)x % 2 == 0) && ((uintptr_t)dy % 2 == 0) && ((uintptr_t)dw % 2 == 0) && tc::encode_im2col_fn() != nullptr;
}

size_t conv2d_wgrad_tc_workspace(const ConvShape& s) {
    const tcwgrad::Plan p = tcwgrad::plan_for(s);
    return p.xb + p.dyb + p.pb + 1024;
}

int conv2d_wgrad_tc(const void* x, const void* dy, void* dw, const ConvShape& s, void* workspace, cudaStream_t st,
                    const ConvLayout& lay) {
    using namespace tcwgrad;
    const Plan p = plan_for(s);
    unsigned char* ws = (unsigned char*)(((uintptr_t)workspace + 1023) & ~(uintptr_t)1023);
    // channels-last ("acdb") x / dy are what the kernel reads: no copy on that side (lay.y_nhwc describes dy)
    __nv_bfloat16* xt = lay.x_nhwc ? (__nv_bfloat16*)const_cast<void*>(x) : (__nv_bfloat16*)ws;
    __nv_bfloat16* dyt = lay.y_nhwc ? (__nv_bfloat16*)const_cast<void*>(dy) : (__nv_bfloat16*)(ws + p.xb);
    float* part = (float*)(ws + p.xb + p.dyb);
    const int HW = s.H * s.W, OHW = s.OH * s.OW;
    {   // x[N][C][HW] -> [N][HW][C] and dy[N][Co][OH*OW] -> [N][OH*OW][Co]
        using tcconv::LayoutJob; using tcconv::layout_rows; using tcconv::pitch8;
        const LayoutJob jobs[2] = {{(const __nv_bfloat16*)x, xt, s.C, HW, pitch8(s.C), lay.x_nhwc ? 0 : s.N},
                                   {(const __nv_bfloat16*)dy, dyt, s.Co, OHW, pitch8(s.Co), lay.y_nhwc ? 0 : s.N}};
        const bool together = s.N <= 32000;                      // grid z
        for (int q = 0; q < (together ? 1 : 2); q++) {
            const LayoutJob a = jobs[q], b = together ? jobs[1] : LayoutJob();
            if (a.n + b.n == 0) continue;
            const int rows = std::max(a.n ? layout_rows(a.R) : 64, b.n ? layout_rows(b.R) : 64);
            const int r = std::max(a.n ? a.R : 0, b.n ? b.R : 0), cols = std::max(a.n ? a.Cn : 0, b.n ? b.Cn : 0);
            const dim3 g((unsigned)((cols + 63) / 64), (unsigned)((r + rows - 1) / rows), (unsigned)(a.n + b.n));
            const auto kernel = rows == 128 ? tcconv::transpose_bf16_batched_kernel<128> : tcconv::transpose_bf16_batched_kernel<64>;
            kernel<<<g, 256, 0, st>>>(a, b, 0, nullptr, nullptr, 0, 0, 0, 0, nullptr, 0, 0);
            B200JT_LAUNCH_CHECK();
        }
    }
    WgradArgs A;
    A.N = s.N; A.C = s.C; A.H = s.H; A.W = s.W; A.Co = s.Co; A.KH = s.KH; A.KW = s.KW; A.OH = s.OH; A.OW = s.OW;
    A.sh = s.sh; A.sw = s.sw; A.ph = s.ph; A.pw = s.pw; A.dh = s.dh; A.dw = s.dw;
    A.blocks = p.blocks; A.tiles_m = p.tiles_m; A.tiles_n = p.tiles_n; A.splits = p.splits; A.groups = p.groups;
    CUtensorMap mx, mdy;
    if (!tcconv::make_map_im2col(&mx, xt, s.N, s.H, s.W, s.C, s.sh, s.sw, s.ph, s.pw, s.dh * (s.KH - 1), s.dw * (s.KW - 1), PIX) ||
        !tcconv::make_map_im2col(&mdy, dyt, s.N, s.OH, s.OW, s.Co, 1, 1, 0, 0, 0, 0, PIX))
        return fail(-4, "conv2d_backward_w: cuTensorMapEncodeIm2col failed");
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [] {
        const std::pair<const void*, int> kernels[] = {
            {(const void*)wgrad_bf16_kernel<256, 1>, Ring<1>::SMEM_BYTES}, {(const void*)wgrad_bf16_kernel<128, 1>, Ring<1>::SMEM_BYTES},
            {(const void*)wgrad_bf16_kernel<256, 2>, Ring<2>::SMEM_BYTES}, {(const void*)wgrad_bf16_kernel<128, 2>, Ring<2>::SMEM_BYTES}};
        for (auto& k : kernels)
            if (attr_err == cudaSuccess) attr_err = cudaFuncSetAttribute(k.first, cudaFuncAttributeMaxDynamicSharedMemorySize, k.second);
    });
    B200JT_CUDA(attr_err);
    const int taps = s.KH * s.KW;
    const unsigned grid = (unsigned)((int64_t)p.groups * p.tiles_m * p.tiles_n * p.splits);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute early;
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization; early.val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(grid); cfg.blockDim = dim3(THREADS); cfg.stream = st; cfg.attrs = &early;
    // An early start saves 0.4 to 1.4 us from a graph, more of direct launches; but the CTAs then stand on the SMs in the order the
    // layout pass left them, and the taps that share x and dy through L2 lie further apart. Nine layers of 0.7e10 to 1.2e11 operations are all
    // faster with it (64 x 64 x 56 x 56 85.6 -> 84.7 us, 128 x 256 x 28 x 28 134.2 -> 133.4); of four with 2.4e11 one is slower
    // (256 x 256 x 28 x 28 241.7 -> 244.8), the others as they were; from 3.6e11 on the power cap's noise hides it.
    cfg.numAttrs = 2.0 * taps * s.C * s.Co * s.N * OHW < 2e11 ? 1 : 0;
    cfg.dynamicSmemBytes = p.taps_per_cta == 2 ? Ring<2>::SMEM_BYTES : Ring<1>::SMEM_BYTES;
    const auto kernel = p.taps_per_cta == 2 ? (p.bn == 256 ? wgrad_bf16_kernel<256, 2> : wgrad_bf16_kernel<128, 2>)
                                            : (p.bn == 256 ? wgrad_bf16_kernel<256, 1> : wgrad_bf16_kernel<128, 1>);
    B200JT_CUDA(cudaLaunchKernelEx(&cfg, kernel, mx, mdy, part, A));
    const int64_t n = (int64_t)taps * s.C * s.Co;
    cfg.gridDim = dim3(grid_for(n, 256)); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = 0; cfg.numAttrs = 1;
    B200JT_CUDA(cudaLaunchKernelEx(&cfg, wgrad_fold_kernel, (const float*)part, (__nv_bfloat16*)dw, p.splits, taps, s.C, s.Co, lay.w_ohwi ? 1 : 0));
    return 0;
}

int tcconv_status_fetch_and_clear() { return tc::status_fetch_and_clear(); }

}  // namespace b200jt
