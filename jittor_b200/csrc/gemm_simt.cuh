// Host entry points of the CUDA-core contraction kernels (gemm_simt.cu) and of the tcgen05 kernels.
#pragma once
#include "common.cuh"

namespace b200jt {

struct ConvShape {
    int N, C, H, W, Co, KH, KW, OH, OW, sh, sw, ph, pw, dh, dw;
    int groups = 1;
};
// Memory layouts other than the default NCHW / OIHW (tensor-core path only): x and y as NHWC ("acdb"), w as OHWI ("ohwi").
struct ConvLayout { bool x_nhwc = false, w_ohwi = false, y_nhwc = false, w_grad = false; };     // w_grad: w[C][Co][taps], taps from the last

int matmul_simt(const void* a, const void* b, void* c, int dtype, int64_t M, int64_t N, int64_t K,
                bool trans_a, bool trans_b, cudaStream_t st);
int batched_matmul_simt(const void* a, const void* b, void* c, int dtype, int64_t batch, int64_t a_batch, int64_t b_batch,
                        int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b, cudaStream_t st);
// tcgen05 path (gemm_tcgen05.cu)
bool matmul_tc_supported(int64_t M, int64_t N, int64_t K, const void* a, const void* b, const void* c);
size_t matmul_tc_workspace(int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b, bool may_split);
int matmul_tc(const void* a, const void* b, void* c, int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b,
              void* workspace, bool may_split, cudaStream_t st);
bool batched_matmul_tc_supported(int64_t batch, int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b,
                                 const void* a, const void* b, const void* c);
int batched_matmul_tc(const void* a, const void* b, void* c, int64_t batch, int64_t a_batch, int64_t b_batch,
                      int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b, cudaStream_t st);
int tc_status_fetch_and_clear();

bool conv2d_tc_supported(const ConvShape& s, const void* x, const void* w, const void* y);
bool conv2d_tc_layout_supported(const ConvShape& s);
bool conv2d_wgrad_tc_layout_supported(const ConvShape& s);
size_t conv2d_tc_workspace(const ConvShape& s);
// `stats_filled`: whether the epilogue fills `stats` (the return value, as everywhere, is 0 or an error, which may be any number)
int conv2d_tc(const void* x, const void* w, void* y, float* stats, const ConvShape& s, void* workspace, cudaStream_t st,
              const ConvLayout& lay, bool* stats_filled);
// weight gradient on tcgen05 (bf16, groups == 1): K = N*OH*OW pixels, split over CTAs, fp32 partial sums folded in a fixed order
bool conv2d_wgrad_tc_supported(const ConvShape& s, const void* x, const void* dy, const void* dw);
size_t conv2d_wgrad_tc_workspace(const ConvShape& s);
// lay: x_nhwc / y_nhwc say that x / dy are channels-last already (no copy), w_ohwi that dw is written [Co][KH][KW][C]
int conv2d_wgrad_tc(const void* x, const void* dy, void* dw, const ConvShape& s, void* workspace, cudaStream_t st,
                    const ConvLayout& lay = ConvLayout());
int tcconv_status_fetch_and_clear();
int peer_status_fetch_and_clear();          // peer_allreduce.cu

// float32 contractions (gemm_f32.cu): tiled fp32x2 FMAs, k split over clusters; sizes beyond its 32-bit offsets stay below
bool matmul_f32_supported(int64_t batch, int64_t M, int64_t N, int64_t K);
double matmul_f32_ns(int64_t M, int64_t N, int64_t K);          // estimated time
size_t matmul_f32_workspace(int64_t M, int64_t N, int64_t K);
int matmul_f32(const void* a, const void* b, void* c, int64_t batch, int64_t a_batch, int64_t b_batch, int64_t M, int64_t N, int64_t K,
               bool trans_a, bool trans_b, void* workspace, size_t workspace_bytes, cudaStream_t st);
// ... and on the tensor cores, operands split into bfloat16 parts (gemm_f32_tc.cu)
bool matmul_f32_tc_wanted(int64_t M, int64_t N, int64_t K);
size_t matmul_f32_tc_workspace(int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b);
int matmul_f32_tc(const void* a, const void* b, void* c, int64_t M, int64_t N, int64_t K, bool trans_a, bool trans_b, void* workspace, cudaStream_t st);
int tcf32_status_fetch_and_clear();
bool conv2d_f32_supported(const ConvShape& s);
int conv2d_f32(const void* x, const void* w, void* y, const ConvShape& s, cudaStream_t st);
bool conv2d_transpose_f32_supported(const ConvShape& s);
int conv2d_transpose_f32(const void* x, const void* w, void* y, const ConvShape& s, cudaStream_t st);
size_t conv2d_wgrad_f32_workspace(const ConvShape& s);
int conv2d_wgrad_f32(const void* x, const void* dy, void* dw, const ConvShape& s, void* workspace, size_t workspace_bytes, cudaStream_t st);

int conv2d_simt(const void* x, const void* w, void* y, int dtype, const ConvShape& s, cudaStream_t st);
int conv2d_backward_w_simt(const void* x, const void* dy, void* dw, int dtype, const ConvShape& s, cudaStream_t st);
int conv2d_transpose_simt(const void* x, const void* w, void* y, int dtype, const ConvShape& s, cudaStream_t st);

}  // namespace b200jt
