// The parameter update of the optimisers for many tensors in one launch. Op by op an SGD step with momentum is two fused chains
// per parameter, each planned, allocated and launched by itself: 12 launches and 0.3 ms of host time for a network of six
// small parameters. Here the pointers of up to kMaxTensors parameters ride in the launch's arguments and a block takes 2048
// elements of one of them. Every step rounds as the op-by-op chain does (no fused multiply-adds): the same bits.
#include "common.cuh"

namespace b200jt {
namespace {

constexpr int kMaxTensors = 48, kChunk = 2048;
enum Kind { SGD = 0, ADAM = 1, ADAMW = 2, RMSPROP = 3 };

struct Pack {
    const float *p[kMaxTensors], *g[kMaxTensors], *s0[kMaxTensors], *s1[kMaxTensors];
    float *po[kMaxTensors], *s0o[kMaxTensors], *s1o[kMaxTensors];
    int64_t n[kMaxTensors];
    int first[kMaxTensors + 1];                 // first block of each tensor
    float h[8];
    int count, kind, nesterov;
};

__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }

__global__ void __launch_bounds__(256) optim_kernel(const __grid_constant__ Pack k) {
    int lo = 0, hi = k.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (k.first[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const int64_t base = (int64_t)(blockIdx.x - k.first[lo]) * kChunk, n = k.n[lo];
    const float* h = k.h;
#pragma unroll 4
    for (int64_t i = base + threadIdx.x; i < base + kChunk && i < n; i += 256) {
        const float p = k.p[lo][i], g = k.g[lo][i];
        if (k.kind == SGD) {                    // h: lr, momentum, weight decay, 1 - dampening
            const float dp = add(mul(p, h[2]), g), v = add(mul(k.s0[lo][i], h[1]), mul(dp, h[3]));
            k.s0o[lo][i] = v;
            k.po[lo][i] = sub(p, mul(k.nesterov ? add(dp, mul(v, h[1])) : v, h[0]));
        } else if (k.kind == RMSPROP) {         // h: lr, alpha, 1 - alpha, eps
            const float v = add(mul(k.s0[lo][i], h[1]), mul(mul(g, g), h[2]));
            k.s0o[lo][i] = v;
            k.po[lo][i] = sub(p, __fdiv_rn(mul(g, h[0]), add(__fsqrt_rn(v), h[3])));
        } else {                                // h: b0, 1 - b0, b1, 1 - b1, step size, eps, decay (Adam: weight decay; AdamW: 1 - lr * wd), sqrt(c1)
            const float q = k.kind == ADAMW ? mul(p, h[6]) : p, d = k.kind == ADAM ? add(mul(p, h[6]), g) : g;
            const float m = add(mul(k.s1[lo][i], h[0]), mul(d, h[1])), v = add(mul(k.s0[lo][i], h[2]), mul(mul(d, d), h[3]));
            k.s1o[lo][i] = m;
            k.s0o[lo][i] = v;
            const float root = __fsqrt_rn(v);
            k.po[lo][i] = sub(q, __fdiv_rn(mul(m, h[4]), add(k.kind == ADAMW ? __fdiv_rn(root, h[7]) : root, h[5])));
        }
    }
}

}  // namespace
}  // namespace b200jt

using namespace b200jt;

extern "C" int b200jt_optim_step(const char* kind, int count, const int64_t* sizes, const float* const* p, const float* const* g,
                                 const float* const* s0, const float* const* s1, float* const* p_out, float* const* s0_out,
                                 float* const* s1_out, const double* hyper, int n_hyper, int nesterov, void* stream) {
    static const char* names[] = {"sgd", "adam", "adamw", "rmsprop"};
    int code = -1;
    for (int i = 0; i < 4; i++) if (kind && !strcmp(kind, names[i])) code = i;
    B200JT_CHECK_ARG(code >= 0, "kind must be sgd, adam, adamw or rmsprop");
    B200JT_CHECK_ARG(count >= 0 && sizes && p && g && s0 && p_out && s0_out && hyper && n_hyper >= 4 && n_hyper <= 8, "missing argument");
    const bool two = code == ADAM || code == ADAMW;
    B200JT_CHECK_ARG(!two || (s1 && s1_out && n_hyper == 8), "Adam keeps two states and takes eight hyper-parameters");
    for (int at = 0; at < count;) {
        Pack k{};
        int64_t blocks = 0;
        for (; at < count && k.count < kMaxTensors; at++) {
            const int64_t n = sizes[at];
            if (n <= 0) continue;
            const int64_t need = (n + kChunk - 1) / kChunk;
            B200JT_CHECK_ARG(need < (1ll << 30), "parameter too large");
            if (blocks + need > 0x7fffffff) break;
            const int i = k.count++;
            k.p[i] = p[at]; k.g[i] = g[at]; k.s0[i] = s0[at]; k.s1[i] = two ? s1[at] : nullptr;
            k.po[i] = p_out[at]; k.s0o[i] = s0_out[at]; k.s1o[i] = two ? s1_out[at] : nullptr;
            k.n[i] = n; k.first[i] = (int)blocks;
            blocks += need;
        }
        if (!k.count) break;
        for (int i = 0; i < n_hyper; i++) k.h[i] = (float)hyper[i];
        k.kind = code; k.nesterov = nesterov;
        optim_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(k);
        B200JT_LAUNCH_CHECK();
    }
    return 0;
}
