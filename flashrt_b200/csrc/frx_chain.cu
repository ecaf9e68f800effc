// The join between the layers of the chained expert-stack benchmark (48 MoE layers, a window of
// three tokens per step): x_next = (x + y) / sqrt(mean((x + y)^2) + 1e-6), an RMS norm with unit
// weight. The reference joins its MoE layers through its attention blocks, which are outside this
// library; this stand-in keeps the activations of a deep stack at unit scale so that every layer
// sees realistic inputs. The order of every floating-point operation is fixed and stated, so a CPU
// restatement gives the same bits: r = x + y in float; lane l of one warp adds r[l]^2, r[l + 32]^2,
// ... in double in that order; the 32 lane sums are combined by a butterfly (offsets 16, 8, 4, 2,
// 1); inv = float(1 / sqrt(sum / n + 1e-6)) in double; x_next = r * inv in float.
#include "frx_common.cuh"

namespace frx {
namespace {

// Two forms with the same order of additions (lane l of a warp adds the squares of elements l, l + 32, ... one after the
// other, then the lanes are added), hence the same bits.
//
// A warp per token, which loads as it adds: n / 128 trips to memory, but 32 tokens at a time on an SM.
__global__ void __launch_bounds__(32) k_chain_rmsnorm_warp(const float* __restrict__ x, const float* __restrict__ y, float* __restrict__ out, int n) {
    pdl_wait();
    pdl_trigger();
    const int t = blockIdx.x, lane = threadIdx.x;
    const float* xr = x + size_t(t) * n;
    const float* yr = y + size_t(t) * n;
    double ss = 0.0;
    for (int i = lane; i < n; i += 32) {
        const float r = __fadd_rn(xr[i], yr[i]);
        ss = __dadd_rn(ss, __dmul_rn(double(r), double(r)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss = __dadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, o));
    const float inv = float(__ddiv_rn(1.0, __dsqrt_rn(__dadd_rn(__ddiv_rn(ss, double(n)), 1e-6))));
    for (int i = lane; i < n; i += 32) out[size_t(t) * n + i] = __fmul_rn(__fadd_rn(xr[i], yr[i]), inv);
}

// A block per token. Every thread loads its share of the row at once and leaves the squares in shared memory for the
// one warp that adds them: the row then costs one trip to memory and n / 32 dependent additions. Verifying three tokens
// through eight layers of 2048 elements: 223 -> 210 us per pass with it.
constexpr int kChainThreads = 512, kChainChunk = 4096;

__global__ void __launch_bounds__(kChainThreads) k_chain_rmsnorm(const float* __restrict__ x, const float* __restrict__ y, float* __restrict__ out, int n) {
    __shared__ double sq[kChainChunk];
    __shared__ float s_inv;
    pdl_wait();
    pdl_trigger();
    const int t = blockIdx.x, lane = threadIdx.x;
    const float* xr = x + size_t(t) * n;
    const float* yr = y + size_t(t) * n;
    constexpr int kHeld = kChainChunk / kChainThreads;   // the last chunk stays in registers until it is written
    float held[kHeld];
    double ss = 0.0;
    const int last = (n - 1) / kChainChunk * kChainChunk;
    for (int c0 = 0; c0 <= last; c0 += kChainChunk) {
#pragma unroll
        for (int j = 0; j < kHeld; ++j) {
            const int i = c0 + threadIdx.x + j * kChainThreads;
            held[j] = i < n ? __fadd_rn(xr[i], yr[i]) : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < kHeld; ++j) sq[threadIdx.x + j * kChainThreads] = __dmul_rn(double(held[j]), double(held[j]));
        __syncthreads();
        if (threadIdx.x < 32) {
            const int m = min(kChainChunk, n - c0);
#pragma unroll 16
            for (int i = lane; i < m; i += 32) ss = __dadd_rn(ss, sq[i]);
        }
        __syncthreads();
    }
    if (threadIdx.x < 32) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss = __dadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, o));
        if (lane == 0) s_inv = float(__ddiv_rn(1.0, __dsqrt_rn(__dadd_rn(__ddiv_rn(ss, double(n)), 1e-6))));
    }
    __syncthreads();
    const float inv = s_inv;
    for (int i = threadIdx.x; i < last; i += kChainThreads) out[size_t(t) * n + i] = __fmul_rn(__fadd_rn(xr[i], yr[i]), inv);
#pragma unroll
    for (int j = 0; j < kHeld; ++j) {
        const int i = last + threadIdx.x + j * kChainThreads;
        if (i < n) out[size_t(t) * n + i] = __fmul_rn(held[j], inv);
    }
}

}  // namespace
}  // namespace frx

using namespace frx;

extern "C" int frx_chain_rmsnorm_unit(const float* x, const float* y, float* x_next, int T, int n, frx_stream_t stream) {
    if (T < 0 || n < 1) return fail(FRX_ERR_ARG, "frx_chain_rmsnorm_unit: T %d, n %d", T, n);
    if (T == 0) return FRX_OK;
    if (!x || !y || !x_next) return fail(FRX_ERR_ARG, "frx_chain_rmsnorm_unit: null pointer");
    // The block form is the faster one while its blocks (four to an SM) are all resident, and the longer the rows, the more
    // trips it saves; beyond that the warp form has more tokens in flight, up to rows whose chunks of additions outweigh it.
    // us, warp / block form, by row length: 512: 2.2 / 2.3 (1 token), 2.6 / 3.5 (512 tokens); 1024: 2.9 / 2.6 (1), 3.0 / 3.1
    // (256), 3.2 / 3.9 (512); 2048: 4.2 / 3.2 (1), 4.7 / 4.7 (512), 5.2 / 6.5 (600), 17.3 / 28.7 (4,096); 4096: 8.0 / 6.4 (592),
    // 17.1 / 25.5 (2,048); 8192: 11.9 / 7.6 (1), 29.9 / 24.2 (1,024), 109.5 / 91.3 (4,096).
    const int per_sm = n >= 2048 ? 4 : n >= 1024 ? 2 : n >= 640 ? 1 : 0;
    if (n >= 8192 || T <= per_sm * sm_count())
        FRX_LAUNCH(kKCombine, stream, launch_pdl(k_chain_rmsnorm, dim3(unsigned(T)), dim3(kChainThreads), 0, stream, x, y, x_next, n));
    else
        FRX_LAUNCH(kKCombine, stream, launch_pdl(k_chain_rmsnorm_warp, dim3(unsigned(T)), dim3(32), 0, stream, x, y, x_next, n));
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}
