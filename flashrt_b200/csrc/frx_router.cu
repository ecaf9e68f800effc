// Router projection in front of the router: logits[t][e] = sum_k W[e][k] * x[t][k], with W in bf16
// and x, the products and the sums in fp32, and in the same launch the shared expert's gate logit
// (one more bf16 row). The reference computes both with one launch of k_bf16_multi
// (arch/qwen4exp/blocks.cu:83-120, called at moe_fast.cu:1039-1042 and moe_stream.cu:145-149): exact
// bf16 x fp32 products, fp32 accumulation, no activation on these two outputs. The order of the
// additions differs from the reference's (and from one GPU generation's launch shape to another in
// the reference itself), so parity is to a tolerance, against a float64 sum.
//
// One block works on tiles of 8 rows x 16 or 64 tokens or 16 rows x 16, 24 or 40. Each of its 8 warps takes an eighth of K and
// walks it in pieces of 32: the piece of x (fp32) and of W (bf16) go through the warp's own shared memory (cp.async),
// a lane accumulates 4 rows x TJ tokens, and at the end the eight partial tiles are added in warp order (fixed, so results
// are reproducible and do not depend on the tile).
// Bound: the latency of a chain of pieces for few tokens (hence four in flight in the small tile); with more, what a
// shared-memory load delivers (128 bytes a clock: 24 clocks of loads and 16 of multiply-adds per 4 x 4 x 4) and the last
// wave. Rows of x are padded so that no two tokens of a quarter-warp share a bank.
// 513 rows of 2560, us: 17 tokens 16.6 -> 7.2, 37 tokens 17.2 -> 9.4, 293 tokens 49 -> 30, 1024 tokens 126 -> 89 (before: one
// tile of 8 x 64 for any number of tokens, one piece in flight).
#include "frx_common.cuh"

#include <algorithm>
#include <mutex>

namespace frx {
namespace {

constexpr int kRtWarps = 8, kRtPiece = 32, kRtPad = 36;   // 36: rows stay 16-byte aligned, no bank conflicts
// RY lanes along the rows (4 rows each), 32 / RY along the tokens (TJ tokens each)
template <int RY, int TJ>
struct RtShape {
    static constexpr int tx = 32 / RY, rows = 4 * RY, tok = tx * TJ, depth = TJ == 1 ? 4 : 2;
    static constexpr int piece = tok * kRtPad * 4 + rows * kRtPiece * 2;   // x (fp32, padded rows), W (bf16)
    static constexpr int warp = depth * piece;
    static constexpr int smem = kRtWarps * warp;
    static constexpr int red = tok + 1;   // row of partial sums: odd, the sums are read across rows
    static_assert(rows % 8 == 0 && tok % 4 == 0, "the copies take 8 rows of W and 4 tokens at a time");
    static_assert(kRtWarps * rows * red * 4 <= smem, "the reduction buffer reuses the pieces' shared memory");
};

__device__ __forceinline__ float bf16_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
// 16 bytes global -> shared without passing through registers; src_bytes = 0 writes zeros
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// rows: E router rows followed by the gate row when w_gate is given (row E). W rows are n bf16 each.
template <int RY, int TJ>
__global__ void __launch_bounds__(kRtWarps * 32, 2) k_router_logits(const uint16_t* __restrict__ w_router, const uint16_t* __restrict__ w_gate,
                                                                  const float* __restrict__ x, int T, int E, int n,
                                                                  float* __restrict__ logits, float* __restrict__ gate_logit) {
    using Sh = RtShape<RY, TJ>;
    extern __shared__ __align__(16) uint8_t smem[];
    pdl_wait();
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t mine = smem_u32(smem) + warp * Sh::warp;
    const int rows_total = E + (w_gate ? 1 : 0), row_tiles = (rows_total + Sh::rows - 1) / Sh::rows, tiles = row_tiles * ((T + Sh::tok - 1) / Sh::tok);
    const int ry = lane / Sh::tx, tx = lane % Sh::tx;   // this lane's tile: rows ry + RY i, tokens tx + Sh::tx j (no bank conflicts)
    const int kslice = n / kRtWarps, pieces = kslice / kRtPiece, kbase = warp * kslice;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int r0 = tile % row_tiles * Sh::rows, t0 = tile / row_tiles * Sh::tok;
        const int wrow = lane >> 2, wk = (lane & 3) * 8;   // this lane's 8 weights of a piece, in rows wrow, wrow + 8, ...
        const uint16_t* wsrc[Sh::rows / 8];
        uint32_t wbytes[Sh::rows / 8];
#pragma unroll
        for (int i = 0; i < Sh::rows / 8; ++i) {
            const int r = r0 + wrow + 8 * i;
            wsrc[i] = (r < E || !w_gate ? w_router + size_t(min(r, E - 1)) * n : w_gate) + kbase + wk;
            wbytes[i] = r < rows_total ? 16u : 0u;
        }
        // the copy of one piece into its buffer: 8 float4 of x per token, 32 bf16 of W per row
        auto fetch = [&](int piece) {
            if (piece < pieces) {
                const uint32_t buf = mine + (piece % Sh::depth) * Sh::piece;
                const int k0 = kbase + piece * kRtPiece;
#pragma unroll
                for (int it = 0; it < Sh::tok / 4; ++it) {
                    const int tok = it * 4 + (lane >> 3), k4 = lane & 7;
                    const bool in = t0 + tok < T;
                    cp_async16(buf + (tok * kRtPad + k4 * 4) * 4, x + size_t(in ? t0 + tok : 0) * n + k0 + k4 * 4, in ? 16u : 0u);
                }
#pragma unroll
                for (int i = 0; i < Sh::rows / 8; ++i)
                    cp_async16(buf + Sh::tok * kRtPad * 4 + ((wrow + 8 * i) * kRtPiece + wk) * 2, wsrc[i] + piece * kRtPiece, wbytes[i]);
            }
            cp_async_commit();
        };
        float acc[4][TJ];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < TJ; ++j) acc[i][j] = 0.0f;
#pragma unroll
        for (int i = 0; i < Sh::depth - 1; ++i) fetch(i);
        for (int piece = 0; piece < pieces; ++piece) {
            fetch(piece + Sh::depth - 1);
            cp_async_wait<Sh::depth - 1>();
            __syncwarp();
            const uint8_t* buf = smem + warp * Sh::warp + (piece % Sh::depth) * Sh::piece;
            const float* xs = reinterpret_cast<const float*>(buf);
            const uint8_t* ws = buf + Sh::tok * kRtPad * 4;
#pragma unroll
            for (int k4 = 0; k4 < kRtPiece / 4; ++k4) {
                float4 wv[4], xv[TJ];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint2 u = *reinterpret_cast<const uint2*>(ws + ((ry + RY * i) * kRtPiece + k4 * 4) * 2);
                    wv[i] = make_float4(bf16_lo(u.x), bf16_hi(u.x), bf16_lo(u.y), bf16_hi(u.y));
                }
#pragma unroll
                for (int j = 0; j < TJ; ++j) xv[j] = *reinterpret_cast<const float4*>(xs + (tx + Sh::tx * j) * kRtPad + k4 * 4);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < TJ; ++j) {
                        acc[i][j] = fmaf(wv[i].x, xv[j].x, acc[i][j]);
                        acc[i][j] = fmaf(wv[i].y, xv[j].y, acc[i][j]);
                        acc[i][j] = fmaf(wv[i].z, xv[j].z, acc[i][j]);
                        acc[i][j] = fmaf(wv[i].w, xv[j].w, acc[i][j]);
                    }
            }
            __syncwarp();   // the buffers are refilled by the next iteration
        }
        // the eight K-slices: partial tiles to shared memory (the pieces are no longer needed), then one
        // thread per (row, token) adds them in warp order
        cp_async_wait<0>();
        __syncthreads();
        float* red = reinterpret_cast<float*>(smem);   // [warp][row][token]
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < TJ; ++j) red[(warp * Sh::rows + ry + RY * i) * Sh::red + tx + Sh::tx * j] = acc[i][j];
        __syncthreads();
        for (int o = threadIdx.x; o < Sh::rows * Sh::tok; o += kRtWarps * 32) {
            const int row = o % Sh::rows, tok = o / Sh::rows, rr = r0 + row, t = t0 + tok;   // (rows of a token are neighbours in the output)
            const float* pr = red + row * Sh::red + tok;
            float sum = pr[0];
#pragma unroll
            for (int w = 1; w < kRtWarps; ++w) sum += pr[w * Sh::rows * Sh::red];
            if (t < T) {
                if (rr < E) logits[size_t(t) * E + rr] = sum;
                else if (rr < rows_total && gate_logit) gate_logit[t] = sum;
            }
        }
        __syncthreads();
    }
}

template <int RY, int TJ>
int router_tiles(int rows, int T) {
    return (rows + RtShape<RY, TJ>::rows - 1) / RtShape<RY, TJ>::rows * ((T + RtShape<RY, TJ>::tok - 1) / RtShape<RY, TJ>::tok);
}

template <int RY, int TJ>
int launch_router(const uint16_t* w_router, const uint16_t* w_gate, const float* x, int T, int E, int n, float* logits, float* gate_logit, cudaStream_t stream) {
    static std::once_flag once[64];
    int dev = 0;
    FRX_CUDA(cudaGetDevice(&dev));
    cudaError_t attr = cudaSuccess;
    if (dev >= 0 && dev < 64)
        std::call_once(once[dev], [&] {
            attr = cudaFuncSetAttribute(k_router_logits<RY, TJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, RtShape<RY, TJ>::smem);
            // two blocks per SM: without this the SM is split for one
            if (attr == cudaSuccess) attr = cudaFuncSetAttribute(k_router_logits<RY, TJ>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        });
    if (attr != cudaSuccess) return cuda_fail(attr, "frx_router_logits: cudaFuncSetAttribute");
    const int tiles = router_tiles<RY, TJ>(E + (w_gate ? 1 : 0), T);
    const int per_sm = std::max(1, (max_smem_optin() + 1024) / (RtShape<RY, TJ>::smem + 1024));
    FRX_LAUNCH(kKRoute, stream, launch_pdl(k_router_logits<RY, TJ>, dim3(unsigned(std::min(tiles, per_sm * sm_count()))), dim3(kRtWarps * 32), size_t(RtShape<RY, TJ>::smem), stream,
                                            w_router, w_gate, x, T, E, n, logits, gate_logit));
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

}  // namespace
}  // namespace frx

using namespace frx;

extern "C" int frx_router_logits(frx_stream_t stream, const void* w_router, const void* w_gate, const float* x, int T, int E, int n,
                                 float* logits, float* gate_logit) {
    if (!w_router || !x || !logits) return fail(FRX_ERR_ARG, "frx_router_logits: null pointer");
    if (w_gate && !gate_logit) return fail(FRX_ERR_ARG, "frx_router_logits: gate weights without a gate output");
    if (T < 0 || E < 1 || n < 256 || n % 256) return fail(FRX_ERR_SHAPE, "frx_router_logits: T %d, E %d, n %d (n a multiple of 256)", T, E, n);
    if ((uintptr_t(w_router) | uintptr_t(w_gate) | uintptr_t(x)) % 16) return fail(FRX_ERR_ARG, "frx_router_logits: pointers must be 16-byte aligned");
    if (T == 0) return FRX_OK;
    const auto* wr = static_cast<const uint16_t*>(w_router);
    const auto* wg = static_cast<const uint16_t*>(w_gate);
    const int rows = E + (w_gate ? 1 : 0), sms = sm_count();
    // few tokens: small tiles, as long as no SM gets a second one
    if (router_tiles<2, 1>(rows, T) <= sms) return launch_router<2, 1>(wr, wg, x, T, E, n, logits, gate_logit, stream);
    // up to eight rows leave half of a tile of 16 empty: eight rows x 64 tokens (8 experts, 16,384 tokens of 1024: 27.3 us in tiles of
    // 16 rows, 16.7 so; 4,096 tokens of 256: 3.8 and 3.6)
    if (rows <= 8) return launch_router<2, 4>(wr, wg, x, T, E, n, logits, gate_logit, stream);
    // else the tile for which the busiest SM finishes first: one of 16 rows costs about TJ + 1 (measured at 37 to 1024 tokens), one of
    // 8 x 64 about 6.5; the latter comes out ahead at 17 to 24 rows (16 experts and the gate, 6,000 tokens of 1024: 17.9 us in tiles
    // of 16 rows, 16.7 so)
    auto cost = [&](int tiles, int each) { return (tiles + sms - 1) / sms * each; };
    const int c2 = cost(router_tiles<4, 2>(rows, T), 6), c3 = cost(router_tiles<4, 3>(rows, T), 8), c5 = cost(router_tiles<4, 5>(rows, T), 12);
    if (cost(router_tiles<2, 4>(rows, T), 13) < std::min({c2, c3, c5})) return launch_router<2, 4>(wr, wg, x, T, E, n, logits, gate_logit, stream);
    if (c2 <= c3 && c2 <= c5) return launch_router<4, 2>(wr, wg, x, T, E, n, logits, gate_logit, stream);
    if (c3 <= c5) return launch_router<4, 3>(wr, wg, x, T, E, n, logits, gate_logit, stream);
    return launch_router<4, 5>(wr, wg, x, T, E, n, logits, gate_logit, stream);
}
