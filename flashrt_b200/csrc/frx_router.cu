// Router projection in front of the router: logits[t][e] = sum_k W[e][k] * x[t][k], with W in bf16
// and x, the products and the sums in fp32, and in the same launch the shared expert's gate logit
// (one more bf16 row). The reference computes both with one launch of k_bf16_multi
// (arch/qwen4exp/blocks.cu:83-120, called at moe_fast.cu:1039-1042 and moe_stream.cu:145-149): exact
// bf16 x fp32 products, fp32 accumulation, no activation on these two outputs. The order of the
// additions differs from the reference's (and from one GPU generation's launch shape to another in
// the reference itself), so parity is to a tolerance, against a float64 sum.
//
// The products run on the tensor cores without losing a bit: an fp32 value is the sum of three bf16 values of eight significant
// bits each (cut off, not rounded; multiply_add below has the exceptions), so W x = W hi + W mid + W lo, every product exact in fp32.
// Three chained MMAs of 16 K start at zero and their result is added to a running fp32 sum: exact products, and four sums per 16 K that may
// round (an MMA in a way that PTX leaves open). Relative error against float64, 2-norm: 1.1e-7 for 2560 terms, 3.2e-7 with 320 multiply-adds
// in a row.
//
// A block works on a tile of 16 MT rows x 8 NT tokens; each of its 8 warps takes an eighth of K and walks it 32 at a time, straight from
// global memory into the MMA's registers: a lane takes eight neighbouring K of a row (one 16-byte load) and of a token (two), which is
// another order of K inside the 32, the same for both operands. At the end the eight partial tiles are added in warp order
// (fixed, so results are reproducible and do not depend on the tile).
// Bound: the latency of a step (a load from the L2, the split, chains of three MMAs) with two pieces in flight, and for many tokens what the
// L2 delivers (all blocks together read x once per row tile and W once per token tile: 63 MB at 293 tokens in tiles of 48 x 32, 200 MB in
// tiles of 16 x 8). 513 rows of 2560, us, against multiply-adds from shared memory: 1 token 6.1 -> 3.7, 37 tokens 9.1 -> 5.2, 293 tokens
// 29.3 -> 15.8, 1024 tokens 87.5 -> 39.3.
#include "frx_common.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace frx {
namespace {

constexpr int kRtWarps = 8, kRtPiece = 32;

// D = A * B + D, bf16 operands, fp32 sums
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The three bf16 pieces of two values, packed. (What is left of an infinity is no number: see multiply_add.) `over` collects
// the bits of the last remainders, whose lower halves are what the third piece has no place for.
__device__ __forceinline__ void split_pair(float a, float b, uint32_t (&p)[3], uint32_t& over) {
    const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    p[0] = __byte_perm(ua, ub, 0x7632);
    const float ra = a - __uint_as_float(ua & 0xffff0000u), rb = b - __uint_as_float(ub & 0xffff0000u);
    const uint32_t va = __float_as_uint(ra), vb = __float_as_uint(rb);
    p[1] = __byte_perm(va, vb, 0x7632);
    const uint32_t la = __float_as_uint(ra - __uint_as_float(va & 0xffff0000u)), lb = __float_as_uint(rb - __uint_as_float(vb & 0xffff0000u));
    p[2] = __byte_perm(la, lb, 0x7632);
    over |= la | lb;
}

// Which lanes of a warp have an activation, of their token t and their part of K, with bits that three pieces do not hold (four lanes a token).
__device__ __noinline__ uint32_t has_rest(const float* x, int t, int n) {
    uint32_t over = 0, p[3];
    const float* xt = x + size_t(t) * n + (threadIdx.x >> 5) * (n / kRtWarps) + (threadIdx.x & 3) * 8;
    for (int k = 0; k < n / kRtWarps; k += kRtPiece)
        for (int h = 0; h < 2; ++h) {
            const float4 v = *reinterpret_cast<const float4*>(xt + k + 4 * h);
            split_pair(v.x, v.y, p, over);
            split_pair(v.z, v.w, p, over);
        }
    return __ballot_sync(0xffffffffu, over & 0xffffu);
}

// One logit by fp32 multiply-adds in order, the eight slices of K each for itself and then one after the other, for what three bf16
// pieces cannot do. A sum that is not finite: an infinite weight times a piece that is zero is no number, where a multiply-add gives the
// infinity, and 16 products together may leave the range of floats where one after the other does not. And a token with an activation
// below 2^-110 whose third piece would need bits below 2^-133, bf16's smallest number. (Four slices side by side, and wide loads:
// what takes the time is that every lane of a warp reads a row of its own. 300 tokens x 513 rows of 2560: 22 us more for one token
// with an infinity, 80 for infinite weights in two rows, 330 if no logit is finite.)
__device__ __noinline__ float multiply_add(const uint16_t* w, const float* x, int n) {
    const int slice = n / kRtWarps;
    float sum = 0.0f;
    for (int s0 = 0; s0 < kRtWarps; s0 += 4) {
        float acc[4] = {};
        for (int k = 0; k < slice; k += 8) {
            uint4 u[4];
            float4 v[4][2];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                u[s] = __ldg(reinterpret_cast<const uint4*>(w + size_t(s0 + s) * slice + k));
                v[s][0] = *reinterpret_cast<const float4*>(x + size_t(s0 + s) * slice + k);
                v[s][1] = *reinterpret_cast<const float4*>(x + size_t(s0 + s) * slice + k + 4);
            }
            auto four = [](float& a, uint32_t lo, uint32_t hi, const float4& v) {
                a = fmaf(__uint_as_float(lo << 16), v.x, a);
                a = fmaf(__uint_as_float(lo & 0xffff0000u), v.y, a);
                a = fmaf(__uint_as_float(hi << 16), v.z, a);
                a = fmaf(__uint_as_float(hi & 0xffff0000u), v.w, a);
            };
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                four(acc[s], u[s].x, u[s].y, v[s][0]);
                four(acc[s], u[s].z, u[s].w, v[s][1]);
            }
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) sum = s0 + s ? sum + acc[s] : acc[s];
    }
    return sum;
}

// rows: E router rows followed by the gate row when w_gate is given (row E). W rows are n bf16 each.
// x is not __restrict__: the kernel in front may write it while this one is already running, so that its loads must neither move
// across pdl_wait() nor take the path for data that no one writes. (513 rows of 2560, 37 / 293 / 1024 tokens: 5.32 / 16.7 / 40.2 us
// with and without; past the L1, ld.global.cg, 5.23 / 16.7 / 40.7, at 512 columns and 8,192 tokens up to 10 % slower.)
template <int MT, int NT>
__global__ void __launch_bounds__(kRtWarps * 32, MT * NT <= 4 ? 2 : 1) k_router_logits(const uint16_t* __restrict__ w_router, const uint16_t* __restrict__ w_gate,
                                                                  const float* x, int T, int E, int n,
                                                                  float* __restrict__ logits, float* __restrict__ gate_logit) {
    // Partial sums are kept per token: [token][row]. With rows of 4 more than a multiple of 16, the four tokens x eight rows that a warp
    // stores at a time fall into 32 banks (odd rows put up to four in one; 513 rows of 512, 293 tokens 5.7 -> 5.2 us, 8,192
    // tokens 97 -> 91; of 2560 16.6 -> 16.5).
    constexpr int kRows = 16 * MT, kTok = 8 * NT, kRed = kRows + 4;
    extern __shared__ float red[];   // [warp][token][row]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int rows_total = E + (w_gate ? 1 : 0), row_tiles = (rows_total + kRows - 1) / kRows;
    const int r0 = int(blockIdx.x) % row_tiles * kRows, t0 = int(blockIdx.x) / row_tiles * kTok;
    const int steps = n / (kRtWarps * kRtPiece);
    const size_t k0 = size_t(warp) * steps * kRtPiece + t4 * 8;
    const uint16_t* wp[MT][2];   // rows beyond the last repeat it, tokens likewise; neither is stored
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = min(r0 + 16 * i + 8 * h + g, rows_total - 1);
            wp[i][h] = (r < E ? w_router + size_t(r) * n : w_gate) + k0;
        }
    const float* xp[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) xp[j] = x + size_t(min(t0 + 8 * j + g, T - 1)) * n + k0;
    struct Piece {
        uint4 w[MT][2];
        float4 x[NT][2];
    };
    auto load = [&](Piece& p, int s) {
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) p.w[i][h] = __ldg(reinterpret_cast<const uint4*>(wp[i][h] + s * kRtPiece));
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) p.x[j][h] = *(reinterpret_cast<const float4*>(xp[j] + s * kRtPiece) + h);
    };
    uint32_t over = 0;
    float acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.0f;
    auto multiply = [&](const Piece& p) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {   // the first and the second four of a lane's eight K
            uint32_t b[NT][2][3];
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                split_pair(p.x[j][h].x, p.x[j][h].y, b[j][0], over);
                split_pair(p.x[j][h].z, p.x[j][h].w, b[j][1], over);
            }
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const uint32_t a0 = h ? p.w[i][0].z : p.w[i][0].x, a2 = h ? p.w[i][0].w : p.w[i][0].y, a1 = h ? p.w[i][1].z : p.w[i][1].x, a3 = h ? p.w[i][1].w : p.w[i][1].y;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int k = 2; k >= 0; --k) mma_bf16(d, a0, a1, a2, a3, b[j][0][k], b[j][1][k]);   // the smallest first
#pragma unroll
                    for (int k = 0; k < 4; ++k) acc[i][j][k] += d[k];
                }
            }
        }
    };
    // W is a weight: its first piece may come in before the kernels in front have ended
    Piece p[2];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) touch_l2(wp[i][h]);
    pdl_wait();
    pdl_trigger();
    load(p[0], 0);
    for (int s = 0; s < steps; s += 2) {
        if (s + 1 < steps) load(p[1], s + 1);
        multiply(p[0]);
        if (s + 2 < steps) load(p[0], s + 2);
        if (s + 1 < steps) multiply(p[1]);
    }
    // the eight slices of K: partial tiles to shared memory, then a thread per (row, token) adds them in warp order
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) red[(warp * kTok + 8 * j + 2 * t4 + (k & 1)) * kRed + 16 * i + 8 * (k >> 1) + g] = acc[i][j][k];
    // Tokens with an activation that three pieces do not hold get no number, for multiply_add below. (One collector a lane for all of its
    // tokens, and which of them it was is found out here: a collector for each cost registers and spilled in the tiles of 32 tokens, 513
    // rows of 2560: 293 tokens 16.5 us against 15.8, 1024 tokens 40.0 against 39.3.)
    if (__any_sync(0xffffffffu, over & 0xffffu)) {
#pragma unroll 1
        for (int j = 0; j < NT; ++j) {
            const uint32_t lanes = has_rest(x, min(t0 + 8 * j + g, T - 1), n);
            __syncwarp();
            for (int c = 0; c < 8; ++c)
                if (lanes >> 4 * c & 15u)
                    for (int row = lane; row < kRows; row += 32) red[(warp * kTok + 8 * j + c) * kRed + row] = NAN;
        }
    }
    __syncthreads();
    for (int o = threadIdx.x; o < kRows * kTok; o += kRtWarps * 32) {
        const int row = o % kRows, tok = o / kRows, rr = r0 + row, t = t0 + tok;   // (rows of a token are neighbours in the output)
        const float* pr = red + tok * kRed + row;
        float sum = pr[0];
#pragma unroll
        for (int w = 1; w < kRtWarps; ++w) sum += pr[w * kTok * kRed];
        if (t < T && rr < rows_total) {
            if (!(fabsf(sum) < INFINITY)) sum = multiply_add(rr < E ? w_router + size_t(rr) * n : w_gate, x + size_t(t) * n, n);
            if (rr < E) logits[size_t(t) * E + rr] = sum;
            else gate_logit[t] = sum;
        }
    }
}

template <int MT, int NT>
constexpr int router_smem() { return kRtWarps * 8 * NT * (16 * MT + 4) * 4; }
template <int MT, int NT>
long long router_tiles(long long rows, long long T) {
    return (rows + 16 * MT - 1) / (16 * MT) * ((T + 8 * NT - 1) / (8 * NT));
}

template <int MT, int NT>
int launch_router(const uint16_t* w_router, const uint16_t* w_gate, const float* x, int T, int E, int n, float* logits, float* gate_logit, cudaStream_t stream) {
    const long long tiles = router_tiles<MT, NT>(E + (w_gate ? 1 : 0), T);
    if (tiles > 0x7fffffffLL) return fail(FRX_ERR_SHAPE, "frx_router_logits: %d rows x %d tokens", E, T);
    if constexpr (router_smem<MT, NT>() > 48 * 1024) {
        static std::once_flag once[64];
        int dev = 0;
        FRX_CUDA(cudaGetDevice(&dev));
        cudaError_t attr = cudaSuccess;
        if (dev >= 0 && dev < 64) std::call_once(once[dev], [&] { attr = cudaFuncSetAttribute(k_router_logits<MT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, router_smem<MT, NT>()); });
        if (attr != cudaSuccess) return cuda_fail(attr, "frx_router_logits: cudaFuncSetAttribute");
    }
    FRX_LAUNCH(kKRoute, stream, launch_pdl(k_router_logits<MT, NT>, dim3(unsigned(tiles)), dim3(kRtWarps * 32), size_t(router_smem<MT, NT>()), stream, w_router, w_gate, x, T, E, n, logits, gate_logit));
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

// The tile for `rows` rows (the gate's among them), as 10 MT + NT.
int router_tile(int rows, int T, int n, int sm_number) {
    // The tile by an estimate in microseconds for every one: steps of K, and waves of a tile per SM (two of the two small ones share an SM,
    // which their figures contain). Fitted to 128, 256 and 512 rows of 512, 2048 and 2560 at 1 to 1024 tokens. Of 932 points with 8 to
    // 2048 rows of 256 to 7168 and 1 to 8192 tokens the one that it picks is 0.9 % slower than the best on average and 14 % at most.
    const double s = n / (kRtWarps * kRtPiece), sms = std::max(sm_number, 1);
    auto waves = [&](long long tiles) { return std::ceil(double(tiles) / sms); };
    const double c11 = 0.5 + 0.08 * s + (0.37 + 0.22 * s) * waves(router_tiles<1, 1>(rows, T)), c22 = 0.82 + 0.14 * s + (0.61 + 0.47 * s) * waves(router_tiles<2, 2>(rows, T)),
                 c32 = (1.8 + 0.73 * s) * waves(router_tiles<3, 2>(rows, T)), c34 = (2.7 + 1.3 * s) * waves(router_tiles<3, 4>(rows, T));
    // up to 16 rows have no second row tile to share the tokens with: long tiles once there are many (7 rows and the gate, 16,384 tokens of 256:
    // 12.2 us in tiles of 16 x 8, 7.0 so; 9,000 tokens of 2560: 19.8)
    if (rows <= 16 && router_tiles<1, 1>(rows, T) > 2 * sms) return 14;
    const double least = std::min({c11, c22, c32, c34});
    return least == c11 ? 11 : least == c22 ? 22 : least == c32 ? 32 : 34;
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
    switch (router_tile(E + (w_gate ? 1 : 0), T, n, sm_count())) {
        case 11: return launch_router<1, 1>(wr, wg, x, T, E, n, logits, gate_logit, stream);
        case 14: return launch_router<1, 4>(wr, wg, x, T, E, n, logits, gate_logit, stream);
        case 22: return launch_router<2, 2>(wr, wg, x, T, E, n, logits, gate_logit, stream);
        case 32: return launch_router<3, 2>(wr, wg, x, T, E, n, logits, gate_logit, stream);
        default: return launch_router<3, 4>(wr, wg, x, T, E, n, logits, gate_logit, stream);
    }
}

extern "C" int frx_router_logits_tile(int T, int rows, int n, int sms) {
    if (T < 1 || rows < 1 || n < 256 || n % 256 || sms < 0) return 0;
    const int tile = router_tile(rows, T, n, sms ? sms : sm_count());
    return tile / 10 * 16 * 100 + tile % 10 * 8;
}
