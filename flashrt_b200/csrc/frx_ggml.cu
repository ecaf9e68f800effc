// ggml-layout entry points of the Q2_0 expert path: the reference's gemv:: and gemm:: functions
// (kernels/cuda/ggml_gemv.h:26-65, kernels/cuda/ggml_gemm.h:27-68) for ggml type 42, as the draft
// head's MoE calls them (arch/qwen4exp/mtp.cu:631-670), and the head's Q8_0 -> Q2_0 requantizer
// (arch/qwen4exp/mtp.cu:129-215) on the device.
//
// Weights stay in ggml's own layout here: rows of 18-byte blocks {fp16 d; 16 code bytes, element j
// in byte j / 4 at bit 2 * (j % 4)}, experts back to back. Activations are ggml's Q8_1 blocks
// {fp16 d; fp16 sum; 32 int8}, rows padded to 512 values. The arithmetic is ggml's
// (third_party/ggml/src/ggml-cuda/vecdotq.cuh:728-771): per 32-value chunk an exact integer sum
// of (q - 1) * a, scaled as d2 * d8 * sumi in float; chunks are added in float.
//
// One kernel serves the gemv entries. A block takes one job (an expert and an activation row) and a
// run of weight rows. The rows are contiguous in memory, so a tile of them is staged
// in shared memory by one 1-D bulk (TMA) copy; a lane owns a pair of neighbouring blocks (36 bytes,
// nine conflict-free 32-bit shared-memory loads) and the activations are kept in shared memory
// transposed so that crumb p of a weight word lines up with one int8x4 word: 16 dp4a per block and
// token, no table look-ups.
#include "frx_common.cuh"

#include <mutex>

namespace frx {
namespace {

#include "frx_group.cuh"

constexpr uint32_t kTypeQ2_0 = 42;   // core/formats.hpp:11-18
constexpr int kQ81Bytes = 36;        // block_q8_1 (third_party/ggml/src/ggml-common.h:256-268)
constexpr int kRowPad = 512;         // MATRIX_ROW_PADDING (third_party/ggml/src/ggml-cuda/common.cuh:186)
constexpr int kDotThreads = 256, kDotWarps = 8;

inline int64_t padded_cols(int64_t ncols) { return (ncols + kRowPad - 1) / kRowPad * kRowPad; }
inline size_t act_row_bytes(int64_t ncols) { return size_t(padded_cols(ncols) / kQ8) * kQ81Bytes; }

// ---- Q8_1 quantizer (third_party/ggml/src/ggml-cuda/quantize.cu:54-101): per 32 values
// d = amax / 127, q = amax == 0 ? 0 : roundf(x / d); the block keeps half(d), half(sum of the inputs).
// With `u`, the input is silu(g) * u first (gemv::swiglu_q8_1, kernels/cuda/ggml_gemv.cu:98-107,
// which uses the fast exponential).
// `early` lets the next kernel's blocks in at once: see launch_q8_1.
__global__ void __launch_bounds__(256) k_q8_1(const float* __restrict__ x, const float* __restrict__ u, int64_t ncols, int64_t padded,
                                              uint8_t* __restrict__ y, int early) {
    pdl_wait();
    if (early) pdl_trigger();
    const int64_t i0 = int64_t(blockDim.x) * blockIdx.x + threadIdx.x, t = blockIdx.y;
    if (i0 >= padded) return;   // padded is a multiple of the block
    float xi = 0.0f;
    if (i0 < ncols) {
        xi = x[t * ncols + i0];
        if (u) xi = __fmul_rn(__fdiv_rn(xi, __fadd_rn(1.0f, __expf(-xi))), u[t * ncols + i0]);
    }
    float amax = fabsf(xi), sum = xi;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
    }
    const float d = __fdiv_rn(amax, 127.0f);
    uint8_t* blk = y + (t * (padded / kQ8) + i0 / kQ8) * kQ81Bytes;
    const int iqs = int(i0 % kQ8);
    blk[4 + iqs] = uint8_t(int8_t(amax == 0.0f ? 0 : int(round_half_away(__fdiv_rn(xi, d)))));
    if (iqs == 0) *reinterpret_cast<__half2*>(blk) = __halves2half2(__float2half_rn(d), __float2half_rn(sum));
}

// ---- the dot-product kernel
struct DotArgs {
    const uint8_t* w;          // expert e's matrix at w + e * expert_stride
    const uint8_t* gate;       // fused SwiGLU: the gate matrix, same strides (or null)
    size_t expert_stride;
    const uint8_t* xq;         // Q8_1 rows
    size_t act_row;            // bytes per activation row
    float* dst;                // [rows of slots][nrows]
    int ncols, nrows;
    int rows_per_tile;         // weight rows staged per step
    int tma;                   // 1: tiles are fetched by bulk copies (alignment checked on the host)
    unsigned long long wait_ns;
    // job j has expert ids[j] (0 without ids), activation row j / act_div, output row j
    const int32_t* ids;
    int act_div;
};

struct DotSmem {
    uint32_t at, d8, sa, w, bar, abort, total;
};
__host__ __device__ inline DotSmem dot_smem(int ncols, int tile_bytes, bool gate) {
    DotSmem s{};
    const uint32_t nch = uint32_t(ncols / kQ8);
    uint32_t off = 0;
    s.at = off;
    off += uint32_t(ncols);
    s.d8 = off;
    off += nch * 4;
    s.sa = off;
    off += nch * 4;
    off = (off + 127u) & ~127u;
    s.w = off;
    off += uint32_t(tile_bytes) * (gate ? 2u : 1u);
    off = (off + 15u) & ~15u;
    s.bar = off;
    off += 16;
    s.abort = off;
    off += 16;
    s.total = off;
    return s;
}

// One pair of neighbouring blocks (36 bytes at a 4-byte boundary) from shared memory: the two
// scales and the eight code words.
__device__ __forceinline__ void load_pair(const uint8_t* p, float& d0, float& d1, uint32_t (&c)[8]) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p);
    uint32_t v[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) v[i] = q[i];
    d0 = __half2float(__ushort_as_half(uint16_t(v[0] & 0xffffu)));
    d1 = __half2float(__ushort_as_half(uint16_t(v[4] >> 16)));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        c[i] = __funnelshift_r(v[i], v[i + 1], 16);   // bytes 2 + 4 i .. 5 + 4 i
        c[4 + i] = v[5 + i];                          // bytes 20 + 4 i ..
    }
}

// sum over the 32 values of one chunk of (q - 1) * a: two code words against eight transposed
// activation words, minus the sum of the activation codes
__device__ __forceinline__ int chunk_sum(uint32_t w0, uint32_t w1, const uint4& a0, const uint4& a1, int suma) {
    constexpr uint32_t M = 0x03030303u;
    int s = 0;
    s = __dp4a(int(w0 & M), int(a0.x), s);
    s = __dp4a(int((w0 >> 2) & M), int(a0.y), s);
    s = __dp4a(int((w0 >> 4) & M), int(a0.z), s);
    s = __dp4a(int((w0 >> 6) & M), int(a0.w), s);
    s = __dp4a(int(w1 & M), int(a1.x), s);
    s = __dp4a(int((w1 >> 2) & M), int(a1.y), s);
    s = __dp4a(int((w1 >> 4) & M), int(a1.z), s);
    s = __dp4a(int((w1 >> 6) & M), int(a1.w), s);
    return s - suma;
}

// Bound with one token (eight jobs): latency, of the chain ids -> weights -> product; so a block asks for its first tile as
// soon as it knows its expert and prepares the activations meanwhile, and its launch overlaps the kernel in front. One
// token through 8 experts of 2560 x 640 (routing, two quantizations, two products, combine): 43.5 -> 31 us.
template <bool GATE>
__global__ void __launch_bounds__(kDotThreads) k_ggml_dot(const DotArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int nb = a.ncols / kQK, np = nb / 2, nch = a.ncols / kQ8;
    const uint32_t row_bytes = uint32_t(nb) * kBlockBytes;
    const uint32_t tile_bytes = uint32_t(a.rows_per_tile) * row_bytes;
    const DotSmem sm = dot_smem(a.ncols, int(tile_bytes), GATE);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + sm.bar);
    volatile int* abort = reinterpret_cast<volatile int*>(smem + sm.abort);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        mbar_init(bar, 1);
        *abort = 0;
        mbar_fence_init();
    }
    pdl_wait();
    const int job = blockIdx.x, e = a.ids ? a.ids[job] : 0;
    const uint8_t* wsrc = a.w + size_t(e) * a.expert_stride;
    const uint8_t* gsrc = GATE ? a.gate + size_t(e) * a.expert_stride : nullptr;
    uint8_t* wt = smem + sm.w;
    uint8_t* gt = wt + tile_bytes;
    const int n_tiles = (a.nrows + a.rows_per_tile - 1) / a.rows_per_tile;
    auto by_tma = [&](int tile) { return a.tma && (tile + 1) * a.rows_per_tile <= a.nrows; };
    auto fetch = [&](int tile) {   // thread 0: a whole tile by bulk copies
        const size_t at = size_t(tile) * tile_bytes;
        mbar_expect_tx(bar, tile_bytes * (GATE ? 2u : 1u));
        bulk_g2s(wt, wsrc + at, tile_bytes, bar);
        if (GATE) bulk_g2s(gt, gsrc + at, tile_bytes, bar);
    };
    if (tid == 0 && by_tma(blockIdx.y)) fetch(blockIdx.y);

    // ---- activations: codes transposed per 16 values (word p of a group = values p, 4 + p, 8 + p,
    // 12 + p), chunk scales, chunk code sums
    uint32_t* at = reinterpret_cast<uint32_t*>(smem + sm.at);
    float* d8 = reinterpret_cast<float*>(smem + sm.d8);
    int* sa = reinterpret_cast<int*>(smem + sm.sa);
    const uint8_t* act = a.xq + size_t(job / a.act_div) * a.act_row;
    for (int c = tid; c < nch; c += kDotThreads) {
        const uint32_t* blk = reinterpret_cast<const uint32_t*>(act + size_t(c) * kQ81Bytes);
        uint32_t v[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) v[i] = blk[i];
        d8[c] = __half2float(__ushort_as_half(uint16_t(v[0] & 0xffffu)));
        int s = 0;
#pragma unroll
        for (int i = 1; i < 9; ++i) s = __dp4a(int(v[i]), 0x01010101, s);
        sa[c] = s;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t u0 = v[1 + 4 * h], u1 = v[2 + 4 * h], u2 = v[3 + 4 * h], u3 = v[4 + 4 * h];
            const uint32_t lo01 = __byte_perm(u0, u1, 0x5140), hi01 = __byte_perm(u0, u1, 0x7362);
            const uint32_t lo23 = __byte_perm(u2, u3, 0x5140), hi23 = __byte_perm(u2, u3, 0x7362);
            uint4 o;
            o.x = __byte_perm(lo01, lo23, 0x5410);
            o.y = __byte_perm(lo01, lo23, 0x7632);
            o.z = __byte_perm(hi01, hi23, 0x5410);
            o.w = __byte_perm(hi01, hi23, 0x7632);
            reinterpret_cast<uint4*>(at)[c * 2 + h] = o;
        }
    }
    __syncthreads();

    // ---- lanes: a lane owns block pairs lane_p, lane_p + stride, ... of row lane_row of a pass
    const int rpp = (np < 32 && 32 % np == 0) ? 32 / np : 1;   // rows per pass of a warp
    const int width = 32 / rpp;                                // lanes per row
    const int lane_row = lane / width, lane_p = lane % width;
    uint32_t phase = 0;
    for (int tile = blockIdx.y; tile < n_tiles; tile += gridDim.y) {
        const int r0 = tile * a.rows_per_tile, rows = min(a.rows_per_tile, a.nrows - r0);
        if (by_tma(tile)) {
            if (tile != int(blockIdx.y)) {
                __syncthreads();   // everyone is done with the previous tile
                if (tid == 0) fetch(tile);
            }
            mbar_wait_bounded(bar, phase, abort, a.wait_ns);
            phase ^= 1u;
        } else {
            const uint32_t bytes = uint32_t(rows) * row_bytes;
            __syncthreads();
            const uint32_t* s0 = reinterpret_cast<const uint32_t*>(wsrc + size_t(r0) * row_bytes);
            for (uint32_t i = tid; i < bytes / 4; i += kDotThreads) reinterpret_cast<uint32_t*>(wt)[i] = s0[i];
            if (GATE) {
                const uint32_t* s1 = reinterpret_cast<const uint32_t*>(gsrc + size_t(r0) * row_bytes);
                for (uint32_t i = tid; i < bytes / 4; i += kDotThreads) reinterpret_cast<uint32_t*>(gt)[i] = s1[i];
            }
            __syncthreads();
        }
        for (int rb = warp * rpp; rb < rows; rb += kDotWarps * rpp) {   // uniform for the warp: the sums below are shuffled
            const int rr = rb + lane_row;
            const bool live = rr < rows;
            float v = 0.0f, g = 0.0f;
            for (int pi = lane_p; live && pi < np; pi += width) {
                float d0, d1, g0 = 0.0f, g1 = 0.0f;
                uint32_t c[8], gc[8];
                load_pair(wt + size_t(rr) * row_bytes + size_t(pi) * 36, d0, d1, c);
                if (GATE) load_pair(gt + size_t(rr) * row_bytes + size_t(pi) * 36, g0, g1, gc);
                const uint4* aj = reinterpret_cast<const uint4*>(at) + pi * 8;
#pragma unroll
                for (int q = 0; q < 4; ++q) {   // the four chunks of the pair
                    const uint4 a0 = aj[2 * q], a1 = aj[2 * q + 1];
                    const float dx = d8[pi * 4 + q];
                    const int sx = sa[pi * 4 + q];
                    v = __fadd_rn(v, __fmul_rn(__fmul_rn(q < 2 ? d0 : d1, dx), float(chunk_sum(c[2 * q], c[2 * q + 1], a0, a1, sx))));   // d2 * d8 * sumi
                    if (GATE) g = __fadd_rn(g, __fmul_rn(__fmul_rn(q < 2 ? g0 : g1, dx), float(chunk_sum(gc[2 * q], gc[2 * q + 1], a0, a1, sx))));
                }
            }
            for (int o = width >> 1; o > 0; o >>= 1) {
                v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
                if (GATE) g = __fadd_rn(g, __shfl_xor_sync(0xffffffffu, g, o));
            }
            if (lane_p == 0 && live) {
                if (GATE) v = __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), v);   // ggml unary.cuh:98-100
                a.dst[size_t(job) * a.nrows + r0 + rr] = v;
            }
        }
    }
    // The next kernel is let in as a block ends, not as it starts: blocks of it that wait beside this kernel's would share the SMs'
    // slots unevenly (eight jobs of 4096 x 1024, 512 blocks: 17.6 us let in at the start, 12.8 at the end; one job 5.1, 5.0).
    pdl_trigger();
}

int dot_tile_rows(int ncols) {
    const int np = ncols / 128;
    const int rpp = (np < 32 && 32 % np == 0) ? 32 / np : 1;
    return kDotWarps * rpp * 2;   // two passes of every warp per tile: 18 KB of weights at the usual shapes
}

template <bool GATE>
int launch_dot(DotArgs a, int grid_x, cudaStream_t stream) {
    a.rows_per_tile = dot_tile_rows(a.ncols);
    const uint32_t row_bytes = uint32_t(a.ncols / kQK) * kBlockBytes, tile_bytes = uint32_t(a.rows_per_tile) * row_bytes;
    a.tma = ((uintptr_t(a.w) | uintptr_t(a.gate) | a.expert_stride | tile_bytes) % 16 == 0) ? 1 : 0;
    a.wait_ns = wait_limit_ns();
    const DotSmem sm = dot_smem(a.ncols, int(tile_bytes), GATE);
    if (int(sm.total) > max_smem_optin() - 1024) return fail(FRX_ERR_SHAPE, "ggml-layout product: ncols %d needs %u bytes of shared memory", a.ncols, sm.total);
    static std::mutex mu;
    static bool set[64] = {};
    int dev = 0;
    FRX_CUDA(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lk(mu);
        if (dev >= 0 && dev < 64 && !set[dev]) {
            FRX_CUDA(cudaFuncSetAttribute(k_ggml_dot<GATE>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem_optin() - 1024));
            // The quantizer in front asks for the same split of the SM, though it uses no shared memory: an SM that runs it could not
            // change its split, and this kernel's early blocks would crowd on the others (4 tokens x 4096 x 1024 with their
            // quantization: 14.1 us, 9.0 so).
            FRX_CUDA(cudaFuncSetAttribute(k_ggml_dot<GATE>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
            FRX_CUDA(cudaFuncSetAttribute(k_q8_1, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
            set[dev] = true;
        }
    }
    const int n_tiles = (a.nrows + a.rows_per_tile - 1) / a.rows_per_tile;
    // enough blocks to fill the GPU, each walking several tiles so the activation set-up is amortised
    const int sms = sm_count() > 0 ? sm_count() : 148;
    int gy = n_tiles;
    while (gy > 1 && (long long)grid_x * gy > 8LL * sms && gy % 2 == 0) gy /= 2;
    FRX_CUDA(launch_pdl(k_ggml_dot<GATE>, dim3(unsigned(grid_x), unsigned(gy)), dim3(kDotThreads), sm.total, stream, a));
    return FRX_OK;
}

int check_dot_shape(const char* who, uint32_t type, int64_t ncols, int64_t nrows) {
    if (type != kTypeQ2_0) return fail(FRX_ERR_SHAPE, "%s: ggml type %u is not built (only Q2_0, type 42)", who, type);
    if (ncols < 128 || ncols % 128 || ncols > 16384 || nrows < 1 || nrows > (1 << 24))
        return fail(FRX_ERR_SHAPE, "%s: ncols %lld must be a multiple of 128 (at most 16384), nrows %lld positive", who, (long long)ncols,
                    (long long)nrows);
    return FRX_OK;
}

// ---- Q8_0 -> Q2_0 (arch/qwen4exp/mtp.cu:129-201): a thread per 64 values. Of 24 candidate scales d the reference takes the
// first with the smallest sum of (x - q d)^2, added in fp32 in index order, q = x / d rounded and clamped to [-1, 2].
//
// The sums are not formed candidate by candidate. With S1 = sum(q x) and S2 = sum(q^2) a sum is X2 - d (2 S1 - d S2), and
// q changes only where |x| passes 0.5 d or x passes 1.5 d: a value adds |x| to S1 and 1 to S2 for every candidate with
// 0.5 d <= |x|, and again |x| and 3 for every one with 1.5 d <= x. The candidates grow with their index, so each
// value goes into at most two of 25 bins (how many candidates it has passed) of the thread's own column in shared
// memory, and 24 suffix sums give S1 and S2 of all candidates, exactly: a bin is a float that counts passes in
// units of 16384 above a sum of 8-bit magnitudes (both below 2^24 together), one half of the block at a time.
// The bin follows from amax / |x|, good to 0.02 of a bin (the candidates are rounded to fp16: 2^-11 of 2.5 * 46 / 3 bins) and
// settled by one exact comparison with the candidate it may just have missed.
// What rounding remains (6 * 2^-24 X2 here: S1 rounds once, 2 S1 <= 4 X2 / d, then twice more; 66 * 2^-24 of the sum in the
// reference's order) decides nothing: candidates closer to the best than twice that are summed again in the reference's
// order and compared as it does.
// Blocks whose candidates are not all normal fp16 numbers are summed so for all 24.
//
// In that sum a division is not needed: the values are d8 * q8 (exact, at most 18 significant bits), a candidate is an
// fp16 value (11 bits): if x / d is not exactly on a rounding boundary (-0.5, 0.5, 1.5) it is at least 2^-18 of itself
// away from it, so a quotient good to 2^-22 gives the reference's code; on a boundary either neighbour leaves the same
// |x - q d|, and only its square is used. The quotient is taken as sat((x / d + 1) / 3) * 3, which clamps it to
// [-1, 2] in the same instruction, rounded by a magic addition; x - q d rounds once in a fused multiply-add because q d
// is exact. The codes of the chosen scale come from the same quotient enlarged by 2^-20, which takes it past a boundary
// it lies on and past none that it does not.
// Bound: issue slots, about 63 per value (six per value and candidate when each candidate was summed). 48 experts of
// 2560 x 640 (236 M values): 1.35 ms with a sum per candidate, 0.51 ms so (0.62 with candidates divided one by one, wider bounds
// and everything unrolled, which the instruction cache did not hold).
constexpr int kRqThreads = 128, kRqCand = 24;
constexpr float kRqCount = 16384.0f;   // a pass in a bin; the magnitudes of 32 values, twice each, stay below 8192
constexpr uint32_t kRqRow = kRqThreads * 4, kRqToBin = kRqCand * kRqRow;
// candidate c is amax / div, div = 2.5f - 1.5f * float(c) / 23.0f, through fp16; and the correctly rounded 1 / div
struct RqDiv {
    float div[kRqCand], inv[kRqCand];
    constexpr RqDiv() : div(), inv() {
        for (int c = 0; c < kRqCand; ++c) {
            div[c] = 2.5f - 1.5f * float(c) / 23.0f;
            inv[c] = float(1.0 / double(div[c]));
        }
    }
};
__constant__ constexpr RqDiv kRqDiv;

// the thread's own column of shared memory, by address (volatile: in program order)
template <uint32_t OFF = 0>
__device__ __forceinline__ float rq_load(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
    return v;
}
template <uint32_t OFF = 0>
__device__ __forceinline__ void rq_store(uint32_t a, float v) {
    asm volatile("st.shared.f32 [%0+%2], %1;" ::"r"(a), "f"(v), "n"(OFF) : "memory");
}
// word i (four values) of a block's half h: the 68 bytes are {d, 32 codes}, {d, 32 codes}
__device__ __forceinline__ uint32_t rq_word(const uint32_t* w, int h, int i) { return h ? w[9 + i] : __funnelshift_r(w[i], w[i + 1], 16); }
// value k of such a word as a float
__device__ __forceinline__ float rq_value(uint32_t biased, int k) { return __uint_as_float(__byte_perm(biased, 0x4B000000u, 0x7440u + k)) - 8388736.0f; }

// the reference's sum for one candidate, in its order
__device__ __forceinline__ float rq_error(const uint32_t* w, float d_lo, float d_hi, float dq) {
    const bool usable = dq > 0.0f && dq < INFINITY;   // else every code is 0 (see the oracle's note on lround)
    const float d = usable ? dq : 0.0f, inv3 = usable ? __fdiv_rn(1.0f, 3.0f * d) : 0.0f;
    float e = 0.0f;
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
        const uint32_t v = rq_word(w, i >> 3, i & 7) ^ 0x80808080u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float x = __fmul_rn(i < 8 ? d_lo : d_hi, rq_value(v, k));
            const float t = __fmaf_rn(__saturatef(__fmaf_rn(x, inv3, 1.0f / 3.0f)), 3.0f, kMagic);   // kMagic + q + 1
            const float r = __fmaf_rn(-__fsub_rn(t, kMagic + 1.0f), d, x);
            e = __fadd_rn(e, __fmul_rn(r, r));
        }
    }
    return e;
}

__global__ void __launch_bounds__(kRqThreads, 6) k_q8_0_to_q2_0(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, size_t nblocks64) {
    __shared__ __align__(16) uint8_t in[kRqThreads * 68];
    __shared__ __align__(16) uint8_t out[kRqThreads * 18];
    __shared__ float half_d[(2 * kRqCand + 1) * kRqThreads];   // [candidate][thread]: 0.5 d; then the bins, [candidates passed][thread]
    const size_t b0 = size_t(blockIdx.x) * kRqThreads;
    const int tid = threadIdx.x, nb = int(min(size_t(kRqThreads), nblocks64 - b0));
    const uint8_t* s = src + b0 * 68;
    if (nb == kRqThreads && uintptr_t(s) % 16 == 0) {
        for (int i = tid; i < kRqThreads * 68 / 16; i += kRqThreads) reinterpret_cast<uint4*>(in)[i] = reinterpret_cast<const uint4*>(s)[i];
    } else if (uintptr_t(s) % 4 == 0) {   // the last blocks of a call, and sources that are not aligned to vectors
        for (int i = tid; i < nb * 17; i += kRqThreads) reinterpret_cast<uint32_t*>(in)[i] = reinterpret_cast<const uint32_t*>(s)[i];
    } else {
        for (int i = tid; i < nb * 68; i += kRqThreads) in[i] = s[i];
    }
    __syncthreads();
    if (tid < nb) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(in) + tid * 17;
        const float d8[2] = {__half2float(__ushort_as_half(uint16_t(w[0] & 0xffffu))), __half2float(__ushort_as_half(uint16_t(w[8] >> 16)))};
        // the largest magnitude and the sum of squares of each half. A signed 16-bit maximum of {byte, byte below it}
        // pairs is decided by the upper byte.
        float mag[2];
        int sq[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t hi = 0x80008000u, lo = 0x7fff7fffu;
            int q = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t v = rq_word(w, h, i), u = v << 8;
                hi = __vmaxs2(__vmaxs2(hi, v), u);
                lo = __vmins2(__vmins2(lo, v), u);
                q = __dp4a(int(v), int(v), q);
            }
            const int top = max(int(hi) >> 24, int(int16_t(hi & 0xffffu)) >> 8), bot = min(int(lo) >> 24, int(int16_t(lo & 0xffffu)) >> 8);
            mag[h] = float(max(top, -bot));
            sq[h] = q;
        }
        const float amax = fmaxf(fmaxf(0.0f, __fmul_rn(fabsf(d8[0]), mag[0])), __fmul_rn(fabsf(d8[1]), mag[1]));
        // the candidates. With 1 / div correctly rounded one residual makes amax * (1 / div) the correctly rounded quotient
        // (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990), if nothing underflows.
        const bool normal = amax >= 0x1p-12f && amax < 32768.0f && fabsf(d8[0]) < INFINITY && fabsf(d8[1]) < INFINITY;
#pragma unroll 4
        for (int c = 0; c < kRqCand; ++c) {
            const float q = __fmul_rn(amax, kRqDiv.inv[c]), exact = __fmaf_rn(__fmaf_rn(-q, kRqDiv.div[c], amax), kRqDiv.inv[c], q);
            half_d[c * kRqThreads + tid] = 0.5f * __half2float(__float2half_rn(normal ? exact : __fdiv_rn(amax, kRqDiv.div[c])));
        }
        uint32_t near_best = (1u << kRqCand) - 1;   // candidates that may have the smallest sum
        if (normal) {
            float first[kRqCand];   // suffix sums of the first half
            const uint32_t cand0 = smem_u32(half_d) + tid * 4, base = cand0 - (0x4B000000u * kRqRow);
            float best = 0.0f, x2 = 0.0f;
            float gain[kRqCand];    // d (2 S1 - d S2)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int c = 0; c <= kRqCand; ++c) rq_store<kRqToBin>(cand0 + c * kRqRow, 0.0f);
                // candidates passed: floor((2.5 - amax / (2 |x|)) * 46 / 3 + 1); 0.03 less, so that the candidate to compare
                // with is the next one, and rounded to nearest, so 0.5 less; in units of 23 for the clamp
                const float c1 = __fdiv_rn(amax, -3.0f * fabsf(d8[h])), off = (2.5f * 46.0f / 3.0f + 0.47f) / 23.0f;
#pragma unroll 1
                for (int i = 0; i < 8; i += 2) {
                    float x[8], one[8];
                    uint32_t a1[8], a3[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float xf = rq_value(rq_word(w, h, i + k / 4) ^ 0x80808080u, k % 4);
                        float r;
                        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fabsf(xf)));
                        x[k] = __fmul_rn(d8[h], xf);
                        one[k] = fabsf(xf) + kRqCount;
                        a1[k] = __float_as_uint(__fmaf_rn(__saturatef(__fmaf_rn(r, c1, off)), 23.0f, 8388608.0f)) * kRqRow + base;
                        a3[k] = __float_as_uint(__fmaf_rn(__saturatef(__fmaf_rn(r, 3.0f * c1, off)), 23.0f, 8388608.0f)) * kRqRow + base;
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        if (fabsf(x[k]) >= rq_load(a1[k])) a1[k] += kRqRow;
                        if (x[k] >= 3.0f * rq_load(a3[k])) a3[k] += kRqRow;
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        rq_store<kRqToBin>(a1[k], rq_load<kRqToBin>(a1[k]) + one[k]);
                        if (x[k] > 0.0f) rq_store<kRqToBin>(a3[k], rq_load<kRqToBin>(a3[k]) + (one[k] + 2.0f * kRqCount));
                    }
                }
                float sum = 0.0f;
#pragma unroll
                for (int c = kRqCand - 1; c >= 0; --c) {
                    sum += rq_load<kRqToBin>(cand0 + (c + 1) * kRqRow);   // exact: an integer below 2^24
                    if (h == 0) {
                        first[c] = sum;
                    } else {
                        const float n0 = __fmaf_rn(first[c], 1.0f / kRqCount, kMagic) - kMagic, n1 = __fmaf_rn(sum, 1.0f / kRqCount, kMagic) - kMagic;
                        const float s1 = __fmaf_rn(fabsf(d8[0]), __fmaf_rn(n0, -kRqCount, first[c]), fabsf(d8[1]) * __fmaf_rn(n1, -kRqCount, sum));   // (both products exact: 11 bits times 13)
                        const float d = 2.0f * rq_load(cand0 + c * kRqRow);
                        gain[c] = d * __fmaf_rn(-d, n0 + n1, 2.0f * s1);
                        best = fmaxf(best, gain[c]);
                    }
                }
                x2 = __fmaf_rn(d8[h] * d8[h], float(sq[h]), x2);
            }
            const float least = best - (8e-7f * x2 + 8.2e-6f * fmaxf(x2 - best, 0.0f));
            near_best = 0;
#pragma unroll
            for (int c = 0; c < kRqCand; ++c) near_best |= uint32_t(gain[c] >= least) << c;
        }
        float best_d = 0.0f;
        if ((near_best & (near_best - 1)) == 0) {
            best_d = 2.0f * half_d[(31 - __clz(near_best)) * kRqThreads + tid];
        } else if (amax > 0.0f) {
            // the first candidate with the smallest error wins; a NaN or infinite error never does
            float best_e = INFINITY;
#pragma unroll 1
            for (uint32_t m = near_best; m; m &= m - 1) {
                const float dq = 2.0f * half_d[(__ffs(m) - 1) * kRqThreads + tid];
                const float e = dq < INFINITY ? rq_error(w, d8[0], d8[1], dq) : INFINITY;
                if (e < best_e) {
                    best_e = e;
                    best_d = dq;
                }
            }
        }
        uint16_t* o = reinterpret_cast<uint16_t*>(out + tid * 18);
        o[0] = __half_as_ushort(__float2half_rn(best_d));
        if (best_d >= 0x1p-14f && best_d < INFINITY) {
            const float inv3 = __fdiv_rn(1.0f + 0x1p-20f, 3.0f * best_d);
#pragma unroll 2
            for (int k = 0; k < 8; ++k) {   // two bytes of four elements each
                const float f = (k < 4 ? d8[0] : d8[1]) * inv3;
                uint32_t v = 0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float xf = rq_value(rq_word(w, k / 4, (k % 4) * 2 + i / 4) ^ 0x80808080u, i % 4);
                    v += __float_as_uint(__fmaf_rn(__saturatef(__fmaf_rn(xf, f, 1.0f / 3.0f)), 3.0f, kMagic)) << (2 * i);   // (kMagic's own bits leave the low 16)
                }
                o[1 + k] = uint16_t(v);
            }
        } else {
            const bool fin = best_d > 0.0f && best_d < INFINITY;
            const float h1 = 0.5f * best_d, h3 = 1.5f * best_d;
#pragma unroll 1
            for (int k = 0; k < 8; ++k) {
                uint32_t v = 0;
                for (int i = 0; i < 8; ++i) {
                    const float xv = __fmul_rn(k < 4 ? d8[0] : d8[1], rq_value(rq_word(w, k / 4, (k % 4) * 2 + i / 4) ^ 0x80808080u, i % 4));
                    const int code = fin ? 1 + int(xv >= h1) + int(xv >= h3) - int(xv <= -h1) : 1;
                    v |= uint32_t(code) << (2 * i);
                }
                o[1 + k] = uint16_t(v);
            }
        }
    }
    __syncthreads();
    uint8_t* d = dst + b0 * 18;
    if (nb == kRqThreads && uintptr_t(d) % 16 == 0) {
        for (int i = tid; i < kRqThreads * 18 / 16; i += kRqThreads) reinterpret_cast<uint4*>(d)[i] = reinterpret_cast<const uint4*>(out)[i];
    } else if (uintptr_t(d) % 2 == 0) {
        for (int i = tid; i < nb * 9; i += kRqThreads) reinterpret_cast<uint16_t*>(d)[i] = reinterpret_cast<const uint16_t*>(out)[i];
    } else {
        for (int i = tid; i < nb * 18; i += kRqThreads) d[i] = out[i];
    }
}

// ---- the grouped product (gemm::moe_run): int8 tensor cores
// A block takes 128 weight rows and up to 64 of the slots of one expert and walks K in chunks of 128 (two
// blocks of weights, 36 bytes per row) through a ring of shared-memory stages filled with cp.async: the
// rows as they are in the file, the activations in the MMA's fragment order, their scales per
// pair of slots. A warp has 32 rows and all the slots, so a row is unpacked once: a lane
// reads its row's nine words (conflict-free, shared by the four lanes of a quad),
// shifts lane t's crumbs into place and masks them, which gives the A operand for a K order of
// {t, 4 + t, 8 + t, 12 + t}; the quantizer writes the activation codes in that order.
// The codes are made signed (code - 1) while they are unpacked, which is cheaper than a sum of the activations per chunk
// and column. The MMA of 32 values starts at kMagicBits and so ends at kMagicBits + sum((q - 1) * a), which
// read as a float is kMagic plus the chunk's exact integer sum.
// What bounds it: issue slots (a 16 x 8 x 64 tile costs two MMAs and eight packed fp32 operations of two slots) and what
// shared memory delivers, about even. 1,000 tokens x 8 of 128 experts of 2560 x 640, per product: 157 us with two warps
// side by side over the slots (each unpacking the rows, half of them idle behind a short item) and the copies' addresses
// computed anew, 118 us now.
constexpr int kGmRows = 128, kGmTok = 64, kGmK = 128, kGmStages = 4, kGmThreads = 128;
constexpr int kGmBytesW = kGmRows * 36;
constexpr int kGmBytesB = kGmTok * kGmK;                     // [block][8 slots][lane] 16 bytes
constexpr int kGmBytesA = 2 * (kGmTok / 2) * 16;             // [block][pair of slots] {a0, a0', a1, a1'}
constexpr int kGmStage = kGmBytesW + kGmBytesB + kGmBytesA;
constexpr int kGmSmem = kGmStages * kGmStage;

// Workspace form of the activations: per row int8 codes in fragment order (word (t * 4 + 2 s + h) of a 64-block
// holds elements 32 s + 16 h + {t, 4 + t, 8 + t, 12 + t}) and the chunk scales d (through fp16, as Q8_1 stores them).
// Quantization is quantize.cu's: d = amax / 127, q = roundf(x / d).
struct GmAct {
    int8_t* q;     // [rows][ncols]
    float* d;      // [rows][ncols / 32]
};
__global__ void __launch_bounds__(256) k_gm_quant(const float* __restrict__ x, int ncols, size_t n_quads, GmAct a) {
    pdl_wait();
    pdl_trigger();
    const size_t quad = size_t(blockIdx.x) * 256 + threadIdx.x;   // four consecutive values; eight lanes one chunk of 32
    if (quad >= n_quads) return;                                  // (a multiple of 32: warps are live as a whole)
    float hv[4];
    if (uintptr_t(x) % 16 == 0) {
        const float4 v = reinterpret_cast<const float4*>(x)[quad];
        hv[0] = v.x, hv[1] = v.y, hv[2] = v.z, hv[3] = v.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) hv[i] = x[quad * 4 + i];
    }
    float am = fmaxf(fmaxf(fabsf(hv[0]), fabsf(hv[1])), fmaxf(fabsf(hv[2]), fabsf(hv[3])));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    const float d = __fdiv_rn(am, 127.0f);
    const int j = int(quad & 7), h = j >> 2, i = j & 3;           // elements 16 h + 4 i + t of the chunk, t = 0 .. 3
    const size_t chunk = quad >> 3;
    int8_t* blk = a.q + (chunk >> 1) * 64 + (chunk & 1) * 8 + h * 4 + i;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int code = am == 0.0f ? 0 : int(round_half_away(__fdiv_rn(hv[t], d)));
        blk[t * 16] = int8_t(code);
    }
    if (j == 0) a.d[chunk] = __half2float(__float2half_rn(d));
}

struct GmArgs {
    const uint8_t* w;        // expert e's matrix at w + e * expert_stride
    size_t expert_stride;
    GmAct act;
    float* dst;              // [slots][nrows]
    int ncols, nrows;
    const int* bounds;       // [E + 1] of the grouped order
    const int* item_off;     // [E + 1] items of kGmTok slots in front of an expert
    const int32_t* perm;
    const int* status;       // [1] = number of items
    int E, K, x_per_slot;
};

// D = A * B + C, A and B signed bytes
__device__ __forceinline__ void mma_s8s8_c4(uint64_t& lo, uint64_t& hi, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                            uint32_t b1, const int4& c) {
    asm volatile(
        "{\n\t.reg .b32 d0, d1, d2, d3;\n\t"
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {d0,d1,d2,d3}, {%2,%3,%4,%5}, {%6,%7}, {%8,%9,%10,%11};\n\t"
        "mov.b64 %0, {d0,d1};\n\t"
        "mov.b64 %1, {d2,d3};\n\t}"
        : "=l"(lo), "=l"(hi)
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c.x), "r"(c.y), "r"(c.z), "r"(c.w));
}
__device__ __forceinline__ void gm_cp4(uint32_t dst, const void* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void gm_cp16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }

__global__ void __launch_bounds__(kGmThreads, 3) k_gm_mma(const GmArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ int s_slot[kGmTok], s_act[kGmTok];
    pdl_wait();
    pdl_trigger();
    const int item = blockIdx.x;
    if (item >= a.status[1] || int(blockIdx.z * gridDim.y + blockIdx.y) * kGmRows >= a.nrows) return;
    int lo = 0, hi = a.E;   // the expert with item_off[e] <= item < item_off[e + 1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (a.item_off[mid] <= item) lo = mid; else hi = mid;
    }
    // an expert's slots in equal items of whole columns of eight: a last item of a few slots would cost as much unpacking
    const int e = lo, first = a.bounds[e], end = a.bounds[e + 1], parts = a.item_off[e + 1] - a.item_off[e];
    const int per = ((end - first + parts - 1) / parts + 7) & ~7;
    const int base = first + (item - a.item_off[e]) * per, m = min(per, end - base);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    if (tid < kGmTok) {   // columns beyond m repeat the last slot and are not stored
        const int slot = a.perm[base + min(tid, m - 1)];
        s_slot[tid] = slot;
        s_act[tid] = a.x_per_slot ? slot : slot / a.K;
    }
    __syncthreads();
    const int r0 = int(blockIdx.z * gridDim.y + blockIdx.y) * kGmRows, rows = min(kGmRows, a.nrows - r0);
    const uint32_t row_bytes = uint32_t(a.ncols / kQK) * kBlockBytes;
    const uint8_t* wsrc = a.w + size_t(e) * a.expert_stride + size_t(r0) * row_bytes;
    const uint32_t s0 = smem_u32(smem);
    const int m8 = (m + 7) & ~7;   // slots whose activations are fetched

    // This thread's copies of a chunk: nine words of the weights (word i of the tile's 128 x 9 by thread i % 128; rows beyond
    // the matrix repeat its last one), 16 bytes of the codes of up to four slots, a scale of up to two.
    // Where they start is found once.
    const int nch = a.ncols / kQ8;
    uint32_t w_at[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        const int idx = tid + i * kGmThreads, row = idx / 9, w = idx - row * 9;
        w_at[i] = uint32_t(min(row, rows - 1)) * row_bytes + w * 4;
    }
    const int8_t* q_at[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q_at[i] = a.act.q + size_t(s_act[(tid >> 3) + 16 * i]) * a.ncols + (tid & 7) * 16;   // vector v: block v >> 2, lane t = v & 3
    size_t d_at[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) d_at[i] = size_t(s_act[(tid >> 2) + 32 * i]) * nch + (tid & 3);                       // one of the four chunks of 32
    const uint32_t q_to = ((tid & 7) >> 2) * (kGmTok * 64) + (tid >> 6) * 512 + (((tid >> 3) & 7) * 4 + (tid & 3)) * 16;
    const uint32_t d_to = ((tid & 2) >> 1) * (kGmTok / 2 * 16) + (tid >> 3) * 16 + (tid & 1) * 8 + ((tid >> 2) & 1) * 4;
    auto fetch = [&](int kc) {
        const uint32_t st = s0 + uint32_t(kc % kGmStages) * kGmStage;
        const uint8_t* wk = wsrc + size_t(kc) * 36;
#pragma unroll
        for (int i = 0; i < 9; ++i) gm_cp4(st + (tid + i * kGmThreads) * 4, wk + w_at[i]);
        const uint32_t sb = st + kGmBytesW;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if ((tid >> 3) + 16 * i < m8) gm_cp16(sb + q_to + i * 1024, q_at[i] + size_t(kc) * kGmK);
        const uint32_t sa = sb + kGmBytesB;
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if ((tid >> 2) + 32 * i < m8) {
                gm_cp4(sa + d_to + i * 256, a.act.d + d_at[i] + size_t(kc) * 4);
            }
    };
    const int chunks = a.ncols / kGmK;
#pragma unroll
    for (int i = 0; i < kGmStages - 1; ++i) {
        if (i < chunks) fetch(i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int wr = warp * 32;         // this warp's rows of the tile
    const int nt = m8 >> 3;           // live columns of eight slots
    uint64_t acc[2][8][2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int n = 0; n < 8; ++n) acc[r][n][0] = acc[r][n][1] = 0ull;
    // the accumulators' start in four registers that stay: as constants they would be loaded again for every MMA
    const uint64_t magic = pack2(kMagic, kMagic), neg_magic = pack2(-kMagic, -kMagic);
    int4 start;
    asm volatile("mov.b32 %0, %4;\n\tmov.b32 %1, %4;\n\tmov.b32 %2, %4;\n\tmov.b32 %3, %4;" : "=r"(start.x), "=r"(start.y), "=r"(start.z), "=r"(start.w) : "r"(kMagicBits));
    for (int kc = 0; kc < chunks; ++kc) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kGmStages - 2) : "memory");
        __syncthreads();   // everyone's share of this chunk has landed, and everyone is done with the chunk before
        if (kc + kGmStages - 1 < chunks) fetch(kc + kGmStages - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const uint8_t* st = smem + (kc % kGmStages) * kGmStage;
        const uint32_t* sw = reinterpret_cast<const uint32_t*>(st) + (wr + g) * 9;
        uint32_t w[2][2][8];      // [group of 16 rows][row g / g + 8][word]: this lane's crumbs, lowest two bits of every byte
        uint64_t dw[2][2][2];     // [group][row][block]: the weight scale, twice
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t v[9];    // {d, 16 code bytes}, {d, 16 code bytes}
#pragma unroll
                for (int i = 0; i < 9; ++i) v[i] = sw[(r * 16 + h * 8) * 9 + i];
                const float d0 = __half2float(__ushort_as_half(uint16_t(v[0] & 0xffffu))), d1 = __half2float(__ushort_as_half(uint16_t(v[4] >> 16)));
                dw[r][h][0] = pack2(d0, d0);
                dw[r][h][1] = pack2(d1, d1);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    w[r][h][i] = __funnelshift_r(v[i], v[i + 1], 16);
                    w[r][h][4 + i] = v[5 + i];
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) w[r][h][i] = (((w[r][h][i] >> (2 * t4)) & 0x03030303u) + 0x7f7f7f7fu) ^ 0x80808080u;   // code - 1 in every byte
            }
        const uint8_t* sb = st + kGmBytesW + lane * 16;
        const uint8_t* sa = st + kGmBytesW + kGmBytesB + t4 * 16;
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int np = 0; np < 8; np += 2) {   // two columns at a time, so that one's loads and products run beside the other's
                if (np >= nt) break;               // (the second may be one that nothing fetched: it is not stored)
#pragma unroll
                for (int n = np; n < np + 2; ++n) {
                    const uint4 bf = *reinterpret_cast<const uint4*>(sb + b * (kGmTok * 64) + n * 512);
                    const ulonglong2 d8 = *reinterpret_cast<const ulonglong2*>(sa + b * (kGmTok / 2 * 16) + n * 64);
                    const uint64_t md = mul2(d8.x, neg_magic);   // exact (two bits times eleven): d * sum in one rounding either way
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        uint64_t lo0, hi0, lo1, hi1;
                        mma_s8s8_c4(lo0, hi0, w[r][0][4 * b], w[r][1][4 * b], w[r][0][4 * b + 1], w[r][1][4 * b + 1], bf.x, bf.y, start);
                        mma_s8s8_c4(lo1, hi1, w[r][0][4 * b + 2], w[r][1][4 * b + 2], w[r][0][4 * b + 3], w[r][1][4 * b + 3], bf.z, bf.w, start);
                        // acc += d2 * (d8[0] * sum0 + d8[1] * sum1)
                        const uint64_t u_lo = fma2(d8.y, sub2(lo1, magic), fma2(lo0, d8.x, md));
                        const uint64_t u_hi = fma2(d8.y, sub2(hi1, magic), fma2(hi0, d8.x, md));
                        acc[r][n][0] = fma2(dw[r][0][b], u_lo, acc[r][n][0]);
                        acc[r][n][1] = fma2(dw[r][1][b], u_hi, acc[r][n][1]);
                    }
                }
            }
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        if (n >= nt) break;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int tok = n * 8 + 2 * t4 + k;
            if (tok >= m) continue;
            float* o = a.dst + size_t(s_slot[tok]) * a.nrows + r0;
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float v0, v1;
                    unpack2(acc[r][n][h], v0, v1);
                    const int row = wr + r * 16 + h * 8 + g;
                    if (row < rows) o[row] = k ? v1 : v0;
                }
        }
    }
}

// ---- grouped plan in a workspace
struct PlanLayout {
    size_t status, chunk_cnt, bounds, item_off, perm, act_q, act_d, total;
    int n_chunks, max_items;
};
PlanLayout plan_layout(int64_t ncols, int64_t rows, int E) {
    PlanLayout L{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += align_up(bytes);
        return o;
    };
    L.n_chunks = int((rows + kChunkSlots - 1) / kChunkSlots);
    L.max_items = int(rows / kGmTok) + E;
    L.status = take(64);
    L.chunk_cnt = take(size_t(L.n_chunks) * E * 4);
    L.bounds = take(size_t(E + 1) * 4);
    L.item_off = take(size_t(E + 1) * 4);
    L.perm = take(size_t(rows) * 4);
    L.act_q = take(size_t(rows) * ncols);
    L.act_d = take(size_t(rows) * (ncols / kQ8) * 4);
    L.total = off;
    return L;
}
constexpr int kPlanMaxExperts = 4096;
GmAct plan_act(uint8_t* base, const PlanLayout& L) {
    return GmAct{reinterpret_cast<int8_t*>(base + L.act_q), reinterpret_cast<float*>(base + L.act_d)};
}

// The next kernel's blocks are let in early only while the whole grid is resident (eight blocks of 256 threads per SM): in a longer
// one they would wait in places that this kernel's own blocks need.
cudaError_t launch_q8_1(const float* x, const float* u, int64_t ncols, int n_tok, void* xq, cudaStream_t stream) {
    const int64_t padded = padded_cols(ncols), blocks = padded / 256 * n_tok;
    return launch_pdl(k_q8_1, dim3(unsigned(padded / 256), unsigned(n_tok)), dim3(256), 0, stream, x, u, ncols, padded, static_cast<uint8_t*>(xq),
                      int(blocks <= 512 || blocks <= 8 * sm_count()));   // (64 SMs are there in any case: one token's call does not ask for the number)
}

}  // namespace
}  // namespace frx

using namespace frx;

extern "C" {

size_t frx_gemv_q8_1_bytes(int64_t ncols, int n_tok) {
    if (ncols < 1 || n_tok < 1) return 0;
    return size_t(n_tok) * act_row_bytes(ncols);
}

int64_t frx_gemv_row_bytes(uint32_t ggml_type, int64_t ncols) {
    if (ggml_type != kTypeQ2_0 || ncols < 0) return 0;
    return ncols / kQK * kBlockBytes;
}

int frx_gemv_quantize_q8_1(const float* x, int64_t ncols, int n_tok, void* xq, frx_stream_t stream) {
    if (ncols < 1 || n_tok < 0) return fail(FRX_ERR_SHAPE, "gemv::quantize_q8_1: ncols %lld, n_tok %d", (long long)ncols, n_tok);
    if (n_tok == 0) return FRX_OK;
    if (!x || !xq || uintptr_t(xq) % 4) return fail(FRX_ERR_ARG, "gemv::quantize_q8_1: null or misaligned pointer");
    FRX_LAUNCH(kKQuant, stream, launch_q8_1(x, nullptr, ncols, n_tok, xq, stream));
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

int frx_gemv_swiglu_q8_1(const float* g, const float* u, int64_t ncols, int n_tok, void* xq, frx_stream_t stream) {
    if (ncols < 1 || n_tok < 0) return fail(FRX_ERR_SHAPE, "gemv::swiglu_q8_1: ncols %lld, n_tok %d", (long long)ncols, n_tok);
    if (n_tok == 0) return FRX_OK;
    if (!g || !u || !xq || uintptr_t(xq) % 4) return fail(FRX_ERR_ARG, "gemv::swiglu_q8_1: null or misaligned pointer");
    FRX_LAUNCH(kKQuant, stream, launch_q8_1(g, u, ncols, n_tok, xq, stream));
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

int frx_gemv_moe_q(uint32_t ggml_type, const void* w, const void* gate, const void* xq, const int32_t* ids, float* dst, int n_tok, int k,
                   int64_t ncols, int64_t nrows, int64_t expert_stride_bytes, int act_per_expert, frx_stream_t stream) {
    if (int rc = check_dot_shape("gemv::moe_q", ggml_type, ncols, nrows)) return rc;
    if (n_tok < 1 || n_tok > 8 || k < 1) return fail(FRX_ERR_SHAPE, "gemv::moe_q: n_tok %d must be 1..8, k %d positive", n_tok, k);
    if (!w || !xq || !ids || !dst) return fail(FRX_ERR_ARG, "gemv::moe_q: null pointer");
    if (expert_stride_bytes < 0 || expert_stride_bytes % kBlockBytes || (uintptr_t(w) | uintptr_t(gate) | uintptr_t(xq)) % 4 || expert_stride_bytes % 4)
        return fail(FRX_ERR_ARG, "gemv::moe_q: the expert stride must be whole blocks and, like the pointers, a multiple of 4 bytes");
    DotArgs a{};
    a.w = static_cast<const uint8_t*>(w);
    a.gate = static_cast<const uint8_t*>(gate);
    a.expert_stride = size_t(expert_stride_bytes);
    a.xq = static_cast<const uint8_t*>(xq);
    a.act_row = act_row_bytes(ncols);
    a.dst = dst;
    a.ncols = int(ncols);
    a.nrows = int(nrows);
    a.ids = ids;
    a.act_div = act_per_expert ? 1 : k;
    if (gate)
        FRX_LAUNCH(kKGateUp, stream, { if (int rc = launch_dot<true>(a, n_tok * k, stream)) return rc; });
    else
        FRX_LAUNCH(kKDown, stream, { if (int rc = launch_dot<false>(a, n_tok * k, stream)) return rc; });
    return FRX_OK;
}

int frx_gemv_moe_q2_0(const void* w, const void* gate, const void* xq, const int32_t* ids, float* dst, int n_ids, int64_t ncols,
                      int64_t nrows, int64_t slot_stride_bytes, int per_channel_act, frx_stream_t stream) {
    if (n_ids < 1) return fail(FRX_ERR_SHAPE, "gemv::moe_q2_0: n_ids %d", n_ids);
    if (int rc = check_dot_shape("gemv::moe_q2_0", kTypeQ2_0, ncols, nrows)) return rc;
    if (!w || !xq || !ids || !dst) return fail(FRX_ERR_ARG, "gemv::moe_q2_0: null pointer");
    if (slot_stride_bytes < 0 || slot_stride_bytes % kBlockBytes || (uintptr_t(w) | uintptr_t(gate) | uintptr_t(xq)) % 4 || slot_stride_bytes % 4)
        return fail(FRX_ERR_ARG, "gemv::moe_q2_0: the slot stride must be whole blocks and, like the pointers, a multiple of 4 bytes");
    DotArgs a{};
    a.w = static_cast<const uint8_t*>(w);
    a.gate = static_cast<const uint8_t*>(gate);
    a.expert_stride = size_t(slot_stride_bytes);
    a.xq = static_cast<const uint8_t*>(xq);
    a.act_row = act_row_bytes(ncols);
    a.dst = dst;
    a.ncols = int(ncols);
    a.nrows = int(nrows);
    a.ids = ids;
    a.act_div = per_channel_act ? 1 : n_ids;   // one activation row for every channel, or one each
    if (gate)
        FRX_LAUNCH(kKGateUp, stream, { if (int rc = launch_dot<true>(a, n_ids, stream)) return rc; });
    else
        FRX_LAUNCH(kKDown, stream, { if (int rc = launch_dot<false>(a, n_ids, stream)) return rc; });
    return FRX_OK;
}

int frx_gemv_matvec_q(uint32_t ggml_type, const void* W, const void* xq, float* y, int64_t ncols, int64_t nrows, int n_tok,
                      frx_stream_t stream) {
    if (int rc = check_dot_shape("gemv::matvec_q", ggml_type, ncols, nrows)) return rc;
    if (n_tok < 1 || n_tok > 8) return fail(FRX_ERR_SHAPE, "gemv::matvec_q: n_tok %d must be 1..8", n_tok);
    if (!W || !xq || !y || (uintptr_t(W) | uintptr_t(xq)) % 4) return fail(FRX_ERR_ARG, "gemv::matvec_q: null or misaligned pointer");
    DotArgs a{};
    a.w = static_cast<const uint8_t*>(W);
    a.expert_stride = 0;
    a.xq = static_cast<const uint8_t*>(xq);
    a.act_row = act_row_bytes(ncols);
    a.dst = y;
    a.ncols = int(ncols);
    a.nrows = int(nrows);
    a.act_div = 1;
    FRX_LAUNCH(kKDown, stream, { if (int rc = launch_dot<false>(a, n_tok, stream)) return rc; });
    return FRX_OK;
}

int frx_gemv_matvec(uint32_t ggml_type, const void* W, const float* x, float* y, int64_t ncols, int64_t nrows, int n_tok, void* scratch,
                    frx_stream_t stream) {
    if (int rc = check_dot_shape("gemv::matvec", ggml_type, ncols, nrows)) return rc;
    if (!scratch) return fail(FRX_ERR_ARG, "gemv::matvec: null scratch");
    if (int rc = frx_gemv_quantize_q8_1(x, ncols, n_tok, scratch, stream)) return rc;
    return frx_gemv_matvec_q(ggml_type, W, scratch, y, ncols, nrows, n_tok, stream);
}

size_t frx_gemm_workspace_bytes(int64_t ncols, int64_t rows) {
    if (ncols < 1 || rows < 1) return 0;
    return plan_layout(ncols, rows, kPlanMaxExperts).total;
}

int frx_gemm_moe_prepare(frx_gemm_moe_plan* plan, uint32_t ggml_type, int n_experts, const float* x, int x_per_slot, const int32_t* ids,
                         int64_t T, int K, int64_t ncols, void* ws, size_t ws_bytes, frx_stream_t stream) {
    if (!plan) return fail(FRX_ERR_ARG, "gemm::moe_prepare: null plan");
    if (int rc = check_dot_shape("gemm::moe_prepare", ggml_type, ncols, 1)) return rc;
    if (n_experts < 1 || n_experts > kPlanMaxExperts || K < 1 || T < 0 || T * K > (int64_t(1) << 28))
        return fail(FRX_ERR_SHAPE, "gemm::moe_prepare: unsupported E %d, K %d, T %lld", n_experts, K, (long long)T);
    if (!x || !ids || !ws || uintptr_t(ws) % kAlign) return fail(FRX_ERR_ARG, "gemm::moe_prepare: null pointer or workspace not 256-byte aligned");
    const int64_t rows = T * K;
    plan->type = ggml_type;
    plan->n_experts = n_experts;
    plan->K = K;
    plan->T = T;
    plan->ncols = ncols;
    plan->rows = rows;
    plan->x_per_slot = x_per_slot ? 1 : 0;
    plan->ws = ws;
    if (T == 0) return FRX_OK;
    const PlanLayout L = plan_layout(ncols, rows, n_experts);
    if (ws_bytes < L.total) return fail(FRX_ERR_WORKSPACE, "gemm::moe_prepare: workspace %zu < %zu", ws_bytes, L.total);
    auto* base = static_cast<uint8_t*>(ws);
    int* status = reinterpret_cast<int*>(base + L.status);
    int* chunk_cnt = reinterpret_cast<int*>(base + L.chunk_cnt);
    int* bounds = reinterpret_cast<int*>(base + L.bounds);
    int* item_off = reinterpret_cast<int*>(base + L.item_off);
    int32_t* perm = reinterpret_cast<int32_t*>(base + L.perm);
    const int S = int(rows), E = n_experts;
    // one row of codes per token, or per (token, expert) slot when every slot has its own activations
    const size_t n_quads = size_t(x_per_slot ? rows : T) * size_t(ncols / 4);
    FRX_LAUNCH(kKQuant, stream, launch_pdl(k_gm_quant, dim3(unsigned((n_quads + 255) / 256)), dim3(256), 0, stream, x, int(ncols), n_quads, plan_act(base, L)));
    FRX_LAUNCH(kKGroup, stream, launch_pdl(k_pf_hist, dim3(L.n_chunks), dim3(256), size_t(E) * 4, stream, ids, S, E, chunk_cnt, status, (const int32_t*)nullptr, 0));
    FRX_LAUNCH(kKGroup, stream, launch_pdl(k_pf_scan, dim3(1), dim3(1024), 0, stream, chunk_cnt, L.n_chunks, E, bounds, item_off, status, L.max_items, kGmTok, TokenBlocks{}));
    FRX_LAUNCH(kKGroup, stream, launch_pdl(k_pf_place, dim3(L.n_chunks), dim3(kChunkSlots), pf_place_smem(E), stream, ids, S, E, (const int*)chunk_cnt, (const int*)bounds, perm,
                                           (const int32_t*)nullptr, 0));
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

int frx_gemm_moe_run(const frx_gemm_moe_plan* plan, const void* W, int64_t expert_stride_bytes, float* y, int64_t nrows, frx_stream_t stream) {
    if (!plan || !plan->ws) return fail(FRX_ERR_ARG, "gemm::moe_run: no plan");
    if (int rc = check_dot_shape("gemm::moe_run", plan->type, plan->ncols, nrows)) return rc;
    if (!W || !y) return fail(FRX_ERR_ARG, "gemm::moe_run: null pointer");
    if (expert_stride_bytes < 0 || expert_stride_bytes % kBlockBytes || uintptr_t(W) % 4 || expert_stride_bytes % 4)
        return fail(FRX_ERR_ARG, "gemm::moe_run: the expert stride must be whole blocks and, like W, a multiple of 4 bytes");
    if (plan->T == 0) return FRX_OK;
    const PlanLayout L = plan_layout(plan->ncols, plan->rows, plan->n_experts);
    auto* base = static_cast<uint8_t*>(plan->ws);
    static std::once_flag once[64];
    int dev = 0;
    FRX_CUDA(cudaGetDevice(&dev));
    cudaError_t attr = cudaSuccess;
    if (dev >= 0 && dev < 64) std::call_once(once[dev], [&] { attr = cudaFuncSetAttribute(k_gm_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, kGmSmem); });
    if (attr != cudaSuccess) return cuda_fail(attr, "gemm::moe_run: cudaFuncSetAttribute");
    GmArgs a{};
    a.w = static_cast<const uint8_t*>(W);
    a.expert_stride = size_t(expert_stride_bytes);
    a.act = plan_act(base, L);
    a.dst = y;
    a.ncols = int(plan->ncols);
    a.nrows = int(nrows);
    a.bounds = reinterpret_cast<const int*>(base + L.bounds);
    a.item_off = reinterpret_cast<const int*>(base + L.item_off);
    a.perm = reinterpret_cast<const int32_t*>(base + L.perm);
    a.status = reinterpret_cast<const int*>(base + L.status);
    a.E = plan->n_experts;
    a.K = plan->K;
    a.x_per_slot = plan->x_per_slot;
    // (a grid has at most 65,535 blocks along y, and nrows may need twice as many tiles)
    const unsigned tiles = unsigned((nrows + kGmRows - 1) / kGmRows), slices = (tiles + 65534) / 65535;
    const dim3 grid(unsigned(L.max_items), (tiles + slices - 1) / slices, slices);
    FRX_LAUNCH(kKDown, stream, launch_pdl(k_gm_mma, grid, dim3(kGmThreads), size_t(kGmSmem), stream, a));
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

int frx_gemm_moe(uint32_t ggml_type, const void* W, int64_t expert_stride_bytes, int n_experts, const float* x, int x_per_slot,
                 const int32_t* ids, int64_t T, int K, float* y, int64_t ncols, int64_t nrows, void* ws, size_t ws_bytes, frx_stream_t stream) {
    frx_gemm_moe_plan plan;
    if (int rc = frx_gemm_moe_prepare(&plan, ggml_type, n_experts, x, x_per_slot, ids, T, K, ncols, ws, ws_bytes, stream)) return rc;
    return frx_gemm_moe_run(&plan, W, expert_stride_bytes, y, nrows, stream);
}

int frx_convert_q8_0_to_q2_0(const void* src_q8_0, void* dst_q2_0, size_t nblocks64, frx_stream_t stream) {
    if (nblocks64 == 0) return FRX_OK;
    if (!src_q8_0 || !dst_q2_0) return fail(FRX_ERR_ARG, "convert_q8_0_to_q2_0: null pointer");
    if (nblocks64 > (size_t(1) << 34)) return fail(FRX_ERR_SHAPE, "convert_q8_0_to_q2_0: too many blocks");
    FRX_LAUNCH(kKLayout, stream, k_q8_0_to_q2_0<<<unsigned((nblocks64 + kRqThreads - 1) / kRqThreads), kRqThreads, 0, stream>>>(static_cast<const uint8_t*>(src_q8_0), static_cast<uint8_t*>(dst_q2_0), nblocks64));
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

}  // extern "C"
