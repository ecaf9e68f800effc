// Prefill-sized grouped expert product (moe_q2::run, kernels/cuda/moe_q2.h:21-30) on the
// 5th-generation tensor cores: tcgen05.mma with fp32 accumulators in tensor memory.
//
// Numerics are the decode path's, i.e. the reference CPU path's: int8 activation codes per 32
// values, exact integer dot products per 32-block, then scale and accumulate in the reference's
// order and roundings. The tensor core does only the exact part. Operands are small integers held
// in e4m3: the weight codes q - 1 in {-1, 0, 1, 2}, and every activation code as the sum of two
// e4m3 values, a multiple of 16 in [-128, 128] and a rest in [-8, 7]. The two products of a
// 32-block go into one accumulator, so it holds the block's integer sum (|sum| <= 8128), exact.
// Each 64-weight block yields two accumulators S0, S1 per (row, token) in tensor memory, which the
// epilogue warps turn into d * (a0 * S0 + a1 * S1) and add to running sums held in registers, block
// after block.
//
// One block per SM works on tiles of 256 matrix rows x up to 48 tokens of one expert, in units of 128
// weights of K. Warps: packed weights (bulk copies), activations and scales (gathered), two MMA
// issuers (one per row tile of 128), eight dequant warps (2-bit codes -> e4m3, written to tensor memory,
// which spares shared memory the A operand's traffic: 48 KB per unit), sixteen epilogue warps. Tensor
// memory: 384 columns of sums (two 64-blocks), 128 of weights. What bounds it: the fp32 pipe in
// principle (four packed operations per two sums, 770 cycles per unit), in practice the issue slots
// (5,400 warp instructions per unit, a packed operation taking two slots) and the hand-off of the two
// sets of sums between the MMAs and the epilogue (about 600 cycles round trip). A unit takes 1,900
// cycles. 16,384 tokens, 512 experts top-10, hidden 2048, width 512: gate/up 1,683 us, down 1,000 us (1,585 and 1,060
// on activations that another kernel had gathered in 237); before, with
// fp16 operands in shared memory, tiles of 128 x 128 and a hand-off per 64 weights: 2,520 and 1,620.
#include "frx_umma.cuh"

#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <mutex>

namespace frx {
namespace {

#include "frx_group.cuh"

constexpr int kTileRows = 128;     // M of the MMA: 8 groups of 16 matrix rows
constexpr int kRowTiles = 2;       // row tiles of a block's tile: 256 matrix rows share the activations
constexpr int kTileTok = 48;       // most tokens of one tile (N of the MMA), a multiple of 16
constexpr int kTokPad = 16;        // every expert's token count is padded to this
constexpr int kBlockBytesB = kTileTok * 128;       // one 64-block: 64 values x 2 e4m3 pieces per token
constexpr int kUnitBytesB = 2 * kBlockBytesB;      // one unit (128 weights of K): 12 KB
constexpr int kBlockBytesS = kTileTok * 8;         // activation scales of one 64-block
constexpr int kUnitBytesS = 2 * kBlockBytesS + kRowTiles * kTileRows * 4;   // and the two block scales of every row
constexpr int kTileBytesW = 8 * kUnitBytes;        // packed weights of one row tile x one unit: 4608 B
constexpr int kUnitBytesW = kRowTiles * kTileBytesW;
constexpr int kStagesW = 8, kStagesB = 8, kStagesS = 16, kStagesA = 2;   // units in flight: packed weights, activations, scales, e4m3 weights
// Scale slots are not handed back by a barrier: activations of unit g are fetched once the MMAs of
// unit g - kStagesB have completed, which waited for the epilogue to read the accumulators of the unit
// before, so every unit up to g - kStagesB - 2 is finished.
static_assert(kStagesS >= kStagesB + 2, "a scale slot may still be in use");
// Tensor memory: the sums of the two 64-blocks of a unit (per row tile two 32-value sums of every
// token), then the e4m3 weights (32 columns of four bytes per row tile and unit).
constexpr int kColsRow = 2 * kTileTok, kColsBlock = kRowTiles * kColsRow, kColsA = kRowTiles * 32, kColA0 = 2 * kColsBlock;
constexpr int kTmemCols = 512;
static_assert(kColA0 + kStagesA * kColsA <= kTmemCols, "tensor memory has 512 columns");
constexpr int kWarpsDequant = 8, kWarpsAux = 4 + kWarpsDequant, kWarpsEpilogue = 16;
constexpr int kThreads = (kWarpsAux + kWarpsEpilogue) * 32;
// registers: 896 threads are launched with 72 each; the auxiliary warps give up 32 of theirs, the
// epilogue warps take 24 more: 384 * 40 + 512 * 96 = 896 * 72
constexpr int kRegsAux = 40, kRegsEpilogue = 96;

// meta words: [1] token blocks
struct PfuLayout {
    size_t status, chunk_cnt, bounds, item_off, perm, meta, tb, xe, xd, hf, he, hd, total;
    int n_chunks, max_tb;
};

PfuLayout pfu_layout(int T, int K, int n, int ff, int E) {
    PfuLayout L{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += align_up(bytes);
        return o;
    };
    const size_t S = size_t(T) * K;
    L.n_chunks = int((S + kChunkSlots - 1) / kChunkSlots);
    L.max_tb = int(S / kTileTok) + E + 1;
    L.status = take(64);
    L.chunk_cnt = take(size_t(L.n_chunks) * E * 4);
    L.bounds = take(size_t(E + 1) * 4);
    L.item_off = take(size_t(E + 1) * 4);
    L.perm = take(S * 4);
    L.meta = take(64);
    L.tb = take(size_t(L.max_tb) * sizeof(int4));
    L.xe = take(size_t(T) * n * 2);
    L.xd = take(size_t(T) * (n / kQ8) * 4);
    L.hf = take(S * ff * 8);   // (gate x, up x) pairs
    L.he = take(S * ff * 2);
    L.hd = take(S * (ff / kQ8) * 4);
    L.total = off;
    return L;
}

// The e4m3 pieces of activation codes. A 64-block of one token is 128 bytes, eight 16-byte chunks
// [half s][piece: 0 the multiple of 16, 1 the rest][c]; inside a half, element 16 q + 4 t + i sits in
// chunk c = t >> 1 at byte (t & 1) * 8 + q * 4 + i: the order in which a lane of the dequant warps
// writes the weights' bytes. This is the place of the four codes of element group (s, q, t).
__device__ __forceinline__ int piece_chunk(int s, int piece, int t) { return s * 4 + piece * 2 + (t >> 1); }
__device__ __forceinline__ int piece_byte(int q, int t) { return (t & 1) * 8 + q * 4; }

// Four int8 codes (as ints in [-127, 127]) -> their multiples of 16 and their rests as e4m3 bytes (exact:
// four significant bits are enough for either).
__device__ __forceinline__ void split_codes(const int (&c)[4], uint32_t& hi, uint32_t& lo) {
    float h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int rest = ((c[i] + 8) & 15) - 8;
        l[i] = float(rest);
        h[i] = float(c[i] - rest);
    }
    auto two = [](float a, float b) { return uint32_t(__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3)); };
    hi = two(h[0], h[1]) | (two(h[2], h[3]) << 16);
    lo = two(l[0], l[1]) | (two(l[2], l[3]) << 16);
}

// Q8 of x rows (q2_0::quantize_q8, quant/q2_0/q2_0.cpp:101-113) straight into e4m3 pieces, token-major
// [T][n / 64][128 bytes], and the block scales d [T][n / 32]. A thread owns four consecutive values,
// eight neighbouring lanes one 32-block. n_quads is a multiple of 32: warps are live as a whole.
__global__ void __launch_bounds__(256) k_pfu_quant_x(const float* __restrict__ x, size_t n_quads, uint8_t* __restrict__ xe,
                                                     float* __restrict__ d, int block64) {
    pdl_wait();
    pdl_trigger();
    const size_t quad = size_t(blockIdx.x) * 256 + threadIdx.x;
    if (quad >= n_quads) return;
    const float4 v = reinterpret_cast<const float4*>(x)[quad];
    float am = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    if (block64) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 8));
    const float dd = __fdiv_rn(am, 127.0f);
    const float id = dd != 0.0f ? __fdiv_rn(1.0f, dd) : 0.0f;
    const int c[4] = {int(round_half_away(__fmul_rn(v.x, id))), int(round_half_away(__fmul_rn(v.y, id))), int(round_half_away(__fmul_rn(v.z, id))),
                      int(round_half_away(__fmul_rn(v.w, id)))};
    uint32_t hi, lo;
    split_codes(c, hi, lo);
    const int j = int(quad & 7), s = int(quad >> 3) & 1, q = j >> 2, t = j & 3;
    uint8_t* blk = xe + (quad >> 4) * 128;
    *reinterpret_cast<uint32_t*>(blk + piece_chunk(s, 0, t) * 16 + piece_byte(q, t)) = hi;
    *reinterpret_cast<uint32_t*>(blk + piece_chunk(s, 1, t) * 16 + piece_byte(q, t)) = lo;
    if (j == 0) d[quad >> 3] = __half2float(__float2half_rn(dd));
}

// The same pieces from codes that arrive already quantized (natural order, as frx_quantize_q8 writes them).
__global__ void __launch_bounds__(256) k_pfu_expand_q8(const int8_t* __restrict__ xq, size_t n_quads, uint8_t* __restrict__ xe) {
    pdl_wait();
    pdl_trigger();
    const size_t quad = size_t(blockIdx.x) * 256 + threadIdx.x;
    if (quad >= n_quads) return;
    const char4 v = reinterpret_cast<const char4*>(xq)[quad];
    const int c[4] = {v.x, v.y, v.z, v.w};
    uint32_t hi, lo;
    split_codes(c, hi, lo);
    const int j = int(quad & 7), s = int(quad >> 3) & 1, q = j >> 2, t = j & 3;
    uint8_t* blk = xe + (quad >> 4) * 128;
    *reinterpret_cast<uint32_t*>(blk + piece_chunk(s, 0, t) * 16 + piece_byte(q, t)) = hi;
    *reinterpret_cast<uint32_t*>(blk + piece_chunk(s, 1, t) * 16 + piece_byte(q, t)) = lo;
}

// silu(g) * u with the fast exponential and reciprocal, within kSwigluErr of swiglu_ref for g >= -80: ex2 and rcp are good to 2^-22 and
// 2^-23 (PTX ISA), -g log2 e rounds by at most 2^-24 of 116, which the exponential makes 2^-17.6, three more roundings.
// silu(g) leaves the normal numbers only for |g| < 2^-125. There -g log2 e is flushed to zero or next to it, the exponential is 1, the
// reciprocal of 2 is exact (as run, not as documented) and g / 2 is rounded alike in both forms, so that no u can bring a difference back.
constexpr float kSwigluErr = 0x1p-16f;
__device__ __forceinline__ float swiglu_fast(float g, float u) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(g * -1.44269504f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return g * r * u;
}

// Q8 of the hidden rows (in the grouped order, the first *n_rows of them) into e4m3 pieces and block scales, like
// k_pfu_quant_x. A thread owns the eight values of element group t of a 32-block (4 t .. + 3 and 16 + 4 t .. + 3), four
// neighbouring lanes one 32-block: silu(gate x) * up x is formed here, the block maximum comes from two shuffles, each piece is
// one 8-byte store.
//
// The codes are those of swiglu_ref, but only two kinds of values need it: those that may be a block's largest (it sets the scale), and
// those whose code could round the other way. All values are formed fast; the ones in question, in a few rounds of at most one per lane
// (between one and two for a warp's 256 values), once more exactly. Bound: HBM (10 bytes a value, 130 us at 163,840 rows of 512) and issue:
// 179 us there, 254 with the double-precision exponential for every value.
__global__ void __launch_bounds__(256) k_pfu_quant_h(const float2* __restrict__ hf, int ff, const int* __restrict__ n_rows, uint8_t* __restrict__ he,
                                                     float* __restrict__ hd, int block64) {
    pdl_wait();
    pdl_trigger();
    const size_t g = size_t(blockIdx.x) * 256 + threadIdx.x, n_blk = size_t(*n_rows) * (ff / kQ8);
    size_t blk = g >> 2;                       // the 32-block, over all rows
    if ((g & ~size_t(31)) >> 2 >= n_blk) return;
    // No exit inside a warp, the shuffles below need it whole: with rows of four blocks (ff = 128) an odd number of them
    // ends in the middle of one. Lanes behind the end repeat the last 64-block and store nothing.
    const bool live = blk < n_blk;
    if (!live) blk = n_blk - 2 + (blk & 1);
    const int t = int(g & 3), s = int(blk & 1);
    const float4* src = reinterpret_cast<const float4*>(hf + blk * kQ8);
    float hv[8];
    float am = 0.0f;
    uint32_t ask = 0;   // values to be formed exactly
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float4 gu = src[q * 8 + t * 2 + i];   // (gate, up) of two hidden values
            hv[q * 4 + 2 * i] = swiglu_fast(gu.x, gu.y);
            hv[q * 4 + 2 * i + 1] = swiglu_fast(gu.z, gu.w);
            ask |= uint32_t(!(gu.x >= -80.0f)) << (q * 4 + 2 * i) | uint32_t(!(gu.z >= -80.0f)) << (q * 4 + 2 * i + 1);
        }
    auto block_max = [&](float v) {
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
        if (block64) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 4));   // eight lanes hold one 64-value scale block
        return v;
    };
    auto exact = [&](int i) {
        const float2 gu = hf[blk * kQ8 + (i >> 2) * 16 + t * 4 + (i & 3)];
        return swiglu_ref(gu.x, gu.y);
    };
#pragma unroll
    for (int i = 0; i < 8; ++i) am = fmaxf(am, fabsf(hv[i]));
    am = block_max(am);
    // (no number, and so large or small that a product of the fast form may have left the range of floats: everything exactly)
    if (am != 0.0f && !(am > 1e-25f && am < 1e25f)) ask = 0xffu;
    // A block of zeros, as rows that pad a prompt have them, asks for none: the exact form could make 2^-149 of them at most, and its codes
    // and scale are zero either way. (The quantizers at 16,384 tokens, half of them zero: 384 us with eight exact values a lane there, 218 so.)
    const float lim = am != 0.0f ? am * (1.0f - 4.0f * kSwigluErr) : 0x1p-149f;
#pragma unroll
    for (int i = 0; i < 8; ++i) ask |= uint32_t(!(fabsf(hv[i]) < lim)) << i;
    am = 0.0f;
    while (__any_sync(0xffffffffu, ask != 0)) {
        if (ask) {
            const int i = __ffs(ask) - 1;
            ask &= ask - 1;
            const float v = exact(i);
            am = fmaxf(am, fabsf(v));
#pragma unroll
            for (int k = 0; k < 8; ++k) hv[k] = k == i ? v : hv[k];
        }
    }
    am = block_max(am);
    // quant/q2_0/q2_0.cpp:101-113: d = amax / 127, id = 1 / d, q = roundf(v * id), d through fp16
    const float d = __fdiv_rn(am, 127.0f);
    const float id = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
    int code[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float c = __fmul_rn(hv[i], id), m = c + kMagic;   // |c| <= 127 and a bit
        code[i] = __float_as_int(m) - kMagicBits;
        ask |= uint32_t(!(fabsf(c - (m - kMagic)) < 0.5f - 2.0f * kSwigluErr * fabsf(c))) << i;
    }
    while (__any_sync(0xffffffffu, ask != 0)) {
        if (ask) {
            const int i = __ffs(ask) - 1;
            ask &= ask - 1;
            const int c = int(round_half_away(__fmul_rn(exact(i), id)));
#pragma unroll
            for (int k = 0; k < 8; ++k) code[k] = k == i ? c : code[k];
        }
    }
    uint32_t hi[2], lo[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) split_codes(*reinterpret_cast<const int(*)[4]>(code + 4 * q), hi[q], lo[q]);
    if (!live) return;
    uint8_t* o = he + (blk >> 1) * 128 + piece_byte(0, t);
    *reinterpret_cast<uint2*>(o + piece_chunk(s, 0, t) * 16) = make_uint2(hi[0], hi[1]);
    *reinterpret_cast<uint2*>(o + piece_chunk(s, 1, t) * 16) = make_uint2(lo[0], lo[1]);
    if (t == 0) hd[blk] = __half2float(__float2half_rn(d));
}

// ---------------------------------------------------------------------------------------------
struct UmmaParams {
    const uint8_t* experts;   // tiled blobs
    size_t stride;
    const int* meta;          // [1] = token blocks
    const int4* tb;           // {expert, first position in the grouped order, slots, slots rounded up to kTokPad}
    const int32_t* perm;      // the slot at every position
    const uint8_t* act;       // e4m3 pieces, a row per token (xe) or per position (he)
    const float* act_scale;   // block scales, likewise
    float2* hf;               // gate/up: (gate x, up x) of every hidden element [positions][ff]
    float* yd;                // down: [slots][n]
    int* status;
    unsigned long long wait_ns;   // the longest a wait on a shared-memory barrier may last
    float neg0;               // -0.0f, an addend the compiler does not know (see scale_add)
    int n, ff, K;
    int y_bf16;               // down: yd holds bf16 rows
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct PfSmem {
    uint32_t w, b, s, slots, bars, tmem, abort, total;
};
__host__ __device__ constexpr PfSmem pf_smem() {
    PfSmem m{};
    uint32_t off = 0;
    m.b = off;
    off += kStagesB * kUnitBytesB;
    m.w = off;
    off += kStagesW * kUnitBytesW;
    m.s = off;
    off += kStagesS * kUnitBytesS;
    m.slots = off;
    off += kStagesS * kTileTok * 4;   // of the last kStagesS token blocks (each has at least one unit)
    m.bars = off;
    off += 64 * 8;
    m.tmem = off;
    off += 16;
    m.abort = off;
    off += 16;
    m.total = off;
    return m;
}

// Barrier indices (a unit is 128 weights of K; its uses of a barrier are numbered by the unit)
enum : int {
    kBarWFull = 0,                                 // + stage: packed weights have landed
    kBarWFree = kBarWFull + kStagesW,              // the dequant warps are done with them
    kBarBFull = kBarWFree + kStagesW,              // B tiles have landed (and been made visible to the tensor core)
    kBarBFree = kBarBFull + kStagesB,              // the MMAs that read them have completed
    kBarSFull = kBarBFree + kStagesB,              // activation scales have landed, row scales are written
    kBarAFull = kBarSFull + kStagesS,              // + row tile * kStagesA + stage: e4m3 weights are in tensor memory
    kBarAFree = kBarAFull + kRowTiles * kStagesA,  // the MMAs that read them have completed
    kBarDFull = kBarAFree + kRowTiles * kStagesA,  // + 64-block of the unit: its sums are complete in tensor memory
    kBarDFree = kBarDFull + 2,                     // the epilogue warps have read them
    kBarCount = kBarDFree + 2
};
static_assert(kBarCount <= 64, "barrier block too small");

// The tiles of a block. A block takes whole token blocks, gridDim.x apart, and walks the row blocks of each (so the
// blocks work on neighbouring token blocks, whose experts' weights and rows are shared in the L2, and nothing has
// to be looked up when only the row block changes); the token blocks that are left over are dealt out tile by tile.
// The entry of the token block after the current one is fetched ahead.
struct TileWalk {
    int tb, rb, tail, e, p0, live, ntok;   // tail: the tile among the left-over ones, or -1
    bool fresh;                            // the token block is another one than in the tile before
    int row_blocks, full, tail_tiles;      // full: token blocks taken whole
    int4 nxt;
    const int4* list;
    __device__ __forceinline__ void begin(const UmmaParams& p, int rows, int n_tb) {
        list = p.tb;
        row_blocks = rows;
        full = n_tb / int(gridDim.x) * int(gridDim.x);
        tail_tiles = (n_tb - full) * rows;
        tb = int(blockIdx.x) - int(gridDim.x);
        rb = rows - 1;
        tail = -1;
        fetch();
    }
    // the token block behind the current one, or -1
    __device__ __forceinline__ int following(int& t) const {
        t = tail;
        if (t < 0) {
            if (tb + int(gridDim.x) < full) return tb + int(gridDim.x);
            t = int(blockIdx.x);
        } else {
            t += int(gridDim.x);
        }
        return t < tail_tiles ? full + t / row_blocks : -1;
    }
    __device__ __forceinline__ void fetch() {
        int t;
        const int n = following(t);
        nxt = n >= 0 ? __ldg(list + n) : make_int4(0, 0, 0, 0);
    }
    __device__ __forceinline__ bool next() {
        fresh = false;
        if (tail < 0 && ++rb < row_blocks) return true;
        int t;
        const int n = following(t);
        if (n < 0) return false;
        tail = n >= full ? t : -1;
        tb = n;
        rb = tail >= 0 ? t % row_blocks : 0;
        fresh = true;
        // (the shuffles tell the compiler that the values are the same in all lanes)
        e = __shfl_sync(0xffffffffu, nxt.x, 0);
        p0 = __shfl_sync(0xffffffffu, nxt.y, 0);
        live = __shfl_sync(0xffffffffu, nxt.z, 0);
        ntok = __shfl_sync(0xffffffffu, nxt.w, 0);
        fetch();
        return true;
    }
    __device__ __forceinline__ int count() const {   // tiles of this block
        const int left = tail_tiles - int(blockIdx.x);
        return full / int(gridDim.x) * row_blocks + (left > 0 ? (left + int(gridDim.x) - 1) / int(gridDim.x) : 0);
    }
};

// 16 code words of 2 bits (the four bytes 4t .. 4t + 3 of a block of one row: field f of byte i is
// element 16 f + 4 t + i) -> the e4m3 bytes of q - 1 in the order of piece_byte: lo = fields 0, 1, hi =
// fields 2, 3. A byte permute looks four codes up at once in a table of four bytes.
__device__ __forceinline__ void codes_to_e4m3(uint32_t w, uint32_t* lo, uint32_t* hi) {
    constexpr uint32_t kTable = 0x403800B8u;   // -1, 0, 1, 2
    const uint32_t y = w & 0x33333333u, z = (w >> 2) & 0x33333333u;
    const uint32_t r0 = __byte_perm(kTable, 0u, y), r1 = __byte_perm(kTable, 0u, y >> 16);   // fields 0 and 2, interleaved
    const uint32_t q0 = __byte_perm(kTable, 0u, z), q1 = __byte_perm(kTable, 0u, z >> 16);   // fields 1 and 3
    lo[0] = __byte_perm(r0, r1, 0x6420);
    lo[1] = __byte_perm(q0, q1, 0x6420);
    hi[0] = __byte_perm(r0, r1, 0x7531);
    hi[1] = __byte_perm(q0, q1, 0x7531);
}

// The sums S0, S1 of NCH * 4 tokens for this thread's row of both row tiles: v[(r * 2 + s) * NCH * 4 + token].
// The loads and the wait for them are one statement, so that nothing that reads the registers can
// move in front of the wait and none of them is copied.
template <int NCH>
__device__ __forceinline__ void tmem_ld_sums(uint32_t t0, uint32_t (&v)[16 * NCH]);
template <>
__device__ __forceinline__ void tmem_ld_sums<1>(uint32_t t0, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%16];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4,%5,%6,%7}, [%17];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8,%9,%10,%11}, [%18];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%12,%13,%14,%15}, [%19];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(t0), "r"(t0 + kTileTok), "r"(t0 + kColsRow), "r"(t0 + kColsRow + kTileTok)
        : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld_sums<2>(uint32_t t0, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%33];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%34];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24,%25,%26,%27,%28,%29,%30,%31}, [%35];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(t0), "r"(t0 + kTileTok), "r"(t0 + kColsRow), "r"(t0 + kColsRow + kTileTok)
        : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld_sums<3>(uint32_t t0, uint32_t (&v)[48]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%48];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8,%9,%10,%11}, [%49];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%12,%13,%14,%15,%16,%17,%18,%19}, [%50];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%20,%21,%22,%23}, [%51];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24,%25,%26,%27,%28,%29,%30,%31}, [%52];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%32,%33,%34,%35}, [%53];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%36,%37,%38,%39,%40,%41,%42,%43}, [%54];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%44,%45,%46,%47}, [%55];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31]), "=r"(v[32]), "=r"(v[33]), "=r"(v[34]), "=r"(v[35]), "=r"(v[36]), "=r"(v[37]), "=r"(v[38]), "=r"(v[39]), "=r"(v[40]), "=r"(v[41]), "=r"(v[42]), "=r"(v[43]), "=r"(v[44]), "=r"(v[45]), "=r"(v[46]), "=r"(v[47])
        : "r"(t0), "r"(t0 + 8), "r"(t0 + kTileTok), "r"(t0 + kTileTok + 8), "r"(t0 + kColsRow), "r"(t0 + kColsRow + 8), "r"(t0 + kColsRow + kTileTok), "r"(t0 + kColsRow + kTileTok + 8)
        : "memory");
}

// acc += d * (a0 * S0 + a1 * S1) for two tokens, with the reference's roundings: a0 * S0 is exact, so the
// fused multiply-add rounds once; the multiply by d and the addition round separately. The multiply
// is written as a fused multiply-add of -0.0, which changes no value and which the assembler, not
// knowing the addend, cannot merge with the addition that follows.
__device__ __forceinline__ uint64_t scale_add(uint64_t acc, const ulonglong2& a, const uint32_t* s0, const uint32_t* s1, uint64_t dd, uint64_t neg0) {
    const uint64_t p0 = pack2(__uint_as_float(s0[0]), __uint_as_float(s0[1])), p1 = pack2(__uint_as_float(s1[0]), __uint_as_float(s1[1]));
    return add2(acc, fma2(dd, fma2(a.y, p1, mul2(a.x, p0)), neg0));
}

// What an epilogue warp does with the units of one tile; NCH chunks of 4 tokens per thread and block,
// for the thread's row of both row tiles (they share the tokens' scales).
struct EpiArgs {
    uint32_t bars, abort, smem_s;   // shared-memory addresses
    unsigned long long wait_ns;
    uint32_t taddr;                 // tensor memory: this warp's lanes, its first token column
    uint32_t tok_off, row_off;      // of the thread's first token pair and of its row inside a unit's scales
    int units;
    bool leader;                    // lane 0
    uint64_t neg0;
    // the tile's results: live tokens of this thread, whether the second row tile exists, where the first token's
    // value goes (gate/up) or its row of every slot starts and the slots are (down), bytes per token or slot
    int live;
    bool second;
    uint8_t* dst;
    uint32_t slots, step;
};
// (The stores are part of it: with the number of tokens known at compile time they are four to five instructions per
// token and row tile. Written once for any number they were thirty, and with all epilogue warps there at the same
// time a tile's end took some 2,000 cycles: a down tile's four units take 8,000.)
template <bool GATE_UP, int NCH>
__device__ __forceinline__ void epilogue_tile(const EpiArgs& q, uint32_t& gu, bool y_bf16) {
    uint64_t acc[4 * NCH];
#pragma unroll
    for (int i = 0; i < 4 * NCH; ++i) acc[i] = 0ull;
#pragma unroll 1
    for (int u = 0; u < q.units; ++u, ++gu) {
        const uint32_t ss = q.smem_s + (gu % kStagesS) * kUnitBytesS, bar_s = q.bars + (kBarSFull + gu % kStagesS) * 8;
        // the scales are complete long ago (the MMAs needed what arrives with them): tested so that this
        // thread acquires them; the test of the first block's sums goes out with it
        const bool ok_s = mbar_test_wait(bar_s, (gu / kStagesS) & 1u), ok_d = mbar_test_wait(q.bars + kBarDFull * 8, gu & 1u);
        if (!ok_s) mbar_spin(bar_s, (gu / kStagesS) & 1u, q.abort, q.wait_ns);
        const uint32_t e0 = lds32(ss + q.row_off), e1 = lds32(ss + q.row_off + kTileRows * 4);
        const __half2 dh0 = *reinterpret_cast<const __half2*>(&e0), dh1 = *reinterpret_cast<const __half2*>(&e1);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            uint32_t v[16 * NCH];
            if (j == 1 || !ok_d) mbar_spin(q.bars + (kBarDFull + j) * 8, gu & 1u, q.abort, q.wait_ns);
            tc_fence_after_sync();
            tmem_ld_sums<NCH>(q.taddr + j * kColsBlock, v);
            tc_fence_before_sync();
            if (q.leader) mbar_arrive(q.bars + (kBarDFree + j) * 8);   // the sums are all in registers: the accumulators go back
            const float d0 = j ? __high2float(dh0) : __low2float(dh0), d1 = j ? __high2float(dh1) : __low2float(dh1);
            const uint64_t dd0 = pack2(d0, d0), dd1 = pack2(d1, d1);
#pragma unroll
            for (int i = 0; i < 2 * NCH; ++i) {
                const ulonglong2 a = lds128(ss + q.tok_off + j * kBlockBytesS + i * 16);
                acc[i] = scale_add(acc[i], a, v + 2 * i, v + 4 * NCH + 2 * i, dd0, q.neg0);
                acc[2 * NCH + i] = scale_add(acc[2 * NCH + i], a, v + 8 * NCH + 2 * i, v + 12 * NCH + 2 * i, dd1, q.neg0);
            }
        }
    }
    // acc[r * 2 NCH + i]: the sums of row tile r for the thread's tokens 2 i, 2 i + 1
    constexpr uint32_t kNextF = GATE_UP ? 64 * 8 : kTileRows * 4, kNextH = kTileRows * 2;   // bytes from a row tile to the next: float (pairs), bf16
    uint8_t* d = q.dst;
#pragma unroll
    for (int i = 0; i < 2 * NCH; ++i) {
        float v[2][2];
        unpack2(acc[i], v[0][0], v[0][1]);
        unpack2(acc[2 * NCH + i], v[1][0], v[1][1]);
        uint2 sl;
        if (!GATE_UP) sl = lds64(q.slots + i * 8);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (!GATE_UP) d = q.dst + size_t(k ? sl.y : sl.x) * q.step;
            if (2 * i + k < q.live) {
                if (!GATE_UP && y_bf16) {
                    *reinterpret_cast<__nv_bfloat16*>(d) = __float2bfloat16_rn(v[0][k]);
                    if (q.second) *reinterpret_cast<__nv_bfloat16*>(d + kNextH) = __float2bfloat16_rn(v[1][k]);
                } else {
                    *reinterpret_cast<float*>(d) = v[0][k];
                    if (q.second) *reinterpret_cast<float*>(d + kNextF) = v[1][k];
                }
            }
            if (GATE_UP) d += q.step;
        }
    }
}

template <bool GATE_UP>
__global__ void __launch_bounds__(kThreads, 1) k_pf_umma(const UmmaParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr PfSmem sm = pf_smem();
    // (the shuffle tells the compiler that the value is the same in all lanes)
    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + sm.tmem);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + sm.abort);
    const uint32_t s0 = smem_u32(smem), bars = s0 + sm.bars, abort = s0 + sm.abort;
    const unsigned long long wait_ns = p.wait_ns;

    const int kdim = GATE_UP ? p.n : p.ff;
    const int units = kdim / kUnitK;
    const int row_tiles = GATE_UP ? (2 * p.ff) / kTileRows : p.n / kTileRows;
    const int row_blocks = (row_tiles + kRowTiles - 1) / kRowTiles;
    const uint32_t group_bytes = uint32_t(units) * kUnitBytes;
    const size_t section = GATE_UP ? 0 : size_t(p.ff / 8) * (size_t(p.n / kUnitK) * kUnitBytes);

    if (threadIdx.x == 0) {
        uint64_t* b = reinterpret_cast<uint64_t*>(smem + sm.bars);
        for (int i = 0; i < kStagesW; ++i) {
            mbar_init(b + kBarWFull + i, 1);
            mbar_init(b + kBarWFree + i, kWarpsDequant);
        }
        for (int i = 0; i < kStagesB; ++i) {
            mbar_init(b + kBarBFull + i, 1);
            mbar_init(b + kBarBFree + i, kRowTiles);
        }
        for (int i = 0; i < kStagesS; ++i) mbar_init(b + kBarSFull + i, 1 + kWarpsDequant);   // the activation warp, the dequant warps
        for (int i = 0; i < kRowTiles * kStagesA; ++i) {
            mbar_init(b + kBarAFull + i, kWarpsDequant / kRowTiles);
            mbar_init(b + kBarAFree + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(b + kBarDFull + i, kRowTiles);
            mbar_init(b + kBarDFree + i, kWarpsEpilogue);
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    pdl_wait();
    pdl_trigger();
    if (warp == 2) tmem_alloc(tmem_slot, kTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    TileWalk t;
    t.begin(p, row_blocks, p.meta[1]);

    // "free" barriers are waited on with the parity of the phase before the one about to be used,
    // which a fresh barrier reports as complete
    if (warp < kWarpsAux) {
        regs_dec<kRegsAux>();
        if (warp == 0) {
            // ---------------- packed weights: one lane per row group. A last row tile that does not exist
            // (n an odd multiple of 128) is computed as a copy of the one before and not stored.
            uint32_t g = 0;
            while (t.next()) {
                const int rt = min(t.rb * kRowTiles + ((lane >> 3) & 1), row_tiles - 1);
                const uint8_t* src = p.experts + size_t(t.e) * p.stride + section + size_t(rt * 8 + (lane & 7)) * group_bytes;
                for (int u = 0; u < units; ++u, ++g) {
                    const uint32_t ws = g % kStagesW, full = bars + (kBarWFull + ws) * 8;
                    mbar_spin(bars + (kBarWFree + ws) * 8, ((g / kStagesW) & 1u) ^ 1u, abort, wait_ns);
                    if (lane == 0) mbar_expect_tx(full, kUnitBytesW);
                    __syncwarp();
                    if (lane < 8 * kRowTiles) bulk_g2s(s0 + sm.w + ws * kUnitBytesW + lane * kUnitBytes, src + size_t(u) * kUnitBytes, kUnitBytes, full);
                }
            }
        } else if (warp == 1) {
            // ---------------- activations: the rows of the tile's tokens, gathered 16 bytes at a time (cp.async) into the MMA's
            // core-matrix order, their scales, and the tile's slots. A unit is handed on kLag units after its copies
            // were issued: they are generic-proxy writes, so each lane waits for its own and makes them visible to the
            // tensor core before the arrival. (A kernel that gathered the rows into this order in memory first took
            // 237 us at 163,840 slots of 2048 and made the products read 671 MB from HBM instead of the L2.)
            constexpr uint32_t kLag = 4;
            static_assert(kLag < kStagesB, "a unit must be handed on before its stage is needed again");
            const uint32_t dst_l = uint32_t(lane >> 3) * 128 + uint32_t(lane & 7) * 16;   // chunk lane / 8 of token lane % 8
            const size_t row_bytes = size_t(kdim) * 2, srow = size_t(kdim / kQ8);
            uint32_t g = 0, tb_no = 0;
            auto hand_on = [&](uint32_t u) {
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(bars + (kBarBFull + u % kStagesB) * 8);
                    mbar_arrive(bars + (kBarSFull + u % kStagesS) * 8);
                }
            };
            int row[kTileTok / 8];   // of token group i: the row of token lane % 8 (tokens beyond the live ones repeat the last)
#pragma unroll
            for (int i = 0; i < kTileTok / 8; ++i) row[i] = 0;
            while (t.next()) {
                const int groups = t.ntok >> 3;
                if (t.fresh) {
                    const uint32_t slots = s0 + sm.slots + (tb_no % kStagesS) * kTileTok * 4;
                    ++tb_no;
#pragma unroll
                    for (int i = 0; i < kTileTok / 8; ++i) {
                        const int pos = t.p0 + min(i * 8 + (lane & 7), t.live - 1);
                        const int slot = i < groups ? p.perm[pos] : 0;
                        row[i] = GATE_UP ? slot / p.K : pos;
                        if (!GATE_UP && i < groups && lane < 8) sts32(slots + (i * 8 + lane) * 4, uint32_t(slot));
                    }
                }
                for (int u = 0; u < units; ++u, ++g) {
                    const uint32_t bs = g % kStagesB, ss = g % kStagesS;
                    mbar_spin(bars + (kBarBFree + bs) * 8, ((g / kStagesB) & 1u) ^ 1u, abort, wait_ns);
                    const uint32_t db = s0 + sm.b + bs * kUnitBytesB + dst_l, ds = s0 + sm.s + ss * kUnitBytesS;
                    const uint8_t* src = p.act + size_t(u) * 256 + (lane >> 3) * 16;
                    const float* ssrc = p.act_scale + size_t(u) * 4 + (lane & 3);
#pragma unroll
                    for (int i = 0; i < kTileTok / 8; ++i) {
                        const int srow_i = __shfl_sync(0xffffffffu, row[i], lane >> 2);
                        if (i < groups) {
                            const uint8_t* r = src + size_t(row[i]) * row_bytes;
#pragma unroll
                            for (int c = 0; c < 4; ++c) cp_async16(db + (c >> 1) * kBlockBytesB + i * 1024 + (c & 1) * 512, r + c * 64);
                            // the scale of 32-block lane % 4 of the unit, of token lane / 4 of the group
                            cp_async4(ds + ((lane >> 1) & 1) * kBlockBytesS + (i * 4 + (lane >> 3)) * 16 + (lane & 1) * 8 + ((lane >> 2) & 1) * 4,
                                      ssrc + size_t(srow_i) * srow);
                        }
                    }
                    cp_async_commit();
                    cp_async_wait<kLag>();
                    if (g >= kLag) hand_on(g - kLag);
                }
            }
            cp_async_wait<0>();
            for (uint32_t u = g > kLag ? g - kLag : 0; u < g; ++u) hand_on(u);
        } else if (warp < 4) {
            // ---------------- MMA issuers, one warp per row tile; one elected lane issues, the warp stays together
            // (so that what it computes is known to be uniform)
            const int r = warp - 2;
            const uint64_t b_desc0 = umma_desc(s0 + sm.b, 128, 1024);
            uint32_t g = 0;
            while (t.next()) {
                const uint32_t idesc = umma_idesc_e4m3(kTileRows, t.ntok);
                for (int u = 0; u < units; ++u, ++g) {
                    const uint32_t bs = g % kStagesB, as = g % kStagesA;
                    const uint32_t bar_b = bars + (kBarBFull + bs) * 8, bar_a = bars + (kBarAFull + r * kStagesA + as) * 8, bar_d = bars + kBarDFree * 8;
                    const uint32_t pb = (g / kStagesB) & 1u, pa = (g / kStagesA) & 1u, pd = (g & 1u) ^ 1u;
                    // (a barrier test has a latency of tens of cycles and this warp is on the critical path:
                    // the three tests go out together, and the second block's in front of the first's MMAs)
                    const bool ok_b = mbar_test_wait(bar_b, pb), ok_a = mbar_test_wait(bar_a, pa), ok_d = mbar_test_wait(bar_d, pd);
                    if (!ok_b) mbar_spin(bar_b, pb, abort, wait_ns);
                    if (!ok_a) mbar_spin(bar_a, pa, abort, wait_ns);
                    if (!ok_d) mbar_spin(bar_d, pd, abort, wait_ns);
                    const bool ok_d1 = mbar_test_wait(bar_d + 8, pd);
                    const uint32_t a0 = tmem + kColA0 + as * kColsA + r * 32;
                    const uint64_t b0 = b_desc0 + uint64_t(bs * (kUnitBytesB >> 4));
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        if (j == 1 && !ok_d1) mbar_spin(bar_d + 8, pd, abort, wait_ns);
                        tc_fence_after_sync();
                        if (elect_one()) {
#pragma unroll
                            for (int s = 0; s < 2; ++s)
#pragma unroll
                                for (int piece = 0; piece < 2; ++piece)   // a 32-block: its multiples of 16, then its rests, into the same sums
                                    umma_f8_ta(tmem + j * kColsBlock + r * kColsRow + s * kTileTok, a0 + j * 16 + s * 8,
                                               b0 + uint64_t((j * kBlockBytesB + (s * 4 + piece * 2) * 128) >> 4), idesc, piece);
                            umma_commit(bars + (kBarDFull + j) * 8);
                            if (j == 1) {
                                umma_commit(bar_a + (kBarAFree - kBarAFull) * 8);
                                umma_commit(bar_b + (kBarBFree - kBarBFull) * 8);
                            }
                        }
                        __syncwarp();
                    }
                }
            }
        } else {
            // ---------------- dequant: packed 2-bit codes -> e4m3 (q - 1) in tensor memory, a thread per row
            const int r = (warp - 4) >> 2, row = (warp & 3) * 32 + lane;
            // of this row inside a stage of packed weights: code words [t] at 16 t, of block j at + 4 j; the two scales
            const uint32_t code_off = uint32_t(r) * kTileBytesW + uint32_t(row >> 4) * kUnitBytes + uint32_t(row & 7) * 64 + uint32_t((row >> 3) & 1) * 8;
            const uint32_t scale_off = uint32_t(r) * kTileBytesW + uint32_t(row >> 4) * kUnitBytes + kUnitCodeBytes + uint32_t(row & 7) * 8 + uint32_t((row >> 3) & 1) * 4;
            const uint32_t a_addr = tmem + (uint32_t((warp & 3) * 32) << 16) + kColA0 + r * 32;
            const uint32_t n_units = uint32_t(t.count()) * uint32_t(units);
            {
#pragma unroll 1
                for (uint32_t g = 0; g < n_units; ++g) {
                    const uint32_t ws = g % kStagesW, as = g % kStagesA, ss = g % kStagesS;
                    const uint32_t bar_w = bars + (kBarWFull + ws) * 8, bar_a = bars + (kBarAFull + r * kStagesA + as) * 8;
                    mbar_spin(bar_w, (g / kStagesW) & 1u, abort, wait_ns);
                    const bool ok_a = mbar_test_wait(bar_a + (kBarAFree - kBarAFull) * 8, ((g / kStagesA) & 1u) ^ 1u);
                    const uint32_t wsrc = s0 + sm.w + ws * kUnitBytesW;
                    uint2 wv[4];   // words of blocks 0, 1
#pragma unroll
                    for (int q = 0; q < 4; ++q) wv[q] = lds64(wsrc + code_off + q * 16);
                    sts32(s0 + sm.s + ss * kUnitBytesS + 2 * kBlockBytesS + (r * kTileRows + row) * 4, lds32(wsrc + scale_off));
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(bars + (kBarSFull + ss) * 8);
                        mbar_arrive(bar_w + (kBarWFree - kBarWFull) * 8);
                    }
                    if (!ok_a) mbar_spin(bar_a + (kBarAFree - kBarAFull) * 8, ((g / kStagesA) & 1u) ^ 1u, abort, wait_ns);
                    tc_fence_after_sync();
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        uint32_t o[16];   // the two halves of the block, eight columns each
#pragma unroll
                        for (int q = 0; q < 4; ++q) codes_to_e4m3(j ? wv[q].y : wv[q].x, o + 2 * q, o + 8 + 2 * q);
                        tmem_st16(a_addr + as * kColsA + j * 16, o);
                    }
                    tmem_st_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_a);
                }
            }
        }
    } else {
        // ---------------- epilogue
        regs_inc<kRegsEpilogue>();
        const int ew = warp - kWarpsAux;
        const int quarter = warp & 3;             // the tensor-memory lanes this warp may read
        const int row = quarter * 32 + lane;      // M row of the row tiles
        EpiArgs q;
        q.bars = bars;
        q.abort = abort;
        q.smem_s = s0 + sm.s;
        q.wait_ns = wait_ns;
        q.units = units;
        q.leader = lane == 0;
        q.row_off = 2 * kBlockBytesS + row * 4;
        q.neg0 = pack2(p.neg0, p.neg0);
        uint32_t g = 0, tb_no = 0;
        while (t.next()) {
            tb_no += t.fresh;   // (of the token blocks so far)
            const int share = t.ntok >> 2, nch = share >> 2;   // four warps share a row's tokens evenly
            const int tok0 = (ew >> 2) * share;
            q.tok_off = tok0 * 8;
            q.taddr = tmem + (uint32_t(quarter * 32) << 16) + uint32_t(tok0);
            q.live = t.live - tok0;
            const int rt = t.rb * kRowTiles;
            q.second = rt + 1 < row_tiles;
            if (GATE_UP) {
                // rows m < 8 of a group are gate rows, m >= 8 the up rows of the same ff rows: a
                // warp's 32 rows are 16 (gate, up) pairs, 128 contiguous bytes per token
                const int m = row & 15, ffrow = rt * 64 + (row >> 4) * 8 + (m & 7);
                q.dst = reinterpret_cast<uint8_t*>(p.hf) + (size_t(t.p0 + tok0) * p.ff + ffrow) * 8 + (m >> 3) * 4;
                q.step = uint32_t(p.ff) * 8;
            } else {
                const uint32_t size = p.y_bf16 ? 2 : 4;
                q.dst = reinterpret_cast<uint8_t*>(p.yd) + size_t(rt * kTileRows + row) * size;
                q.step = uint32_t(p.n) * size;
                q.slots = s0 + sm.slots + (((tb_no - 1) % kStagesS) * kTileTok + tok0) * 4;
            }
            switch (nch) {
                case 1: epilogue_tile<GATE_UP, 1>(q, g, p.y_bf16 != 0); break;
                case 2: epilogue_tile<GATE_UP, 2>(q, g, p.y_bf16 != 0); break;
                default: epilogue_tile<GATE_UP, 3>(q, g, p.y_bf16 != 0); break;
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag) {
        // A wait ran out: bulk copies and MMAs may still be in flight. Give them time to land
        // before tensor memory and the block's shared memory are released.
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) {
        }
        __syncthreads();
    }
    if (warp == 2) tmem_free(tmem, kTmemCols);
    if (threadIdx.x == 0 && *abort_flag) p.status[0] = kDevWaitTimeout;
}


int set_pf_attr() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    FRX_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= 0 && dev < 64 && done[dev]) return FRX_OK;
    FRX_CUDA(cudaFuncSetAttribute(k_pf_umma<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(pf_smem().total)));
    FRX_CUDA(cudaFuncSetAttribute(k_pf_umma<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(pf_smem().total)));
    if (dev >= 0 && dev < 64) done[dev] = true;
    return FRX_OK;
}

}  // namespace
}  // namespace frx

using namespace frx;

// Which form. The tensor-memory form pays per unit of 256 rows x 128 weights whatever the number of tokens in the tile, and its
// tiles (token blocks x blocks of 256 rows) are whole SMs' work; the streaming form reads an expert again for every eight
// tokens, but its tasks are small enough to fill the chip with any number of experts. So: 32 tokens per expert on average,
// and the shorter of two estimates in microseconds on 148 SMs:
//   tensor memory   units of K x 1.2 per tile and round of tiles over the SMs (at least one, on average half a round more than
//                   full ones), for either product, and 4 more than the other form for its launches;
//   streaming       0.02 + 0.26 (n ff / 2^20) per item of eight slots, of which an expert's last one is half full.
// Measured (us, uniform routing, streaming / tensor memory; slots per expert at 2048 / 512): one expert 64: 32 / 47, 255: 37 / 55;
// 4 experts 255: 60 / 64, 300: 65 / 64; 16 experts 96: 75 / 86, 200: 122 / 113; 32 experts 40: 72 / 68; 64 experts 32: 97 / 95,
// 64: 153 / 140; 512 experts 24: 420 / 393, 32: 531 / 435. 512 / 256: 4 experts 255: 37 / 40, 16 experts 128: 45 / 42, 64 experts
// 32: 45 / 42. 2560 / 640: one expert 96: 36 / 58, 64 experts 64: 218 / 194. Of 900 such points the estimate is off the faster
// form by 0.7 % on average and 15 % at most; the mean number of tokens alone was off by 62 % (one expert).
// With skewed routing the forms meet at the same mean.
constexpr int kUmmaMinTokensPerExpert = 32;
static bool umma_pays(long long slots, int E, int n, int ff) {
    if (slots < (long long)kUmmaMinTokensPerExpert * E) return false;
    const double sms = std::max(sm_count(), 1), blocks = double(slots) / kTileTok + 0.5 * E, items = double(slots) / kTokPerItem + 0.5 * E;
    auto rounds = [&](int row_blocks) { return std::max(1.0, blocks * row_blocks / sms + 0.5); };
    const int row_tiles = n / kTileRows;
    const double umma = 1.2 * (rounds(2 * ff / (kRowTiles * kTileRows)) * (n / kUnitK) + rounds((row_tiles + 1) / 2) * (ff / kUnitK));
    const double stream = items * (0.02 + 0.26 * double(n) * ff / (1 << 20)) * (148.0 / sms);
    return umma + 4.0 < stream || !prefill_stream_fits(n, ff);
}

extern "C" {

// the streaming form lives in frx_decode.cu
size_t frx_moe_prefill_stream_workspace_bytes(int T, int K, int n, int ff, int E);
int frx_moe_prefill_stream_ex(const void* experts, size_t stride, int E, int n, int ff, const float* x, const int32_t* ids, int T, int K,
                              void* yd, void* ws, size_t ws_bytes, frx_stream_t stream, int block64, int yd_bf16);
int frx_moe_prefill_stream_q8_ep(const void* experts_local, size_t stride, int E_local, const int32_t* e_map, int E_all, int n, int ff,
                                 const int8_t* xq, const float* xd, const int32_t* ids, int T, int K, float* yd, void* ws, size_t ws_bytes,
                                 frx_stream_t stream);

int frx_moe_prefill_form(int T, int K, int n, int ff, int E, int E_local) {
    if (T < 1 || K < 1 || E < 1 || E_local < 1) return 1;
    return umma_pays((long long)T * K * E_local / E, E_local, n, ff) ? 2 : 1;
}

size_t frx_moe_prefill_umma_workspace_bytes(int T, int K, int n, int ff, int E) {
    if (T < 1 || K < 1 || n < kUnitK || ff < kUnitK || E < 1) return 0;
    return pfu_layout(T, K, n, ff, E).total;
}

int frx_moe_prefill_umma(const void* experts, size_t stride, int E, int n, int ff, const float* x, const int32_t* ids, int T, int K,
                         float* yd, void* ws, size_t ws_bytes, frx_stream_t stream) {
    return frx_moe_prefill_umma_ex(experts, stride, E, n, ff, x, ids, T, K, yd, ws, ws_bytes, stream, 0, 0);
}

static void quant_h(const float2* hf, const int* n_rows, int max_rows, int ff, uint8_t* he, float* hd, int block64, frx_stream_t stream) {
    const size_t groups = size_t(max_rows) * size_t(ff / 8);
    FRX_LAUNCH(kKQuant, stream, launch_pdl(k_pfu_quant_h, dim3(unsigned((groups + 255) / 256)), dim3(256), 0, stream, hf, ff, n_rows, he, hd, block64));
}

int frx_debug_quantize_hidden(const float* pairs, const int* n_rows, int max_rows, int ff, void* pieces, float* scales, int block64, frx_stream_t stream) {
    if (!pairs || !n_rows || !pieces || !scales) return fail(FRX_ERR_ARG, "frx_debug_quantize_hidden: null pointer");
    if (max_rows < 0 || max_rows > 1 << 20 || ff < kUnitK || ff % kUnitK || ff > 8192) return fail(FRX_ERR_SHAPE, "frx_debug_quantize_hidden: %d rows of %d", max_rows, ff);
    if ((uintptr_t(pairs) | uintptr_t(pieces)) % 16 || uintptr_t(scales) % 4) return fail(FRX_ERR_ARG, "frx_debug_quantize_hidden: pairs and pieces must be 16-byte aligned");
    if (max_rows == 0) return FRX_OK;
    quant_h(reinterpret_cast<const float2*>(pairs), n_rows, max_rows, ff, static_cast<uint8_t*>(pieces), scales, block64, stream);
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

static int prefill_umma_impl(const void* experts, size_t stride, int E, const int32_t* e_map, int E_all, int n, int ff, const float* x,
                             const int8_t* xq_in, const float* xd_in, const int32_t* ids, int T, int K, void* yd, void* ws, size_t ws_bytes,
                             frx_stream_t stream, int block64, int yd_bf16) {
    if (!experts || !ids || !yd || !ws) return fail(FRX_ERR_ARG, "frx_moe_prefill: null pointer");
    if (n < kUnitK || ff < kUnitK || n % kUnitK || ff % kUnitK || n > 8192 || ff > 8192)
        return fail(FRX_ERR_SHAPE, "frx_moe_prefill: n %d and ff %d must be multiples of %d, at most 8192", n, ff, kUnitK);
    if (K < 1 || K > 32 || T < 0 || E < 1 || E > 4096 || E_all < E || E_all > 4096 || size_t(T) * K > (size_t(1) << 28))
        return fail(FRX_ERR_SHAPE, "frx_moe_prefill: unsupported T %d, K %d, E %d", T, K, E);
    if ((uintptr_t(experts) | stride) % 16 || uintptr_t(ws) % kAlign)
        return fail(FRX_ERR_ARG, "frx_moe_prefill: experts and stride must be 16-byte aligned, ws 256-byte aligned");
    if (uintptr_t(x) % 16 || uintptr_t(xq_in) % 4) return fail(FRX_ERR_ARG, "frx_moe_prefill: x must be 16-byte aligned, xq 4-byte aligned");
    if (stride < frx_q2_expert_bytes(n, ff)) return fail(FRX_ERR_ARG, "frx_moe_prefill: stride %zu < blob %zu", stride, frx_q2_expert_bytes(n, ff));
    if (T == 0) return FRX_OK;
    const PfuLayout L = pfu_layout(T, K, n, ff, E);
    if (ws_bytes < L.total) return fail(FRX_ERR_WORKSPACE, "frx_moe_prefill: workspace %zu < %zu", ws_bytes, L.total);
    if (int rc = set_pf_attr()) return rc;
    auto* base = static_cast<uint8_t*>(ws);
    int* status = reinterpret_cast<int*>(base + L.status);
    int* chunk_cnt = reinterpret_cast<int*>(base + L.chunk_cnt);
    int* bounds = reinterpret_cast<int*>(base + L.bounds);
    int* item_off = reinterpret_cast<int*>(base + L.item_off);
    int32_t* perm = reinterpret_cast<int32_t*>(base + L.perm);
    int* meta = reinterpret_cast<int*>(base + L.meta);
    int4* tb = reinterpret_cast<int4*>(base + L.tb);
    const int S = T * K;
    uint8_t* xe = base + L.xe;
    float* xd = reinterpret_cast<float*>(base + L.xd);
    const size_t nquads = size_t(T) * (n / 4);
    const unsigned qgrid = unsigned((nquads + 255) / 256);
    if (xq_in)   // the activations arrived already quantized
        FRX_LAUNCH(kKQuant, stream, launch_pdl(k_pfu_expand_q8, dim3(qgrid), dim3(256), 0, stream, xq_in, nquads, xe));
    else
        FRX_LAUNCH(kKQuant, stream, launch_pdl(k_pfu_quant_x, dim3(qgrid), dim3(256), 0, stream, x, nquads, xe, xd, block64));
    FRX_LAUNCH(kKGroup, stream, launch_pdl(k_pf_hist, dim3(L.n_chunks), dim3(256), size_t(E) * 4, stream, ids, S, E, chunk_cnt, status, e_map, E_all));
    FRX_LAUNCH(kKGroup, stream, launch_pdl(k_pf_scan, dim3(1), dim3(1024), 0, stream, chunk_cnt, L.n_chunks, E, bounds, item_off, status, 1 << 30, kTokPerItem,
                                           TokenBlocks{kTileTok, kTokPad, meta, tb, L.max_tb}));
    FRX_LAUNCH(kKGroup, stream, launch_pdl(k_pf_place, dim3(L.n_chunks), dim3(kChunkSlots), pf_place_smem(E), stream, ids, S, E, (const int*)chunk_cnt, (const int*)bounds, perm, e_map, E_all));
    UmmaParams p{};
    p.experts = static_cast<const uint8_t*>(experts);
    p.stride = stride;
    p.meta = meta;
    p.tb = tb;
    p.perm = perm;
    p.hf = reinterpret_cast<float2*>(base + L.hf);
    p.yd = static_cast<float*>(yd);
    p.y_bf16 = yd_bf16 ? 1 : 0;
    p.status = status;
    p.wait_ns = wait_limit_ns();
    p.neg0 = -0.0f;
    p.n = n;
    p.ff = ff;
    p.K = K;
    const dim3 blocks{unsigned(sm_count())};
    p.act = xe;
    p.act_scale = xq_in ? xd_in : xd;
    FRX_LAUNCH(kKGateUp, stream, launch_pdl(k_pf_umma<true>, blocks, dim3(kThreads), pf_smem().total, stream, p));
    quant_h(p.hf, bounds + E, S, ff, base + L.he, reinterpret_cast<float*>(base + L.hd), block64, stream);
    p.act = base + L.he;
    p.act_scale = reinterpret_cast<const float*>(base + L.hd);
    FRX_LAUNCH(kKDown, stream, launch_pdl(k_pf_umma<false>, blocks, dim3(kThreads), pf_smem().total, stream, p));
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

int frx_moe_prefill_umma_ex(const void* experts, size_t stride, int E, int n, int ff, const float* x, const int32_t* ids, int T, int K,
                            void* yd, void* ws, size_t ws_bytes, frx_stream_t stream, int block64, int yd_bf16) {
    if (!x) return fail(FRX_ERR_ARG, "frx_moe_prefill: null pointer");
    return prefill_umma_impl(experts, stride, E, nullptr, E, n, ff, x, nullptr, nullptr, ids, T, K, yd, ws, ws_bytes, stream, block64, yd_bf16);
}

// ---- expert-parallel prefill on activations that arrive quantized: this rank holds E_local
// experts (e_map[id] = index here, or -1), the T tokens are all the tokens whose slots may land here
int frx_moe_prefill_q8_ep(const void* experts_local, size_t stride, int E_local, const int32_t* e_map, int E_all, int n, int ff,
                          const int8_t* xq, const float* xd, const int32_t* ids, int T, int K, float* yd, void* ws, size_t ws_bytes,
                          frx_stream_t stream, int form) {
    if (!xq || !xd || !e_map) return fail(FRX_ERR_ARG, "frx_moe_prefill_q8_ep: null pointer");
    if (form < 0 || form > 2) return fail(FRX_ERR_ARG, "frx_moe_prefill_q8_ep: form %d", form);
    // the expected number of slots per local expert is T * K / E_all (the counts stay on the device)
    const bool umma = form == 2 || (form == 0 && frx_moe_prefill_form(T, K, n, ff, E_all, E_local) == 2);
    if (umma) return prefill_umma_impl(experts_local, stride, E_local, e_map, E_all, n, ff, nullptr, xq, xd, ids, T, K, yd, ws, ws_bytes, stream, 0, 0);
    return frx_moe_prefill_stream_q8_ep(experts_local, stride, E_local, e_map, E_all, n, ff, xq, xd, ids, T, K, yd, ws, ws_bytes, stream);
}

// ---- the public entry: both forms compute the same bits, see umma_pays

size_t frx_moe_prefill_workspace_bytes(int T, int K, int n, int ff, int E) {
    const size_t a = frx_moe_prefill_stream_workspace_bytes(T, K, n, ff, E), b = frx_moe_prefill_umma_workspace_bytes(T, K, n, ff, E);
    if (!a || !b) return 0;
    return a > b ? a : b;
}

int frx_moe_prefill(const void* experts, size_t stride, int E, int n, int ff, const float* x, const int32_t* ids, int T, int K,
                    float* yd, void* ws, size_t ws_bytes, frx_stream_t stream) {
    return frx_moe_prefill_ex(experts, stride, E, n, ff, x, ids, T, K, yd, ws, ws_bytes, stream, 0, 0);
}

int frx_moe_prefill_ex(const void* experts, size_t stride, int E, int n, int ff, const float* x, const int32_t* ids, int T, int K,
                       void* yd, void* ws, size_t ws_bytes, frx_stream_t stream, int block64, int yd_bf16) {
    if (frx_moe_prefill_form(T, K, n, ff, E, E) == 2)
        return frx_moe_prefill_umma_ex(experts, stride, E, n, ff, x, ids, T, K, yd, ws, ws_bytes, stream, block64, yd_bf16);
    return frx_moe_prefill_stream_ex(experts, stride, E, n, ff, x, ids, T, K, yd, ws, ws_bytes, stream, block64, yd_bf16);
}

}  // extern "C"
