// Q2_0 storage on the device: ggml -> planar repack, planar <-> tiled relayout, dequantisation.
// All three are pure permutations or element-wise decodes, so they are bit-exact by construction;
// the tests check them against the CPU oracle byte for byte.
#include "frx_common.cuh"

#include <algorithm>

namespace frx {
namespace {

// ---- q2_0::repack (quant/q2_0/q2_0.cpp:34-39,51-62): one thread per output 32-bit word.
// Planar word w of a block (bytes 4w..4w+3) takes, for g = 0..3, the four 2-bit fields of ggml
// code byte 4g + w and puts them at bit 2g of its four bytes.
__global__ void k_repack(const uint8_t* __restrict__ ggml, size_t nblk, uint8_t* __restrict__ planar) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;   // (block, word)
    if (i >= nblk * 4) return;
    const size_t blk = i >> 2;
    const int w = int(i & 3);
    const uint8_t* b = ggml + blk * kBlockBytes;
    uint32_t out = 0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        const uint32_t byte = b[2 + 4 * g + w];
        const uint32_t spread = (byte & 3u) | ((byte >> 2) & 3u) << 8 | ((byte >> 4) & 3u) << 16 | ((byte >> 6) & 3u) << 24;
        out |= spread << (2 * g);
    }
    reinterpret_cast<uint32_t*>(planar)[i] = out;
    if (w == 0) reinterpret_cast<uint16_t*>(planar + nblk * 16)[blk] = uint16_t(b[0]) | uint16_t(b[1]) << 8;
}

// Geometry of one tiled expert.
struct Geo {
    int n, ff;
    int gu_groups, gu_units;   // ff/8 groups of n/128 units
    int dn_groups, dn_units;   // n/16 groups of ff/128 units
    size_t gu_mat;             // bytes of one planar gate/up matrix
    __host__ __device__ Geo(int n_, int ff_)
        : n(n_), ff(ff_), gu_groups(ff_ / 8), gu_units(n_ / kUnitK), dn_groups(n_ / 16), dn_units(ff_ / kUnitK),
          gu_mat(size_t(ff_) * (n_ / kQK) * kBlockBytes) {}
    __host__ __device__ size_t total_units() const { return size_t(gu_groups) * gu_units + size_t(dn_groups) * dn_units; }
};

// A warp per unit: lane L moves the 16 bytes of codes of lane L, lanes 0..15 a scale word each (two fp16).
// Neighbouring warps of a block take neighbouring units, i.e. the same matrix rows further along K, so
// the 32 bytes a row gives to a unit share their lines in the L1. TO_TILED: planar -> tiled;
// otherwise tiled -> planar. Bound: HBM, two passes over the weights. (A thread per word, each with its own
// 64-bit divisions to find its place, took twice as long.)
template <bool TO_TILED>
__global__ void __launch_bounds__(256) k_tile(const uint8_t* __restrict__ src, size_t src_stride, uint8_t* __restrict__ dst, size_t dst_stride, int n, int ff,
                                              int units_per_expert, int n_experts) {
    const int unit = blockIdx.x * 8 + int(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (unit >= units_per_expert) return;
    const Geo G(n, ff);
    const int gu_total = G.gu_groups * G.gu_units;
    const bool gu = unit < gu_total;
    const int k = gu ? unit : unit - gu_total, per = gu ? G.gu_units : G.dn_units, grp = k / per, u = k - grp * per;
    const int nb = (gu ? n : ff) / kQK, rows = gu ? ff : n;
    // M row m of the unit: gate rows, then up rows (m >= 8), or 16 down rows
    auto mat_row = [&](int m, size_t& mat) {
        mat = gu ? (m < 8 ? 0 : G.gu_mat) : 2 * G.gu_mat;
        return gu ? grp * 8 + (m & 7) : grp * 16 + m;
    };
    const int g = lane >> 2, t = lane & 3;
    size_t code_off[2], scale_off = 0;   // of the planar blob: block 2u of rows g, g + 8 (this lane's word); its scale word
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        size_t mat;
        const int row = mat_row(g + 8 * h, mat);
        code_off[h] = mat + (size_t(row) * nb + 2 * u) * 16 + size_t(t) * 4;
    }
    if (lane < 16) {   // scale word s holds [g = s / 2][h = s % 2][j = 0, 1]
        size_t mat;
        const int row = mat_row((lane >> 1) + 8 * (lane & 1), mat);
        scale_off = mat + size_t(rows) * nb * 16 + (size_t(row) * nb + 2 * u) * 2;
    }
    const size_t tiled_off = size_t(unit) * kUnitBytes;
    for (int e = blockIdx.y; e < n_experts; e += gridDim.y) {
        const uint8_t* s = src + size_t(e) * src_stride;
        uint8_t* d = dst + size_t(e) * dst_stride;
        if (TO_TILED) {
            uint4 v;
            v.x = *reinterpret_cast<const uint32_t*>(s + code_off[0]);
            v.y = *reinterpret_cast<const uint32_t*>(s + code_off[0] + 16);
            v.z = *reinterpret_cast<const uint32_t*>(s + code_off[1]);
            v.w = *reinterpret_cast<const uint32_t*>(s + code_off[1] + 16);
            uint32_t* o = reinterpret_cast<uint32_t*>(d + tiled_off);
            if (uintptr_t(o) % 16 == 0) {
                reinterpret_cast<uint4*>(o)[lane] = v;
            } else {
                o[lane * 4] = v.x, o[lane * 4 + 1] = v.y, o[lane * 4 + 2] = v.z, o[lane * 4 + 3] = v.w;
            }
            if (lane < 16) o[128 + lane] = *reinterpret_cast<const uint32_t*>(s + scale_off);
        } else {
            const uint32_t* i = reinterpret_cast<const uint32_t*>(s + tiled_off);
            *reinterpret_cast<uint32_t*>(d + code_off[0]) = i[lane * 4];
            *reinterpret_cast<uint32_t*>(d + code_off[0] + 16) = i[lane * 4 + 1];
            *reinterpret_cast<uint32_t*>(d + code_off[1]) = i[lane * 4 + 2];
            *reinterpret_cast<uint32_t*>(d + code_off[1] + 16) = i[lane * 4 + 3];
            if (lane < 16) *reinterpret_cast<uint32_t*>(d + scale_off) = i[128 + lane];
        }
    }
}

// Dequantise one matrix of a tiled expert: one thread per (row, block), 64 floats out.
// which: 0 gate, 1 up, 2 down.
__global__ void k_dequant(const uint8_t* __restrict__ blob, int n, int ff, int which, float* __restrict__ out) {
    const int rows = which == 2 ? n : ff, cols = which == 2 ? ff : n, nb = cols / kQK;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * nb) return;
    const int row = i / nb, b = i % nb, u = b >> 1, j = b & 1;
    const Geo G(n, ff);
    size_t unit;
    int m;
    if (which == 2) {
        unit = size_t(G.gu_groups) * G.gu_units + size_t(row / 16) * G.dn_units + u;
        m = row % 16;
    } else {
        unit = size_t(row / 8) * G.gu_units + u;
        m = (row % 8) + (which == 1 ? 8 : 0);
    }
    const uint8_t* up = blob + unit * kUnitBytes;
    const int g = m & 7, h = m >> 3;
    const __half d = *reinterpret_cast<const __half*>(up + kUnitCodeBytes + g * 8 + (h * 2 + j) * 2);
    const float df = __half2float(d);
    float* o = out + size_t(row) * cols + size_t(b) * kQK;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const uint32_t word = *reinterpret_cast<const uint32_t*>(up + (g * 4 + t) * 16 + (h * 2 + j) * 4);
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int q = int((word >> (8 * k + 2 * p)) & 3u);
                o[16 * p + 4 * t + k] = __fmul_rn(float(q - 1), df);
            }
    }
}

int check_shape(const char* who, int n, int ff) {
    if (n < kUnitK || ff < kUnitK || n % kUnitK || ff % kUnitK)
        return fail(FRX_ERR_SHAPE, "%s: n %d and ff %d must be positive multiples of %d", who, n, ff, kUnitK);
    return FRX_OK;
}

template <bool TO_TILED>
int tile_launch(const char* who, const void* src, size_t src_stride, void* dst, size_t dst_stride, int n_experts, int n, int ff,
                cudaStream_t stream) {
    if (!src || !dst) return fail(FRX_ERR_ARG, "%s: null pointer", who);
    if (n_experts < 0) return fail(FRX_ERR_ARG, "%s: n_experts %d", who, n_experts);
    if (int rc = check_shape(who, n, ff)) return rc;
    const size_t blob = frx_q2_expert_bytes(n, ff);
    if (src_stride < blob || dst_stride < blob || (src_stride | dst_stride) % 4 || (uintptr_t(src) | uintptr_t(dst)) % 4)
        return fail(FRX_ERR_ARG, "%s: strides %zu / %zu must be >= %zu and, like the pointers, 4-byte aligned", who, src_stride,
                    dst_stride, blob);
    if (n_experts == 0) return FRX_OK;
    const Geo G(n, ff);
    const int units = int(G.total_units());
    k_tile<TO_TILED><<<dim3(unsigned((units + 7) / 8), unsigned(std::min(n_experts, 65535))), 256, 0, stream>>>(
        static_cast<const uint8_t*>(src), src_stride, static_cast<uint8_t*>(dst), dst_stride, n, ff, units, n_experts);
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

}  // namespace
}  // namespace frx

using namespace frx;

extern "C" {

int frx_q2_repack(const void* ggml_rows, int rows, int cols, void* planar, frx_stream_t stream) {
    if (!ggml_rows || !planar) return fail(FRX_ERR_ARG, "frx_q2_repack: null pointer");
    if (rows < 0 || cols < kQK || cols % kQK) return fail(FRX_ERR_SHAPE, "frx_q2_repack: rows %d, cols %d", rows, cols);
    if (uintptr_t(planar) % 4) return fail(FRX_ERR_ARG, "frx_q2_repack: planar must be 4-byte aligned");
    const size_t nblk = size_t(rows) * (cols / kQK);
    if (nblk == 0) return FRX_OK;
    k_repack<<<unsigned((nblk * 4 + 255) / 256), 256, 0, stream>>>(static_cast<const uint8_t*>(ggml_rows), nblk,
                                                                  static_cast<uint8_t*>(planar));
    FRX_CUDA(cudaGetLastError());
    return FRX_OK;
}

int frx_q2_tile_experts(const void* src_planar, size_t src_stride, void* dst_tiled, size_t dst_stride, int n_experts, int n,
                        int ff, frx_stream_t stream) {
    return tile_launch<true>("frx_q2_tile_experts", src_planar, src_stride, dst_tiled, dst_stride, n_experts, n, ff, stream);
}

int frx_q2_untile_experts(const void* src_tiled, size_t src_stride, void* dst_planar, size_t dst_stride, int n_experts, int n,
                          int ff, frx_stream_t stream) {
    return tile_launch<false>("frx_q2_untile_experts", src_tiled, src_stride, dst_planar, dst_stride, n_experts, n, ff, stream);
}

int frx_q2_dequant_expert(const void* tiled_blob, int n, int ff, float* gate, float* up, float* down, frx_stream_t stream) {
    if (!tiled_blob) return fail(FRX_ERR_ARG, "frx_q2_dequant_expert: null blob");
    if (int rc = check_shape("frx_q2_dequant_expert", n, ff)) return rc;
    if (uintptr_t(tiled_blob) % 16) return fail(FRX_ERR_ARG, "frx_q2_dequant_expert: blob must be 16-byte aligned");
    float* outs[3] = {gate, up, down};
    for (int which = 0; which < 3; ++which) {
        if (!outs[which]) continue;
        const int rows = which == 2 ? n : ff, nb = (which == 2 ? ff : n) / kQK;
        k_dequant<<<(rows * nb + 127) / 128, 128, 0, stream>>>(static_cast<const uint8_t*>(tiled_blob), n, ff, which, outs[which]);
        FRX_CUDA(cudaGetLastError());
    }
    return FRX_OK;
}

}  // extern "C"
