// The decode layer for few tokens as two kernels. Include inside namespace frx { namespace { ... } }
// after the quantizers, the Item definitions and frx_route.cuh.
//
// With a few tokens the layer is a chain of dependent latencies over 10 to 40 MB of weights: route, group,
// quantize, gate/up, quantize, down, combine. Everything small is done again by every block instead of
// once by one block with a kernel boundary behind it:
//   k_small_up    every block routes all tokens, groups the slots into items of at most two tokens,
//                 quantizes x into its own shared memory, and takes tasks of 32 hidden values (four row
//                 groups) of one item; the hidden values are formed and quantized where they are made.
//   k_small_down  every block routes and groups again while k_small_up is still running (the logits
//                 were complete before it) and brings its weights into shared memory; it owns 16 output
//                 rows of every item, so the weighted sum over a token's experts needs no other block.
// Both split K over warps: the terms d * (a0 * S0 + a1 * S1) of a row's blocks are independent, only their sum
// has an order. The terms go through shared memory and one thread per (row, token) adds them in block
// order, so a slot's row is the same bits as that of k_stream. (Routing weights may differ from k_route_topk's in their last
// bit: the double-precision softmax sum is added in another order.) Four row groups (up) or four items (down)
// are chained into one accumulator as in units_mma_n2.

constexpr int kSmallTok = 2;                          // tokens of an item
constexpr int kSmallMaxT = 8, kSmallMaxSlots = 96;    // tokens, and routed slots
constexpr int kUpProd = 8, kUpThreads = (kUpProd + 4 + 1) * 32;        // 8 warps of products, 4 of sums, 1 that fetches weights
constexpr int kUpHelpers = 64;                        // threads that only quantize x: see launch_small
constexpr int kUpBarThreads = (kUpProd + 4) * 32;
constexpr int kDnProd = 12, kDnThreads = (kDnProd + 1) * 32;
constexpr int kSmallGroups = 3;                       // tokens routed at a time, by four warps each
// Registers: blocks of both kernels are to be resident side by side, 480 + 416 threads of at most 72. (Two more warps of products
// instead of the two that only quantize: 5 units of 16 on one scheduler instead of 4, 2 % slower at three tokens.) (16 warps of products and
// 64 registers, with spills, were measured: 14.6 us per layer against 13.3 for one token, no gain for three.)

struct SmallParams {
    const float* logits;          // router input, or null: ids / wts are given
    const int32_t* ids;           // [T][K] (without logits)
    const float* wts;
    const uint8_t* const* hit_ptr;   // moe_hits: [T][K] expert blobs, hit_n[t] of them live (else null)
    const int32_t* hit_n;
    int32_t* ids_out;             // with logits: the routing, written by one block
    float* wts_out;
    const uint8_t* experts;
    size_t stride;
    const uint8_t* shared;        // shared expert, or null
    const float* x;               // [T][n]
    const float* gate_logit;      // [T] or null
    int8_t* xq;                   // the Q8 form of x as the workspace documents it, written by one block (or null)
    float* xa;
    float* xc;
    int8_t* hq;                   // [slots][ff] hidden codes in fragment order
    float4* hs;                   // [slots][ff / 64] {a0, a1 / 16, -(kMagic + sum of codes) of both halves}
    float* out;                   // [T][n] (not moe_hits)
    float* y;                     // [T * K][n] per-slot rows, or null
    int* status;
    unsigned long long wait_ns;
    int T, K, E, n, ff;
    int ring;                     // k_small_up: tasks in the weight ring; k_small_down: quads of items
    int tbufs;                    // k_small_up: buffers of terms (1 or 2)
};

// Loads of the routing inputs. k_small_down makes them before its wait, while the kernel in front still runs, and the same
// addresses are rewritten from layer to layer and step to step: they are complete in the L2 by then (the kernel in front waited
// for whatever wrote them before it let this one start), but this SM's L1 may still hold the lines that an earlier layer
// read. So they bypass it. (A few hundred words per block, none read twice from here: eight layers of 2048 / 512 take one token
// 111.3 us through the L1 and 110.8 past it, three tokens 200.7 and 201.1.)
__device__ __forceinline__ float ld_l2(const float* p) {
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_l2(const float4* p) {
    float4 v;
    asm volatile("ld.global.cg.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ int32_t ld_l2(const int32_t* p) {
    int32_t v;
    asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ const uint8_t* ld_l2(const uint8_t* const* p) {
    const uint8_t* v;
    asm volatile("ld.global.cg.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}

// What every block works out for itself.
struct SmallItem {
    const uint8_t* blob;
    int m;
    int slot[kSmallTok], tok[kSmallTok];
};
struct __align__(16) SmallRoute {
    uint32_t lm[128];                    // the largest key of every thread
    unsigned long long cand[256];        // the candidates: key, then the complement of the expert (ties to the lower one)
    double sum[4];
    uint32_t wmax[4];
    float p[32];
};
struct SmallPlan {
    int32_t ids[kSmallMaxSlots + 4];     // expert of every routed slot (-1: dead), padded to a multiple of four with -1
    int32_t start[kSmallMaxSlots + 4];   // the expert where a slot is the first of an item, else a large number
    float wts[kSmallMaxSlots];
    const uint8_t* ptr[kSmallMaxSlots];  // moe_hits: the expert of every routed slot (null: dead)
    SmallItem item[kSmallMaxSlots + kSmallMaxT / kSmallTok + 4];
    int16_t ord[kSmallMaxSlots];         // a token's slots by ascending expert id
    int n_items;
};

// The K most probable experts of every token, by G groups of four warps (the order and the ties are
// route_warp's). A thread holds VT consecutive logits (E <= 128 VT). An expert among the first K of all is
// in a thread whose largest logit is among the first K largest ones, so: the rank of a thread's
// largest among the 128 by counting, the VT K logits of the threads that rank below K, their ranks by
// counting again. Two barriers of four warps instead of K dependent rounds of reductions (hidden 2048, 512 experts, one
// token: 4.0 us from the wait to the ids before).
// weights: also the softmax weights (k_small_down, and the block that reports them).
template <int VT, int G>
__device__ __forceinline__ void small_route(const SmallParams& p, SmallPlan& s, SmallRoute* route, bool weights) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = warp >> 2, gw = warp & 3, gl = gw * 32 + lane;
    if (group >= G) return;
    SmallRoute& r = route[group];
    for (int t = group; t < p.T; t += G) {
        const float* l = p.logits + size_t(t) * p.E;
        uint32_t key[VT];
        const int e0 = gl * VT;
        if (VT % 4 == 0 && p.E % 4 == 0 && uintptr_t(p.logits) % 16 == 0) {
#pragma unroll
            for (int q = 0; q < VT / 4; ++q) {
                const bool in = e0 + 4 * q < p.E;
                const float4 v = in ? ld_l2(reinterpret_cast<const float4*>(l + e0 + 4 * q)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                key[(4 * q) % VT] = in ? order_key(v.x + 0.0f) : 0u;
                key[(4 * q + 1) % VT] = in ? order_key(v.y + 0.0f) : 0u;
                key[(4 * q + 2) % VT] = in ? order_key(v.z + 0.0f) : 0u;
                key[(4 * q + 3) % VT] = in ? order_key(v.w + 0.0f) : 0u;
            }
        } else {
#pragma unroll
            for (int i = 0; i < VT; ++i) key[i] = e0 + i < p.E ? order_key(ld_l2(l + e0 + i) + 0.0f) : 0u;
        }
        uint32_t lm = key[0];
#pragma unroll
        for (int i = 1; i < VT; ++i) lm = max(lm, key[i]);
        r.lm[gl] = lm;
        if (weights) {
            const uint32_t wm = __reduce_max_sync(0xffffffffu, lm);
            if (lane == 0) r.wmax[gw] = wm;
        }
        named_bar_sync(9 + group, 128);
        // threads in front of this one hold smaller experts: they win ties. (match.any would say so for this warp's lanes,
        // but takes over a thousand cycles for 32 different values.)
        const uint4* l4 = reinterpret_cast<const uint4*>(r.lm);
        const uint32_t lt = lm - 1u;
        int cnt = 0;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            const uint4 v = l4[j];
            const int d = gl - 4 * j;   // how many of the four are in front
            cnt += int(v.x > (d > 0 ? lt : lm)) + int(v.y > (d > 1 ? lt : lm)) + int(v.z > (d > 2 ? lt : lm)) + int(v.w > (d > 3 ? lt : lm));
        }
        if (lm != 0u && cnt < p.K) {
#pragma unroll
            for (int i = 0; i < VT; ++i) r.cand[cnt * VT + i] = (static_cast<unsigned long long>(key[i]) << 32) | (0xffffffffu - uint32_t(e0 + i));
        }
        float mx = 0.0f;
        if (weights) {
            mx = key_value(max(max(r.wmax[0], r.wmax[1]), max(r.wmax[2], r.wmax[3])));
            double part = 0.0;
#pragma unroll
            for (int i = 0; i < VT; ++i)
                if (key[i] != 0u) part += double(expf(key_value(key[i]) - mx));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            if (lane == 0) r.sum[gw] = part;
        }
        named_bar_sync(9 + group, 128);
        const int nc = p.K * VT;
        for (int c = gl; c < nc; c += 128) {
            const unsigned long long me = r.cand[c];
            int rank = 0;
#pragma unroll 8
            for (int j = 0; j < nc; ++j) rank += int(r.cand[j] > me);
            const uint32_t k = uint32_t(me >> 32);
            if (k != 0u && rank < p.K) {
                s.ids[t * p.K + rank] = int(0xffffffffu - uint32_t(me));
                if (weights) r.p[rank] = float(double(expf(key_value(k) - mx)) / ((r.sum[0] + r.sum[1]) + (r.sum[2] + r.sum[3])));
            }
        }
        if (weights) {
            named_bar_sync(9 + group, 128);
            if (gl < p.K) {
                float wsum = 0.0f;
                for (int k = 0; k < p.K; ++k) wsum += r.p[k];
                s.wts[t * p.K + gl] = __fdiv_rn(r.p[gl], fmaxf(wsum, 6.103515625e-5f));
            }
        }
        if (t + G < p.T) named_bar_sync(9 + group, 128);   // the buffers are used again
    }
}

// Routes (or takes over the given routing) and groups the slots into items of at most kSmallTok
// tokens: experts in ascending id (moe_hits: in order of first appearance), then the shared expert.
// `work` is called by every warp beside it. VT: logits per thread, 0 without a router. route: scratch.
template <int VT, int G, class Work>
__device__ __forceinline__ void small_plan(const SmallParams& p, SmallPlan& s, SmallRoute* route, bool weights, bool report, Work work) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nt = blockDim.x, TK = p.T * p.K;
    constexpr int kNone = 0x7fffffff;
    const bool one_warp = TK <= 32;
    if constexpr (VT > 0) {
        small_route<VT, G>(p, s, route, weights);
        if (tid < 4) s.ids[TK + tid] = -1;
    } else if (p.hit_ptr) {
        if (!one_warp) {   // an id for every pointer: the first slot that has it
            for (int i = tid; i < TK; i += nt) s.ptr[i] = i % p.K < ld_l2(p.hit_n + i / p.K) ? ld_l2(p.hit_ptr + i) : nullptr;
            __syncthreads();
            for (int i = tid; i < TK + 4; i += nt) {
                int id = -1;
                if (i < TK && s.ptr[i]) {
                    id = 0;
                    while (s.ptr[id] != s.ptr[i]) ++id;
                }
                s.ids[i] = id;
            }
        }
    } else {
        for (int i = tid; i < TK + 4; i += nt) {
            int e = i < TK ? ld_l2(p.ids + i) : -1;
            if (i < TK) {
                s.wts[i] = ld_l2(p.wts + i);
                if (e < 0 || e >= p.E) {
                    if (report) {
                        p.status[0] = kDevBadExpertId;
                        p.status[2] = i;
                    }
                    e = -1;
                }
            }
            s.ids[i] = e;
        }
    }
    const int sh = p.shared ? (p.T + kSmallTok - 1) / kSmallTok : 0;
    auto put = [&](int slot, int e, int base, int pos, int cnt, const uint8_t* blob) {
        SmallItem& it = s.item[base];
        const int at = pos % kSmallTok;
        it.slot[at] = slot;
        it.tok[at] = slot / p.K;
        if (at == 0) {
            it.blob = blob ? blob : p.experts + size_t(e) * p.stride;
            it.m = min(kSmallTok, cnt - pos);
            if (it.m == 1) it.slot[1] = slot, it.tok[1] = slot / p.K;   // the second column repeats the first and is not used
        }
    };
    auto put_shared = [&](int i, int n_start) {
        SmallItem& it = s.item[n_start + i];
        it.blob = p.shared;
        it.m = min(kSmallTok, p.T - i * kSmallTok);
        it.slot[0] = TK + i * kSmallTok;
        it.slot[1] = it.slot[0] + it.m - 1;
        it.tok[0] = it.slot[0] - TK;
        it.tok[1] = it.slot[1] - TK;
    };
    if (one_warp) {
        // warp 0 groups while the others work; it needs the ids of all groups of warps
        if (warp < 4 * G && warp != 0) {
            named_bar_arrive(13, 4 * G * 32);
        } else if (warp == 0) {
            const int t0 = lane / p.K * p.K;
            named_bar_sync(13, 4 * G * 32);
            int e = -1, cnt = 0, pos = 0;
            const uint8_t* ptr = nullptr;
            if (VT == 0 && p.hit_ptr) {   // an id for every pointer: the first slot that has it
                if (lane < TK && lane % p.K < ld_l2(p.hit_n + lane / p.K)) ptr = ld_l2(p.hit_ptr + lane);
#pragma unroll 4
                for (int j = TK - 1; j >= 0; --j)
                    if (__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(ptr), j) == reinterpret_cast<unsigned long long>(ptr) && ptr) e = j;
                if (lane < TK) s.ids[lane] = e;
                if (lane < 4) s.ids[TK + lane] = -1;
                __syncwarp();
            } else if (lane < TK) {
                e = s.ids[lane];
            }
            const int4* v4 = reinterpret_cast<const int4*>(s.ids);
#pragma unroll 4
            for (int j = 0; j < (TK + 3) / 4; ++j) {
                const int4 v = v4[j];
                const int d = lane - 4 * j;
                cnt += int(v.x == e) + int(v.y == e) + int(v.z == e) + int(v.w == e);
                pos += int(v.x == e && d > 0) + int(v.y == e && d > 1) + int(v.z == e && d > 2) + int(v.w == e && d > 3);
            }
            const bool starts = e >= 0 && pos % kSmallTok == 0;
            const unsigned sm = __ballot_sync(0xffffffffu, starts);
            int base = pos / kSmallTok, rank = 0;
#pragma unroll 5
            for (int j = 0; j < TK; ++j) {
                const int ej = s.ids[j];
                base += int(ej < e) & int(sm >> j & 1u);
                rank += int(unsigned(j - t0) < unsigned(p.K)) & (int(ej < e) | (int(ej == e) & int(j < lane)));
            }
            if (lane < TK) s.ord[t0 + rank] = int16_t(lane);
            if (e >= 0) put(lane, e, base, pos, cnt, ptr);
            const int n_start = __popc(sm);
            if (lane < sh) put_shared(lane, n_start);
            if (lane == 0) s.n_items = n_start + sh;
        }
        work();
        __syncthreads();
    } else {
        work();
        __syncthreads();
        const int q4 = (TK + 3) >> 2;
        int e = -1, cnt = 0, pos = 0;
        if (tid < TK) {
            e = s.ids[tid];
            const int4* v4 = reinterpret_cast<const int4*>(s.ids);
            for (int j = 0; j < q4; ++j) {
                const int4 v = v4[j];
                const int b = 4 * j;
                cnt += int(v.x == e) + int(v.y == e) + int(v.z == e) + int(v.w == e);
                pos += int(v.x == e && b < tid) + int(v.y == e && b + 1 < tid) + int(v.z == e && b + 2 < tid) + int(v.w == e && b + 3 < tid);
            }
            // the token's slots by ascending expert id (then k): the order of the weighted sum
            const int t0 = tid / p.K * p.K;
            int rank = 0;
            for (int j = t0; j < t0 + p.K; ++j) {
                const int ej = s.ids[j];
                rank += int(ej < e || (ej == e && j < tid));
            }
            s.ord[t0 + rank] = int16_t(tid);
        }
        const bool starts = e >= 0 && pos % kSmallTok == 0;
        if (tid < TK + 4) s.start[tid] = starts ? e : kNone;
        const int n_start = __syncthreads_count(starts);
        if (e >= 0) {
            const int4* v4 = reinterpret_cast<const int4*>(s.start);
            int base = pos / kSmallTok;
            for (int j = 0; j < q4; ++j) {
                const int4 v = v4[j];
                base += int(v.x < e) + int(v.y < e) + int(v.z < e) + int(v.w < e);
            }
            put(tid, e, base, pos, cnt, VT == 0 && p.hit_ptr ? s.ptr[e] : nullptr);
        }
        if (tid < sh) put_shared(tid, n_start);
        if (tid == 0) s.n_items = n_start + sh;
        __syncthreads();
    }
    if (VT > 0 && report) {
        for (int i = tid; i < TK; i += nt) {
            p.ids_out[i] = s.ids[i];
            p.wts_out[i] = s.wts[i];
        }
    }
}

// One unit (two 64-blocks) of four row groups at `units`, `stride` bytes apart: calls emit(j, t) for block j with
// t = {row g token 0, row g token 1, row g + 8 token 0, row g + 8 token 1} of row group t4 (see units_mma_n2
// for the arithmetic). bf: for blocks 0, 1 the lane's B fragment, of token g & 1 for row group g >> 1;
// v: the scales of row group t4's tokens 0, 1 for blocks 0, 1.
template <class Emit>
__device__ __forceinline__ void quad_terms(const uint8_t* units, uint32_t stride, int lane, const uint4 (&bf)[2], const float4 (&v)[2][2], Emit emit) {
    constexpr uint32_t M0 = 0x03030303u, M1 = 0x30303030u;
    const int g = lane >> 2, t4 = lane & 3, mine = g >> 1;
    uint4 c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = *reinterpret_cast<const uint4*>(units + j * stride + lane * 16);
    const uint2 sc = *reinterpret_cast<const uint2*>(units + t4 * stride + kUnitCodeBytes + g * 8);
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
        uint32_t a0[16], a1[16], b0[8], b1[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const bool live = mine == j;
            b0[2 * j] = live ? bf[jj].x : 0u;
            b0[2 * j + 1] = live ? bf[jj].y : 0u;
            b1[2 * j] = live ? bf[jj].z : 0u;
            b1[2 * j + 1] = live ? bf[jj].w : 0u;
            const uint32_t w0 = jj ? c[j].y : c[j].x, w1 = jj ? c[j].w : c[j].z;
            const uint32_t y0 = w0 >> 2, y1 = w1 >> 2;
            a0[4 * j] = w0 & M0;
            a0[4 * j + 1] = w1 & M0;
            a0[4 * j + 2] = y0 & M0;
            a0[4 * j + 3] = y1 & M0;
            a1[4 * j] = w0 & M1;
            a1[4 * j + 1] = w1 & M1;
            a1[4 * j + 2] = y0 & M1;
            a1[4 * j + 3] = y1 & M1;
        }
        uint64_t lo0, hi0, lo1, hi1;
        mma_u8s8_chain4(lo0, hi0, a0, b0, kMagicBits);
        mma_u8s8_chain4(lo1, hi1, a1, b1, kMagicBits);
        const __half2 s_lo = *reinterpret_cast<const __half2*>(&sc.x), s_hi = *reinterpret_cast<const __half2*>(&sc.y);
        const float d_lo = jj ? __high2float(s_lo) : __low2float(s_lo), d_hi = jj ? __high2float(s_hi) : __low2float(s_hi);
        const float4 v0 = v[jj][0], v1 = v[jj][1];
        const uint64_t ax = pack2(v0.x, v1.x), ay = pack2(v0.y, v1.y), nx = pack2(v0.z, v1.z), ny = pack2(v0.w, v1.w);
        float t[4];
        unpack2(fma2(ay, add2(lo1, ny), mul2(ax, add2(lo0, nx))), t[0], t[1]);
        unpack2(fma2(ay, add2(hi1, ny), mul2(ax, add2(hi0, nx))), t[2], t[3]);
        t[0] = __fmul_rn(d_lo, t[0]);
        t[1] = __fmul_rn(d_lo, t[1]);
        t[2] = __fmul_rn(d_hi, t[2]);
        t[3] = __fmul_rn(d_hi, t[3]);
        emit(jj, t);
    }
}

// Place of the four codes of element group (s, hi, t) of 64-block b in the fragment order (a word index).
__device__ __forceinline__ int frag_word(int b, int s, int hi, int t) { return (b * 4 + t) * 4 + s * 2 + hi; }

struct SmallUpSmem {
    uint32_t plan, xs, sc, terms, red, bars, abort, ring, total;
    int xstride;
};
__host__ __device__ inline SmallUpSmem small_up_smem(int T, int n, int ring, int tbufs) {
    SmallUpSmem m{};
    uint32_t off = 0;
    m.plan = off;
    off += (uint32_t(sizeof(SmallPlan)) + 15u) & ~15u;
    m.xstride = n + 64;                                // codes of a token: neighbouring tokens fall into different halves of the banks
    m.xs = off;
    off += uint32_t(T) * uint32_t(m.xstride);
    m.sc = off;
    off += uint32_t(T) * uint32_t(n / kQK) * 16;       // {a0, a1 / 16, biases} per block
    m.terms = off;
    off += uint32_t(tbufs) * uint32_t(n / kQK) * 512;  // [buffer][block][token, pair of groups][gate / up, group, row] float
    if (off < m.terms + kSmallGroups * uint32_t(sizeof(SmallRoute))) off = m.terms + kSmallGroups * uint32_t(sizeof(SmallRoute));   // (the routing's scratch lies there first)
    m.red = off;
    off += 2 * 2 * 4 * 4;                              // [buffer][amax, sum][sum warp]
    m.bars = off;
    off += uint32_t(ring) * 16;                        // full, empty
    m.abort = off;
    off += 16;
    off = (off + 127u) & ~127u;
    m.ring = off;
    off += uint32_t(ring) * 4u * uint32_t(n / kUnitK) * kUnitBytes;
    m.total = off;
    return m;
}

template <int VT>
__global__ void __maxnreg__(72) k_small_up(const SmallParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const SmallUpSmem sm = small_up_smem(p.T, p.n, p.ring, p.tbufs);
    SmallPlan& plan = *reinterpret_cast<SmallPlan*>(smem + sm.plan);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t full = smem_u32(smem + sm.bars), empty = full + p.ring * 8, abort = smem_u32(smem + sm.abort);
    if (tid == 0) {
        for (int i = 0; i < p.ring; ++i) {
            mbar_init(reinterpret_cast<uint64_t*>(smem + sm.bars) + i, 1);
            mbar_init(reinterpret_cast<uint64_t*>(smem + sm.bars) + p.ring + i, kUpProd);
        }
        sts32(abort, 0u);
        mbar_fence_init();
    }
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const bool first = blockIdx.x == 0;
    if (first && tid == 0 && p.status[3] != kCookie) {   // first use of this workspace
        p.status[0] = kDevOk;
        p.status[2] = 0;
        p.status[3] = kCookie;
    }
    if constexpr (VT == 0) {   // (the status is reset before a bad id can be reported)
        if (first) __syncthreads();
    }
    const int nb = p.n / kQK, units = p.n / kUnitK;
    // x into Q8 fragments, 32 quads of four values (a chunk) per warp at a time; the first chunks are loaded before the
    // routing, so that their latency passes beside it
    const int cpr = p.n / 128, chunks = p.T * cpr;
    constexpr int kAhead = 4;
    const int warps = int(blockDim.x >> 5);
    // (one token: the four warps that route it take no chunks; while warp 0 groups alone it takes none)
    const int w0 = p.T == 1 && VT > 0 ? 4 : p.T * p.K <= 32 ? 1 : 0, nw = warps - w0;
    const int c_first = warp >= w0 ? warp - w0 : chunks;
    float4 xv[kAhead];
    auto load_x = [&](int c0) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) xv[i] = c0 + i * nw < chunks ? reinterpret_cast<const float4*>(p.x)[size_t(c0 + i * nw) * 32 + lane] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    auto quant_x = [&](int c0, auto count) {   // chunks nw apart, step by step together: each is one long dependent chain
        constexpr int N = decltype(count)::value;
        const float4 (&v)[kAhead] = xv;
        float am[N], d[N], id[N];
        int sum[N] = {};
        uint32_t word[N] = {};
#pragma unroll
        for (int k = 0; k < N; ++k) am[k] = fmaxf(fmaxf(fabsf(v[k].x), fabsf(v[k].y)), fmaxf(fabsf(v[k].z), fabsf(v[k].w)));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int k = 0; k < N; ++k) am[k] = fmaxf(am[k], __shfl_xor_sync(0xffffffffu, am[k], o));
#pragma unroll
        for (int k = 0; k < N; ++k) {
            d[k] = __fdiv_rn(am[k], 127.0f);
            id[k] = d[k] != 0.0f ? __fdiv_rn(1.0f, d[k]) : 0.0f;
            const float hv[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int code = int(round_half_away(__fmul_rn(hv[i], id[k])));
                sum[k] += code;
                word[k] |= uint32_t(code & 0xff) << (8 * i);
            }
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int k = 0; k < N; ++k) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const int c = c0 + k * nw;
            if (c >= chunks) break;
            const int tok = c / cpr, q = (c - tok * cpr) * 32 + lane;   // quad of the row
            const int rb = q >> 3, j = q & 7, b = rb >> 1, s = rb & 1;
            reinterpret_cast<uint32_t*>(smem + sm.xs + tok * sm.xstride)[frag_word(b, s, j >> 2, j & 3)] = word[k];
            if (j == 0) {
                const float ds = __half2float(__float2half_rn(d[k])), av = s ? ds * 0.0625f : ds;
                const int ss = s ? 16 * sum[k] : sum[k];
                float* f = reinterpret_cast<float*>(smem + sm.sc) + (size_t(tok) * nb + b) * 4;
                f[s] = av;
                f[2 + s] = -(kMagic + float(ss));
                if (first && p.xq) {
                    p.xa[size_t(tok) * 2 * nb + rb] = av;
                    p.xc[size_t(tok) * 2 * nb + rb] = __int_as_float(kMagicBits - ss);
                }
            }
            if (first && p.xq) reinterpret_cast<uint32_t*>(p.xq + size_t(tok) * p.n)[frag_word(b, s, j >> 2, j & 3)] = word[k];
        }
    };
    load_x(c_first);
    small_plan<VT, kSmallGroups>(p, plan, reinterpret_cast<SmallRoute*>(smem + sm.terms), first, first, [&]() {
        for (int c0 = c_first; c0 < chunks; c0 += kAhead * nw) {
            if (c0 != c_first) load_x(c0);
            if (c0 + 2 * nw < chunks) quant_x(c0, std::integral_constant<int, kAhead>());
            else quant_x(c0, std::integral_constant<int, 2>());
        }
    });

    const int fbs = p.ff / kQ8, n_tasks = plan.n_items * fbs;
    const uint32_t group_bytes = uint32_t(units) * kUnitBytes, task_bytes = 4 * group_bytes;
    float* terms = reinterpret_cast<float*>(smem + sm.terms);
    const int tbufs = p.tbufs;
    // task = item * fbs + block of 32 hidden values, a stride of gridDim.x apart
    const int item0 = int(blockIdx.x) / fbs, fb0 = int(blockIdx.x) % fbs, d_item = int(gridDim.x) / fbs, d_fb = int(gridDim.x) % fbs;
    auto advance = [&](int& item, int& fb) {
        item += d_item;
        fb += d_fb;
        if (fb >= fbs) fb -= fbs, ++item;
    };
    // named barriers: 1 + buffer = its terms are complete, 3 + buffer = they have been added up
    if (warp < kUpProd) {
        // ---------------- products: this warp's units of the task's four row groups
        const int g = lane >> 2, t4 = lane & 3;
        int round = 0, slot = 0, item = item0, fb = fb0;
        uint32_t phase = 0;
        for (int task = blockIdx.x; task < n_tasks; task += gridDim.x, ++round, advance(item, fb)) {
            const int buf = tbufs == 2 ? round & 1 : 0;
            const SmallItem& it = plan.item[item];
            const int tok[2] = {it.tok[0], it.tok[1]};
            const uint8_t* xb = smem + sm.xs + tok[g & 1] * sm.xstride + t4 * 16;
            const float4* s0 = reinterpret_cast<const float4*>(smem + sm.sc) + tok[0] * nb;
            const float4* s1 = reinterpret_cast<const float4*>(smem + sm.sc) + tok[1] * nb;
            const uint8_t* w = smem + sm.ring + slot * task_bytes;
            // (of a term's place: token * 64 + pair of groups * 32 + (gate / up, swapped in odd pairs) * 16 + group of the pair * 8 + row)
            float* tb = terms + buf * nb * 128 + (t4 >> 1) * 32 + (t4 & 1) * 8 + g;
            const int up_off = (t4 >> 1) ? 0 : 16, gate_off = 16 - up_off;
            mbar_spin(full + slot * 8, phase, abort, p.wait_ns);
            if (round >= tbufs) named_bar_sync(3 + buf, kUpBarThreads);
            for (int u = warp; u < units; u += kUpProd) {
                uint4 bf[2];
                float4 v[2][2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    bf[j] = *reinterpret_cast<const uint4*>(xb + (2 * u + j) * 64);
                    v[j][0] = s0[2 * u + j];
                    v[j][1] = s1[2 * u + j];
                }
                quad_terms(w + u * kUnitBytes, group_bytes, lane, bf, v, [&](int j, const float (&t)[4]) {
                    float* o = tb + (2 * u + j) * 128;
                    o[gate_off] = t[0];
                    o[64 + gate_off] = t[1];
                    o[up_off] = t[2];
                    o[64 + up_off] = t[3];
                });
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + slot * 8);
            named_bar_arrive(1 + buf, kUpBarThreads);
            if (++slot == p.ring) {
                slot = 0;
                phase ^= 1u;
            }
        }
    } else if (warp < kUpProd + 4) {
        // ---------------- sums: one (row, token) per thread; warp = token * 2 + pair of groups, lanes l and l ^ 16 hold
        // gate and up of hidden value pair * 16 + (l & 15) of the task's 32
        const int sw = warp - kUpProd, tk = sw >> 1, pr = sw & 1, hid = pr * 16 + (lane & 15);
        const bool is_up = ((lane >> 4) ^ pr) != 0;
        int round = 0, item = item0, fb = fb0;
        for (int task = blockIdx.x; task < n_tasks; task += gridDim.x, ++round, advance(item, fb)) {
            const int buf = tbufs == 2 ? round & 1 : 0;
            const SmallItem& it = plan.item[item];
            const float* tb = terms + buf * nb * 128 + sw * 32 + lane;
            float* red = reinterpret_cast<float*>(smem + sm.red) + (round & 1) * 8;   // [amax, sum][sum warp]
            named_bar_sync(1 + buf, kUpBarThreads);
            float v = 0.0f;
#pragma unroll 8
            for (int b = 0; b < nb; ++b) v = __fadd_rn(v, tb[b * 128]);
            if (task + tbufs * int(gridDim.x) < n_tasks) named_bar_arrive(3 + buf, kUpBarThreads);
            if (tk >= it.m) continue;   // (both warps of the token)
            const float other = __shfl_xor_sync(0xffffffffu, v, 16);
            // the hidden value, and the Q8 of its block of 32 (quant/q2_0/q2_0.cpp:101-113), which the token's two warps hold
            const float h = swiglu_ref(is_up ? other : v, is_up ? v : other);
            float am = fabsf(h);
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
            if (lane == 0) red[sw] = am;
            named_bar_sync(5 + tk, 64);
            am = fmaxf(am, red[sw ^ 1]);
            const float d = __fdiv_rn(am, 127.0f);
            const float id = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
            const int code = int(round_half_away(__fmul_rn(h, id)));
            int sum = code;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane == 0) reinterpret_cast<int*>(red)[4 + sw] = sum;
            uint32_t word = uint32_t(code & 0xff) << (8 * (lane & 3));
            word |= __shfl_xor_sync(0xffffffffu, word, 1);
            word |= __shfl_xor_sync(0xffffffffu, word, 2);
            named_bar_sync(7 + tk, 64);
            const int sl = it.slot[tk], b = fb >> 1, s = fb & 1, e4 = hid >> 2;   // quad e4 of the block of 32
            if (lane < 16 && (lane & 3) == 0) reinterpret_cast<uint32_t*>(p.hq + size_t(sl) * p.ff)[frag_word(b, s, e4 >> 2, e4 & 3)] = word;
            if (pr == 0 && lane == 0) {
                const int all = sum + reinterpret_cast<const int*>(red)[4 + (sw ^ 1)];
                const float ds = __half2float(__float2half_rn(d));
                float* f = reinterpret_cast<float*>(p.hs + size_t(sl) * (p.ff / kQK) + b);
                f[s] = s ? ds * 0.0625f : ds;
                f[2 + s] = -(kMagic + float(s ? 16 * all : all));
            }
        }
    } else if (warp == kUpProd + 4 && lane == 0) {
        // ---------------- the weights of a task: four consecutive row groups of its expert
        int slot = 0, item = item0, fb = fb0;
        uint32_t phase = 0;
        for (int task = blockIdx.x; task < n_tasks; task += gridDim.x, advance(item, fb)) {
            mbar_spin(empty + slot * 8, phase ^ 1u, abort, p.wait_ns);
            const uint8_t* src = plan.item[item].blob + size_t(fb) * task_bytes;
            const uint32_t dst = smem_u32(smem + sm.ring) + slot * task_bytes;
            mbar_expect_tx(full + slot * 8, task_bytes);
#pragma unroll
            for (int j = 0; j < 4; ++j) bulk_g2s(dst + j * group_bytes, src + size_t(j) * group_bytes, group_bytes, full + slot * 8);
            if (++slot == p.ring) {
                slot = 0;
                phase ^= 1u;
            }
        }
    }
    __syncwarp();
    __syncthreads();
    if (lds32(abort)) {   // a wait ran out: report it, and let copies still in flight land
        if (tid == 0) p.status[0] = kDevWaitTimeout;
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) {
        }
    }
}

struct SmallDownSmem {
    uint32_t plan, terms, hq, hs, y, list, bars, abort, ring, total;
    int tstride;
};
__host__ __device__ inline SmallDownSmem small_down_smem(int slots, int ff, int ring) {
    SmallDownSmem m{};
    uint32_t off = 0;
    m.plan = off;
    off += (uint32_t(sizeof(SmallPlan)) + 15u) & ~15u;
    m.tstride = (ff / kQK) * 16 + 8;                    // [slot][block][16 rows] float (8 more: neighbouring slots in other banks)
    m.terms = off;
    off += uint32_t(slots) * uint32_t(m.tstride) * 4;
    if (off < m.terms + kSmallGroups * uint32_t(sizeof(SmallRoute))) off = m.terms + kSmallGroups * uint32_t(sizeof(SmallRoute));
    m.hq = off;
    off += uint32_t(slots) * uint32_t(ff);
    m.hs = off;
    off += uint32_t(slots) * uint32_t(ff / kQK) * 16;
    m.y = off;
    off += uint32_t(slots) * 64;                        // [slot][16 rows]
    m.list = off;
    off += uint32_t(kSmallMaxSlots + kSmallMaxT) * 8;   // {weight, slot} in the order of a token's sum; then the shared expert's weights
    m.bars = off;
    off += (uint32_t(2 * ring + 1) * 8 + 15u) & ~15u;   // weights of a quad: full, then free; the hidden rows
    m.abort = off;
    off += 16;
    off = (off + 127u) & ~127u;
    m.ring = off;
    off += uint32_t(ring) * 4u * uint32_t(ff / kUnitK) * kUnitBytes;
    m.total = off;
    return m;
}

template <int VT>
__global__ void __maxnreg__(72) k_small_down(const SmallParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int TK = p.T * p.K, slots = TK + (p.shared ? p.T : 0);
    const SmallDownSmem sm = small_down_smem(slots, p.ff, p.ring);
    SmallPlan& plan = *reinterpret_cast<SmallPlan*>(smem + sm.plan);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const uint32_t full = smem_u32(smem + sm.bars), empty = full + p.ring * 8, bar_h = empty + p.ring * 8, abort = smem_u32(smem + sm.abort);
    const int units = p.ff / kUnitK, nb = p.ff / kQK, r0 = blockIdx.x * 16;
    if (tid == 0) {
        uint64_t* b = reinterpret_cast<uint64_t*>(smem + sm.bars);
        for (int i = 0; i < p.ring; ++i) {
            mbar_init(b + i, 1);
            mbar_init(b + p.ring + i, kDnProd);
        }
        mbar_init(b + 2 * p.ring, 1);
        sts32(abort, 0u);
        mbar_fence_init();
    }
    __syncthreads();
    // (before the wait: the logits, ids and expert pointers were complete before the kernel in front let this one start)
    small_plan<VT, kSmallGroups>(p, plan, reinterpret_cast<SmallRoute*>(smem + sm.terms), true, false, []() {});
    pdl_trigger();
    const int n_items = plan.n_items, quads = (n_items + 3) / 4;
    const uint32_t item_bytes = uint32_t(units) * kUnitBytes;
    float* terms = reinterpret_cast<float*>(smem + sm.terms);
    if (warp == kDnProd) {
        // ---------------- the weights: this block's 16 rows of four items at a time (the first ones do not wait for
        // anything); the hidden rows of all slots, written by the kernel in front
        const size_t off = size_t(p.ff / 8) * (size_t(p.n / kUnitK) * kUnitBytes) + size_t(blockIdx.x) * item_bytes;
        int slot = 0;
        uint32_t phase = 0;
        for (int q = 0; q < max(quads, p.ring); ++q) {
            if (q == p.ring) slot = 0, phase ^= 1u;
            if (q >= p.ring) mbar_spin(empty + slot * 8, phase ^ 1u, abort, p.wait_ns);
            if (q < quads) {
                const int live = min(4, n_items - q * 4);
                if (lane == 0) mbar_expect_tx(full + slot * 8, live * item_bytes);
                __syncwarp();
                if (lane < live)
                    bulk_g2s(smem_u32(smem + sm.ring) + (slot * 4 + lane) * item_bytes, plan.item[q * 4 + lane].blob + off, item_bytes, full + slot * 8);
            }
            if (q == p.ring - 1) {
                pdl_wait();
                if (lane == 0) {
                    const uint32_t q_bytes = uint32_t(slots * p.ff), s_bytes = uint32_t(slots * nb * 16);
                    asm volatile("fence.proxy.async;" ::: "memory");
                    mbar_expect_tx(bar_h, q_bytes + s_bytes);
                    bulk_g2s(smem_u32(smem + sm.hq), p.hq, q_bytes, bar_h);
                    bulk_g2s(smem_u32(smem + sm.hs), p.hs, s_bytes, bar_h);
                }
            }
            if (++slot == p.ring && q >= p.ring) slot = 0, phase ^= 1u;
        }
    } else {
        if (p.out) {   // (what the sums at the end need, before the wait)
            float2* list = reinterpret_cast<float2*>(smem + sm.list);
            for (int i = tid; i < TK; i += kDnProd * 32) {
                const int slot = plan.ord[i];
                list[i] = make_float2(plan.wts[slot], __int_as_float(plan.ids[slot] >= 0 ? slot : -1));
            }
            if (tid < p.T && p.shared) list[TK + tid].x = p.gate_logit ? sigmoid_ref(ld_l2(p.gate_logit + tid)) : 1.0f;
        }
        pdl_wait();
        mbar_spin(bar_h, 0u, abort, p.wait_ns);
        // ---------------- products: unit u of four items; lane (g, t4) finishes rows g, g + 8 of item t4
        auto quad = [&](int q, int slot, int next, int end) {   // units next, next + kDnProd, ... in front of `end`, counted over all quads
            const SmallItem& ib = plan.item[min(4 * q + (g >> 1), n_items - 1)];   // whose activations this lane brings
            const SmallItem& it = plan.item[min(4 * q + t4, n_items - 1)];         // whose rows it finishes
            const uint8_t* hb = smem + sm.hq + ib.slot[g & 1] * p.ff + t4 * 16;
            const float4* h0 = reinterpret_cast<const float4*>(smem + sm.hs) + it.slot[0] * nb;
            const float4* h1 = reinterpret_cast<const float4*>(smem + sm.hs) + it.slot[1] * nb;
            const bool live = 4 * q + t4 < n_items, two = live && it.m > 1;
            float* o0 = terms + it.slot[0] * sm.tstride + g;
            float* o1 = terms + it.slot[1] * sm.tstride + g;
            for (; next < end; next += kDnProd) {
                const int u = next - q * units;
                uint4 bf[2];
                float4 v[2][2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    bf[j] = *reinterpret_cast<const uint4*>(hb + (2 * u + j) * 64);
                    v[j][0] = h0[2 * u + j];
                    v[j][1] = h1[2 * u + j];
                }
                quad_terms(smem + sm.ring + slot * 4 * item_bytes + u * kUnitBytes, item_bytes, lane, bf, v, [&](int j, const float (&t)[4]) {
                    const int b = (2 * u + j) * 16;
                    if (live) {
                        o0[b] = t[0];
                        o0[b + 8] = t[2];
                    }
                    if (two) {
                        o1[b] = t[1];
                        o1[b + 8] = t[3];
                    }
                });
            }
            return next;
        };
        int next = warp;
        if (quads <= p.ring) {   // no slot is used twice: a warp goes from one of its units to the next
            while (next < quads * units) {
                const int q = next / units;
                mbar_spin(full + q * 8, 0u, abort, p.wait_ns);
                next = quad(q, q, next, (q + 1) * units);
            }
        } else {                 // every warp walks all quads in order, so that it never waits for a later use of a slot than the next one
            int slot = 0;
            uint32_t phase = 0;
            for (int q = 0; q < quads; ++q) {
                mbar_spin(full + slot * 8, phase, abort, p.wait_ns);
                next = quad(q, slot, next, (q + 1) * units);
                __syncwarp();
                if (lane == 0) mbar_arrive(empty + slot * 8);
                if (++slot == p.ring) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
        }
    }
    __syncthreads();
    float* ybuf = reinterpret_cast<float*>(smem + sm.y);
    for (int i = tid; i < slots * 16; i += kDnThreads) {
        const int slot = i >> 4, r = i & 15;
        if (slot < TK && plan.ids[slot] < 0) continue;
        const float* tb = terms + slot * sm.tstride + r;
        float acc = 0.0f;
#pragma unroll 4
        for (int b = 0; b < nb; ++b) acc = __fadd_rn(acc, tb[b * 16]);
        ybuf[i] = acc;
        if (p.y && slot < TK) p.y[size_t(slot) * p.n + r0 + r] = acc;
    }
    if (p.out) {
        __syncthreads();
        // the token's experts in ascending id, then the shared one (see k_combine_ordered)
        const float2* list = reinterpret_cast<const float2*>(smem + sm.list);
        for (int i = tid; i < p.T * 16; i += kDnThreads) {
            const int t = i >> 4, r = i & 15;
            float acc = 0.0f;
#pragma unroll 4
            for (int k = 0; k < p.K; ++k) {
                const float2 w = list[t * p.K + k];
                const int slot = __float_as_int(w.y);
                const float v = ybuf[max(slot, 0) * 16 + r];
                if (slot >= 0) acc = __fadd_rn(acc, __fmul_rn(w.x, v));
            }
            if (p.shared) acc = __fadd_rn(acc, __fmul_rn(ybuf[(TK + t) * 16 + r], list[TK + t].x));
            p.out[size_t(t) * p.n + r0 + r] = acc;
        }
    }
    if (lds32(abort)) {
        if (tid == 0) p.status[0] = kDevWaitTimeout;
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) {
        }
    }
}
