// Grouping of (token, expert) slots by expert for any number of tokens: stable in slot order, no
// host synchronisation, no atomics on data, the same result on every run. Shared by the streaming
// and the tensor-memory forms of the prefill-sized entry point and the ggml-layout products. Include
// inside namespace frx { namespace { ... } }. Three small kernels, chained by programmatic dependent
// launch: what bounds them is their start and one or two round trips to memory each.
#pragma once

constexpr int kCookie = 0x46525831;   // marks a workspace whose status words have been initialised

// ---------------------------------------------------------------------------------------------
// Slots are cut into chunks of 1024, these into parts of 128.
constexpr int kChunkSlots = 1024, kPartSlots = 128, kParts = kChunkSlots / kPartSlots;

// Expert parallel: with `e_map` (one entry per expert of the whole layer, E_all of them), ids name
// experts of the whole layer, e_map[id] is the index of the expert among those held here or -1, and
// slots of experts held elsewhere take no part; E is then the number of experts held here.
__device__ __forceinline__ int local_expert(int id, int E, const int32_t* __restrict__ e_map, int E_all, bool& bad) {
    if (!e_map) {
        bad = id < 0 || id >= E;
        return bad ? -1 : id;
    }
    bad = id < 0 || id >= E_all;
    return bad ? -1 : e_map[id];
}

// per chunk: how many of its slots go to each expert
__global__ void __launch_bounds__(256) k_pf_hist(const int32_t* __restrict__ ids, int S, int E, int* __restrict__ chunk_cnt,
                                                 int* __restrict__ status, const int32_t* __restrict__ e_map = nullptr, int E_all = 0) {
    extern __shared__ int hist[];
    for (int e = threadIdx.x; e < E; e += blockDim.x) hist[e] = 0;
    pdl_wait();
    pdl_trigger();
    if (blockIdx.x == 0 && threadIdx.x == 0 && status[3] != kCookie) {
        status[0] = kDevOk;
        status[2] = 0;
        status[3] = kCookie;
    }
    const int s0 = blockIdx.x * kChunkSlots;
    int id[kChunkSlots / 256];
#pragma unroll
    for (int i = 0; i < kChunkSlots / 256; ++i) {
        const int s = s0 + threadIdx.x + i * 256;
        id[i] = s < S ? ids[s] : 0;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kChunkSlots / 256; ++i) {
        const int s = s0 + threadIdx.x + i * 256;
        if (s >= S) break;
        bool bad;
        const int e = local_expert(id[i], E, e_map, E_all, bad);
        if (bad) {
            status[0] = kDevBadExpertId;
            status[2] = s;
        } else if (e >= 0) {
            atomicAdd(&hist[e], 1);   // integer counts: exact whatever the order
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) chunk_cnt[size_t(blockIdx.x) * E + e] = hist[e];
}

// Sum of v over the threads in front of this one, and over all of them (`total`), for a block of 1024; tot: scratch.
__device__ __forceinline__ int block_scan(int v, int* tot, int& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    __syncthreads();   // (tot may still be read from the scan before)
    if (lane == 31) tot[warp] = inc;
    __syncthreads();
    int w = tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += u;
    }
    total = __shfl_sync(0xffffffffu, w, 31);
    return inc - v + (warp ? __shfl_sync(0xffffffffu, w, warp - 1) : 0);
}

// The token blocks of the tensor-memory form: every expert's slots cut into blocks of at most tok, as equal as multiples
// of `unit` allow (a tile costs its fixed steps whatever its width).
struct TokenBlocks {
    int tok, unit;
    int* meta;          // [1]: number of blocks; null: no blocks are wanted
    int4* tb;           // {expert, first position in the grouped order, slots, slots rounded up to the unit}
    int max_tb;
};

// per expert: exclusive offsets of its slots over the chunks (written back into chunk_cnt), its
// bounds in the grouped order, and the range of its items of per_item slots. bounds, item_off: [E + 1].
__global__ void __launch_bounds__(1024) k_pf_scan(int* __restrict__ chunk_cnt, int n_chunks, int E, int* __restrict__ bounds,
                                                  int* __restrict__ item_off, int* __restrict__ status, int max_items, int per_item, const TokenBlocks blocks) {
    __shared__ int tot[32];
    pdl_wait();
    pdl_trigger();
    const int tid = threadIdx.x;
    const int per = (E + 1023) / 1024, e0 = tid * per, e1 = min(E, e0 + per);
    int slots = 0, items = 0, tbs = 0;
    constexpr int kBatch = 16;   // loads in flight: the running sum is a chain, the loads need not be
    auto tb_count = [&](int c) { return (c + blocks.tok - 1) / blocks.tok; };
    for (int e = e0; e < e1; ++e) {
        int run = 0;
        for (int c0 = 0; c0 < n_chunks; c0 += kBatch) {
            int v[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) v[i] = c0 + i < n_chunks ? chunk_cnt[size_t(c0 + i) * E + e] : 0;
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                if (c0 + i < n_chunks) chunk_cnt[size_t(c0 + i) * E + e] = run;
                run += v[i];
            }
        }
        bounds[e] = run;   // the count for now
        slots += run;
        items += (run + per_item - 1) / per_item;
        if (blocks.meta) tbs += tb_count(run);
    }
    int n_slots, n_items, n_tb = 0;
    int at_s = block_scan(slots, tot, n_slots), at_i = block_scan(items, tot, n_items), at_t = 0;
    if (blocks.meta) at_t = block_scan(tbs, tot, n_tb);
    const bool fits = n_items <= max_items && n_tb <= blocks.max_tb;
    for (int e = e0; e < e1; ++e) {
        const int c = bounds[e];
        bounds[e] = at_s;
        item_off[e] = at_i;
        if (blocks.meta && fits) {
            // block j gets units * (j + 1) / nb - units * j / nb units, by running remainders: the products leave 32 bits from
            // 1.3 million slots on
            const int nb = tb_count(c), units = (c + blocks.unit - 1) / blocks.unit, each = nb ? units / nb : 0, more = units - each * nb;
            for (int j = 0, lo = 0, rest = 0; j < nb; ++j) {
                rest += more;
                const int width = (each + int(rest >= nb)) * blocks.unit;
                if (rest >= nb) rest -= nb;
                blocks.tb[at_t++] = make_int4(e, at_s + lo, min(width, c - lo), width);
                lo += width;
            }
        }
        at_s += c;
        at_i += (c + per_item - 1) / per_item;
    }
    if (tid == 0) {
        bounds[E] = n_slots;
        item_off[E] = n_items;
        if (!fits) status[0] = kDevTooManyItems;
        status[1] = fits ? n_items : 0;
        if (blocks.meta) blocks.meta[1] = fits ? n_tb : 0;
    }
}

// per chunk: every slot's position in the grouped order (by expert, then slot order). A thread per slot counts the equal
// ids in front of it in its part of 128 (a warp of match.any per 32 slots, 32 steps in a row, took 27 us), and adds
// the counts of the parts in front. `done(slot, expert, its index among the expert's slots)` is called for every placed one.
template <class Done>
__device__ __forceinline__ void pf_place(const int32_t* __restrict__ ids, int S, int E, const int* __restrict__ chunk_off, const int* __restrict__ bounds,
                                         int32_t* __restrict__ perm, const int32_t* __restrict__ e_map, int E_all, Done done) {
    extern __shared__ __align__(16) int32_t place_smem[];   // [1024] local experts, then bytes [kParts][E]: slots of the expert in the part
    uint8_t* part_cnt = reinterpret_cast<uint8_t*>(place_smem + kChunkSlots);
    const int tid = threadIdx.x, c = blockIdx.x, s = c * kChunkSlots + tid, part = tid / kPartSlots, in = tid % kPartSlots;
    for (int i = tid; i < kParts * E / 4 + 1; i += kChunkSlots) reinterpret_cast<uint32_t*>(part_cnt)[i] = 0u;
    bool bad = false;
    int e = s < S ? local_expert(ids[s], E, e_map, E_all, bad) : -1;
    if (e >= E) e = -1;
    place_smem[tid] = e;
    const int base = e >= 0 ? bounds[e] + chunk_off[size_t(c) * E + e] : 0, first = e >= 0 ? bounds[e] : 0;
    __syncthreads();
    const int4* mine = reinterpret_cast<const int4*>(place_smem + part * kPartSlots);
    int rank = 0, all = 0;
#pragma unroll 8
    for (int j = 0; j < kPartSlots / 4; ++j) {
        const int4 v = mine[j];
        const int d = in - 4 * j;
        all += int(v.x == e) + int(v.y == e) + int(v.z == e) + int(v.w == e);
        rank += int(v.x == e && d > 0) + int(v.y == e && d > 1) + int(v.z == e && d > 2) + int(v.w == e && d > 3);
    }
    if (e >= 0 && rank + 1 == all) part_cnt[part * E + e] = uint8_t(all);
    __syncthreads();
    if (e < 0) return;
    int pos = base + rank;
    for (int p = 0; p < part; ++p) pos += part_cnt[p * E + e];
    perm[pos] = s;
    done(s, e, pos - first);
}
inline size_t pf_place_smem(int E) { return size_t(kChunkSlots) * 4 + size_t(kParts) * E + 16; }

__global__ void __launch_bounds__(kChunkSlots) k_pf_place(const int32_t* __restrict__ ids, int S, int E, const int* __restrict__ chunk_off,
                                                          const int* __restrict__ bounds, int32_t* __restrict__ perm,
                                                          const int32_t* __restrict__ e_map = nullptr, int E_all = 0) {
    pdl_wait();
    pdl_trigger();
    pf_place(ids, S, E, chunk_off, bounds, perm, e_map, E_all, [](int, int, int) {});
}
