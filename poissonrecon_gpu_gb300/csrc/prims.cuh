// Device primitives: exclusive scan, stable LSD radix sort of (u64 key, u32
// index) pairs, and compaction.
// All work on the caller's stream; temporary memory comes from the stream's
// memory pool (cudaMallocAsync).
#pragma once
#include <utility>
#include <vector>

#include "common.cuh"

namespace prgpu {

// ------------------------------- memory ------------------------------------
// The device allocations an API call has made on this host thread and not yet
// freed (null outside a call); when the call fails, it frees the ones its stages
// left behind.
struct LiveAllocs {
    std::vector<std::pair<void*, cudaStream_t>> v;
};
extern thread_local LiveAllocs* g_live;
// PRGPU_HOOK_FAIL_ALLOC: allocations left before the one that fails (0: off)
extern std::atomic<long long> g_fail_alloc_countdown;

template <class T>
inline T* dalloc(i64 n, cudaStream_t s) {
    void* p = nullptr;
    if (n <= 0) n = 1;
    if (g_fail_alloc_countdown.load(std::memory_order_relaxed) > 0 && --g_fail_alloc_countdown == 0) {
        set_last_error("cudaMallocAsync(%lld bytes): failure injected by PRGPU_HOOK_FAIL_ALLOC",
                       (long long)((size_t)n * sizeof(T)));
        throw Error{PRGPU_ERR_NOMEM, {0}};
    }
    cudaError_t e = cudaMallocAsync(&p, (size_t)n * sizeof(T), s);
    if (e != cudaSuccess) {
        set_last_error("cudaMallocAsync(%lld bytes): %s", (long long)((size_t)n * sizeof(T)),
                       cudaGetErrorString(e));
        throw Error{PRGPU_ERR_NOMEM, {0}};
    }
    if (g_live) g_live->v.emplace_back(p, s);
    return (T*)p;
}
template <class T>
inline void dfree(T*& p, cudaStream_t s) {
    if (p) {
        if (g_live)
            for (size_t k = g_live->v.size(); k-- > 0;)
                if (g_live->v[k].first == (void*)p) {
                    g_live->v.erase(g_live->v.begin() + (long)k);
                    break;
                }
        cudaFreeAsync((void*)p, s);
    }
    p = nullptr;
}

// ------------------------------- scan ---------------------------------------
constexpr int SCAN_BLOCK = 512;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_BLOCK * SCAN_ITEMS;

template <class T>
__device__ __forceinline__ T block_exclusive_sum(T v, T* smem_warp, T* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        T w = lane < nw ? smem_warp[lane] : T(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) smem_warp[lane] = w;
    }
    __syncthreads();
    T warp_off = warp ? smem_warp[warp - 1] : T(0);
    *total = smem_warp[(blockDim.x >> 5) - 1];
    __syncthreads();
    return warp_off + x - v;
}

template <class TI, class TO>
__global__ void k_tile_reduce(const TI* __restrict__ in, i64 n, TO* __restrict__ partial) {
    __shared__ TO sw[32];
    i64 base = (i64)blockIdx.x * SCAN_TILE + (i64)threadIdx.x * SCAN_ITEMS;
    TO s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k)
        if (base + k < n) s += (TO)in[base + k];
    TO tot;
    block_exclusive_sum<TO>(s, sw, &tot);
    if (threadIdx.x == 0) partial[blockIdx.x] = tot;
}

// 'partial' (null: one tile): the tiles' sums, scanned when 'scanned', else summed here up to this tile
template <class TI, class TO>
__global__ void k_tile_scan(const TI* __restrict__ in, i64 n, TO* __restrict__ out,
                            const TO* __restrict__ partial, bool scanned, TO* __restrict__ total_out) {
    __shared__ TO sw[32];
    i64 base = (i64)blockIdx.x * SCAN_TILE + (i64)threadIdx.x * SCAN_ITEMS;
    TO off = TO(0);
    if (partial && scanned) {
        off = partial[blockIdx.x];
    } else if (partial) {
        TO p = TO(0);
        for (unsigned k = threadIdx.x; k < blockIdx.x; k += SCAN_BLOCK) p += partial[k];
        block_exclusive_sum<TO>(p, sw, &off);
    }
    TO v[SCAN_ITEMS];
    TO s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        v[k] = (base + k < n) ? (TO)in[base + k] : TO(0);
        s += v[k];
    }
    TO tot;
    TO pre = block_exclusive_sum<TO>(s, sw, &tot);
    TO run = off + pre;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
    if (total_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) *total_out = run;
}

// out[i] = sum_{k<i} in[k]; *total_dev (device pointer, optional) receives the sum.
// 'in' and 'out' may alias.  Up to SCAN_SELF tiles each tile sums the sums of the tiles before it (at most
// two loads a thread) instead of waiting for a scan of them: two launches in place of three, which is
// what short scans cost (a few us each; a pass over 5,000 points makes 20 of them).
constexpr i64 SCAN_SELF = 1024;
template <class TI, class TO>
void exclusive_scan(const TI* in, TO* out, i64 n, TO* total_dev, cudaStream_t s) {
    if (n <= 0) {
        if (total_dev) CK(cudaMemsetAsync(total_dev, 0, sizeof(TO), s));
        return;
    }
    i64 nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (nb == 1) {
        k_tile_scan<TI, TO><<<1, SCAN_BLOCK, 0, s>>>(in, n, out, nullptr, false, total_dev);
        CK_LAUNCH();
        return;
    }
    TO* part = dalloc<TO>(nb, s);
    k_tile_reduce<TI, TO><<<(unsigned)nb, SCAN_BLOCK, 0, s>>>(in, n, part);
    CK_LAUNCH();
    const bool scanned = nb > SCAN_SELF;
    if (scanned) exclusive_scan<TO, TO>(part, part, nb, (TO*)nullptr, s);
    k_tile_scan<TI, TO><<<(unsigned)nb, SCAN_BLOCK, 0, s>>>(in, n, out, part, scanned, total_dev);
    CK_LAUNCH();
    dfree(part, s);
}

// ----------------------------- radix sort -----------------------------------
// Stable LSD sort of (key, index) pairs, 8 bits a pass, one launch per pass behind one that counts the digits
// of all passes (the scheme of Adinets and Merrill's Onesweep, 2022, with the look-back of Merrill and
// Garland's single-pass scan, 2016).  A tile ranks its 4,096 keys warp by warp (a warp's 512 consecutive keys against counters of
// its own, without a barrier), publishes its count per digit, adds the counts of the tiles before it
// (look-back) and writes its elements from shared memory in digit order, so that each digit's run is written
// at once.  24 bytes move per element and pass, where a count, a scan and a scatter moved 32 and wrote
// every element by itself.  Tiles are numbered as their blocks start, so a tile waits for running ones
// only; a wait that runs out (sort_poll_limit) ends in counting the earlier tiles' keys instead.
// Bound by the latency of a tile's phases (load, rank, look back, write) at two blocks per SM: three (80
// registers, spilling) and tiles of 2,048 are slower, 0.47 and 0.48 ms on the second line.  Against three
// launches a pass: 15 K keys of 20 bits 0.099 -> 0.040 ms, 9.2 M of 36 bits (corners of the 1M torus)
// 0.585 -> 0.42, 80 M of 39 bits 4.5 -> 3.3.
constexpr int RS_BLOCK = 256;
constexpr int RS_WARPS = RS_BLOCK / 32;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_BLOCK * RS_ITEMS;
constexpr int RS_BINS = 256;
static_assert(RS_BLOCK == RS_BINS, "a thread per digit value");
constexpr int RS_PASSES = 8;
constexpr int RS_LOOK = 16;              // tiles a look-back step reads at once
constexpr size_t RS_SHARED = RS_TILE * (sizeof(u64) + sizeof(uint32_t));

struct RsCounts {
    unsigned hist[RS_PASSES][RS_BINS];   // of the digits, all keys
    unsigned ticket[RS_PASSES];          // tiles started
};

static __global__ void __launch_bounds__(RS_BLOCK) k_rs_hist(const u64* __restrict__ keys, i64 n, int nbits,
                                                             RsCounts* __restrict__ counts) {
    __shared__ unsigned h[RS_PASSES][RS_BINS];
#pragma unroll
    for (int p = 0; p < RS_PASSES; ++p) h[p][threadIdx.x] = 0;
    __syncthreads();
    const i64 stride = (i64)gridDim.x * RS_BLOCK * 4;
    for (i64 e0 = (i64)blockIdx.x * RS_BLOCK * 4; e0 < n; e0 += stride) {
        u64 k[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const i64 e = e0 + i * RS_BLOCK + threadIdx.x;
            k[i] = e < n ? keys[e] : ~0ull;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool valid = e0 + i * RS_BLOCK + threadIdx.x < n;
            for (int p = 0; 8 * p < nbits; ++p) {
                const unsigned mask = nbits - 8 * p < 8 ? (1u << (nbits - 8 * p)) - 1u : 255u;
                const unsigned dig = valid ? (unsigned)(k[i] >> (8 * p)) & mask : RS_BINS;
                // the upper digits of neighbouring keys agree: one addition for the warp
                if (__all_sync(0xffffffffu, dig == __shfl_sync(0xffffffffu, dig, 0))) {
                    if (valid && (threadIdx.x & 31) == 0) atomicAdd(&h[p][dig], 32u);
                } else if (valid) {
                    atomicAdd(&h[p][dig], 1u);
                }
            }
        }
    }
    __syncthreads();
    for (int p = 0; 8 * p < nbits; ++p)
        if (h[p][threadIdx.x]) atomicAdd(&counts->hist[p][threadIdx.x], h[p][threadIdx.x]);
}

// Elements of digit t in the tiles before 'tile'; false after 'limit' polls in a row that found no further tile.  A
// tile's word is its tag << 32 | count: tag 2 pass + 1 with the tile's own count, 2 pass + 2 with the count of all tiles
// up to it; words of earlier passes have lower tags.
__device__ __forceinline__ bool rs_look_back(const u64* status, unsigned tag, int tile, int limit, unsigned& before) {
    const unsigned t = threadIdx.x;
    before = 0;
    int at = tile - 1, polls = 0;
    while (at >= 0) {
        if (polls >= limit) return false;
        u64 w[RS_LOOK];
#pragma unroll
        for (int j = 0; j < RS_LOOK; ++j)
            w[j] = at - j >= 0 ? *(volatile const u64*)&status[(i64)(at - j) * RS_BINS + t] : (u64)(tag + 1) << 32;
        int got = 0;
        bool open = true, done = false;
#pragma unroll
        for (int j = 0; j < RS_LOOK; ++j) {
            const unsigned wt = (unsigned)(w[j] >> 32);
            open = open && wt >= tag;
            if (open) {
                before += (unsigned)w[j];
                ++got;
                if (wt > tag) {
                    done = true;
                    open = false;
                }
            }
        }
        if (done) return true;
        at -= got;
        polls = got ? 0 : polls + 1;
    }
    return true;
}

// vin null: the index of each element (the first pass)
static __global__ void __launch_bounds__(RS_BLOCK, 2) k_rs_pass(const u64* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                                i64 n, int pass, unsigned mask, int poll_limit,
                                                                RsCounts* __restrict__ counts, u64* status,
                                                                u64* __restrict__ kout, uint32_t* __restrict__ vout) {
    extern __shared__ u64 rs_shared[];
    u64* skey = rs_shared;
    uint32_t* sval = reinterpret_cast<uint32_t*>(rs_shared + RS_TILE);
    __shared__ unsigned wcnt[RS_WARPS][RS_BINS];
    __shared__ unsigned lbase[RS_BINS], gbase[RS_BINS], sw[32];
    __shared__ int s_tile;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, shift = 8 * pass;
    const unsigned lt = (1u << lane) - 1u, tag = 2u * pass + 1u;
    if (t == 0) s_tile = (int)atomicAdd(&counts->ticket[pass], 1u);
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) wcnt[w][t] = 0;
    __syncthreads();
    const int tile = s_tile;
    const i64 first = (i64)tile * RS_TILE, mine = first + warp * (32 * RS_ITEMS) + lane;
    u64 key[RS_ITEMS];
    uint32_t val[RS_ITEMS];
    unsigned short rank[RS_ITEMS];
#pragma unroll
    for (int i = 0; i < RS_ITEMS; ++i) {
        const i64 e = mine + 32 * i;
        key[i] = e < n ? kin[e] : 0;
        val[i] = e < n ? (vin ? vin[e] : (uint32_t)e) : 0;
    }
#pragma unroll
    for (int i = 0; i < RS_ITEMS; ++i) {
        const bool valid = mine + 32 * i < n;
        const unsigned dig = (unsigned)(key[i] >> shift) & mask;
        const unsigned peers = __match_any_sync(0xffffffffu, valid ? dig : RS_BINS);
        const unsigned r = wcnt[warp][dig];
        __syncwarp();
        if (valid && (peers & lt) == 0) wcnt[warp][dig] = r + __popc(peers);
        __syncwarp();
        rank[i] = (unsigned short)(r + __popc(peers & lt));
    }
    __syncthreads();
    unsigned total = 0;                  // of digit t in this tile
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
        const unsigned c = wcnt[w][t];
        wcnt[w][t] = total;
        total += c;
    }
    u64* mineword = status + (i64)tile * RS_BINS + t;
    if (tile > 0) *(volatile u64*)mineword = ((u64)tag << 32) | total;
    unsigned all;
    const unsigned local = block_exclusive_sum<unsigned>(total, sw, &all);
    lbase[t] = local;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RS_ITEMS; ++i) {
        if (mine + 32 * i < n) {
            const unsigned dig = (unsigned)(key[i] >> shift) & mask;
            const unsigned p = lbase[dig] + wcnt[warp][dig] + rank[i];
            skey[p] = key[i];
            sval[p] = val[i];
        }
    }
    const unsigned start = block_exclusive_sum<unsigned>(counts->hist[pass][t], sw, &all);
    unsigned before;
    const bool known = rs_look_back(status, tag, tile, poll_limit, before);
    if (known) *(volatile u64*)mineword = ((u64)(tag + 1) << 32) | (before + total);
    gbase[t] = start + before - local;   // modulo 2^32
    if (__syncthreads_or(!known)) {      // a wait ran out: the block counts the keys of the tiles before its own
        gbase[t] = 0;
        __syncthreads();
        for (i64 e = t; e < first; e += RS_BLOCK) atomicAdd(&gbase[(unsigned)(kin[e] >> shift) & mask], 1u);
        __syncthreads();
        before = gbase[t];
        if (!known) *(volatile u64*)mineword = ((u64)(tag + 1) << 32) | (before + total);
        gbase[t] = start + before - local;
        __syncthreads();
    }
    const int m = (int)min(n - first, (i64)RS_TILE);
    for (int q = t; q < m; q += RS_BLOCK) {
        const u64 k = skey[q];
        const unsigned pos = gbase[(unsigned)(k >> shift) & mask] + q;
        kout[pos] = k;
        vout[pos] = sval[q];
    }
}

// Sorts n keys (below 2^31) by bits [0, nbits) and gives the index each came from, stable.  The result ends in
// (keys, vals); the four buffers may change roles.
inline void radix_sort_pairs(u64*& keys, uint32_t*& vals, u64*& ktmp, uint32_t*& vtmp, i64 n, int nbits, cudaStream_t s) {
    if (n <= 0) return;
    nbits = std::max(nbits, 1);
    const i64 nb = (n + RS_TILE - 1) / RS_TILE;
    static_assert(sizeof(RsCounts) % sizeof(u64) == 0, "the tiles' words follow the counts");
    const i64 head = sizeof(RsCounts) / sizeof(u64);
    u64* work = dalloc<u64>(head + nb * RS_BINS, s);
    RsCounts* counts = reinterpret_cast<RsCounts*>(work);
    CK(cudaMemsetAsync(work, 0, (size_t)(head + nb * RS_BINS) * sizeof(u64), s));
    k_rs_hist<<<grid_for(n, RS_BLOCK * 8, 152 * 8), RS_BLOCK, 0, s>>>(keys, n, nbits, counts);
    CK_LAUNCH();
    CK(cudaFuncSetAttribute(k_rs_pass, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RS_SHARED));
    const int limit = sort_poll_limit();
    for (int pass = 0; 8 * pass < nbits; ++pass) {
        const unsigned mask = nbits - 8 * pass < 8 ? (1u << (nbits - 8 * pass)) - 1u : 255u;
        k_rs_pass<<<(unsigned)nb, RS_BLOCK, RS_SHARED, s>>>(keys, pass ? vals : nullptr, n, pass, mask, limit, counts,
                                                            work + head, ktmp, vtmp);
        CK_LAUNCH();
        std::swap(keys, ktmp);
        std::swap(vals, vtmp);
    }
    dfree(work, s);
}

// ---------------------------- small helpers ---------------------------------
template <class T>
__global__ void k_fill(T* p, i64 n, T v) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) p[i] = v;
}
template <class T>
inline void fill(T* p, i64 n, T v, cudaStream_t s) {
    if (n <= 0) return;
    k_fill<T><<<grid_for(n, 256), 256, 0, s>>>(p, n, v);
    CK_LAUNCH();
}

template <class T>
inline T read_scalar(const T* dptr, cudaStream_t s) {
    T h;
    CK(cudaMemcpyAsync(&h, dptr, sizeof(T), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    return h;
}

}  // namespace prgpu
