// Octree stage: normalisation, Morton keys, radix sort, level-by-level node
// arrays and 27-neighbour tables.  Replaces pipelineBuildNodeArray
// (main.cu:511-841) and the kernels it launches (main.cu:126-509).
//
// The node arrays are derived directly from the sorted leaf keys: at every
// depth the non-empty nodes are the runs of equal key prefixes, and each
// non-empty node owns one full group of 8 child slots one depth below.
// Parents, children, point ranges and finest-slot ranges follow from the run
// structure, so no hash table or atomic is needed and every field is exact
// (the reference's racy parent assignment, main.cu:331,357, is not reproduced:
// every slot receives its true parent).
//
// A point starts a run at every depth from the first at which its key differs
// from its predecessor's, so one pass over the points counts the runs of all
// depths, and a second one writes all depths' runs; one launch then fills the
// nodes of all depths.  Depth by depth (flags, scan, the count read back, runs,
// slots, fill) the stage was a chain of some ten launches and a host round trip
// per depth: 0.50 of the 2.65 ms of 5,000 points at maxDepth 6.
#include <algorithm>
#include <cmath>
#include <vector>

#include "context.h"
#include "prims.cuh"

namespace prgpu {

// --------------------------- bounding box -----------------------------------
__device__ __forceinline__ unsigned f2ord(float f) {
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ inline float ord2f(unsigned u) {
    unsigned b = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float f;
    memcpy(&f, &b, 4);
    return f;
#endif
}

__global__ void k_bbox(const float* __restrict__ xyz, i64 n, unsigned* __restrict__ mm) {
    unsigned mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0, 0, 0};
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            unsigned o = f2ord(xyz[3 * i + a]);
            mn[a] = min(mn[a], o);
            mx[a] = max(mx[a], o);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        for (int o = 16; o; o >>= 1) {
            mn[a] = min(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
            mx[a] = max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
        }
    }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            atomicMin(&mm[a], mn[a]);
            atomicMax(&mm[3 + a], mx[a]);
        }
    }
}

// scale and corner of the cube from the box (ordered bits of min x y z, max x y z), as the reference's host
// code computes them (main.cu:530-553)
struct Cube {
    float corner[3], scale;
};
__host__ __device__ inline Cube cube_of(const unsigned* mm) {
    Cube c;
    float scale = 1;
    for (int a = 0; a < 3; ++a) {
        const float mn = ord2f(mm[a]), mx = ord2f(mm[3 + a]);
        if (!a || scale < mx - mn) scale = float(mx - mn);
        c.corner[a] = float(mx + mn) / 2;
    }
    scale *= 1.25f;
    for (int a = 0; a < 3; ++a) c.corner[a] -= scale / 2;
    c.scale = scale;
    return c;
}

// ----------------- normalisation + Morton key (main.cu:132-173,555-569) ------
__global__ void k_normalise_encode(const float* __restrict__ in_xyz, const float* __restrict__ in_nrm, i64 n,
                                   const unsigned* __restrict__ mm, float nscale, int D,
                                   float* __restrict__ p_out, float* __restrict__ n_out, u64* __restrict__ keys) {
    const Cube cube = cube_of(mm);
    const float cx = cube.corner[0], cy = cube.corner[1], cz = cube.corner[2], scale = cube.scale;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        float p[3] = {(in_xyz[3 * i] - cx) / scale, (in_xyz[3 * i + 1] - cy) / scale, (in_xyz[3 * i + 2] - cz) / scale};
        float nx = in_nrm[3 * i], ny = in_nrm[3 * i + 1], nz = in_nrm[3 * i + 2];
        float sq = nx * nx + ny * ny + nz * nz;   // unfused (--fmad=false), as on the reference host
        float len = (float)sqrt((double)sq);
        if (len > 1e-6f) len = 1.0f / len;
        len = len * nscale;
        p_out[3 * i] = p[0];
        p_out[3 * i + 1] = p[1];
        p_out[3 * i + 2] = p[2];
        n_out[3 * i] = nx * len;
        n_out[3 * i + 1] = ny * len;
        n_out[3 * i + 2] = nz * len;
        u64 key = 0;
        float mx = 0.5f, my = 0.5f, mz = 0.5f, w = 0.25f;
        for (int l = D - 1; l >= 0; --l) {
            if (p[0] > mx) { key |= 1ull << (3 * l + 2); mx += w; } else mx -= w;
            if (p[1] > my) { key |= 1ull << (3 * l + 1); my += w; } else my -= w;
            if (p[2] > mz) { key |= 1ull << (3 * l); mz += w; } else mz -= w;
            w *= 0.5f;
        }
        keys[i] = key;
    }
}

__global__ void k_gather_points(const uint32_t* __restrict__ idx, i64 n, const float* __restrict__ p_in,
                                const float* __restrict__ n_in, float* __restrict__ p_out, float* __restrict__ n_out) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        i64 s = idx[i];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            p_out[3 * i + a] = p_in[3 * s + a];
            n_out[3 * i + a] = n_in[3 * s + a];
        }
    }
}

// ------------------------------- runs ---------------------------------------
// first depth at which sorted point i differs from its predecessor: 0 for the first point, D + 1 when the
// keys are equal (the point starts no run)
__device__ __forceinline__ int first_depth(const u64* __restrict__ keys, i64 i, int D) {
    if (i == 0) return 0;
    const u64 x = keys[i] ^ keys[i - 1];
    return x ? D - (63 - __clzll((i64)x)) / 3 : D + 1;
}

constexpr int LV_BLOCK = 256;
constexpr int LV_ROUNDS = 4;
constexpr int LV_TILE = LV_BLOCK * LV_ROUNDS;
constexpr int LV_MAX = PRGPU_MAX_DEPTH + 1;   // depths 0..15

// runs that start in each tile of LV_TILE points, per depth: cnt[d * ntiles + tile]
__global__ void __launch_bounds__(LV_BLOCK) k_run_count(const u64* __restrict__ keys, i64 n, int D, i64 ntiles,
                                                        int* __restrict__ cnt) {
    __shared__ int h[LV_MAX];
    if (threadIdx.x < LV_MAX) h[threadIdx.x] = 0;
    __syncthreads();
    int mine = 0;   // lane d: the warp's runs of depth d
    for (int q = 0; q < LV_ROUNDS; ++q) {
        const i64 i = (i64)blockIdx.x * LV_TILE + q * LV_BLOCK + threadIdx.x;
        const int L = i < n ? first_depth(keys, i, D) : D + 1;
        for (int d = 0; d <= D; ++d) {
            const int c = __popc(__ballot_sync(0xffffffffu, L <= d));
            if ((int)(threadIdx.x & 31) == d) mine += c;
        }
    }
    if ((int)(threadIdx.x & 31) <= D) atomicAdd(&h[threadIdx.x & 31], mine);
    __syncthreads();
    if ((int)threadIdx.x <= D) cnt[(i64)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// exclusive scan of each depth's counts over the tiles, in place (a block per depth); totals to U[d]
__global__ void __launch_bounds__(1024) k_run_offsets(int* __restrict__ cnt, i64 ntiles, int* __restrict__ U) {
    __shared__ int sw[32];
    int* c = cnt + (i64)blockIdx.x * ntiles;
    int run = 0;
    for (i64 t0 = 0; t0 < ntiles; t0 += 1024) {
        const i64 t = t0 + threadIdx.x;
        const int v = t < ntiles ? c[t] : 0;
        int total;
        const int e = block_exclusive_sum<int>(v, sw, &total);
        if (t < ntiles) c[t] = run + e;
        run += total;
    }
    if (threadIdx.x == 0) U[blockIdx.x] = run;
}

// the runs of all depths
struct Levels {
    u64* key[LV_MAX];     // unique prefix (levels below masked)
    int* pidx[LV_MAX];    // first point
    int* slot[LV_MAX];    // slot among the depth's nodes: 8 * the parent's run + child code
    int* first[LV_MAX];   // depths < D: first run one depth below
    int* lo[LV_MAX];      // depths < D: first run of depth D - 1 below (its own number at D - 1)
    int U[LV_MAX];        // runs
    i64 base[LV_MAX + 1]; // first node of each depth
};

__global__ void __launch_bounds__(LV_BLOCK) k_runs(const u64* __restrict__ keys, i64 n, int D, i64 ntiles,
                                                   const int* __restrict__ off, Levels lv, int* __restrict__ point_node) {
    __shared__ int wcnt[LV_BLOCK / 32][LV_MAX];
    __shared__ int run[LV_MAX];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if ((int)threadIdx.x <= D) run[threadIdx.x] = off[(i64)threadIdx.x * ntiles + blockIdx.x];
    const unsigned upto = 0xffffffffu >> (31 - lane);
    for (int q = 0; q < LV_ROUNDS; ++q) {
        const i64 i = (i64)blockIdx.x * LV_TILE + q * LV_BLOCK + threadIdx.x;
        const int L = i < n ? first_depth(keys, i, D) : D + 1;
        for (int d = 0; d <= D; ++d) {
            const int c = __popc(__ballot_sync(0xffffffffu, L <= d));
            if (lane == d) wcnt[w][d] = c;
        }
        __syncthreads();
        int before = 0, all = 0;   // lane d: runs of depth d before this warp, and in the round
        if (lane <= D) {
            for (int k = 0; k < LV_BLOCK / 32; ++k) {
                if (k < w) before += wcnt[k][lane];
                all += wcnt[k][lane];
            }
            before += run[lane];
        }
        const u64 key = i < n ? keys[i] : 0ull;
        const unsigned b1 = __ballot_sync(0xffffffffu, L < D);
        const int last = __shfl_sync(0xffffffffu, before, D - 1) + __popc(b1 & upto) - 1;   // its run of depth D - 1
        int up = 0;                // this point's run one depth above
        for (int d = 0; d <= D; ++d) {
            const unsigned b = __ballot_sync(0xffffffffu, L <= d);
            const int r = __shfl_sync(0xffffffffu, before, d) + __popc(b & upto) - 1;
            const int slot = d ? 8 * up + (int)((key >> (3 * (D - d))) & 7) : 0;
            if (L <= d) {
                lv.key[d][r] = d ? key & ~((1ull << (3 * (D - d))) - 1) : 0ull;
                lv.pidx[d][r] = (int)i;
                lv.slot[d][r] = slot;
                if (d < D) lv.lo[d][r] = last;
                if (L < d) lv.first[d - 1][up] = r;   // the first run below the run that starts above
            }
            if (d == D && i < n) point_node[i] = (int)lv.base[D] + slot;
            up = r;
        }
        __syncthreads();
        if (w == 0 && lane <= D) run[lane] += all;
        __syncthreads();
    }
}

// Every depth's nodes (one thread per slot of the depths 1..D); the empty-slot
// conventions follow updateEmptyNodeInfo (main.cu:433-490)
__global__ void k_fill_nodes(Levels lv, int D, i64 N, i64 M, NodeArrays nd) {
    for (i64 i = 1 + (i64)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (i64)gridDim.x * blockDim.x) {
        int d = 1;
        while (d < D && lv.base[d + 1] <= i) ++d;
        const i64 s = i - lv.base[d], g = s >> 3;
        const int k = (int)(s & 7), shift = 3 * (D - d);
        nd.key[i] = lv.key[d - 1][g] | ((u64)k << shift);
        nd.depth[i] = (int8_t)d;
        nd.parent[i] = (int)(lv.base[d - 1] + lv.slot[d - 1][g]);
        // the parent's children are the runs [f0, f1) of this depth, in slot order: the first at or after
        // slot k, and the first after it
        const int Ud = lv.U[d], f0 = lv.first[d - 1][g], f1 = g + 1 < lv.U[d - 1] ? lv.first[d - 1][g + 1] : Ud;
        int r = f0;
        while (r < f1 && (lv.slot[d][r] & 7) < k) ++r;
        const bool self = r < f1 && (lv.slot[d][r] & 7) == k;
        const int p0 = r < Ud ? lv.pidx[d][r] : (int)N, p1 = r + 1 < Ud ? lv.pidx[d][r + 1] : (int)N;
        nd.pidx[i] = p0;
        nd.pnum[i] = self ? p1 - p0 : 0;
        if (d == D) {
            nd.didx[i] = (int)s;
            nd.dnum[i] = 1;
        } else {
            // finest slots: 8 per run of depth D - 1
            const int l0 = r < Ud ? lv.lo[d][r] : lv.U[D - 1], l1 = r + 1 < Ud ? lv.lo[d][r + 1] : lv.U[D - 1];
            nd.didx[i] = 8 * l0;
            nd.dnum[i] = self ? 8 * (l1 - l0) : 0;
        }
        nd.child0[i] = (self && d < D) ? (int)(lv.base[d + 1] + 8 * (i64)r) : -1;
    }
}

__global__ void k_root(NodeArrays nd, i64 N, i64 countD, i64 M) {
    nd.key[0] = 0;
    nd.depth[0] = 0;
    nd.parent[0] = -1;
    nd.pidx[0] = 0;
    nd.pnum[0] = (int)N;
    nd.didx[0] = 0;
    nd.dnum[0] = (int)countD;
    nd.child0[0] = 1;
    for (int j = 0; j < 27; ++j) nd.neigh[(i64)j * M] = (j == 13) ? 0 : -1;
}

// computeNeighbor (main.cu:492-509): neighbour j of a node is a child of one of
// its parent's neighbours
// Neighbours of depth d from those of depth d-1 (main.cu:492-509): neighbour j of
// child s of P is child (s + off_j) & 1 of P's neighbour (s + off_j) >> 1 per axis,
// the values the reference's LUTs tabulate (main.cu:80-99).  The 8 children of a
// node are contiguous, so a warp takes 4 sibling groups: the first children of
// each parent's 27 neighbours are loaded once per group into shared memory, then
// every lane writes its node's 27 neighbours (coalesced along the nodes).
__global__ void __launch_bounds__(256) k_neighbours(NodeArrays nd, i64 lo, i64 ng) {
    __shared__ int cn[8][4][27];
    const i64 M = nd.M;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
    for (i64 tile = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile * 4 < ng; tile += nwarps) {
        for (int e = lane; e < 4 * 27; e += 32) {
            const i64 g = tile * 4 + e / 27;
            int v = -1;
            if (g < ng) {
                const int p = nd.parent[lo + 8 * g];
                const int np = nd.neigh[(i64)(e % 27) * M + p];
                if (np != -1) v = nd.child0[np];
            }
            cn[w][e / 27][e % 27] = v;
        }
        __syncwarp();
        const i64 g = tile * 4 + (lane >> 3);
        if (g < ng) {
            const int s = lane & 7, sx = s >> 2, sy = (s >> 1) & 1, sz = s & 1;
            const i64 i = lo + 8 * g + s;
#pragma unroll
            for (int j = 0; j < 27; ++j) {
                const int ax = sx + j / 9 - 1, ay = sy + (j / 3) % 3 - 1, az = sz + j % 3 - 1;
                const int jp = 9 * ((ax >> 1) + 1) + 3 * ((ay >> 1) + 1) + ((az >> 1) + 1);
                const int c0 = cn[w][lane >> 3][jp];
                nd.neigh[(i64)j * M + i] = c0 == -1 ? -1 : c0 + (((ax & 1) << 2) | ((ay & 1) << 1) | (az & 1));
            }
        }
        __syncwarp();
    }
}

void stage_octree(Ctx& c) {
    cudaStream_t s = c.stream;
    const int D = c.D;
    const i64 N = c.N;
    // ---- bounding box; scale and centre as the reference host code, on the device and below
    unsigned* mm = dalloc<unsigned>(6, s);
    const unsigned init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0, 0, 0};
    CK(cudaMemcpyAsync(mm, init, sizeof init, cudaMemcpyHostToDevice, s));
    k_bbox<<<grid_for(N, 256, 152 * 8), 256, 0, s>>>(c.in_xyz, N, mm);
    CK_LAUNCH();
    // ---- normalise + keys, sort, gather
    float* ptmp = dalloc<float>(3 * N, s);
    float* ntmp = dalloc<float>(3 * N, s);
    u64* keys = dalloc<u64>(N, s);
    u64* ktmp = dalloc<u64>(N, s);
    uint32_t* idx = dalloc<uint32_t>(N, s);
    uint32_t* itmp = dalloc<uint32_t>(N, s);
    k_normalise_encode<<<grid_for(N, 256), 256, 0, s>>>(c.in_xyz, c.in_nrm, N, mm, (float)(2 << D), D, ptmp, ntmp, keys);
    CK_LAUNCH();
    const int ks = c.kbegin("point_sort", (double)N * 12 * 2);
    radix_sort_pairs(keys, idx, ktmp, itmp, N, 3 * D, s);
    c.kend(ks);
    dfree(ktmp, s);
    dfree(itmp, s);
    dfree(c.pts, s); dfree(c.nrm, s); dfree(c.sort_idx, s);
    c.pts = dalloc<float>(3 * N, s);
    c.nrm = dalloc<float>(3 * N, s);
    c.sort_idx = idx;
    k_gather_points<<<grid_for(N, 256), 256, 0, s>>>(idx, N, ptmp, ntmp, c.pts, c.nrm);
    CK_LAUNCH();
    dfree(ptmp, s);
    dfree(ntmp, s);

    // ---- runs per depth; their counts and the bounding box come back in one read
    const i64 ntiles = (N + LV_TILE - 1) / LV_TILE;
    int* cnt = dalloc<int>((D + 1) * ntiles, s);
    int* dU = dalloc<int>(LV_MAX, s);
    k_run_count<<<(unsigned)ntiles, LV_BLOCK, 0, s>>>(keys, N, D, ntiles, cnt);
    CK_LAUNCH();
    k_run_offsets<<<D + 1, 1024, 0, s>>>(cnt, ntiles, dU);
    CK_LAUNCH();
    Levels lv{};
    unsigned h[6];
    CK(cudaMemcpyAsync(h, mm, sizeof h, cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(lv.U, dU, (D + 1) * sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    dfree(mm, s);
    dfree(dU, s);
    {
        const Cube cube = cube_of(h);
        for (int a = 0; a < 3; ++a) c.center[a] = cube.corner[a];
        c.scale = cube.scale;
        if (!(c.scale > 0.f) || !std::isfinite(c.scale) || !std::isfinite(c.center[0]) ||
            !std::isfinite(c.center[1]) || !std::isfinite(c.center[2])) {
            set_last_error("degenerate bounding box (all points coincide or are not finite)");
            throw Error{PRGPU_ERR_ARG, {0}};
        }
    }
    // ---- sizes
    c.count.assign(D + 1, 0);
    c.base.assign(D + 2, 0);
    c.count[0] = 1;
    for (int d = 1; d <= D; ++d) c.count[d] = 8 * (i64)lv.U[d - 1];
    for (int d = 1; d <= D + 1; ++d) c.base[d] = c.base[d - 1] + c.count[d - 1];
    const i64 M = c.base[D + 1];
    if (M > 0x7fffffffLL) {
        set_last_error("node array of %lld nodes exceeds 32-bit indexing", (long long)M);
        throw Error{PRGPU_ERR_LIMIT, {0}};
    }
    c.free_nodes();
    NodeArrays& nd = c.nodes;
    nd.M = M;
    nd.key = dalloc<u64>(M, s);
    nd.pidx = dalloc<int>(M, s);
    nd.pnum = dalloc<int>(M, s);
    nd.didx = dalloc<int>(M, s);
    nd.dnum = dalloc<int>(M, s);
    nd.parent = dalloc<int>(M, s);
    nd.child0 = dalloc<int>(M, s);
    nd.depth = dalloc<int8_t>(M, s);
    nd.neigh = dalloc<int>(27 * M, s);
    // ---- the runs of all depths, each point's leaf, and the nodes
    dfree(c.point_node, s);
    c.point_node = dalloc<int>(N, s);
    for (int d = 0; d <= D + 1; ++d) lv.base[d] = c.base[d];
    for (int d = 0; d <= D; ++d) {
        lv.key[d] = dalloc<u64>(lv.U[d], s);
        lv.pidx[d] = dalloc<int>(lv.U[d], s);
        lv.slot[d] = dalloc<int>(lv.U[d], s);
        if (d < D) {
            lv.first[d] = dalloc<int>(lv.U[d], s);
            lv.lo[d] = dalloc<int>(lv.U[d], s);
        }
    }
    k_runs<<<(unsigned)ntiles, LV_BLOCK, 0, s>>>(keys, N, D, ntiles, cnt, lv, c.point_node);
    CK_LAUNCH();
    k_root<<<1, 1, 0, s>>>(nd, N, c.count[D], M);
    CK_LAUNCH();
    k_fill_nodes<<<grid_for(M - 1, 256), 256, 0, s>>>(lv, D, N, M, nd);
    CK_LAUNCH();
    dfree(cnt, s);
    dfree(keys, s);
    for (int d = 0; d <= D; ++d) {
        dfree(lv.key[d], s); dfree(lv.pidx[d], s); dfree(lv.slot[d], s); dfree(lv.first[d], s); dfree(lv.lo[d], s);
    }
    // ---- neighbours, top-down
    const int kn = c.kbegin("neighbours", (double)M * (108 + 8 + 4 + 4));
    for (int d = 1; d <= D; ++d) {
        k_neighbours<<<grid_for(c.count[d] / 8 * 8, 256), 256, 0, s>>>(nd, c.base[d], c.count[d] / 8);
        CK_LAUNCH();
    }
    c.kend(kn);
}

}  // namespace prgpu
