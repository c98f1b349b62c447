// Iso-surface stage: implicit function at the points, iso-value, octree corner
// values, marching cubes on the finest nodes and on subdivided coarse leaves.
// Replaces main.cu:1334-1381 and 1438-4561.
//
// Differences in mechanism (not in result) from the reference:
//   * corners, edges and faces are not materialised as records; each cell finds
//     the owner of a corner/edge/face (the minimum key among the cells that
//     share it, as initVertexOwner/initEdgeArray/initFaceArray do) from its
//     neighbour table or its sibling group's, and a corner value is evaluated
//     once, by its owner;
//   * edge vertices are de-duplicated by sorting edge keys (batch, lattice
//     edge) instead of by owner back-links, one sort for the whole mesh;
//   * subdivided leaves are never expanded into node arrays: their finest cells
//     are enumerated implicitly, and the real nodes around them are reached by
//     descending from the leaf's neighbour table.
// Every vertex value, crossing position and triangle follows the reference's
// arithmetic and owner rules.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "context.h"
#include "mc_table.h"
#include "prims.cuh"

namespace prgpu {

__constant__ int c_tri_count[256];
__constant__ signed char c_tri_edges[256][16];
__constant__ signed char c_edge_v[12][2];
__constant__ signed char c_pfk[8][6];        // parentFaceKind, reference layout
__constant__ signed char c_vid[8];           // cube-vertex id of corner kind j
__constant__ signed char c_face_edges[6][4];

// the tables go to each device's constant memory once (contexts may run on several host threads)
static std::mutex g_mc_mu;
static bool g_mc_uploaded[64] = {false};
static void upload_mc_tables() {
    prgpu_mc::Tables T;
    prgpu_mc::build(T);
    signed char te[256][16], ev[12][2], pfk[8][6], vid[8], fe[6][4];
    for (int c = 0; c < 256; ++c)
        for (int k = 0; k < 16; ++k) te[c][k] = (signed char)T.tri_edges[c][k];
    for (int e = 0; e < 12; ++e) { ev[e][0] = (signed char)T.edge_v[e][0]; ev[e][1] = (signed char)T.edge_v[e][1]; }
    for (int s = 0; s < 8; ++s) {
        int xyz[3] = {s & 1, (s >> 1) & 1, (s >> 2) & 1};
        for (int j = 0; j < 6; ++j) pfk[s][j] = (signed char)((xyz[j >> 1] == (j & 1)) ? j : -1);
    }
    pfk[7][0] = 0;   // the reference table's last row also lists face 0 (MarchingCubes.cuh:716)
    for (int j = 0; j < 8; ++j) vid[j] = (signed char)prgpu_mc::vertex_id(j & 1, (j >> 1) & 1, (j >> 2) & 1);
    for (int f = 0; f < 6; ++f) {
        int a = f >> 1, sd = f & 1, n = 0;
        for (int e = 0; e < 12; ++e) {
            int o = e >> 2;
            if (o == a) continue;
            int a0 = (o == 0) ? 1 : 0;
            int off = (a == a0) ? (e & 1) : ((e >> 1) & 1);
            if (off == sd) fe[f][n++] = (signed char)e;
        }
    }
    CK(cudaMemcpyToSymbol(c_tri_count, T.tri_count, sizeof T.tri_count));
    CK(cudaMemcpyToSymbol(c_tri_edges, te, sizeof te));
    CK(cudaMemcpyToSymbol(c_edge_v, ev, sizeof ev));
    CK(cudaMemcpyToSymbol(c_pfk, pfk, sizeof pfk));
    CK(cudaMemcpyToSymbol(c_vid, vid, sizeof vid));
    CK(cudaMemcpyToSymbol(c_face_edges, fe, sizeof fe));
}
static void ensure_mc_tables() {
    int dev = 0;
    CK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_mc_mu);
    if (dev < 0 || dev >= 64) throw Error{PRGPU_ERR_LIMIT, {0}};
    if (!g_mc_uploaded[dev]) {
        upload_mc_tables();
        g_mc_uploaded[dev] = true;
    }
}

// ----------------------------- evaluation ----------------------------------
struct EvalArgs {
    NodeArrays nd;
    int D;
    const CPoly* basis;
    const float* x;
    const float* x27;      // nodes [0, nx27): x of the 27 neighbours (0: none), 28 floats per node; or null
    i64 nx27;
    const float4* lb;      // basis values at finest-lattice points by cell (see lattice_at), or null
    int stable;            // params.stable_basis: closed-form basis values (basis_stable)
};

// Basis values at the finest-lattice points, by depth-d cell c and point u = c w + k of its closure
// (0 <= k <= w = 2^(D-d)): the values at u of the functions c - 1, c, c + 1 and c + 2, those a walk at u
// through cell c multiplies with (c + 2 reaches u only at k = w; it serves corners whose owner is the
// next cell), 0 for functions that do not exist or do not reach u.  One 16-byte load per axis and level
// in place of three looked-up scalars.  Depth d starts at sum_{l<d} (2^D + 2^l) = d 2^D + 2^d - 1.
__device__ __host__ __forceinline__ i64 lattice_offset(int D, int d) { return (i64)d * (1ll << D) + (1ll << d) - 1; }
__device__ __forceinline__ float4 lattice_at(const EvalArgs& a, int d, int c, int k) {
    return a.lb[lattice_offset(a.D, d) + (i64)c * ((1 << (a.D - d)) + 1) + k];
}
// entry t of lattice_at
__device__ __forceinline__ float lattice_entry(const EvalArgs& a, int d, int c, int k, int t) {
    return reinterpret_cast<const float*>(a.lb)[4 * (lattice_offset(a.D, d) + (i64)c * ((1 << (a.D - d)) + 1) + k) + t];
}

// B_{d,n}(u / 2^D), 0 <= n < 2^d, for any finest-lattice coordinate u: from the table where u lies in the
// support [(n-1)w, (n+2)w], evaluated elsewhere (the table's values are the evaluated ones)
__device__ __forceinline__ float lattice_basis(const EvalArgs& a, int d, int n, int u) {
    const int w = 1 << (a.D - d);
    const int k = u - (n - 1) * w;
    if (k >= 0 && k <= 3 * w) {
        int c = min(u >> (a.D - d), (1 << d) - 1);   // a cell that holds u
        if (c > n + 1) --c;                          // u is the support's right end: the cell left of it
        return lattice_entry(a, d, c, u - c * w, n - c + 1);
    }
    if (a.stable) return basis_stable(d, n, (float)u * (1.0f / (float)(1 << a.D)));
    return cpoly_value<3>(a.basis[(1 << d) - 1 + n], (float)u * (1.0f / (float)(1 << a.D)));
}

__global__ void k_lattice_basis(const CPoly* __restrict__ basis, int D, i64 total, float* __restrict__ lb, int stable) {
    const float inv = 1.0f / (float)(1 << D);
    for (i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x; e < 4 * total; e += (i64)gridDim.x * blockDim.x) {
        const i64 q = e >> 2;
        int d = 0;
        while (q >= lattice_offset(D, d + 1)) ++d;
        const int w = 1 << (D - d);
        const i64 r = q - lattice_offset(D, d);
        const int c = (int)(r / (w + 1)), k = (int)(r % (w + 1)), n = c + (int)(e & 3) - 1;
        const int u = c * w + k, ks = u - (n - 1) * w;
        float v = 0.f;
        if (n >= 0 && n < (1 << d) && ks >= 0 && ks <= 3 * w) {
            const float x = (float)u * inv;
            v = stable ? basis_stable(d, n, x) : cpoly_value<3>(basis[(1 << d) - 1 + n], x);
        }
        lb[e] = v;
    }
}

// values at finest-lattice coordinate u of the functions c - 1, c, c + 1 of depth d (0 outside 0..2^d - 1)
__device__ __forceinline__ void lattice_row(const EvalArgs& a, int d, int c, int u, float bv[3]) {
    const int k = u - (c << (a.D - d));
    if ((unsigned)k <= (1u << (a.D - d))) {
        const float4 f = lattice_at(a, d, c, k);
        bv[0] = f.x; bv[1] = f.y; bv[2] = f.z;
        return;
    }
#pragma unroll 1
    for (int t = 0; t < 3; ++t) {
        const int n = c + t - 1;
        const float v = (n >= 0 && n < (1 << d)) ? lattice_basis(a, d, n, u) : 0.f;
        if (t == 0) bv[0] = v;
        else if (t == 1) bv[1] = v;
        else bv[2] = v;
    }
}

// x of the 27 neighbours of every node below the finest depth, contiguous per
// node (the evaluation walks read one 112-byte row per ancestor)
constexpr int X27_STRIDE = 28;
__global__ void k_build_x27(NodeArrays nd, const float* __restrict__ x, i64 n, float* __restrict__ x27) {
    for (i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x; e < n * X27_STRIDE; e += (i64)gridDim.x * blockDim.x) {
        const i64 i = e / X27_STRIDE;
        const int j = (int)(e % X27_STRIDE);
        float v = 0.f;
        if (j < 27) {
            const int nb = nd.neigh[(i64)j * nd.M + i];
            if (nb != -1) v = x[nb];
        }
        x27[e] = v;
    }
}

// sum over the 27 neighbours of real node 'node' (at depth d, coordinates xyz)
// of x_n * B_n(q), in neighbour order with the reference's FMA
// (calculatePointsImplicitFunctionValue main.cu:1351-1377)
__device__ __forceinline__ float level_sum(const EvalArgs& a, i64 node, int d, const int xyz[3], const float q[3],
                                           float val) {
    const int fb = (1 << d) - 1, lim = 1 << d;
    float bv[3][3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax)
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            int c = xyz[ax] + t - 1;
            bv[ax][t] = (c >= 0 && c < lim)
                            ? (a.stable ? basis_stable(d, c, q[ax]) : cpoly_value<3>(a.basis[fb + c], q[ax]))
                            : 0.f;
        }
    if (node < a.nx27) {
        // absent neighbours read 0: adding a zero product leaves the sum unchanged
        const float4* row = reinterpret_cast<const float4*>(a.x27 + node * X27_STRIDE);
        float xs[28];
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const float4 t = row[k];
            xs[4 * k] = t.x; xs[4 * k + 1] = t.y; xs[4 * k + 2] = t.z; xs[4 * k + 3] = t.w;
        }
#pragma unroll
        for (int j = 0; j < 27; ++j) val = fmaf(xs[j] * bv[0][j / 9] * bv[1][(j / 3) % 3], bv[2][j % 3], val);
        return val;
    }
    const i64 M = a.nd.M;
#pragma unroll
    for (int j = 0; j < 27; ++j) {
        const int nb = a.nd.neigh[(i64)j * M + node];
        if (nb == -1) continue;
        const float vx = bv[0][j / 9], vy = bv[1][(j / 3) % 3], vz = bv[2][j % 3];
        val = fmaf(a.x[nb] * vx * vy, vz, val);
    }
    return val;
}

// the x27 rows for nodes [0, n) on the stage's stream; null when n is 0
inline float* build_x27(const Ctx& c, i64 n) {
    if (n <= 0) return nullptr;
    float* x27 = dalloc<float>(n * X27_STRIDE, c.stream);
    k_build_x27<<<grid_for(n * X27_STRIDE, 256), 256, 0, c.stream>>>(c.nodes, c.x, n, x27);
    CK_LAUNCH();
    return x27;
}

// level_sum at a finest-lattice point u (q = u / 2^D), basis values from the table
__device__ __forceinline__ float level_sum_u(const EvalArgs& a, i64 node, int d, const int xyz[3], const int u[3],
                                             float val) {
    float bv[3][3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) lattice_row(a, d, xyz[ax], u[ax], bv[ax]);
    if (node < a.nx27) {
        const float4* row = reinterpret_cast<const float4*>(a.x27 + node * X27_STRIDE);
        float xs[28];
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const float4 t = row[k];
            xs[4 * k] = t.x; xs[4 * k + 1] = t.y; xs[4 * k + 2] = t.z; xs[4 * k + 3] = t.w;
        }
#pragma unroll
        for (int j = 0; j < 27; ++j) val = fmaf(xs[j] * bv[0][j / 9] * bv[1][(j / 3) % 3], bv[2][j % 3], val);
        return val;
    }
    const i64 M = a.nd.M;
#pragma unroll
    for (int j = 0; j < 27; ++j) {
        const int nb = a.nd.neigh[(i64)j * M + node];
        if (nb == -1) continue;
        val = fmaf(a.x[nb] * bv[0][j / 9] * bv[1][(j / 3) % 3], bv[2][j % 3], val);
    }
    return val;
}
// from a node to the root: a parent is one depth up and its cell coordinates are the
// child's halved, so the node's key is decoded once
__device__ __forceinline__ float walk_up_u(const EvalArgs& a, i64 node, const int u[3], float val) {
    if (node == -1) return val;
    int d = a.nd.depth[node];
    int xyz[3];
    key_coords(a.nd.key[node], d, a.D, xyz);
    while (node != -1) {
        val = level_sum_u(a, node, d, xyz, u, val);
        node = a.nd.parent[node];
        --d;
        xyz[0] >>= 1; xyz[1] >>= 1; xyz[2] >>= 1;
    }
    return val;
}

__device__ __forceinline__ float walk_up(const EvalArgs& a, i64 node, const float q[3], float val) {
    if (node == -1) return val;
    int d = a.nd.depth[node];
    int xyz[3];
    key_coords(a.nd.key[node], d, a.D, xyz);
    while (node != -1) {
        val = level_sum(a, node, d, xyz, q, val);
        node = a.nd.parent[node];
        --d;
        xyz[0] >>= 1; xyz[1] >>= 1; xyz[2] >>= 1;
    }
    return val;
}

// the iso-value sum: sum of f(p), or of w(p) f(p) with density weights (mean 1)
__global__ void k_point_values(EvalArgs a, const float* __restrict__ pts, const int* __restrict__ point_node, i64 n,
                               const float* __restrict__ weight, float* __restrict__ out, double* __restrict__ sum) {
    double loc = 0;
    for (i64 k = (i64)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (i64)gridDim.x * blockDim.x) {
        const float q[3] = {pts[3 * k], pts[3 * k + 1], pts[3 * k + 2]};
        const float v = walk_up(a, point_node[k], q, 0.f);
        out[k] = v;
        if (weight) loc += (double)v * (double)weight[k];
        else loc += (double)v;
    }
    for (int o = 16; o; o >>= 1) loc += __shfl_xor_sync(0xffffffffu, loc, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(sum, loc);
}

void stage_points(Ctx& c) {
    cudaStream_t s = c.stream;
    dfree(c.point_value, s);
    c.point_value = dalloc<float>(c.N, s);
    double* sum = dalloc<double>(1, s);
    CK(cudaMemsetAsync(sum, 0, sizeof(double), s));
    float* x27 = build_x27(c, c.base[c.D]);
    EvalArgs a{c.nodes, c.D, c.basis, c.x, x27, x27 ? c.base[c.D] : 0, nullptr, c.params.stable_basis};
    const int kt = c.kbegin("point_values", (double)c.N * (12 + 4 + 4) + (double)c.nodes.M * (4 + 4 + 8 + 108));
    k_point_values<<<grid_for(c.N, 128, 1ll << 30), 128, 0, s>>>(a, c.pts, c.point_node, c.N, c.point_weight,
                                                                 c.point_value, sum);
    CK_LAUNCH();
    c.kend(kt);
    double h = read_scalar(sum, s);
    dfree(sum, s);
    dfree(x27, s);
    c.iso = (float)h / (float)c.N;
}

// ------------------------------ corners -------------------------------------
// A corner's value is its owner's (computeVertexImplicitFunctionValue main.cu:2259-2326): the walk from the owner to
// the root, then, where the owner has children, the descent through children[childrenVertexKind[kind]] added here
__device__ __forceinline__ float corner_descent(const EvalArgs& a, i64 node, int d, int kind, int cx, int cy, int cz,
                                                const int u[3], float val) {
    const int exceed = c_vid[kind];
    int c[3] = {cx, cy, cz};
    for (int dd = d + 1; dd <= a.D; ++dd) {
        const int c0 = a.nd.child0[node];
        if (c0 == -1) break;
        node = c0 + exceed;   // child 'exceed': its coordinates are the parent's doubled plus its bits
        c[0] = (c[0] << 1) | ((exceed >> 2) & 1);
        c[1] = (c[1] << 1) | ((exceed >> 1) & 1);
        c[2] = (c[2] << 1) | (exceed & 1);
        val = level_sum_u(a, node, dd, c, u, val);
    }
    return val;
}

// Cells in tiles of CELL_TILE: the kernels that find the categories sum each tile's triangles, the sums are
// scanned, and the emission kernels place a tile's active cells and triangles by a scan in the block.  (Lists
// of active cells and triangle offsets, built by flags, scans and gathers over all cells, took a dozen
// launches and as many bytes as the cells' corner values.)
constexpr int CELL_BLOCK = 256;
constexpr int CELL_ITEMS = 4;
constexpr int CELL_TILE = CELL_ITEMS * CELL_BLOCK;
__device__ __forceinline__ void tile_triangles(int n, int* __restrict__ tile_tri) {
    __shared__ int s_n[CELL_BLOCK / 32];
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0) s_n[threadIdx.x >> 5] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int k = 0; k < CELL_BLOCK / 32; ++k) t += s_n[k];
        tile_tri[blockIdx.x] = t;
    }
}
// The tile's active cells: cell (in the tile) of each of its triangles, and each cell's first triangle, in
// shared memory; returns the tile's triangles.  All threads call.
struct TileShared {
    unsigned short cell[5 * CELL_TILE];   // of triangle t (a cell has at most 5)
    unsigned short first[CELL_TILE];      // first triangle of a cell
    int sw[32];
};
__device__ __forceinline__ int tile_active(const unsigned char* __restrict__ cat, i64 total, TileShared& sm) {
    const i64 c0 = (i64)blockIdx.x * CELL_TILE + CELL_ITEMS * threadIdx.x;
    int nt[CELL_ITEMS], mine = 0;
#pragma unroll
    for (int k = 0; k < CELL_ITEMS; ++k) {
        nt[k] = c0 + k < total ? c_tri_count[cat[c0 + k]] : 0;
        mine += nt[k];
    }
    int all;
    int at = block_exclusive_sum<int>(mine, sm.sw, &all);
#pragma unroll
    for (int k = 0; k < CELL_ITEMS; ++k) {
        const int cell = CELL_ITEMS * (int)threadIdx.x + k;
        sm.first[cell] = (unsigned short)at;
        for (int t = 0; t < nt[k]; ++t) sm.cell[at++] = (unsigned short)cell;
    }
    __syncthreads();
    return all;
}

// cube category of each finest cell, the tile's triangles
__global__ void __launch_bounds__(CELL_BLOCK) k_finest_cells(const float* __restrict__ cell_v, i64 n,
                                                             unsigned char* __restrict__ cat, int* __restrict__ tile_tri) {
    int tri = 0;
    for (int q = 0; q < CELL_TILE / CELL_BLOCK; ++q) {
        const i64 l = (i64)blockIdx.x * CELL_TILE + q * CELL_BLOCK + threadIdx.x;
        if (l >= n) break;
        const float4 v0 = reinterpret_cast<const float4*>(cell_v + 8 * l)[0], v1 = reinterpret_cast<const float4*>(cell_v + 8 * l)[1];
        const float cv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        int cc = 0;
#pragma unroll
        for (int kind = 0; kind < 8; ++kind)
            if (cv[kind] < 0.f) cc |= 1 << c_vid[kind];
        cat[l] = (unsigned char)cc;
        tri += c_tri_count[cc];
    }
    tile_triangles(tri, tile_tri);
}

// ------------------------------- faces ---------------------------------------
// owner record of face j of node n: (owner node, face kind in its frame)
__device__ __forceinline__ void face_owner(const NodeArrays& nd, i64 n, int j, int& o, int& k) {
    const int ax = j >> 1, sd = j & 1;
    int dxyz[3] = {0, 0, 0};
    dxyz[ax] = sd ? 1 : -1;
    const int jj = 9 * (dxyz[0] + 1) + 3 * (dxyz[1] + 1) + (dxyz[2] + 1);
    const int nb = nd.neigh[(i64)jj * nd.M + n];
    if (nb != -1 && nd.key[nb] < nd.key[n]) { o = nb; k = j ^ 1; }
    else { o = (int)n; k = j; }
}
__device__ __forceinline__ int face_has_parent(const NodeArrays& nd, int o, int k, int D) {
    if (nd.parent[o] == -1) return -1;
    const int d = nd.depth[o];
    const int son = (int)((nd.key[o] >> (3 * (D - d))) & 7);
    return c_pfk[son][k] != -1 ? 1 : -1;
}

// surface-intersection marks (generateTrianglePos main.cu:2736-2755)
__global__ void k_mark_faces(NodeArrays nd, int D, i64 lo, i64 hi, const unsigned char* __restrict__ cat,
                             int* __restrict__ fflag) {
    for (i64 i = lo + (i64)blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += (i64)gridDim.x * blockDim.x) {
        const int cc = cat[i - lo];
        const int nt = c_tri_count[cc];
        if (!nt) continue;
        int used = 0;
        for (int t = 0; t < 3 * nt; ++t) used |= 1 << c_tri_edges[cc][t];
        for (int j = 0; j < 6; ++j) {
            int m = 0;
            for (int q = 0; q < 4; ++q) m |= (used >> c_face_edges[j][q]) & 1;
            if (!m) continue;
            int o, k;
            face_owner(nd, i, j, o, k);
            fflag[6 * (i64)o + k] = 1;
            int par = nd.parent[i];
            while (face_has_parent(nd, o, k, D) != -1) {
                face_owner(nd, par, j, o, k);
                par = nd.parent[par];
                fflag[6 * (i64)o + k] = 1;
            }
        }
    }
}

// leaves above the finest depth: sign change at their corners or a marked face
// (ProcessLeafNodesAtOtherDepth main.cu:2957-2986, ifSubdivide :2988-2992)
__global__ void __launch_bounds__(128) k_coarse_leaves(NodeArrays nd, i64 lo, i64 hi, const float* __restrict__ leaf_v,
                                const int* __restrict__ fflag, int* __restrict__ has_tri, int* __restrict__ has_int,
                                int* __restrict__ is_root) {
    for (i64 i = lo + (i64)blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += (i64)gridDim.x * blockDim.x) {
        if (nd.child0[i] != -1) { is_root[i] = 0; continue; }
        const float4 v0 = reinterpret_cast<const float4*>(leaf_v + 8 * i)[0], v1 = reinterpret_cast<const float4*>(leaf_v + 8 * i)[1];
        const float cv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        float v[8];
#pragma unroll
        for (int kind = 0; kind < 8; ++kind) v[kind ^ ((kind >> 1) & 1)] = cv[kind];   // c_vid: the cube's vertex order
        const int sign = v[0] < 0 ? -1 : 1;
        int ht = 0;
        for (int j = 1; j < 8; ++j)
            if ((float)sign * v[j] < 0) { ht = 1; break; }
        int hi2 = 0;
        for (int j = 0; j < 6; ++j) {
            int o, k;
            face_owner(nd, i, j, o, k);
            if (fflag[6 * (i64)o + k]) { hi2 = 1; break; }
        }
        has_tri[i] = ht;
        has_int[i] = hi2;
        is_root[i] = (ht || hi2) ? 1 : 0;
    }
}

// ------------------------ subdivided leaves (virtual) ------------------------
struct VRoot {
    int node;          // real empty leaf
    int depth;         // r
    int batch;         // vertex-sharing batch id (1-based)
    int pad;
};

struct VArgs {
    EvalArgs e;
    const VRoot* roots;
    int nroots;
    const int* batch_root_flag;   // per node: batch id if the node is a root of a depth batch (>= 3), else 0
    float iso;
};

// real node at depth d with coordinates c[] reached from the depth-r node a
// (its ancestor), or -1
__device__ __forceinline__ i64 descend(const NodeArrays& nd, i64 a, int r, int d, const int c[3]) {
    i64 node = a;
    for (int l = r + 1; l <= d; ++l) {
        const int c0 = nd.child0[node];
        if (c0 == -1) return -1;
        const int b = d - l;
        const int k = (((c[0] >> b) & 1) << 2) | (((c[1] >> b) & 1) << 1) | ((c[2] >> b) & 1);
        node = c0 + k;
    }
    return node;
}

// is the finest cell 'cell' (depth-D coordinates) a member of the batch of root R?
// If so returns the root node that contains it (R or another root of R's depth batch).
__device__ __forceinline__ int batch_member(const VArgs& v, const VRoot& R, const int Lc[3], const int cell[3]) {
    const int D = v.e.D, sh = D - R.depth;
    const int lim = 1 << D;
    if (cell[0] < 0 || cell[1] < 0 || cell[2] < 0 || cell[0] >= lim || cell[1] >= lim || cell[2] >= lim) return -1;
    const int A[3] = {cell[0] >> sh, cell[1] >> sh, cell[2] >> sh};
    const int dx = A[0] - Lc[0], dy = A[1] - Lc[1], dz = A[2] - Lc[2];
    if (!dx && !dy && !dz) return R.node;
    if (R.depth < 3) return -1;                 // single-root batch
    const int j = 9 * (dx + 1) + 3 * (dy + 1) + (dz + 1);
    const int nb = v.e.nd.neigh[(i64)j * v.e.nd.M + R.node];
    if (nb == -1) return -1;
    return (v.batch_root_flag[nb] == R.batch) ? nb : -1;
}

// value at finest corner q (lattice coordinates) for a walk starting at the
// finest cell 'oc' inside root node L (computeSubdivideVertexImplicitFunctionValue
// main.cu:2328-2442): virtual levels contribute only the real nodes around them
__device__ float virtual_corner_value(const VArgs& v, int L, int r, const int oc[3], const int qc[3]) {
    const EvalArgs& a = v.e;
    const NodeArrays& nd = a.nd;
    const int D = a.D;
    int Lc[3];
    key_coords(nd.key[L], r, D, Lc);
    float val = 0.f;
    for (int d = D; d > r; --d) {
        const int sh = D - d;
        const int V[3] = {oc[0] >> sh, oc[1] >> sh, oc[2] >> sh};
        const int lim = 1 << d;
        // a virtual cell whose 3x3x3 block lies inside the leaf has no real neighbour
        const int span = 1 << (d - r);
        bool inner = true;
        for (int ax = 0; ax < 3; ++ax) {
            const int lo = Lc[ax] * span;
            if (V[ax] - 1 < lo || V[ax] + 1 >= lo + span) inner = false;
        }
        if (inner) continue;
        float bv[3][3];
        for (int ax = 0; ax < 3; ++ax) lattice_row(a, d, V[ax], qc[ax], bv[ax]);
        for (int j = 0; j < 27; ++j) {
            const int N[3] = {V[0] + j / 9 - 1, V[1] + (j / 3) % 3 - 1, V[2] + j % 3 - 1};
            if (N[0] < 0 || N[1] < 0 || N[2] < 0 || N[0] >= lim || N[1] >= lim || N[2] >= lim) continue;
            const int s2 = d - r;
            const int A[3] = {N[0] >> s2, N[1] >> s2, N[2] >> s2};
            const int ddx = A[0] - Lc[0], ddy = A[1] - Lc[1], ddz = A[2] - Lc[2];
            if (!ddx && !ddy && !ddz) continue;    // inside the subdivided leaf: no coefficient
            const int jj = 9 * (ddx + 1) + 3 * (ddy + 1) + (ddz + 1);
            const int an = nd.neigh[(i64)jj * nd.M + L];
            if (an == -1) continue;
            const i64 node = descend(nd, an, r, d, N);
            if (node < 0) continue;
            const float vx = bv[0][j / 9], vy = bv[1][(j / 3) % 3], vz = bv[2][j % 3];
            val = fmaf(a.x[node] * vx * vy, vz, val);
        }
    }
    // the leaf itself and its real ancestors
    val = walk_up_u(a, L, qc, val);
    return val;
}

__device__ __forceinline__ u64 cell_key_D(const int c[3], int D) { return coords_key(c[0], c[1], c[2], D, D); }

// ---- subdivided leaves in bricks: the leaf's lattice of finest cells is cut
// into bricks of B^3 cells, B = min(lattice edge, 8).
//
// Most corners of a subdivided leaf lie far from the surface.  Each brick is
// bounded before any of its corners is evaluated:
//   * every term of a corner value is x_n * B_x * B_y * B_z with the
//     single-precision basis values the evaluation uses, so the range of a term
//     over the corners that include it is an interval product; terms that only
//     some corners include get intervals widened to 0;
//   * the rounding of the FMA chain is at most (K + 4) u sum|term| for K terms
//     (u = 2^-24);
//   * a brick whose bound proves that every corner value has the same sign as
//     (value - iso) is culled: none of its cells carries a triangle and its
//     corners are never read.
// The surviving ("live") bricks are evaluated exactly, in the order of
// virtual_corner_value, so culling changes no value.  Corners on the leaf's
// lower faces may be owned by a cell of another leaf of the same depth batch
// ("foreign" corners): their virtual depths read the same window (a real node
// is the same node in either leaf's frame, and every cell inside either leaf
// reads 0), their real ancestors are the owner's.  Such a corner is a corner
// of the owner leaf's brick that contains its owner cell, where the owner's own
// bound covers it; so a brick with foreign corners is culled only when its own
// bound and those of the owner bricks prove the same sign.
//
// The basis values a brick's corners use along one axis depend only on the
// leaf, the axis and the brick's index along it (a "brick row"):
//   BT[d][t][k]   basis value at corner k of the function of cell V_k + t - 1
//                 (depth d > r, V_k = (corner - 1) >> (D - d), t = 0..3; t = 3
//                 serves owner cells V_k + 1) or of ancestor cell + t - 1
//                 (depth d <= r); read per live brick from the lattice table
//   RA[l][t]      range over k of BT[l][t][k], l <= r
//   RW[d][n]      range (with 0) of the depth-d function of window cell n over
//                 the corners whose owner cell is within one cell of it
// RA and RW are tabulated once per row by k_brick_rows for the bounds.
constexpr int BR = 8;              // largest brick edge (cells); corners per axis up to BR+1
constexpr int BR1 = BR + 1;
constexpr int BR_CORNERS = BR1 * BR1 * BR1;
constexpr int BR_LEVELS = 16;      // depths 0..15
constexpr int BR_WEXT = BR + 4;    // window cells per axis in the row tables (at most 11 are used)
// window cells over all virtual depths of a brick of edge 8 whose first corner is a multiple of 8: per
// axis the owner cells of its corners (8 cells and the one below) and one more to each side, 11, 7 and 5
// cells at the finest depths and 4 at the others: 11^3 + 7^3 + 5^3 + 12 * 4^3 = 2567
constexpr int BR_XW = 2568;
// Row table of a brick or super-brick of edge E, 24 floats per depth d > r (the ancestors, d <= r, are one
// polynomial per leaf):
//   d <= D - lg E  PW[n]  window cell n < 4: Bernstein form over the brick's corners (b0, b1, b2, M,
//                         see bern_fit) of its function, masked as RW is; the function's knots are
//                         multiples of its cell width 2^(D-d) >= E, so it is one quadratic piece there
//   d >  D - lg E  RW[n]  as above (12 cells, range with 0; bricks only)
constexpr int PROW = 24;
constexpr int PW = 4;              // window cells per axis at the depths of knot spacing >= E
constexpr int ANC_STRIDE = 32;     // per root: Bernstein coefficients C[27] of the ancestors, S3, count, FIT
constexpr int SUPER = 4 * BR;      // edge of a super-brick (leaves of lattice edge >= 64)
constexpr int BELOW = 5;           // depths below a node whose range of x k_x_below keeps

__device__ __forceinline__ int brick_edge(int D, int r) { return min(1 << (D - r), BR); }

// 16 bytes from global to shared memory without a register in between; async_wait returns when this thread's are there
__device__ __forceinline__ void async_copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Roots are in depth order and every root of depth d has the same number of bricks
// (8^lg[d]) and super-bricks (8^slg[d]), so the root of a brick follows from the
// per-depth counts without a search.
struct DepthLayout {
    int first[17];                 // first root of depth d
    int lg[17], slg[17];           // log2 of bricks (super-bricks) per leaf edge at depth d
    i64 boff[17], soff[17];        // bricks (super-bricks) of the roots above depth d
    i64 roff[17], sroff[17];       // brick rows (super-brick rows) of the roots above depth d
};
struct BrickIndex {                // bricks of all subdivided leaves, numbered root by root
    const i64* prefix;             // first brick of each root
    const i64* row_prefix;         // first brick row of each root (3 * bricks per edge rows each)
    int nroots;
    const float* rows;             // brick-row tables, PROW (D+1) floats each
    const int* up;                 // per root: its node and its ancestors by depth, BR_LEVELS each
    const float* anc;              // per root: the ancestor polynomial, ANC_STRIDE floats
    const float2* below;           // k_x_below
    i64 below0;                    // its first node
    const float2* bsum;            // k_basis_sums, per depth
    DepthLayout dl;
};
struct VBrick {
    int root;                      // index into roots
    int b[3];                      // brick coordinates in the leaf
};
__device__ __forceinline__ VBrick brick_of(const VArgs& v, const BrickIndex& bx, i64 g) {
    const DepthLayout& L = bx.dl;
    int d = 0;
    while (d < v.e.D - 1 && L.boff[d + 1] <= g) ++d;   // roots are coarse nodes: depth < D
    const i64 loc = g - L.boff[d];
    const int lg = L.lg[d];
    VBrick b;
    b.root = L.first[d] + (int)(loc >> (3 * lg));
    const i64 l = loc & ((1ll << (3 * lg)) - 1);
    const int m = (1 << lg) - 1;
    b.b[0] = (int)(l >> (2 * lg));
    b.b[1] = (int)(l >> lg) & m;
    b.b[2] = (int)l & m;
    return b;
}
__device__ __forceinline__ const float* brick_row(const float* rows, const i64* row_prefix, int D, int root, int nb,
                                                  int ax, int b) {
    return rows + (row_prefix[root] + (i64)ax * nb + b) * (i64)(PROW * (D + 1));
}

__device__ __forceinline__ float f4_at(const float4& f, int i) { return i == 0 ? f.x : (i == 1 ? f.y : f.z); }

// Bernstein form over the corners k = 0..K (K a power of two <= 2^15) of a function tabulated
// there, val(k), that is one quadratic piece over them in exact arithmetic: b0 = v(0), b2 = v(K),
// b1 = 2 v(K/2) - (b0 + b2) / 2 (the quadratic Q through the three), returned as (b0, b1, b2, delta)
// with delta >= max_k |Q(k) - v(k)|.  The tabulated values are the reference's float evaluations of
// shifted polynomials, whose error grows about 4x per depth (near 1e-3 at depth 8 of a depth-10
// tree), so delta is that noise rather than rounding.  Q(k) = b0 B0 + b1 B1 + b2 B2 with
// B0 = (K-k)^2 / K^2, B1 = 2k(K-k) / K^2, B2 = k^2 / K^2 (exact in float for K <= 2^12, else rounded
// once); its float evaluation is within 4u max|b| of Q (the 5u max|b| term), a float |a - b| is
// within u of exact (the factor 1 + 2^-20), and the factor 1 + 2^-16 covers the last roundings.
template <class F>
__device__ __forceinline__ float4 bern_fit(F val, int K) {
    const float v0 = val(0), vm = val(K >> 1), vK = val(K);
    const float b1 = 2.0f * vm - 0.5f * (v0 + vK);
    const float mb = fmaxf(fmaxf(fabsf(v0), fabsf(vK)), fabsf(b1));
    const float inv = 1.0f / ((float)K * (float)K);   // a power of two: exact
    float dmax = 0.f;
    for (int k = 0; k <= K; ++k) {
        const float vk = val(k);
        const float B0 = (float)((K - k) * (K - k)) * inv, B1 = (float)(2 * k * (K - k)) * inv,
                    B2 = (float)(k * k) * inv;
        const float q = fmaf(v0, B0, fmaf(b1, B1, vK * B2));
        dmax = fmaxf(dmax, fabsf(q - vk));
    }
    const float u = 5.9604644775390625e-08f;   // 2^-24
    const float delta = (dmax * (1.0f + 9.5367431640625e-07f) + 5.0f * u * mb) * (1.0f + 1.52587890625e-05f);
    return make_float4(v0, b1, vK, delta);
}

// M = max|b_i| + delta for an entry (b0, b1, b2, delta) of bern_fit: it bounds |Q| (a Bernstein
// form lies within its coefficients' range) and |v(k)| <= |Q(k)| + delta; rounded up
__device__ __forceinline__ float bern_m(const float4& f) {
    return (fmaxf(fmaxf(fabsf(f.x), fabsf(f.y)), fabsf(f.z)) + f.w) * (1.0f + 9.5367431640625e-07f);
}

// real node at depth d with coordinates N near leaf L (depth r, coords Lc), or -1 (none, or inside L)
__device__ i64 shell_node(const VArgs& v, int L, int r, const int Lc[3], int d, const int N[3]) {
    const NodeArrays& nd = v.e.nd;
    const int lim = 1 << d;
    if (N[0] < 0 || N[1] < 0 || N[2] < 0 || N[0] >= lim || N[1] >= lim || N[2] >= lim) return -1;
    const int s2 = d - r;
    const int dx = (N[0] >> s2) - Lc[0], dy = (N[1] >> s2) - Lc[1], dz = (N[2] >> s2) - Lc[2];
    if (!dx && !dy && !dz) return -1;
    if (dx < -1 || dx > 1 || dy < -1 || dy > 1 || dz < -1 || dz > 1) return -1;   // not a neighbour's cell
    const int an = nd.neigh[(i64)(9 * (dx + 1) + 3 * (dy + 1) + (dz + 1)) * nd.M + L];
    if (an == -1) return -1;
    return descend(nd, an, r, d, N);
}

// can a corner of brick b[] (nb bricks per edge) be owned by a cell of another
// leaf of the batch?  The candidate cells of a corner lie in the leaf or in a
// neighbour at offset (dx,dy,dz): -1 on an axis only for corners on the leaf's
// lower face there, +1 only for corners on its upper face.  A cell outside the
// leaf can have the least key only if one offset is -1 (Morton order is
// monotone per axis).  So: only if such a neighbour is a root of the same batch
// (batch_member's rule)
// (the test for the neighbour at offset j, given that it is such a root)
__device__ __forceinline__ bool foreign_neighbour(int j, const int b[3], int nb) {
    const int off[3] = {j / 9 - 1, (j / 3) % 3 - 1, j % 3 - 1};
    bool lower = false, allowed = true;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        if (off[ax] == -1) { lower = true; if (b[ax] != 0) allowed = false; }
        if (off[ax] == 1 && b[ax] != nb - 1) allowed = false;
    }
    return lower && allowed;
}

// window of depth d around a brick (edge B) along one axis: origin and extent
// of the cells the brick's owner cells can reach; 'cross' when that reaches outside the leaf
__device__ __forceinline__ void window_axis(int g0, int B, int Lc_ax, int r, int d, int D, int& wlo, int& ext, bool& cross) {
    const int sh = D - d, span = 1 << (d - r);
    const int llo = Lc_ax * span;
    // the first corner's owner cell: the one below it, or its own on the leaf's lower face
    const int Vlo = (g0 == (llo << sh)) ? (g0 >> sh) : ((g0 - 1) >> sh), Vhi = (g0 + B - 1) >> sh;
    cross = (Vlo - 1 < llo || Vhi + 1 >= llo + span);
    wlo = Vlo - 1;
    ext = Vhi - Vlo + 3;
}

// BT[d][0..3][k] of the brick row starting at corner g0 (see above): the corner is in the closure of its
// ancestor cell (d <= r) or of the cell below it.  The corner 0 has no cell below it: the functions
// -2..1 there are those of cell 0 moved by one.
__device__ __forceinline__ float4 brick_bt(const EvalArgs& a, int r, int Lc_ax, int g0, int d, int k) {
    const int u = g0 + k, sh = a.D - d;
    const int c = (d <= r) ? (Lc_ax >> (r - d)) : ((u - 1) >> sh);
    if (c < 0) {
        const float4 f = lattice_at(a, d, 0, 0);
        return make_float4(0.f, f.x, f.y, f.z);
    }
    return lattice_at(a, d, c, u - (c << sh));
}

// a / n for 0 <= a < 2^14 and 1 <= n <= 2^10 through the reciprocal inv = 1/n:
// (a + 0.5)/n lies at least 0.5/n from an integer and the float product is
// within 2^-9 of it, so truncation gives the quotient
__device__ __forceinline__ int small_div(int a, float inv) { return __float2int_rz(((float)a + 0.5f) * inv); }

// the part of a window box [wlo, wlo+ext) outside the leaf's box [llo, llo+span)
// (per axis, at one depth) as at most 6 disjoint boxes
struct Box3 {
    int lo[3];
    int n[3];
};
__device__ __forceinline__ int outside_boxes(const int wlo[3], const int ext[3], const int llo[3], int span,
                                             Box3 out[6]) {
    int lo[3] = {wlo[0], wlo[1], wlo[2]}, hi[3] = {wlo[0] + ext[0], wlo[1] + ext[1], wlo[2] + ext[2]};
    int nb = 0;
    for (int ax = 0; ax < 3; ++ax) {
        const int a = max(lo[ax], llo[ax]), b = min(hi[ax], llo[ax] + span);
        if (a >= b) {   // no overlap along this axis: the rest is outside
            Box3 bx;
            for (int q = 0; q < 3; ++q) { bx.lo[q] = lo[q]; bx.n[q] = hi[q] - lo[q]; }
            out[nb++] = bx;
            return nb;
        }
        if (lo[ax] < a) {
            Box3 bx;
            for (int q = 0; q < 3; ++q) { bx.lo[q] = lo[q]; bx.n[q] = hi[q] - lo[q]; }
            bx.n[ax] = a - lo[ax];
            out[nb++] = bx;
        }
        if (b < hi[ax]) {
            Box3 bx;
            for (int q = 0; q < 3; ++q) { bx.lo[q] = lo[q]; bx.n[q] = hi[q] - lo[q]; }
            bx.lo[ax] = b;
            bx.n[ax] = hi[ax] - b;
            out[nb++] = bx;
        }
        lo[ax] = a;
        hi[ax] = b;
    }
    return nb;   // what is left lies inside the leaf
}

// root k's batch id on its node (depth >= 3; shallower roots are single-root batches)
__global__ void k_batch_flags(const VRoot* __restrict__ roots, int nroots, int* __restrict__ bflag) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nroots; k += gridDim.x * blockDim.x)
        if (roots[k].depth >= 3) bflag[roots[k].node] = roots[k].batch;
}

// edge of the bricks (super == 0) or of the super-bricks (super == 1: 4^3 bricks of 8^3
// cells, in leaves with lattice edge >= 64; 0 elsewhere)
__device__ __forceinline__ int row_edge(int D, int r, int super) {
    return super ? ((D - r >= 6) ? SUPER : 0) : brick_edge(D, r);
}

// one thread per (brick row, depth); rows numbered root by root (row_prefix), 3 x bricks-per-edge each
// (rows of a single-brick leaf whose real corners change sign are skipped: k_brick_bound leaves
// such a brick unproven without reading them)
__global__ void k_brick_rows(VArgs v, DepthLayout dl, i64 nrows, int super, const int* __restrict__ has_tri,
                             float* __restrict__ rows) {
    const EvalArgs& a = v.e;
    const int D = a.D;
    const i64* off = super ? dl.sroff : dl.roff;
    for (i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x; e < nrows * (D + 1); e += (i64)gridDim.x * blockDim.x) {
        const i64 row = e / (D + 1);
        const int d = (int)(e % (D + 1));
        // the root from the per-depth layout: 3 * 2^lg rows per root of depth dd
        int dd = 0;
        while (dd < D - 1 && off[dd + 1] <= row) ++dd;
        const int nbk = 1 << (super ? dl.slg[dd] : dl.lg[dd]);
        const i64 loc = row - off[dd];
        const int root = dl.first[dd] + (int)(loc / (3 * nbk));
        const int rl = (int)(loc % (3 * nbk));
        const int4 rd = make_int4(root, rl / nbk, rl % nbk, 0);   // root, axis, brick index
        const VRoot R = v.roots[rd.x];
        if (!super && nbk == 1 && has_tri[R.node]) continue;
        const int ax = rd.y, r = R.depth, S = 1 << (D - r), B = row_edge(D, r, super);
        int Lc[3];
        key_coords(a.nd.key[R.node], r, D, Lc);
        const int g0 = Lc[ax] * S + rd.z * B;
        const int c0 = rd.z * B;
        float* out = rows + row * (i64)(PROW * (D + 1));
        if (d <= r) continue;   // the leaf's ancestor polynomial (k_brick_xl)
        {
            int wlo, ext;
            bool cross;
            window_axis(g0, B, Lc[ax], r, d, D, wlo, ext, cross);
            const int sh = D - d, lim = 1 << d;
            // the term of window cell N at corner k: its basis value where the corner's owner cell
            // (the lower-face corner owns its own cell) is within one cell of N, else 0
            auto term = [&](int N, int k) {
                const int Va = (k == 0 && c0 == 0) ? (g0 >> sh) : ((g0 + k - 1) >> sh);
                return (N < Va - 1 || N > Va + 1) ? 0.f : lattice_entry(a, d, Va, g0 + k - (Va << sh), N - Va + 1);
            };
            if ((1 << sh) >= B) {
                float4* pw = reinterpret_cast<float4*>(out + d * PROW);
                for (int n = 0; n < PW; ++n) {
                    const int N = wlo + n;
                    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (n < ext && N >= 0 && N < lim) f = bern_fit([&](int k) { return term(N, k); }, B);
                    pw[n] = f;
                }
                continue;
            }
            if (super) continue;   // k_super_bound reads no ranges
            float* rw = out + d * PROW;
            for (int n = 0; n < BR_WEXT; ++n) {
                const int N = wlo + n;
                float mn = 0.f, mx = 0.f;             // 0: corners without this term
                if (n < ext && N >= 0 && N < lim) {
                    for (int k = 0; k <= B; ++k) {
                        const float b = term(N, k);
                        mn = fminf(mn, b);
                        mx = fmaxf(mx, b);
                    }
                }
                rw[n * 2] = mn;
                rw[n * 2 + 1] = mx;
            }
        }
    }
}

// per root: its node and its ancestors, by depth (their x27 rows hold the neighbours' x of each level)
__global__ void k_root_up(NodeArrays nd, const VRoot* __restrict__ roots, int nroots, int* __restrict__ up) {
    for (i64 k = (i64)blockIdx.x * blockDim.x + threadIdx.x; k < nroots; k += (i64)gridDim.x * blockDim.x) {
        int node = roots[k].node;
        for (int l = roots[k].depth; l >= 0; --l) {
            up[k * BR_LEVELS + l] = node;
            node = nd.parent[node];
        }
    }
}

// Per root: the leaf's ancestor polynomial (anc, for the bounds).  Every ancestor function is one
// quadratic piece per axis over the leaf (its knots are multiples of its cell width, and the leaf
// lies in one such cell), so the ancestors' sum is one tri-quadratic over the leaf, kept in
// Bernstein form over t = (corner - leaf origin) / S per axis:
//   C[9i + 3j + l] = sum over levels and neighbours of x * bx_i * by_j * bz_l   (bern_fit's b)
// (lane k computes coefficient k, per level as sum_jx bx_i (sum_jy by_j (sum_jz x bz_l))), then
// S3 = sum |x| Mx My Mz, the number of terms and FIT = sum |x| (dx My Mz + Mx dy Mz + Mx My dz)
// (d the fits' residuals, M = bern_m), which bounds |sum x (vx vy vz - Qx Qy Qz)| at every corner.
// Single-brick leaves whose corners change sign are never bounded: their entry is not written.
// The x of the levels are rows of x27, which siblings and cousins share in L2; the copy of them per
// root that the evaluation read before (1,728 bytes, 3.6 GB written and read at 4 M points, maxDepth
// 11) was half of this kernel (11.3 -> 6.1 ms without it); the nine coefficients a lane needs of a level
// read as scalars and not picked from vectors in the inner loop take it to 2.1 ms.
constexpr int XL_WARPS = 4;
__global__ void __launch_bounds__(32 * XL_WARPS) k_brick_xl(VArgs v, int nroots, const int* __restrict__ has_tri,
                                                             const int* __restrict__ up, float* __restrict__ anc) {
    // one warp per root: it stages the levels' x, fits the ancestor functions of all levels (lanes
    // over level and axis), then forms the polynomial
    __shared__ float4 sx[XL_WARPS][BR_LEVELS * 7];
    __shared__ float4 sfit[XL_WARPS][BR_LEVELS * 9];   // [level][axis][t]
    __shared__ float sm_[XL_WARPS][BR_LEVELS * 9];     // their bern_m
    const NodeArrays& nd = v.e.nd;
    const int D = v.e.D;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const i64 warp = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
    const int i = min(lane / 9, 2), j = (lane / 3) % 3, lz = lane % 3;
    for (i64 ri = warp; ri < nroots; ri += nwarps) {
        const VRoot R = v.roots[ri];
        const int r = R.depth, S = 1 << (D - r);
        if (S <= BR && has_tri[R.node]) continue;
        __syncwarp();   // the previous root's readers are done
        for (int t = lane; t < 7 * (r + 1); t += 32)
            sx[w][t] = reinterpret_cast<const float4*>(v.e.x27 + (i64)up[ri * BR_LEVELS + t / 7] * X27_STRIDE)[t % 7];
        int Lc[3];
        key_coords(nd.key[R.node], r, D, Lc);
        for (int f = lane; f < 9 * (r + 1); f += 32) {
            const int l = f / 9, ax = (f % 9) / 3, t = f % 3, g0 = Lc[ax] * S, c = Lc[ax] >> (r - l);
            const float* tab = reinterpret_cast<const float*>(v.e.lb + lattice_offset(D, l) +
                                                              (i64)c * ((1 << (D - l)) + 1) + (g0 - (c << (D - l)))) + t;
            const float4 b = bern_fit([&](int k) { return tab[4 * k]; }, S);
            sfit[w][f] = b;
            sm_[w][f] = bern_m(b);
        }
        __syncwarp();
        float c = 0.f, s3 = 0.f, fit = 0.f;
        int cnt = 0;
        if (lane < 27) {
            // the lane's coefficient of each function is one scalar: nine loads a level
            const float* F = reinterpret_cast<const float*>(sfit[w]);
            const float* Mf = sm_[w];
            for (int l = 0; l <= r; ++l, F += 36, Mf += 9) {
                float xs[28];
#pragma unroll
                for (int q = 0; q < 7; ++q) {
                    const float4 f = sx[w][7 * l + q];
                    xs[4 * q] = f.x; xs[4 * q + 1] = f.y; xs[4 * q + 2] = f.z; xs[4 * q + 3] = f.w;
                }
                float bx[3], by[3], bz[3];
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    bx[t] = F[4 * t + i];
                    by[t] = F[4 * (3 + t) + j];
                    bz[t] = F[4 * (6 + t) + lz];
                }
                float acc = 0.f;
#pragma unroll
                for (int jx = 0; jx < 3; ++jx) {
                    float ys = 0.f;
#pragma unroll
                    for (int jy = 0; jy < 3; ++jy) {
                        float zs = 0.f;
#pragma unroll
                        for (int jz = 0; jz < 3; ++jz) zs = fmaf(xs[9 * jx + 3 * jy + jz], bz[jz], zs);
                        ys = fmaf(by[jy], zs, ys);
                    }
                    acc = fmaf(bx[jx], ys, acc);
                }
                c += acc;
                const float ax = fabsf(reinterpret_cast<const float*>(sx[w] + 7 * l)[lane]);   // the neighbour at offset (i, j, lz)
                if (ax != 0.f) {
                    const float Mx = Mf[i], My = Mf[3 + j], Mz = Mf[6 + lz];
                    const float dx = F[4 * i + 3], dy = F[4 * (3 + j) + 3], dz = F[4 * (6 + lz) + 3];
                    s3 += ax * Mx * My * Mz;
                    fit += ax * (dx * My * Mz + Mx * dy * Mz + Mx * My * dz);
                    ++cnt;
                }
            }
        }
        for (int o = 16; o; o >>= 1) {
            s3 += __shfl_xor_sync(0xffffffffu, s3, o);
            fit += __shfl_xor_sync(0xffffffffu, fit, o);
            cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        }
        anc[ri * ANC_STRIDE + lane] =
            lane < 27 ? c : (lane == 27 ? s3 : (lane == 28 ? (float)cnt : (lane == 29 ? fit : 0.f)));
    }
}

// Owner of corner qc of leaf R: the cell with the least key among the 8 around the corner that belong to
// the leaf or to another root of its batch (member[j]: batch_member's answer for the neighbour at offset
// j, 13 = the leaf itself).  The keys are the OR of one spread coordinate per axis, two of each.
__device__ __forceinline__ int corner_owner_cell(int D, int r, const int Lc[3], const int qc[3], const int* member,
                                                 int oc[3]) {
    const int sh = D - r, lim = 1 << D;
    u64 key[3][2];
    int off[3][2];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int c = qc[ax] - e;
            key[ax][e] = morton_spread3((uint32_t)max(c, 0)) << (2 - ax);
            off[ax][e] = (c < 0 || c >= lim) ? -1 : (c >> sh) - Lc[ax] + 1;   // 0..2, or outside the cube
        }
    u64 best = ~0ull;
    int own = -1, eb = 0;
#pragma unroll
    for (int eo = 0; eo < 8; ++eo) {
        const int ex = eo & 1, ey = (eo >> 1) & 1, ez = eo >> 2;
        if ((off[0][ex] | off[1][ey] | off[2][ez]) < 0) continue;
        const int m = member[9 * off[0][ex] + 3 * off[1][ey] + off[2][ez]];
        const u64 kk = key[0][ex] | key[1][ey] | key[2][ez];
        if (m >= 0 && kk < best) { best = kk; own = m; eb = eo; }
    }
    if (own >= 0) {
        oc[0] = qc[0] - (eb & 1);
        oc[1] = qc[1] - ((eb >> 1) & 1);
        oc[2] = qc[2] - (eb >> 2);
    }
    return own;
}

// Shell terms of a bound at virtual depth d: the window cells outside the leaf that hold a
// real node, each term x * X * Y * Z over the row tables' ranges RW.
//  * Nodes: a cell's node is found by descending from the leaf's neighbour at depth r, through
//    two levels of "anchors" the warp finds first: the cells of depth d - 4 covering the window
//    (at most 2 per axis, one lane each; when d - r > 4) and of depth d - 2 (at most 4 per axis,
//    two per lane, each descending 2 levels from its depth d - 4 anchor; when d - r > 2).  A
//    cell then descends 2 levels from its anchor; cells under an absent anchor are skipped,
//    and a window without any anchor is skipped whole.  The path through the anchors is the
//    same path, so the node is the same.
//  * The lanes run over the cells of all boxes in turn (a lane's next cell continues into the
//    next box), so boxes smaller than a warp leave fewer lanes idle.
//  * rw[ax]: the depth's RW ranges of the window cells along each axis.
//  * An RW range always contains 0 (lo <= 0 <= hi), and float rounding is monotone, so
//    [a, b] x [lo, hi] = [min(b lo, a hi), max(a lo, b hi)]: exactly the min and max of the four
//    rounded products, in 4 multiplies and 2 min/max instead of 4 and 6.
// The window's extent is at most 12 < 16 cells per axis: at most 2 anchors of depth d - 4 and
// 4 of depth d - 2 per axis.
constexpr int SHELL_ANCHORS = 8 + 64;   // ints of shared memory per warp
__device__ __forceinline__ void shell_terms(const VArgs& v, int L, int r, const int Lc[3], int d, int D,
                                            const int wlo[3], const int ext[3], const float2* const rw[3],
                                            int lane, int* __restrict__ anchor, float& lo, float& hi, float& amax,
                                            int& cnt) {
    const float* __restrict__ xv = v.e.x;
    const NodeArrays& nd = v.e.nd;
    const bool anch = d - r > 2;
    int blo[3] = {0, 0, 0};
    if (anch) {
        int* a4 = anchor;        // depth d - 4
        int* a2 = anchor + 8;    // depth d - 2, 4 x 4 x 4
        // only anchors that cover window cells are looked up: those lie in the leaf's
        // neighbours (the window reaches at most 2 cells beyond the leaf)
        int alo[3], ahi[3], bhi[3];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            alo[ax] = wlo[ax] >> 4;   // floor, also below 0
            blo[ax] = wlo[ax] >> 2;
            ahi[ax] = (wlo[ax] + ext[ax] - 1) >> 4;
            bhi[ax] = (wlo[ax] + ext[ax] - 1) >> 2;
        }
        __syncwarp();                 // the previous depth's readers are done
        if (d - r > 4) {
            int an = -1;
            if (lane < 8) {
                const int A[3] = {alo[0] + ((lane >> 2) & 1), alo[1] + ((lane >> 1) & 1), alo[2] + (lane & 1)};
                if (A[0] <= ahi[0] && A[1] <= ahi[1] && A[2] <= ahi[2]) an = (int)shell_node(v, L, r, Lc, d - 4, A);
            }
            if (__ballot_sync(0xffffffffu, an >= 0) == 0) return;   // no real node near this window
            if (lane < 8) a4[lane] = an;
            __syncwarp();
        }
        int any = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int q = lane + 32 * h;
            const int B[3] = {blo[0] + (q >> 4), blo[1] + ((q >> 2) & 3), blo[2] + (q & 3)};
            int bn = -1;
            if (B[0] > bhi[0] || B[1] > bhi[1] || B[2] > bhi[2]) {
                // covers no window cell
            } else if (d - r > 4) {
                const int an = a4[(((B[0] >> 2) - alo[0]) << 2) | (((B[1] >> 2) - alo[1]) << 1) | ((B[2] >> 2) - alo[2])];
                bn = an < 0 ? -1 : (int)descend(nd, an, d - 4, d - 2, B);
            } else {
                bn = (int)shell_node(v, L, r, Lc, d - 2, B);
            }
            a2[q] = bn;
            any |= bn >= 0;
        }
        if (__ballot_sync(0xffffffffu, any) == 0) return;
        __syncwarp();
    }
    const int span = 1 << (d - r);
    const int llo[3] = {Lc[0] * span, Lc[1] * span, Lc[2] * span};
    Box3 bxs[6];
    const int nbx = outside_boxes(wlo, ext, llo, span, bxs);
    const int* a2 = anchor + 8;
    int g = lane, first = 0;
    for (int q = 0; q < nbx; ++q) {
        const Box3 bx = bxs[q];
        const int n12 = bx.n[1] * bx.n[2], ncell = bx.n[0] * n12;
        const float inv12 = 1.0f / (float)n12, inv2 = 1.0f / (float)bx.n[2];
        for (; g < first + ncell; g += 32) {
            const int t = g - first;
            const int i0 = small_div(t, inv12), rem = t - i0 * n12, i1 = small_div(rem, inv2),
                      i2 = rem - i1 * bx.n[2];
            const int N[3] = {bx.lo[0] + i0, bx.lo[1] + i1, bx.lo[2] + i2};
            i64 node;
            if (anch) {
                const int bn = a2[(((N[0] >> 2) - blo[0]) << 4) | (((N[1] >> 2) - blo[1]) << 2) | ((N[2] >> 2) - blo[2])];
                if (bn < 0) continue;
                node = descend(nd, bn, d - 2, d, N);
            } else {
                node = shell_node(v, L, r, Lc, d, N);
            }
            if (node < 0) continue;
            const float x = xv[node];
            const float2 X = rw[0][N[0] - wlo[0]], Y = rw[1][N[1] - wlo[1]], Z = rw[2][N[2] - wlo[2]];
            const float p0 = x * X.x, p1 = x * X.y;
            float a = fminf(p0, p1), b = fmaxf(p0, p1);
            const float a1 = fminf(b * Y.x, a * Y.y), b1 = fmaxf(a * Y.x, b * Y.y);
            a = fminf(b1 * Z.x, a1 * Z.y);
            b = fmaxf(a1 * Z.x, b1 * Z.y);
            lo += a;
            hi += b;
            amax += fmaxf(fabsf(a), fabsf(b));
            ++cnt;
        }
        first += ncell;
    }
}

// Per node of the depths [D - BELOW, D): the least and the largest x, with 0, among its descendants k = 1..
// BELOW depths down (below[BELOW * node + k - 1]; one launch per depth, finest first).  A node whose
// descendants hold a value that is not finite gets an infinite range, which proves nothing.
__global__ void k_x_below(NodeArrays nd, const float* __restrict__ x, i64 lo, i64 hi, i64 node0, int kmax,
                          float2* __restrict__ below) {
    for (i64 i = lo + (i64)blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += (i64)gridDim.x * blockDim.x) {
        const int c0 = nd.child0[i];
        float2* out = below + BELOW * (i - node0);
        float2 r = make_float2(0.f, 0.f);
        if (c0 != -1)
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float v = x[c0 + c];
                if (!(fabsf(v) < INFINITY)) r = make_float2(-INFINITY, INFINITY);
                r = make_float2(fminf(r.x, v), fmaxf(r.y, v));
            }
        out[0] = r;
        for (int k = 1; k < kmax; ++k) {
            r = make_float2(0.f, 0.f);
            if (c0 != -1)
                for (int c = 0; c < 8; ++c) {
                    const float2 q = below[BELOW * (c0 + c - node0) + k - 1];
                    r = make_float2(fminf(r.x, q.x), fmaxf(r.y, q.y));
                }
            out[k] = r;
        }
    }
}

// Per depth, over all lattice points of all cells: the largest sum of the magnitudes of the three basis
// values a walk multiplies with along an axis, and the largest sum of their negative parts (float noise of
// the tabulated values; the B-spline itself is not negative), rounded up.  One block per depth.
__global__ void k_basis_sums(const float4* __restrict__ lb, int D, float2* __restrict__ out) {
    __shared__ float s_r[256], s_n[256];
    const int d = blockIdx.x;
    float r = 0.f, n = 0.f;
    for (i64 e = lattice_offset(D, d) + threadIdx.x; e < lattice_offset(D, d + 1); e += blockDim.x) {
        const float4 f = lb[e];
        r = fmaxf(r, fabsf(f.x) + fabsf(f.y) + fabsf(f.z));
        n = fmaxf(n, fmaxf(-f.x, 0.f) + fmaxf(-f.y, 0.f) + fmaxf(-f.z, 0.f));
    }
    s_r[threadIdx.x] = r;
    s_n[threadIdx.x] = n;
    __syncthreads();
    for (int o = 128; o; o >>= 1) {
        if ((int)threadIdx.x < o) {
            s_r[threadIdx.x] = fmaxf(s_r[threadIdx.x], s_r[threadIdx.x + o]);
            s_n[threadIdx.x] = fmaxf(s_n[threadIdx.x], s_n[threadIdx.x + o]);
        }
        __syncthreads();
    }
    const float up = 1.0f + 9.5367431640625e-07f;
    if (threadIdx.x == 0) out[d] = make_float2(s_r[0] * up, s_n[0] * up);
}

// sign of a bound lo = min C + flo, hi = max C + fhi against iso: C the Bernstein coefficients over
// the brick of its coarse polynomial P (the leaf's ancestors and the shell terms of knot spacing
// >= E; P lies within their range over the brick's box), [flo, fhi] the interval sum of the finer
// shell terms.  The margin is (2 cnt + 2 BR_WEXT + 8) u A over A = 1.01 (amax + s3) (the evaluation's
// FMA chain over all the terms, and the interval part's own arithmetic), plus fit (the fits'
// residuals: the corner values' coarse terms lie within fit of P), plus (cnt + 96) u s3 for P's
// coefficients, s3 = sum |x| Mx My Mz over its terms: (cnt + 56)u for forming them (at most 9 roundings
// per level and 16 levels for the ancestors, 12 per shell depth and one per further depth), 40u for the
// restriction to the brick (three axes of 3 rounded factors and FMAs; the blossom rows are
// non-negative and sum to 1) and adding the two parts.  Every operation of the margin rounds by at
// most u relative and every term is non-negative, so scaling by 1 + 2^-16 bounds the exact value from
// above; the tests are made as lo - iso > m and iso - hi > m, whose float differences are within u of
// exact, which the last term's extra 2u covers.  (A non-finite bound compares false: not proven.)
__device__ __forceinline__ signed char bound_sign_poly(float lo, float hi, float amax, float s3, float fit, int cnt,
                                                       float iso) {
    const float u = 5.9604644775390625e-08f;   // 2^-24
    const float A = (amax + s3) * 1.01f;
    const float m = ((2.0f * (float)cnt + (2.0f * BR_WEXT + 8.0f)) * u * A + ((float)cnt + 96.0f) * u * s3 * 1.01f +
                     fit * 1.01f + 6.0f * u * (fabsf(lo) + fabsf(hi) + 2.0f * fabsf(iso)) + 1e-30f) *
                    (1.0f + 1.52587890625e-05f);
    if (lo - iso > m) return 1;
    if (iso - hi > m) return -1;
    return 0;
}

// row q of the blossom matrix that takes quadratic Bernstein coefficients over [0, S] to those over
// [A, B] (0 <= A < B <= S, S a power of two <= 2^15): the blossom of the basis at (A, A), (A, B),
// (B, B), divided by S^2 (exact in float for S <= 2^11, else rounded once); non-negative, sums to 1
__device__ __forceinline__ void blossom_row(unsigned a, unsigned b, unsigned s, int q, float out[3]) {
    unsigned n0, n1, n2;   // below 2^31
    if (q == 0) { n0 = (s - a) * (s - a); n1 = 2 * a * (s - a); n2 = a * a; }
    else if (q == 1) { n0 = (s - a) * (s - b); n1 = a * (s - b) + b * (s - a); n2 = a * b; }
    else { n0 = (s - b) * (s - b); n1 = 2 * b * (s - b); n2 = b * b; }
    const float inv = 1.0f / ((float)s * (float)s);
    out[0] = (float)n0 * inv;
    out[1] = (float)n1 * inv;
    out[2] = (float)n2 * inv;
}

// shared memory of a warp that bounds bricks
struct BoundShared {
    float X[64], T1[48], T2[36];
    int id[2][64];                 // nodes of the window cells at a depth, 4 x 4 x 4 (-1: none)
    int anchor[SHELL_ANCHORS];
};

// The bound over the corners the leaf owns of the box of edge E at g0 (a brick or super-brick, one warp):
// 1 (all above iso), -1 (all below) or 0 (not proven).
//  * The coarse part, exact up to rounding and the tabulated values' noise: the leaf's ancestor
//    polynomial (per root, k_brick_xl), restricted to the box, and the shell terms of the depths of knot
//    spacing >= E.  Each window cell outside the leaf with a real node contributes x Qx Qy Qz, Q the
//    cell's PW entries (Bernstein form over the box).  The window spans at most PW = 4 cells per axis
//    there (the box lies in one cell of depth d, and its first corner's owner may lie in the cell below),
//    so the terms form a 4^3 grid X of x (0: no node, or inside the leaf; two cells per lane), contracted
//    one axis at a time through shared memory:
//      T1[n0 n1 l] = sum_n2 X Qz_l(n2),  T2[n0 j l] = sum_n1 T1 Qy_j(n1),  C_ijl += sum_n0 T2 Qx_i(n0)
//    (lane k < 27 holds coefficient k = 9i + 3j + l).  s3 gains |x| Mx My Mz, fit
//    |x| (dx My Mz + Mx dy Mz + Mx My dz) (as k_brick_xl's), cnt the number of terms.  The windows are
//    nested, so a cell's node is the child of a cell of the window above, from the leaf's 27 neighbours.
//    Bounded by the range of the Bernstein coefficients.
//  * The finer shell terms only widen the bound (a term that some corners lack ranges over 0), so a box
//    whose coarse part already straddles iso is left unproven without them.
//  * First the finer terms together: at a corner the 27 terms of depth d are at most the largest |x| near
//    the box times the product of the axes' sums of basis magnitudes (k_basis_sums), on the side of x's
//    sign but for the basis values' negative noise.  The largest and least x come from the range of x
//    below the nodes of the last coarse window (k_x_below) that the fine window touches: one load per
//    depth and cell, where the terms themselves take a descent each.  In a dense shell this is also the
//    tighter bound: a sum of intervals counts every cell of the window at its best corner.
//  * Then, for a brick, the terms one by one (shell_terms).
// Measured, bricks of leaves of edge >= 16 with their super-bricks: 4 M points, maxDepth 11, 8.3 M bricks
// 15.9 -> 3.8 ms (92 % of the super-bricks decided, 36 % when they were bounded by interval products and
// those at a leaf's face given up); 30 M points, maxDepth 12, 67 M bricks 147 -> 17; 1M torus 1.95 -> 0.42.
__device__ __forceinline__ signed char bound_box(const VArgs& v, const BrickIndex& bix, int root, const VRoot& R,
                                                 const int b[3], int E, const float* const row[3], int lane,
                                                 BoundShared& sm) {
    const EvalArgs& a = v.e;
    const NodeArrays& nd = a.nd;
    const int D = a.D, r = R.depth, S = 1 << (D - r), L = R.node;
    const int dpoly = D - (31 - __clz(E));   // depths of knot spacing >= E
    int Lc[3];
    key_coords(nd.key[L], r, D, Lc);
    const int g0[3] = {Lc[0] * S + b[0] * E, Lc[1] * S + b[1] * E, Lc[2] * S + b[2] * E};
    float s3 = 0.f, fit = 0.f, coef = 0.f;
    int cnt = 0;
    int plo[3] = {Lc[0] - 1, Lc[1] - 1, Lc[2] - 1}, cur = 0;
    __syncwarp();   // the previous box's readers are done
    {
        const int n = lane < 27 ? nd.neigh[(i64)lane * nd.M + L] : -1;
        sm.id[0][lane] = sm.id[0][lane + 32] = -1;
        __syncwarp();
        if (lane < 27) sm.id[0][(lane / 9) * 16 + ((lane / 3) % 3) * 4 + lane % 3] = n;
        __syncwarp();   // (a single-brick leaf has no coarse depth: the finer terms below are the next to read)
    }
    bool inside = false;
    for (int d = r + 1; d <= dpoly; ++d) {
        int wlo[3], ext[3];
        bool cross = false;
        for (int ax = 0; ax < 3; ++ax) {
            bool c;
            window_axis(g0[ax], E, Lc[ax], r, d, D, wlo[ax], ext[ax], c);
            cross |= c;
        }
        if (!cross) { inside = true; break; }   // nested windows: the finer ones lie inside the leaf too
        if (ext[0] > PW || ext[1] > PW || ext[2] > PW) return 0;   // (cannot happen)
        const float4* pw[3];
        for (int ax = 0; ax < 3; ++ax) pw[ax] = reinterpret_cast<const float4*>(row[ax] + d * PROW);
        __syncwarp();
        bool any = false;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int g = lane + 32 * h, n0 = g >> 4, n1 = (g >> 2) & 3, n2 = g & 3;
            float x = 0.f;
            int node = -1;
            if (n0 < ext[0] && n1 < ext[1] && n2 < ext[2]) {
                const int N[3] = {wlo[0] + n0, wlo[1] + n1, wlo[2] + n2};
                const int p = sm.id[cur][((N[0] >> 1) - plo[0]) * 16 + ((N[1] >> 1) - plo[1]) * 4 + ((N[2] >> 1) - plo[2])];
                const int c0 = p < 0 ? -1 : nd.child0[p];   // (the leaf itself has none: cells inside it come out absent)
                if (c0 != -1) {
                    node = c0 + (((N[0] & 1) << 2) | ((N[1] & 1) << 1) | (N[2] & 1));
                    x = a.x[node];
                }
            }
            sm.X[g] = x;
            sm.id[cur ^ 1][g] = node;
            if (x != 0.f) {
                const float4 QX = pw[0][n0], QY = pw[1][n1], QZ = pw[2][n2];
                const float Mx = bern_m(QX), My = bern_m(QY), Mz = bern_m(QZ), ax = fabsf(x);
                s3 += ax * Mx * My * Mz;
                fit += ax * (QX.w * My * Mz + Mx * QY.w * Mz + Mx * My * QZ.w);
                ++cnt;
                any = true;
            }
        }
        cur ^= 1;
        plo[0] = wlo[0]; plo[1] = wlo[1]; plo[2] = wlo[2];
        if (!__any_sync(0xffffffffu, any)) continue;   // no real node near the box at this depth
        __syncwarp();
        for (int e = lane; e < 48; e += 32) {
            const int nn = e / 3, l = e - 3 * nn;   // nn = 4 n0 + n1
            float t = 0.f;
#pragma unroll
            for (int n2 = 0; n2 < 4; ++n2) t = fmaf(sm.X[4 * nn + n2], f4_at(pw[2][n2], l), t);
            sm.T1[e] = t;
        }
        __syncwarp();
        for (int e = lane; e < 36; e += 32) {
            const int n0 = e / 9, j = (e / 3) % 3, l = e % 3;
            float t = 0.f;
#pragma unroll
            for (int n1 = 0; n1 < 4; ++n1) t = fmaf(sm.T1[(4 * n0 + n1) * 3 + l], f4_at(pw[1][n1], j), t);
            sm.T2[e] = t;
        }
        __syncwarp();
        if (lane < 27) {
            const int i = lane / 9, jl = lane % 9;
            float t = 0.f;
#pragma unroll
            for (int n0 = 0; n0 < 4; ++n0) t = fmaf(sm.T2[9 * n0 + jl], f4_at(pw[0][n0], i), t);
            coef += t;
        }
    }
    // the ancestor polynomial's coefficients over the box (lane k < 27: coefficient k = 9i + 3j + l), one
    // axis at a time through the blossom rows (the identity for a single-brick leaf), plus the shell part
    const float* an = bix.anc + (i64)root * ANC_STRIDE;
    float c = lane < 27 ? an[lane] : 0.f;
    if (S > E) {
        const int i = lane / 9, j = (lane / 3) % 3, l = lane % 3;
        float t[3];
        blossom_row(b[2] * E, (b[2] + 1) * E, S, l, t);
        {
            const int q = lane - l;
            const float c0 = __shfl_sync(0xffffffffu, c, q), c1 = __shfl_sync(0xffffffffu, c, (q + 1) & 31),
                        c2 = __shfl_sync(0xffffffffu, c, (q + 2) & 31);
            c = fmaf(c2, t[2], fmaf(c1, t[1], c0 * t[0]));
        }
        blossom_row(b[1] * E, (b[1] + 1) * E, S, j, t);
        {
            const int q = lane - 3 * j;
            const float c0 = __shfl_sync(0xffffffffu, c, q), c1 = __shfl_sync(0xffffffffu, c, (q + 3) & 31),
                        c2 = __shfl_sync(0xffffffffu, c, (q + 6) & 31);
            c = fmaf(c2, t[2], fmaf(c1, t[1], c0 * t[0]));
        }
        blossom_row(b[0] * E, (b[0] + 1) * E, S, i, t);
        {
            const int q = lane - 9 * i;
            const float c0 = __shfl_sync(0xffffffffu, c, q), c1 = __shfl_sync(0xffffffffu, c, (q + 9) & 31),
                        c2 = __shfl_sync(0xffffffffu, c, (q + 18) & 31);
            c = fmaf(c2, t[2], fmaf(c1, t[1], c0 * t[0]));
        }
    }
    c += coef;
    float cmin = lane < 27 ? c : INFINITY, cmax = lane < 27 ? c : -INFINITY;
    for (int o = 16; o; o >>= 1) {
        s3 += __shfl_xor_sync(0xffffffffu, s3, o);
        fit += __shfl_xor_sync(0xffffffffu, fit, o);
        // (a value that is not a number must not drop out of the range)
        const float p = __shfl_xor_sync(0xffffffffu, cmin, o), q = __shfl_xor_sync(0xffffffffu, cmax, o);
        cmin = (p < cmin || p != p) ? p : cmin;
        cmax = (q > cmax || q != q) ? q : cmax;
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt) + (int)an[28];
    s3 += an[27];
    fit += an[29];
    const signed char coarse = bound_sign_poly(cmin, cmax, 0.f, s3, fit, cnt, v.iso);
    if (coarse == 0 || inside) return coarse;
    // the finer terms together
    {
        float flo = 0.f, fhi = 0.f, famax = 0.f;
        int fcnt = 0;
        for (int d = dpoly + 1; d <= D; ++d) {
            const int k = d - dpoly;
            int wlo[3], ext[3];
            bool cross = false;
            for (int ax = 0; ax < 3; ++ax) {
                bool cr;
                window_axis(g0[ax], E, Lc[ax], r, d, D, wlo[ax], ext[ax], cr);
                cross |= cr;
            }
            if (!cross) break;
            unsigned neg = 0, pos = 0;   // bits of the largest magnitudes on either side
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int g = lane + 32 * h;
                const int N[3] = {plo[0] + (g >> 4), plo[1] + ((g >> 2) & 3), plo[2] + (g & 3)};
                const int node = sm.id[cur][g];
                bool touch = node >= 0;
#pragma unroll
                for (int ax = 0; ax < 3; ++ax) touch &= N[ax] >= (wlo[ax] >> k) && N[ax] <= ((wlo[ax] + ext[ax] - 1) >> k);
                if (touch) {
                    const float2 q = bix.below[BELOW * (node - bix.below0) + k - 1];
                    neg = max(neg, __float_as_uint(-q.x) & 0x7fffffffu);
                    pos = max(pos, __float_as_uint(q.y) & 0x7fffffffu);
                }
            }
            const float xn = __uint_as_float(__reduce_max_sync(0xffffffffu, neg)),
                        xp = __uint_as_float(__reduce_max_sync(0xffffffffu, pos)), xm = fmaxf(xn, xp);
            if (xm == 0.f) continue;
            const float2 bs = bix.bsum[d];
            const float up = 1.0f + 9.5367431640625e-07f;
            const float r3 = bs.x * bs.x * bs.x * up, n3 = 3.f * bs.y * bs.x * bs.x * up;
            flo -= (xn * r3 + xm * n3) * up;
            fhi += (xp * r3 + xm * n3) * up;
            famax += xm * r3 * up;
            fcnt += 27;
        }
        const signed char sg = bound_sign_poly(cmin + flo, cmax + fhi, famax, s3, fit, cnt + fcnt, v.iso);
        if (sg != 0 || E > BR) return sg;
    }
    // the finer terms one by one; only window cells outside the leaf can hold a real node
    float lo = 0.f, hi = 0.f, amax = 0.f;
    int fcnt = 0;
    for (int d = max(dpoly, r) + 1; d <= D; ++d) {
        int wlo[3], ext[3];
        bool cross = false;
        for (int ax = 0; ax < 3; ++ax) {
            bool cr;
            window_axis(g0[ax], E, Lc[ax], r, d, D, wlo[ax], ext[ax], cr);
            cross |= cr;
        }
        if (!cross) break;
        const float2* rw[3];
        for (int ax = 0; ax < 3; ++ax) rw[ax] = reinterpret_cast<const float2*>(row[ax] + d * PROW);
        shell_terms(v, L, r, Lc, d, D, wlo, ext, rw, lane, sm.anchor, lo, hi, amax, fcnt);
    }
    for (int o = 16; o; o >>= 1) {
        lo += __shfl_xor_sync(0xffffffffu, lo, o);
        hi += __shfl_xor_sync(0xffffffffu, hi, o);
        amax += __shfl_xor_sync(0xffffffffu, amax, o);
    }
    fcnt = __reduce_add_sync(0xffffffffu, fcnt);
    return bound_sign_poly(cmin + lo, cmax + hi, amax, s3, fit, cnt + fcnt, v.iso);
}

// One warp per super-brick (4^3 bricks of leaves with lattice edge >= 64): decided, its bricks get its sign;
// undecided, it joins the list whose bricks k_brick_bound takes.
constexpr int BB_BLOCK = 256;
__global__ void __launch_bounds__(BB_BLOCK, 4) k_super_bound(VArgs v, BrickIndex bix, const i64* __restrict__ srow_prefix,
                                                            const float* __restrict__ srows, i64 nsuper,
                                                            signed char* __restrict__ sign, int* __restrict__ nopen,
                                                            i64* __restrict__ open) {
    __shared__ BoundShared sm[BB_BLOCK / 32];
    const int D = v.e.D;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const DepthLayout& dl = bix.dl;
    const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
    for (i64 si = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; si < nsuper; si += nwarps) {
        int dd = 0;
        while (dd < D - 1 && dl.soff[dd + 1] <= si) ++dd;
        const i64 loc = si - dl.soff[dd];
        const int slg = dl.slg[dd], ns = 1 << slg;
        const int root = dl.first[dd] + (int)(loc >> (3 * slg));
        const VRoot R = v.roots[root];
        const i64 l = loc & ((1ll << (3 * slg)) - 1);
        const int b[3] = {(int)(l >> (2 * slg)), (int)(l >> slg) & (ns - 1), (int)l & (ns - 1)};
        const float* row[3];
        for (int ax = 0; ax < 3; ++ax) row[ax] = brick_row(srows, srow_prefix, D, root, ns, ax, b[ax]);
        const signed char sg = bound_box(v, bix, root, R, b, SUPER, row, lane, sm[w]);
        const int nb = 4 * ns;
        const i64 first = bix.prefix[root] + ((i64)(4 * b[0]) * nb + 4 * b[1]) * nb + 4 * b[2];
        if (sg != 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int g = lane + 32 * h;
                sign[first + ((i64)(g >> 4) * nb + ((g >> 2) & 3)) * nb + (g & 3)] = sg;
            }
        } else if (lane == 0) {
            open[atomicAdd(nopen, 1)] = first;
        }
    }
}

// One warp per brick: sign[bi] = 1 (all above iso), -1 (all below) or 0 (not proven), for the bricks of
// the undecided super-bricks ('open': their first bricks) and those of [first, nbricks).
// A single-brick leaf whose own real corners change sign ('has_tri') is left unproven at once:
// its brick's corners include the leaf's corners, so its bound straddles iso (and a brick left
// unproven is only evaluated exactly, which changes no value).
// The launch has up to 256 blocks per SM: bricks differ in cost, and with 8 blocks per SM striding over
// all of them the last blocks ran alone (22.0 -> 15.9 ms at 4 M points, 2.41 -> 1.90 on the 1M torus).
__global__ void __launch_bounds__(BB_BLOCK, 4) k_brick_bound(VArgs v, BrickIndex bix, const int* __restrict__ nopen,
                                                          const i64* __restrict__ open, i64 first, i64 nbricks,
                                                          const int* __restrict__ has_tri,
                                                          signed char* __restrict__ sign) {
    __shared__ BoundShared sm[BB_BLOCK / 32];
    const int D = v.e.D;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const i64 nsub = nopen ? 64ll * *nopen : 0;
    const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
    for (i64 it = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < nsub + (nbricks - first); it += nwarps) {
        i64 bi = first + it - nsub;
        if (it < nsub) {
            const i64 f = open[it >> 6];
            const VBrick F = brick_of(v, bix, f);
            const i64 nb = 1ll << bix.dl.lg[v.roots[F.root].depth];
            const int g = (int)it & 63;
            bi = f + ((i64)(g >> 4) * nb + ((g >> 2) & 3)) * nb + (g & 3);
        }
        const VBrick B = brick_of(v, bix, bi);
        const VRoot R = v.roots[B.root];
        const int r = R.depth, E = brick_edge(D, r), nb = (1 << (D - r)) / E;
        signed char sg = 0;
        if (!(nb == 1 && has_tri[R.node])) {
            const float* row[3];
            for (int ax = 0; ax < 3; ++ax) row[ax] = brick_row(bix.rows, bix.row_prefix, D, B.root, nb, ax, B.b[ax]);
            sg = bound_box(v, bix, B.root, R, B.b, E, row, lane, sm[w]);
        }
        if (lane == 0) sign[bi] = sg;
    }
}

// culled: the brick's own bound is proven and, where some of its corners may be
// owned by another leaf L' of the batch, every brick of L' that can hold such
// an owner cell is proven with the same sign
__global__ void k_brick_cull(VArgs v, BrickIndex bix, const int* __restrict__ root_of, const signed char* __restrict__ sign,
                             i64 nbricks, unsigned char* __restrict__ culled) {
    const int D = v.e.D;
    const NodeArrays& nd = v.e.nd;
    for (i64 bi = (i64)blockIdx.x * blockDim.x + threadIdx.x; bi < nbricks; bi += (i64)gridDim.x * blockDim.x) {
        const int sg = sign[bi];
        if (sg == 0) { culled[bi] = 0; continue; }
        const VBrick B = brick_of(v, bix, bi);
        const VRoot R = v.roots[B.root];
        const int E = brick_edge(D, R.depth), nb = (1 << (D - R.depth)) / E;
        bool ok = true;
        if (R.depth >= 3 && !(B.b[0] && B.b[1] && B.b[2])) {
            for (int j = 0; j < 27 && ok; ++j) {
                const int off[3] = {j / 9 - 1, (j / 3) % 3 - 1, j % 3 - 1};
                bool lower = false, allowed = true;
                for (int ax = 0; ax < 3; ++ax) {
                    if (off[ax] == -1) { lower = true; if (B.b[ax] != 0) allowed = false; }
                    if (off[ax] == 1 && B.b[ax] != nb - 1) allowed = false;
                }
                if (!lower || !allowed) continue;
                const int n = nd.neigh[(i64)j * nd.M + R.node];
                if (n == -1 || v.batch_root_flag[n] != R.batch) continue;
                const int k2 = root_of[n];
                // bricks of the neighbour holding owner cells within one cell of this brick
                int lo3[3], hi3[3];
                for (int ax = 0; ax < 3; ++ax) {
                    if (off[ax] == -1) { lo3[ax] = hi3[ax] = nb - 1; }
                    else if (off[ax] == 1) { lo3[ax] = hi3[ax] = 0; }
                    else { lo3[ax] = max(B.b[ax] - 1, 0); hi3[ax] = min(B.b[ax] + 1, nb - 1); }
                }
                for (int x = lo3[0]; x <= hi3[0] && ok; ++x)
                    for (int y = lo3[1]; y <= hi3[1] && ok; ++y)
                        for (int z = lo3[2]; z <= hi3[2] && ok; ++z)
                            if (sign[bix.prefix[k2] + ((i64)x * nb + y) * nb + z] != sg) ok = false;
            }
        }
        culled[bi] = ok ? 1 : 0;
    }
}

// root index of each subdivided leaf's node (-1 elsewhere)
__global__ void k_root_of(const VRoot* __restrict__ roots, int nroots, int* __restrict__ root_of) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nroots; k += gridDim.x * blockDim.x)
        root_of[roots[k].node] = k;
}

// live brick: root and brick coordinates
struct LiveBrick {
    int root;
    int b[3];
};
// The live bricks in brick order.  Roots come in depth order, so the bricks of edge 8 come first, then those
// of edge 4 and of edge 2: a brick's corner values and cells are numbered in closed form.
struct LiveIndex {
    const LiveBrick* live;
    i64 n8, n4, n2;
    __host__ __device__ i64 lattices() const { return 729 * n8 + 125 * n4 + 27 * n2; }
    __host__ __device__ i64 cells() const { return 512 * n8 + 64 * n4 + 8 * n2; }
    __device__ __forceinline__ i64 lat(i64 li) const {   // first corner value
        if (li < n8) return 729 * li;
        li -= n8;
        return 729 * n8 + (li < n4 ? 125 * li : 125 * n4 + 27 * (li - n4));
    }
    // brick of cell e; its edge's logarithm and the cell in it
    __device__ __forceinline__ i64 brick(i64 e, int& lg, int& loc) const {
        if (e < 512 * n8) { lg = 3; loc = (int)(e & 511); return e >> 9; }
        e -= 512 * n8;
        if (e < 64 * n4) { lg = 2; loc = (int)(e & 63); return n8 + (e >> 6); }
        e -= 64 * n4;
        lg = 1;
        loc = (int)(e & 7);
        return n8 + n4 + (e >> 3);
    }
};
// a corner of live brick li owned by another leaf of the batch, and the corner of that leaf's brick which
// is the same point: brick << 10 | corner
struct ForeignCorner {
    int li;
    int e;
    u64 src;
};
__device__ __forceinline__ u64 foreign_src(int D, int r, int E, const DepthLayout& dl, int owner_root, const int oc[3],
                                           const int qc[3]) {
    const int sh = D - r, lg = dl.lg[r], E1 = E + 1;
    int b[3], k[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const int l0 = (oc[ax] >> sh) << sh;         // the owner leaf's first cell
        b[ax] = (oc[ax] - l0) / E;
        k[ax] = qc[ax] - (l0 + b[ax] * E);
    }
    const i64 brick = dl.boff[r] + ((i64)(owner_root - dl.first[r]) << (3 * lg)) +
                      (((((i64)b[0]) << lg) + b[1]) << lg) + b[2];
    return ((u64)brick << 10) | (u64)((k[0] * E1 + k[1]) * E1 + k[2]);
}
// append the lanes' foreign corners (a whole warp calls): one atomic per warp
__device__ __forceinline__ void push_foreign(bool isf, int li, int e, u64 src, unsigned long long* nforeign,
                                             ForeignCorner* foreign, i64 cap) {
    const unsigned fm = __ballot_sync(0xffffffffu, isf);
    if (!fm) return;
    const int lane = threadIdx.x & 31, leader = __ffs(fm) - 1;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(nforeign, (unsigned long long)__popc(fm));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (isf) {
        const unsigned long long f = base + (unsigned long long)__popc(fm & ((1u << lane) - 1u));
        if ((i64)f < cap) foreign[f] = ForeignCorner{li, e, src};
    }
}

// Values of a live brick's corners, the same bit for bit as virtual_corner_value's: for every level, the
// 27 terms in order, each fma((x bx) by, bz, value).
//
// A thread takes a column of corners along z.  A term's (x bx) by is the same for all corners of the
// column that read the same x, so a level costs a column 54 products (the ancestors, whose 27 x are the
// leaf's) or 18 per window cell along z (the virtual depths) and then 27 FMAs per corner, where a thread
// per corner spends 54 products and 27 FMAs on each.  The values of the column are independent chains.
// On the virtual depths the column slides along z: the products of the three z neighbours stay in
// registers and move by one when the owner cell does.  Terms that virtual_corner_value skips (levels
// whose 3x3x3 block lies inside the owner's leaf, cells inside the leaf, absent nodes) read 0 here,
// and adding a zero product leaves the sum unchanged.
template <int E>
struct BrickShared {
    static constexpr int K1 = E + 1;          // corners per axis
    // window cells over the virtual depths and in the largest window above the finest depth; edge 4: the
    // leaf itself, 6^3 + 4^3
    static constexpr int XW = (E == BR) ? BR_XW : 280, PW3 = (E == BR) ? 343 : 64;
    float4 Bt[3 * BR_LEVELS * K1];            // [axis][depth][k], the four t of a corner in one vector
    float4 xL[BR_LEVELS * 7];                 // neighbours of the leaf and its ancestors (0: none), 27 + 1 per level
    float Xw[XW];                             // window coefficients, virtual depths (0: none or inside the leaf)
    int child[2][PW3];                        // first child of the window cells of the depth above (-1: none)
    int wlo[BR_LEVELS][3];                    // window origin (cell coordinates at that depth)
    int wext[BR_LEVELS][3];
    int woff[BR_LEVELS];                      // offset into Xw, -1 when no corner reaches outside the leaf
    int member[27];                           // batch_member of the leaf at each neighbour offset
    int total, fposs;
};

// one level of a column whose corners all read the 27 x in xs: val[kz] += the 27 terms
template <int K1>
__device__ __forceinline__ void column_level(const float xs[28], const float4& bx, const float4& by, const float4* bz,
                                             float val[K1]) {
    const float x3[3] = {bx.x, bx.y, bx.z}, y3[3] = {by.x, by.y, by.z};
    float p[27];
#pragma unroll
    for (int j = 0; j < 27; ++j) p[j] = xs[j] * x3[j / 9] * y3[(j / 3) % 3];
#pragma unroll
    for (int kz = 0; kz < K1; ++kz) {
        const float4 b = bz[kz];
        const float z3[3] = {b.x, b.y, b.z};
        float v = val[kz];
#pragma unroll
        for (int j = 0; j < 27; ++j) v = fmaf(p[j], z3[j % 3], v);
        val[kz] = v;
    }
}

// Bricks of edge 8 (96 threads, 81 columns) and 4 (a warp, 25 columns).  4 M points, maxDepth 11: 109 K
// bricks of edge 8 in 3.5 ms (7.9 with a thread per corner and a descent per window cell; 3.8 with 16 blocks
// per SM striding over the bricks, some of them left with one more at the end), 0.4 M of edge 4 in 3.  At most 85 registers, so that 7 blocks share an SM: with 128 (5 blocks) the edge-8 bricks take
// 8.7 ms, set-up and window loads waiting.
template <int E, int NT>
__global__ void __launch_bounds__(NT, E == BR ? 7 : 24) k_brick_eval(VArgs v, BrickIndex bix, const int* __restrict__ root_of,
                                                   LiveIndex lx, i64 first, i64 nlist, float* __restrict__ blat,
                                                   unsigned long long* __restrict__ nforeign,
                                                   ForeignCorner* __restrict__ foreign, i64 foreign_cap) {
    __shared__ BrickShared<E> sm;
    constexpr int K1 = E + 1;
    static_assert(K1 * K1 <= NT, "a thread per column");
    const EvalArgs& a = v.e;
    const int D = a.D;
    for (i64 it = blockIdx.x; it < nlist; it += gridDim.x) {
        const int li = (int)(first + it);
        const LiveBrick lb = lx.live[li];
        const VRoot R = v.roots[lb.root];
        const int r = R.depth, S = 1 << (D - r), L = R.node, nb = S / E;
        int Lc[3];
        key_coords(a.nd.key[L], r, D, Lc);
        const int g0[3] = {Lc[0] * S + lb.b[0] * E, Lc[1] * S + lb.b[1] * E, Lc[2] * S + lb.b[2] * E};
        __syncthreads();   // the previous brick's readers are done
        if (threadIdx.x < 32) {
            // the leaf's neighbours: first children, batch membership (batch_member's rule)
            const int lane = threadIdx.x;
            bool fp = false;
            if (lane < 27) {
                const int n = a.nd.neigh[(i64)lane * a.nd.M + L];
                int m = lane == 13 ? L : -1;
                if (r >= 3 && n != -1 && lane != 13 && v.batch_root_flag[n] == R.batch) {
                    m = n;
                    fp = foreign_neighbour(lane, lb.b, nb);
                }
                sm.member[lane] = m;
                sm.child[r & 1][lane] = n == -1 ? -1 : a.nd.child0[n];
            }
            fp = __any_sync(0xffffffffu, fp);
            // window layout, a lane per depth
            int wl[3] = {0, 0, 0}, we[3] = {0, 0, 0}, size = 0;
            bool cross = false;
            if (lane > r && lane <= D) {
                for (int ax = 0; ax < 3; ++ax) {
                    bool c;
                    window_axis(g0[ax], E, Lc[ax], r, lane, D, wl[ax], we[ax], c);
                    cross |= c;
                }
                if (cross) size = we[0] * we[1] * we[2];
            }
            int inc = size;
            for (int o = 1; o < 16; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane < BR_LEVELS) {
                for (int ax = 0; ax < 3; ++ax) { sm.wlo[lane][ax] = wl[ax]; sm.wext[lane][ax] = we[ax]; }
                sm.woff[lane] = cross ? inc - size : -1;
            }
            if (lane == BR_LEVELS - 1) sm.total = inc;
            if (lane == 0) sm.fposs = fp;
        }
        for (int e = threadIdx.x; e < 7 * (r + 1); e += NT)
            sm.xL[e] = reinterpret_cast<const float4*>(a.x27 + (i64)bix.up[(i64)lb.root * BR_LEVELS + e / 7] * X27_STRIDE)[e % 7];
        for (int e = threadIdx.x; e < 3 * K1 * (D + 1); e += NT) {
            const int d = e / (3 * K1), ax = (e % (3 * K1)) / K1, k = e % K1;
            sm.Bt[(ax * BR_LEVELS + d) * K1 + k] = brick_bt(a, r, Lc[ax], g0[ax], d, k);
        }
        __syncthreads();
        const bool fposs = sm.fposs;
        if (sm.total > BrickShared<E>::XW) {   // cannot happen for aligned bricks: reported, brick skipped
            if (threadIdx.x == 0) atomicAdd(nforeign + 1, 1ull);
            continue;
        }
        // the windows from the coarsest depth down: a cell's node is the child of its parent, a cell of the
        // window above (the windows are nested; below depth r, the leaf's 27 neighbours), so a depth costs
        // a cell one more load instead of a descent from the leaf's neighbour.  The leaf has no children:
        // cells inside it come out absent.
        {
            int plo[3] = {Lc[0] - 1, Lc[1] - 1, Lc[2] - 1}, p1 = 3, p2 = 3;
            for (int d = r + 1; d <= D; ++d) {
                const int off = sm.woff[d];
                if (off < 0) break;            // and so are the finer ones
                const int wl[3] = {sm.wlo[d][0], sm.wlo[d][1], sm.wlo[d][2]};
                const int e0 = sm.wext[d][0], e1 = sm.wext[d][1], e2 = sm.wext[d][2], n12 = e1 * e2, ncell = e0 * n12;
                const float inv12 = 1.0f / (float)n12, inv2 = 1.0f / (float)e2;
                const int* up = sm.child[(d - 1) & 1];
                int* down = sm.child[d & 1];
                for (int t = threadIdx.x; t < ncell; t += NT) {
                    const int i0 = small_div(t, inv12), rem = t - i0 * n12, i1 = small_div(rem, inv2), i2 = rem - i1 * e2;
                    const int N[3] = {wl[0] + i0, wl[1] + i1, wl[2] + i2};
                    const int c0 = up[(((N[0] >> 1) - plo[0]) * p1 + ((N[1] >> 1) - plo[1])) * p2 + ((N[2] >> 1) - plo[2])];
                    float x = 0.f;
                    int c = -1;
                    if (c0 != -1) {
                        const int node = c0 + (((N[0] & 1) << 2) | ((N[1] & 1) << 1) | (N[2] & 1));
                        x = a.x[node];
                        if (d < D) c = a.nd.child0[node];
                    }
                    sm.Xw[off + t] = x;
                    if (d < D) down[t] = c;
                }
                plo[0] = wl[0]; plo[1] = wl[1]; plo[2] = wl[2];
                p1 = e1;
                p2 = e2;
                __syncthreads();
            }
        }
        // this thread's column (threads beyond the last column repeat it and store nothing)
        const bool col = threadIdx.x < K1 * K1;
        const int ci = col ? threadIdx.x : K1 * K1 - 1, kx = ci / K1, ky = ci % K1;
        const int qx = g0[0] + kx, qy = g0[1] + ky;
        // the leaf's lower faces: there a corner's own cell is the one above it
        const bool lowx = lb.b[0] == 0 && kx == 0, lowy = lb.b[1] == 0 && ky == 0, lowz = lb.b[2] == 0;
        float val[K1];
#pragma unroll
        for (int kz = 0; kz < K1; ++kz) val[kz] = 0.f;
#pragma unroll 1
        for (int d = D; d > r; --d) {
            const int off = sm.woff[d];
            if (off < 0) continue;
            const int sh = D - d;
            const int V0 = (qx - 1 + lowx) >> sh, V1 = (qy - 1 + lowy) >> sh;
            // the row holds the functions around the cell below the corner: one further on the lower face
            const float4 fx = sm.Bt[d * K1 + kx], fy = sm.Bt[(BR_LEVELS + d) * K1 + ky];
            const float x3[3] = {lowx ? fx.y : fx.x, lowx ? fx.z : fx.y, lowx ? fx.w : fx.z};
            const float y3[3] = {lowy ? fy.y : fy.x, lowy ? fy.z : fy.y, lowy ? fy.w : fy.z};
            const int e1 = sm.wext[d][1], e2 = sm.wext[d][2];
            const float* xw = sm.Xw + off + ((V0 - 1 - sm.wlo[d][0]) * e1 + (V1 - 1 - sm.wlo[d][1])) * e2;
            float p[3][9];                  // (x bx) by of the z neighbours below, at and above the owner cell
            auto slice = [&](int z, float q[9]) {
#pragma unroll
                for (int j = 0; j < 9; ++j) q[j] = xw[((j / 3) * e1 + j % 3) * e2 + z] * x3[j / 3] * y3[j % 3];
            };
            int zc = ((g0[2] - 1 + lowz) >> sh) - 1 - sm.wlo[d][2];   // window cell of p[0]
            slice(zc, p[0]);
            slice(zc + 1, p[1]);
            slice(zc + 2, p[2]);
#pragma unroll
            for (int kz = 0; kz < K1; ++kz) {
                const int qz = g0[2] + kz;
                const int zk = ((qz - 1 + (lowz && kz == 0)) >> sh) - 1 - sm.wlo[d][2];
                if (kz > 0 && zk != zc) {   // the owner cell moved up by one
                    zc = zk;
#pragma unroll
                    for (int j = 0; j < 9; ++j) { p[0][j] = p[1][j]; p[1][j] = p[2][j]; }
                    slice(zc + 2, p[2]);
                }
                const float4 fz = sm.Bt[(2 * BR_LEVELS + d) * K1 + kz];
                const bool lz = lowz && kz == 0;
                const float z3[3] = {lz ? fz.y : fz.x, lz ? fz.z : fz.y, lz ? fz.w : fz.z};
                float t = val[kz];
#pragma unroll
                for (int j = 0; j < 27; ++j) t = fmaf(p[j % 3][j / 3], z3[j % 3], t);
                val[kz] = t;
            }
        }
        // the leaf itself and its real ancestors
#pragma unroll 1
        for (int l = r; l >= 0; --l) {
            float xs[28];
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                const float4 f = sm.xL[7 * l + q];
                xs[4 * q] = f.x; xs[4 * q + 1] = f.y; xs[4 * q + 2] = f.z; xs[4 * q + 3] = f.w;
            }
            column_level<K1>(xs, sm.Bt[l * K1 + kx], sm.Bt[(BR_LEVELS + l) * K1 + ky], sm.Bt + (2 * BR_LEVELS + l) * K1, val);
        }
        float* out = blat + lx.lat(li) + (i64)ci * K1;
        unsigned fmask = 0;                 // corners of the column that another leaf owns
        if (fposs) {
#pragma unroll 1
            for (int kz = 0; kz < K1; ++kz) {
                const bool low = lowx || lowy || (lowz && kz == 0);
                if (!__any_sync(0xffffffffu, col && low)) continue;
                const int qc[3] = {qx, qy, g0[2] + kz};
                int oc[3] = {0, 0, 0};
                int own = L;
                if (col && low) own = corner_owner_cell(D, r, Lc, qc, sm.member, oc);
                // owned by another leaf of the batch: filled by k_foreign_fill
                const bool isf = own != L;
                const u64 src = isf ? foreign_src(D, r, E, bix.dl, root_of[own], oc, qc) : 0ull;
                push_foreign(isf, li, ci * K1 + kz, src, nforeign, foreign, foreign_cap);
                if (isf) fmask |= 1u << kz;
            }
        }
        if (col) {
#pragma unroll
            for (int kz = 0; kz < K1; ++kz)
                if (!((fmask >> kz) & 1)) out[kz] = val[kz] - v.iso;
        }
    }
}

// Bricks of edge 2 (leaves one depth above the finest), three to a warp, nine columns of three corners each.
// The only virtual depth is the finest, and its window, the 4x4x4 cells around the leaf, are the children
// of the leaf's 27 neighbours, so a cell's x is two loads away without a descent.  A level costs a warp 45
// instructions of arithmetic per brick where a lane per corner takes 81 on 27 of 32 lanes, and its set-up
// is shared by three.  The x27 rows and basis entries of all levels are fetched by asynchronous copies at
// once, beside the gathers of the window, so that a warp waits for one latency instead of one per level.
// 4 M points, maxDepth 11, 1.6 M such bricks, with the edge-4 bricks: 7.1 -> 5.9 ms (19.7 with a lane per
// corner); without a bound on the registers (119): 0.5 ms less than at 96.
constexpr int E2_WARPS = 2;
struct E2Warp {                        // a warp's share of shared memory, before the levels
    float x[3][64];                    // finest-depth window
    int child[3][27], member[3][27];   // the leaf's neighbours: first child, leaf of the batch (-1: none)
    int up[3][BR_LEVELS];
    int pad[2];
};
constexpr int E2_ROWS = 3 * 7, E2_BASIS = 3 * 9;   // float4 per level: x27 rows (below the finest), basis entries
static_assert(sizeof(E2Warp) % 16 == 0, "the levels follow at 16-byte alignment");
inline size_t edge2_shared(int D) { return E2_WARPS * (sizeof(E2Warp) + 16 * (size_t)(E2_ROWS * D + E2_BASIS * (D + 1))); }
static_assert(E2_WARPS * (sizeof(E2Warp) + 16 * (E2_ROWS * PRGPU_MAX_DEPTH + E2_BASIS * (PRGPU_MAX_DEPTH + 1))) <= 48 * 1024,
              "dynamic shared memory without an opt-in");
__global__ void __launch_bounds__(32 * E2_WARPS) k_edge2_eval(VArgs v, BrickIndex bix, const int* __restrict__ root_of,
                                                              LiveIndex lx, i64 first, i64 nlist,
                                                              float* __restrict__ blat,
                                                              unsigned long long* __restrict__ nforeign,
                                                              ForeignCorner* __restrict__ foreign, i64 foreign_cap) {
    extern __shared__ float4 e2_shared[];
    const EvalArgs& a = v.e;
    const int D = a.D, r = D - 1;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    char* mine = reinterpret_cast<char*>(e2_shared) +
                 w * (sizeof(E2Warp) + 16 * (size_t)(E2_ROWS * D + E2_BASIS * (D + 1)));
    E2Warp& sm = *reinterpret_cast<E2Warp*>(mine);
    float4* s_row = reinterpret_cast<float4*>(mine + sizeof(E2Warp));   // [level][brick][7]
    float4* s_bt = s_row + E2_ROWS * D;                                 // [level][brick][axis][corner]
    const int gi = min(lane / 9, 2), ci = lane - 9 * gi < 9 ? lane - 9 * gi : 8, kx = ci / 3, ky = ci % 3;
    const int rb = min(lane / 7, 2), rq = lane % 7;    // the row entry this lane fetches (lanes below 21)
    const i64 nwarps = (i64)gridDim.x * E2_WARPS;
    for (i64 it = ((i64)blockIdx.x * E2_WARPS + w) * 3; it < nlist; it += nwarps * 3) {
        const int nbr = (int)min(nlist - it, (i64)3);
        __syncwarp();                       // the previous bricks' readers are done
        for (int e = lane; e < nbr * BR_LEVELS; e += 32) {
            const int b = e / BR_LEVELS, l = e % BR_LEVELS;
            if (l <= r) sm.up[b][l] = bix.up[(i64)lx.live[first + it + b].root * BR_LEVELS + l];
        }
        __syncwarp();
        const bool on = lane < 27 && gi < nbr;
        const int g = min(gi, nbr - 1);
        int Lc[3];
        key_coords(a.nd.key[sm.up[g][r]], r, D, Lc);
        const int g0[3] = {2 * Lc[0], 2 * Lc[1], 2 * Lc[2]};
        const int u[3] = {g0[0] + kx, g0[1] + ky, g0[2]};
        int nb[3], ch[3];                   // neighbours and their first children, loads side by side
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const int e = lane + 32 * m;
            nb[m] = e < nbr * 27 ? a.nd.neigh[(i64)(e % 27) * a.nd.M + sm.up[e / 27][r]] : -1;
        }
        {
            // lanes below 27: entry k = ky of axis kx of brick g
            const int ax = kx, k = ky, gax = ax == 0 ? g0[0] : ax == 1 ? g0[1] : g0[2];
            for (int l = 0; l <= r; ++l) {
                const int sh = D - l, c = gax >> sh;
                if (lane < 27)
                    async_copy16(s_bt + l * E2_BASIS + lane, &a.lb[lattice_offset(D, l) + (i64)c * ((1 << sh) + 1) + (gax + k - (c << sh))]);
                if (lane < 21 && rb < nbr)
                    async_copy16(s_row + l * E2_ROWS + lane,
                                 reinterpret_cast<const float4*>(a.x27 + (i64)sm.up[rb][l] * X27_STRIDE) + rq);
            }
            // the finest depth: owner cell = the one below the corner, its own on the leaf's lower face
            if (lane < 27)
                async_copy16(s_bt + D * E2_BASIS + lane, &a.lb[lattice_offset(D, D) + 2 * (i64)(gax + (k == 2)) + (k - (k == 2))]);
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) ch[m] = nb[m] == -1 ? -1 : a.nd.child0[nb[m]];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const int e = lane + 32 * m, b = e / 27, j = e % 27;
            if (e >= nbr * 27) break;
            sm.child[b][j] = ch[m];
            // batch_member's rule (r >= 3: the roots of a depth are one batch)
            sm.member[b][j] = j == 13 ? sm.up[b][r] : (r >= 3 && nb[m] != -1 && v.batch_root_flag[nb[m]] == v.roots[lx.live[first + it + b].root].batch) ? nb[m] : -1;
        }
        __syncwarp();
        {
            float xv[6];
#pragma unroll
            for (int m = 0; m < 6; ++m) {
                const int b = m >> 1, cell = lane + 32 * (m & 1), bx = cell >> 4, by = (cell >> 2) & 3, bz = cell & 3;
                const int c0 = b < nbr ? sm.child[b][9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1) + ((bz + 1) >> 1)] : -1;
                xv[m] = c0 == -1 ? 0.f : a.x[c0 + ((((bx + 1) & 1) << 2) | (((by + 1) & 1) << 1) | ((bz + 1) & 1))];
            }
#pragma unroll
            for (int m = 0; m < 6; ++m) sm.x[m >> 1][lane + 32 * (m & 1)] = xv[m];
        }
        async_wait();
        __syncwarp();
        const int li = (int)(first + it + g);
        const i64 lat = lx.lat(li);
        float val[3] = {0.f, 0.f, 0.f};
        {
            const int sx = kx == 2, sy = ky == 2;
            const float4* bt = s_bt + D * E2_BASIS + 9 * g;
            const float4 fx = bt[kx], fy = bt[3 + ky];
            const float x3[3] = {fx.x, fx.y, fx.z}, y3[3] = {fy.x, fy.y, fy.z};
            float p[4][9];
#pragma unroll
            for (int z = 0; z < 4; ++z)
#pragma unroll
                for (int j = 0; j < 9; ++j)
                    p[z][j] = sm.x[g][(sx + j / 3) * 16 + (sy + j % 3) * 4 + z] * x3[j / 3] * y3[j % 3];
#pragma unroll
            for (int kz = 0; kz < 3; ++kz) {
                const int sz = kz == 2;
                const float4 fz = bt[6 + kz];
                const float z3[3] = {fz.x, fz.y, fz.z};
#pragma unroll
                for (int j = 0; j < 27; ++j) val[kz] = fmaf(p[sz + j % 3][j / 3], z3[j % 3], val[kz]);
            }
        }
#pragma unroll 1
        for (int l = r; l >= 0; --l) {
            const float4* row = s_row + l * E2_ROWS + 7 * g;
            float xs[28];
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                const float4 f = row[q];
                xs[4 * q] = f.x; xs[4 * q + 1] = f.y; xs[4 * q + 2] = f.z; xs[4 * q + 3] = f.w;
            }
            const float4* bt = s_bt + l * E2_BASIS + 9 * g;
            column_level<3>(xs, bt[kx], bt[3 + ky], bt + 6, val);
        }
        unsigned fmask = 0;
#pragma unroll
        for (int kz = 0; kz < 3; ++kz) {
            const int qc[3] = {u[0], u[1], u[2] + kz};
            int oc[3] = {0, 0, 0};
            int own = -1;
            const bool low = on && (kx == 0 || ky == 0 || kz == 0);
            if (low) own = corner_owner_cell(D, r, Lc, qc, sm.member[g], oc);
            const bool isf = low && own != sm.up[g][r];
            const u64 src = isf ? foreign_src(D, r, 2, bix.dl, root_of[own], oc, qc) : 0ull;
            push_foreign(isf, li, ci * 3 + kz, src, nforeign, foreign, foreign_cap);
            if (isf) fmask |= 1u << kz;
        }
        if (on) {
            float* out = blat + lat + ci * 3;
#pragma unroll
            for (int kz = 0; kz < 3; ++kz)
                if (!((fmask >> kz) & 1)) out[kz] = val[kz] - v.iso;
        }
    }
}

// Corners by sibling groups, four to a warp.  A group's 2x2x2 cells have 3x3x3 corners.
// The cells around them are the 4x4x4 block of the children of the parent's 27 neighbours (the group table:
// sibling groups are whole), so which exist and which of them precede the group in key order are 27 bits, and
// a corner is the group's own when none of its 8 cells that exists precedes the group; its owner is then the
// lowest of the group's cells at it.  The window, the ancestors' x27 rows and the walk are those of the
// edge-2 bricks above: a column of up to three corners along z per lane, here only the columns that own any (a surface fills about
// half of the 36), and each value goes to the cells of the block that share the corner, without a look at
// their neighbour tables.
// COARSE: the groups above the finest depth (a warp's may lie at two depths), of whose corners only those that a
// leaf shares are wanted; an owner with children adds its descent, the corners one to a lane.  Corners and flags of
// the coarse leaves, 50k sphere 0.088 -> 0.051 ms, 100k superquadric 0.215 -> 0.177, 1M torus 0.48 -> 0.46 (4M
// displaced sphere 2.3 either way, bound by the descents).
// Finest cells: 1M torus 0.90 -> 0.56 ms, 4M displaced sphere 3.9 -> 2.4, where a pass over the nodes' neighbours and keys
// found the owners and a thread per owned corner walked up alone.  Two thirds of it is arithmetic; fetching
// every group's rows, shared or not, cost 0.16 ms on the torus, and the basis entries a level ahead gain nothing.
constexpr int FC_GROUPS = 4, FC_WARPS = 2;
struct FcWarp {
    unsigned long long leaf[FC_GROUPS];         // COARSE: the leaves among the cells of the block
    unsigned long long before[FC_GROUPS];       // cells of the block that exist and precede the group, a bit each
    float x[FC_GROUPS][65];                     // windows; a warp reads 0, 4, 16 and 20 on of each, in banks of their own
    int gn[FC_GROUPS * GN_ROW];
    int up[FC_GROUPS][BR_LEVELS];               // the parent and its ancestors, by depth
    int depth[FC_GROUPS];
    int cell[FC_GROUPS][3];                     // coordinates of the group's first cell
    unsigned char row[FC_GROUPS][BR_LEVELS];    // the group whose copy of the ancestor's row serves this one
    float val[96];                              // COARSE: corners of a round of columns
    unsigned char corner[96];
    unsigned short col[40];                     // group, column and owned corners of the columns that own any
};
constexpr int FC_ROWS = FC_GROUPS * 7;          // float4 per level
static_assert(sizeof(FcWarp) % 16 == 0, "the rows follow at 16-byte alignment");
static_assert(FC_WARPS * (sizeof(FcWarp) + 16 * FC_ROWS * PRGPU_MAX_DEPTH) <= 48 * 1024,
              "dynamic shared memory without an opt-in");
inline unsigned group_blocks(i64 ng) { return (unsigned)((ng + FC_GROUPS * FC_WARPS - 1) / (FC_GROUPS * FC_WARPS)); }
inline size_t group_shared(int D) { return FC_WARPS * (sizeof(FcWarp) + 16 * (size_t)FC_ROWS * D); }
// out: eight values per cell from node out0 on
template <bool COARSE>
__global__ void __launch_bounds__(32 * FC_WARPS) k_group_corners(EvalArgs a, const int* __restrict__ gn_rows, i64 gfirst,
                                                                 i64 ng, float iso, float* __restrict__ out, i64 out0) {
    extern __shared__ float4 fc_shared[];
    const int D = a.D;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    char* mine = reinterpret_cast<char*>(fc_shared) + w * (sizeof(FcWarp) + 16 * (size_t)FC_ROWS * D);
    FcWarp& sm = *reinterpret_cast<FcWarp*>(mine);
    float4* s_row = reinterpret_cast<float4*>(mine + sizeof(FcWarp));   // [level][group][7]
    const i64 g1 = ((i64)blockIdx.x * FC_WARPS + w) * FC_GROUPS;
    if (g1 >= ng) return;
    const int nbr = (int)min(ng - g1, (i64)FC_GROUPS);
#pragma unroll
    for (int m = 0; m < (FC_GROUPS * GN_ROW + 31) / 32; ++m) {
        const int e = lane + 32 * m;
        if (e < FC_GROUPS * GN_ROW) sm.gn[e] = e < nbr * GN_ROW ? gn_rows[(gfirst + g1) * GN_ROW + e] : -1;
    }
    if (lane < nbr) {
        const i64 first = 1 + 8 * (gfirst + g1 + lane);
        const int d = COARSE ? a.nd.depth[first] : D;
        sm.depth[lane] = d;
        int n = (int)first;
        for (int l = D - 1; l >= 0; --l) {
            if (!COARSE || l < d) n = a.nd.parent[n];
            sm.up[lane][l] = !COARSE || l < d ? n : -1;
        }
        int c[3];
        key_coords(a.nd.key[first], d, D, c);
        for (int ax = 0; ax < 3; ++ax) sm.cell[lane][ax] = c[ax];
    }
    __syncwarp();
    int node[2 * FC_GROUPS];                    // this lane's cells of the blocks, -1: absent
#pragma unroll
    for (int m = 0; m < 2 * FC_GROUPS; ++m) {
        const int g = m >> 1, cell = lane + 32 * (m & 1), bx = cell >> 4, by = (cell >> 2) & 3, bz = cell & 3;
        const int cn = sm.gn[g * GN_ROW + 9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1) + ((bz + 1) >> 1)];
        node[m] = cn == -1 ? -1 : cn + ((((bx + 1) & 1) << 2) | (((by + 1) & 1) << 1) | ((bz + 1) & 1));
        const unsigned b = __ballot_sync(0xffffffffu, cn != -1 && cn < sm.gn[g * GN_ROW + 13]);
        if (lane == 0) reinterpret_cast<unsigned*>(sm.before)[m] = b;
    }
    auto stage = [&]() {
        {
            // neighbouring groups share their upper ancestors: a row is fetched by the first group that has it
            const int b = lane / 7, q = lane % 7;
            if (b < nbr)
                for (int l = 0; l < sm.depth[b]; ++l) {
                    const int n = sm.up[b][l];
                    int first = b;
                    while (first > 0 && sm.up[first - 1][l] == n) --first;
                    if (first == b)
                        async_copy16(s_row + l * FC_ROWS + lane, reinterpret_cast<const float4*>(a.x27 + (i64)n * X27_STRIDE) + q);
                    if (q == 0) sm.row[b][l] = (unsigned char)first;
                }
        }
        {
            float xv[2 * FC_GROUPS];
#pragma unroll
            for (int m = 0; m < 2 * FC_GROUPS; ++m) xv[m] = node[m] == -1 ? 0.f : a.x[node[m]];
#pragma unroll
            for (int m = 0; m < 2 * FC_GROUPS; ++m) sm.x[m >> 1][lane + 32 * (m & 1)] = xv[m];
        }
    };
    if (!COARSE) stage();
    if (COARSE) {
        bool leaf[2 * FC_GROUPS];
#pragma unroll
        for (int m = 0; m < 2 * FC_GROUPS; ++m) leaf[m] = node[m] != -1 && a.nd.child0[node[m]] == -1;
#pragma unroll
        for (int m = 0; m < 2 * FC_GROUPS; ++m) {
            const unsigned b = __ballot_sync(0xffffffffu, leaf[m]);
            if (lane == 0) reinterpret_cast<unsigned*>(sm.leaf)[m] = b;
        }
    }
    __syncwarp();
    int ncol = 0;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int e = lane + 32 * m, g = e / 9, kx = e % 9 / 3, ky = e % 3;
        int bits = 0;
        if (e < 9 * nbr)
#pragma unroll
            for (int kz = 0; kz < 3; ++kz) {
                const unsigned long long at = 0x330033ull << (16 * kx + 4 * ky + kz);   // the 2x2x2 cells at the corner
                if (!(sm.before[g] & at) && (!COARSE || (sm.leaf[g] & at))) bits |= 1 << kz;
            }
        const unsigned some = __ballot_sync(0xffffffffu, bits != 0);
        if (bits) sm.col[ncol + __popc(some & ((1u << lane) - 1u))] = (unsigned short)(e << 3 | bits);
        ncol += __popc(some);
    }
    if (COARSE) {                               // nothing to fetch where no corner is wanted
        if (ncol == 0) return;
        stage();
    }
    async_wait();
    __syncwarp();
    for (int c0 = 0; c0 < ncol; c0 += 32) {
        const int entry = sm.col[min(c0 + lane, ncol - 1)];
        const int bits = c0 + lane < ncol ? entry & 7 : 0, e = entry >> 3, g = e / 9, kx = e % 9 / 3, ky = e % 3;
        const int g0[3] = {sm.cell[g][0], sm.cell[g][1], sm.cell[g][2]};
        const int d = COARSE ? sm.depth[g] : D, sh0 = D - d;   // corner k of the group: (g0 + k) << sh0 on the lattice
        float val[3] = {0.f, 0.f, 0.f};
        {
            // the group's depth: owner cell = the one below the corner, its own on the group's lower face
            const int sx = kx == 2, sy = ky == 2;
            const float4 fx = lattice_at(a, d, g0[0] + sx, (kx - sx) << sh0),
                         fy = lattice_at(a, d, g0[1] + sy, (ky - sy) << sh0);
            const float x3[3] = {fx.x, fx.y, fx.z}, y3[3] = {fy.x, fy.y, fy.z};
            float p[4][9];
#pragma unroll
            for (int z = 0; z < 4; ++z)
#pragma unroll
                for (int j = 0; j < 9; ++j)
                    p[z][j] = sm.x[g][(sx + j / 3) * 16 + (sy + j % 3) * 4 + z] * x3[j / 3] * y3[j % 3];
#pragma unroll
            for (int kz = 0; kz < 3; ++kz) {
                const int sz = kz == 2;
                const float4 fz = lattice_at(a, d, g0[2] + sz, (kz - sz) << sh0);
                const float z3[3] = {fz.x, fz.y, fz.z};
#pragma unroll
                for (int j = 0; j < 27; ++j) val[kz] = fmaf(p[sz + j % 3][j / 3], z3[j % 3], val[kz]);
            }
        }
#pragma unroll 1
        for (int l = d - 1; l >= 0; --l) {
            const int sh = D - l;
            int c[3], k[3];
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                c[ax] = g0[ax] >> (d - l);
                k[ax] = (g0[ax] << sh0) - (c[ax] << sh);
            }
            const float4* bz = &a.lb[lattice_offset(D, l) + (i64)c[2] * ((1 << sh) + 1) + k[2]];
            const float4 b3[3] = {bz[0], bz[1 << sh0], bz[2 << sh0]};
            const float4* row = s_row + l * FC_ROWS + 7 * sm.row[g][l];
            float xs[28];
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                const float4 f = row[q];
                xs[4 * q] = f.x; xs[4 * q + 1] = f.y; xs[4 * q + 2] = f.z; xs[4 * q + 3] = f.w;
            }
            column_level<3>(xs, lattice_at(a, l, c[0], k[0] + (kx << sh0)), lattice_at(a, l, c[1], k[1] + (ky << sh0)), b3, val);
        }
        auto scatter = [&](int g, int kx, int ky, int kz, float v) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {       // the cells at the corner, in block coordinates
                const int bx = kx + (q & 1), by = ky + ((q >> 1) & 1), bz = kz + (q >> 2);
                const int cn = sm.gn[g * GN_ROW + 9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1) + ((bz + 1) >> 1)];
                if (cn == -1 || (COARSE && !((sm.leaf[g] >> (16 * bx + 4 * by + bz)) & 1))) continue;
                const int cell = cn + ((((bx + 1) & 1) << 2) | (((by + 1) & 1) << 1) | ((bz + 1) & 1));
                out[8 * ((i64)cell - out0) + (q ^ 7)] = v;
            }
        };
        if (!COARSE) {
#pragma unroll
            for (int kz = 0; kz < 3; ++kz)
                if ((bits >> kz) & 1) scatter(g, kx, ky, kz, val[kz] - iso);
            continue;
        }
        // a descent is a walk of its own: the corners one to a lane
        __syncwarp();
        int n = 0;
#pragma unroll
        for (int kz = 0; kz < 3; ++kz) {
            const bool own = (bits >> kz) & 1;
            const unsigned some = __ballot_sync(0xffffffffu, own);
            if (own) {
                const int at = n + __popc(some & ((1u << lane) - 1u));
                sm.val[at] = val[kz];
                sm.corner[at] = (unsigned char)(3 * e + kz);
            }
            n += __popc(some);
        }
        __syncwarp();
        for (int q = lane; q < n; q += 32) {
            const int e = sm.corner[q] / 3, kz = sm.corner[q] % 3, g = e / 9, kx = e % 9 / 3, ky = e % 3;
            const int sx = kx == 2, sy = ky == 2, sz = kz == 2, d = sm.depth[g], sh0 = D - d;
            const int X = sm.cell[g][0], Y = sm.cell[g][1], Z = sm.cell[g][2];
            const int u[3] = {(X + kx) << sh0, (Y + ky) << sh0, (Z + kz) << sh0};
            const float v = corner_descent(a, sm.gn[g * GN_ROW + 13] + (sx << 2 | sy << 1 | sz), d,
                                           (kx - sx) | (ky - sy) << 1 | (kz - sz) << 2, X + sx, Y + sy, Z + sz, u, sm.val[q]);
            scatter(g, kx, ky, kz, v - iso);
        }
    }
}

// corners on a leaf's lower faces owned by a cell of another leaf L' of the
// batch: the same value is a corner of L''s brick holding the owner cell, where
// L' owns it -- copied when that brick is live, evaluated otherwise
// (count[0]: the corners; count[2]: those evaluated.  The grids do not depend on the counts, which the host
// has not read.)  A few in a hundred are evaluated, at a hundred times the cost of a copy.  LIST: they are listed by
// the launch that copies and evaluated by one of their own, one to a thread, instead of each holding up a warp of
// copies: 27 M corners (4M displaced sphere) 2.36 -> 1.50 ms, 101 M 8.5 -> 5.3, 1.3 M (1M torus) 0.174 -> 0.150.
// Below FF_LISTED lower-face corners of live bricks one launch that does both is the faster, the evaluation's chain of loads
// being most of either: 0.44 M corners 0.065 against 0.085 ms.  A launch with a list takes the corners [at, end), at most
// FF_SPAN, whose numbers from 'at' on the list holds; count[3] of them.  (PRGPU_HOOK_FOREIGN_SPAN: lists for every size, of
// shorter spans.)
constexpr i64 FF_SPAN = 1ll << 31, FF_LISTED = 1ll << 21;
// the owner brick's corner, evaluated by its own leaf
__device__ __forceinline__ float foreign_value(const VArgs& v, const BrickIndex& bix, u64 src) {
    const int D = v.e.D, e = (int)(src & 1023);
    const VBrick B = brick_of(v, bix, (i64)(src >> 10));
    const VRoot R = v.roots[B.root];
    const int r = R.depth, S = 1 << (D - r), E = brick_edge(D, r), E1 = E + 1;
    int Lc[3];
    key_coords(v.e.nd.key[R.node], r, D, Lc);
    const int kk[3] = {e / (E1 * E1), (e / E1) % E1, e % E1};
    int oc[3], qc[3];
    for (int ax = 0; ax < 3; ++ax) {
        const int l0 = Lc[ax] * S;
        qc[ax] = l0 + B.b[ax] * E + kk[ax];
        oc[ax] = max(qc[ax] - 1, l0);
    }
    return virtual_corner_value(v, R.node, r, oc, qc) - v.iso;
}
template <bool LIST>
__global__ void k_foreign_fill(VArgs v, BrickIndex bix, LiveIndex lx, const unsigned char* __restrict__ culled,
                               const int* __restrict__ live_pos, const ForeignCorner* __restrict__ foreign, i64 at, i64 end,
                               float* __restrict__ blat, unsigned* __restrict__ list, unsigned long long* __restrict__ count) {
    const i64 n = min((i64)count[0], end);
    for (i64 f0 = at + (i64)blockIdx.x * blockDim.x; f0 < n; f0 += (i64)gridDim.x * blockDim.x) {
        const i64 f = f0 + threadIdx.x;
        bool slow = false;
        if (f < n) {
            const ForeignCorner fe = foreign[f];
            const i64 brick = (i64)(fe.src >> 10);
            slow = culled[brick];
            if (!slow) {
                blat[lx.lat(fe.li) + fe.e] = blat[lx.lat(live_pos[brick]) + (int)(fe.src & 1023)];
            } else if (!LIST) {
                atomicAdd(&count[2], 1ull);
                blat[lx.lat(fe.li) + fe.e] = foreign_value(v, bix, fe.src);
            }
        }
        if (!LIST) continue;
        const unsigned m = __ballot_sync(0xffffffffu, slow);
        if (!m) continue;
        const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
        unsigned base = 0;
        if (lane == leader) {
            base = (unsigned)atomicAdd(&count[3], (unsigned long long)__popc(m));
            atomicAdd(&count[2], (unsigned long long)__popc(m));
        }
        base = __shfl_sync(0xffffffffu, base, leader);
        if (slow) list[base + __popc(m & ((1u << lane) - 1u))] = (unsigned)(f - at);
    }
}
__global__ void k_foreign_eval(VArgs v, BrickIndex bix, LiveIndex lx, const ForeignCorner* __restrict__ foreign, i64 at,
                               const unsigned* __restrict__ list, float* __restrict__ blat,
                               const unsigned long long* __restrict__ count) {
    const i64 n = (i64)count[3];
    for (i64 q = (i64)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (i64)gridDim.x * blockDim.x) {
        const ForeignCorner fe = foreign[at + list[q]];
        blat[lx.lat(fe.li) + fe.e] = foreign_value(v, bix, fe.src);
    }
}

// live bricks in brick order
__global__ void k_live_bricks(VArgs v, BrickIndex bix, const unsigned char* __restrict__ culled,
                              const int* __restrict__ pos, i64 nbricks, LiveBrick* __restrict__ live) {
    for (i64 bi = (i64)blockIdx.x * blockDim.x + threadIdx.x; bi < nbricks; bi += (i64)gridDim.x * blockDim.x) {
        if (culled[bi]) continue;
        const VBrick B = brick_of(v, bix, bi);
        LiveBrick lb;
        lb.root = B.root;
        lb.b[0] = B.b[0]; lb.b[1] = B.b[1]; lb.b[2] = B.b[2];
        live[pos[bi]] = lb;
    }
}
__global__ void k_live_flags(const unsigned char* __restrict__ culled, i64 n, int* __restrict__ f) {
    for (i64 k = (i64)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (i64)gridDim.x * blockDim.x)
        f[k] = culled[k] ? 0 : 1;
}

// ---- virtual cells: the cells of the live bricks
__global__ void __launch_bounds__(CELL_BLOCK) k_virtual_cells(LiveIndex lx, const float* __restrict__ lat, i64 total,
                                                              unsigned char* __restrict__ cat, int* __restrict__ tile_tri) {
    int tri = 0;
    for (int q = 0; q < CELL_TILE / CELL_BLOCK; ++q) {
        const i64 e = (i64)blockIdx.x * CELL_TILE + q * CELL_BLOCK + threadIdx.x;
        if (e >= total) break;
        int lg, loc;
        const i64 li = lx.brick(e, lg, loc);
        const int E = 1 << lg, E1 = E + 1;
        const float* L = lat + lx.lat(li) + ((loc >> (2 * lg)) * E1 + ((loc >> lg) & (E - 1))) * E1 + (loc & (E - 1));
        int cc = 0;
#pragma unroll
        for (int kind = 0; kind < 8; ++kind)
            if (L[((kind & 1) * E1 + ((kind >> 1) & 1)) * E1 + (kind >> 2)] < 0.f) cc |= 1 << c_vid[kind];
        cat[e] = (unsigned char)cc;
        tri += c_tri_count[cc];
    }
    tile_triangles(tri, tile_tri);
}

// ---------------------------- triangle emission ------------------------------
struct EmitArgs {
    int D;
    int local_bits;
    int weld;           // 1: keys without the batch (vertices shared across batches)
    i64 tri_offset;     // first global triangle of this emission
    u64* keys;          // 3 per triangle
    float* pos;         // 3 floats per emission
};

__device__ __forceinline__ u64 edge_key(const int lp[3], int o, int D, int batch, int local_bits) {
    const u64 S1 = (u64)(1 << D) + 1;
    u64 k = (((u64)lp[0] * S1 + (u64)lp[1]) * S1 + (u64)lp[2]) * 3 + (u64)o;
    return ((u64)batch << local_bits) | k;
}

// interpolatePoint (main.cu:2584-2597) with p1/p2 in the edge owner's frame
__device__ __forceinline__ void crossing(const int lo_pt[3], int o, bool reversed, float v_lo, float v_hi, int D,
                                         float out[3]) {
    const float inv = 1.0f / (float)(1 << D);
    float p1[3] = {(float)lo_pt[0] * inv, (float)lo_pt[1] * inv, (float)lo_pt[2] * inv};
    float p2[3] = {p1[0], p1[1], p1[2]};
    p2[o] = (float)(lo_pt[o] + 1) * inv;
    float f1 = v_lo, f2 = v_hi;
    if (reversed) {
        float t = p1[o]; p1[o] = p2[o]; p2[o] = t;
        f1 = v_hi; f2 = v_lo;
    }
    for (int i = 0; i < 3; ++i) out[i] = p1[i];
    const float pivot = f1 / (f1 - f2);
    const float another = 1.f - pivot;
    out[o] = fmaf(p2[o], pivot, p1[o] * another);
}

// lattice lower end of edge e of a cell at c[], its orientation and off bits
__device__ __forceinline__ void edge_geom(int e, const int c[3], int lp[3], int& o, int& a0, int& a1, int& b0, int& b1) {
    o = e >> 2;
    a0 = (o == 0) ? 1 : 0;
    a1 = (o == 2) ? 1 : 2;
    b0 = e & 1;
    b1 = (e >> 1) & 1;
    lp[0] = c[0]; lp[1] = c[1]; lp[2] = c[2];
    lp[a0] += b0;
    lp[a1] += b1;
}

// Emission: a thread per triangle corner, in the order of the output, so that a warp writes 32 consecutive
// keys, slots and positions.  (A thread per cell writes its corners one by one, every store of a warp
// spread over 32 sectors: 0.52 ms for the 9.2 M corners of the 1M torus, 220 MB.)
// Corner k of the cell's triangles: its edge's key and crossing.  rev(a0, a1, b0, b1): the edge at offsets
// b0, b1 along the axes a0, a1 runs reversed in its owner's frame; only edges along x do (crossing's
// frame), so only they look for their owner.
template <class V, class R>
__device__ __forceinline__ void emit_corner(const EmitArgs& em, const int c[3], V value, int cc, int k, i64 slot, int batch,
                                            R rev) {
    const int e = c_tri_edges[cc][k];
    int lp[3], o, a0, a1, b0, b1;
    edge_geom(e, c, lp, o, a0, a1, b0, b1);
    const int ev0 = (b0 << a0) | (b1 << a1);   // corner kind of the lower end
    const int ev1 = ev0 | (1 << o);
    float p[3];
    crossing(lp, o, o == 0 && rev(a0, a1, b0, b1), value(ev0), value(ev1), em.D, p);
    em.keys[slot] = edge_key(lp, o, em.D, batch, em.local_bits);
    em.pos[3 * slot] = p[0];
    em.pos[3 * slot + 1] = p[1];
    em.pos[3 * slot + 2] = p[2];
}

// real finest cells
__global__ void __launch_bounds__(CELL_BLOCK) k_emit_real(NodeArrays nd, EmitArgs em, i64 lo, i64 total,
                                                          const unsigned char* __restrict__ cat,
                                                          const i64* __restrict__ tile_first, const float* __restrict__ cell_v) {
    __shared__ TileShared sm;
    const int n = 3 * tile_active(cat, total, sm);
    const i64 slot0 = 3 * (em.tri_offset + tile_first[blockIdx.x]);
    for (int q = threadIdx.x; q < n; q += CELL_BLOCK) {
        const int cell = sm.cell[q / 3];
        const i64 s = (i64)blockIdx.x * CELL_TILE + cell, i = lo + s;
        int c[3];
        key_coords(nd.key[i], em.D, em.D, c);
        const float* cv = cell_v + 8 * s;
        emit_corner(em, c, [&](int kind) { return cv[kind]; }, cat[s], q - 3 * sm.first[cell], slot0 + q, 0,
                    [&](int a0, int a1, int b0, int b1) {
                        // edge owner among the real cells sharing it
                        u64 best = ~0ull;
                        int own_b0 = b0;
                        for (int t = 0; t < 4; ++t) {
                            const int d0 = b0 - (t & 1), d1 = b1 - ((t >> 1) & 1);
                            int dxyz[3] = {0, 0, 0};
                            dxyz[a0] = d0;
                            dxyz[a1] = d1;
                            const int nb = nd.neigh[(i64)(9 * (dxyz[0] + 1) + 3 * (dxyz[1] + 1) + (dxyz[2] + 1)) * nd.M + i];
                            if (nb == -1) continue;
                            const u64 kk = nd.key[nb];
                            if (kk < best) { best = kk; own_b0 = b0 - d0; }
                        }
                        return own_b0 == 1;
                    });
    }
}

__global__ void __launch_bounds__(CELL_BLOCK) k_emit_virtual(VArgs v, EmitArgs em, LiveIndex lx, const float* __restrict__ lat,
                                                             i64 total, const unsigned char* __restrict__ cat,
                                                             const i64* __restrict__ tile_first) {
    __shared__ TileShared sm;
    const int n = 3 * tile_active(cat, total, sm);
    const int D = em.D;
    const i64 slot0 = 3 * (em.tri_offset + tile_first[blockIdx.x]);
    for (int q = threadIdx.x; q < n; q += CELL_BLOCK) {
        const int cell = sm.cell[q / 3];
        const i64 e = (i64)blockIdx.x * CELL_TILE + cell;
        int lg, loc;
        const i64 li = lx.brick(e, lg, loc);
        const int E = 1 << lg, E1 = E + 1;
        const int l3[3] = {loc >> (2 * lg), (loc >> lg) & (E - 1), loc & (E - 1)};
        const LiveBrick lb = lx.live[li];
        const VRoot R = v.roots[lb.root];
        const int S = 1 << (D - R.depth);
        int Lc[3];
        key_coords(v.e.nd.key[R.node], R.depth, D, Lc);
        const int c[3] = {Lc[0] * S + lb.b[0] * E + l3[0], Lc[1] * S + lb.b[1] * E + l3[1], Lc[2] * S + lb.b[2] * E + l3[2]};
        const float* L = lat + lx.lat(li) + (l3[0] * E1 + l3[1]) * E1 + l3[2];
        emit_corner(em, c, [&](int kind) { return L[((kind & 1) * E1 + ((kind >> 1) & 1)) * E1 + (kind >> 2)]; }, cat[e],
                    q - 3 * sm.first[cell], slot0 + q, em.weld ? 0 : R.batch, [&](int a0, int a1, int b0, int b1) {
                        u64 best = ~0ull;
                        int own_b0 = b0;
                        for (int t = 0; t < 4; ++t) {
                            const int d0 = b0 - (t & 1), d1 = b1 - ((t >> 1) & 1);
                            int oc[3] = {c[0], c[1], c[2]};
                            oc[a0] += d0;
                            oc[a1] += d1;
                            if (batch_member(v, R, Lc, oc) < 0) continue;
                            const u64 kk = cell_key_D(oc, D);
                            if (kk < best) { best = kk; own_b0 = b0 - d0; }
                        }
                        return own_b0 == 1;
                    });
    }
}

// after sorting: vertex id per sorted element, positions of the first element
__global__ void k_vertex_ids(const u64* __restrict__ keys, const uint32_t* __restrict__ slot, i64 n,
                             const int* __restrict__ pos_scan, const float* __restrict__ epos, float scale,
                             float3 center, int32_t* __restrict__ tri_vid, float* __restrict__ vpos) {
    for (i64 k = (i64)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (i64)gridDim.x * blockDim.x) {
        const bool head = (k == 0) || keys[k] != keys[k - 1];
        const int vid = pos_scan[k] + (head ? 1 : 0) - 1;
        tri_vid[slot[k]] = vid;
        if (head) {
            // input coordinates: p*scale + centre (PlyWriteTriangles plyfile.cu:2801-2812), unfused
            const uint32_t sl = slot[k];
            vpos[3 * (i64)vid] = __fadd_rn(__fmul_rn(epos[3 * (i64)sl], scale), center.x);
            vpos[3 * (i64)vid + 1] = __fadd_rn(__fmul_rn(epos[3 * (i64)sl + 1], scale), center.y);
            vpos[3 * (i64)vid + 2] = __fadd_rn(__fmul_rn(epos[3 * (i64)sl + 2], scale), center.z);
        }
    }
}
// subdivision roots: node index and depth, in node order
__global__ void k_root_list(NodeArrays nd, const int* __restrict__ is_root, const int* __restrict__ pos, i64 n,
                            int2* __restrict__ out) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
        if (is_root[i]) out[pos[i]] = make_int2((int)i, (int)nd.depth[i]);
}
// subdivision roots are in node order, hence in depth order: the index of the
// first root at depth d is the root prefix at the first node of depth d, and
// every per-root count (bricks, rows, batch) is a closed form of the depth
struct DepthStarts {
    i64 base[17];
};
__global__ void k_depth_firsts(const int* __restrict__ rpos, DepthStarts b, int D, int* __restrict__ out) {
    const int d = threadIdx.x;
    if (d <= D) out[d] = rpos[b.base[d]];
}
struct RootLayout {
    int first[17];    // first root at depth d
    int batch[17];    // batch of the roots at depth d >= 3
    i64 off[4][17];   // bricks, brick rows, super-bricks, super rows of the roots above depth d
    i64 per[4][17];   // the same per root at depth d
};
__global__ void k_make_roots(const int2* __restrict__ dr, int nr, int D, RootLayout L, VRoot* __restrict__ roots,
                             i64* __restrict__ pre) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nr; k += gridDim.x * blockDim.x) {
        const int2 r = dr[k];
        const int d = r.y;
        VRoot R;
        R.node = r.x;
        R.depth = d;
        R.batch = d < 3 ? k + 1 : L.batch[d];   // one batch per root above depth 3, one per depth from 3
        R.pad = 0;
        roots[k] = R;
        const i64 local = k - L.first[d];
#pragma unroll
        for (int q = 0; q < 4; ++q) pre[(i64)q * (nr + 1) + k] = L.off[q][d] + local * L.per[q][d];
        if (k == 0)
#pragma unroll
            for (int q = 0; q < 4; ++q) pre[(i64)q * (nr + 1) + nr] = L.off[q][D];
    }
}

__global__ void k_key_heads(const u64* __restrict__ keys, i64 n, int* __restrict__ f) {
    for (i64 k = (i64)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (i64)gridDim.x * blockDim.x)
        f[k] = (k == 0 || keys[k] != keys[k - 1]) ? 1 : 0;
}
void stage_mesh(Ctx& c) {
    ensure_mc_tables();
    cudaStream_t s = c.stream;
    const int D = c.D;
    const NodeArrays& nd = c.nodes;
    const i64 M = nd.M, lo = c.base[D], nD = c.count[D];
    const int kx = c.kbegin("mesh_tables", 0.0);
    float* x27 = build_x27(c, lo);
    EvalArgs ea{c.nodes, D, c.basis, c.x, x27, x27 ? lo : 0, nullptr, c.params.stable_basis};
    float4* lb = nullptr;
    {
        const i64 total = lattice_offset(D, D + 1);
        lb = dalloc<float4>(total, s);
        k_lattice_basis<<<grid_for(4 * total, 256), 256, 0, s>>>(c.basis, D, total, reinterpret_cast<float*>(lb),
                                                                 c.params.stable_basis);
        CK_LAUNCH();
        ea.lb = lb;
    }
    c.kend(kx);
    // ---- finest corner values, categories
    float* cell_v = dalloc<float>(8 * nD, s);
    unsigned char* cat = dalloc<unsigned char>(nD, s);
    const i64 rtiles = (nD + CELL_TILE - 1) / CELL_TILE;
    int* rtri = dalloc<int>(rtiles, s);             // triangles of each tile of real cells
    i64* rfirst = dalloc<i64>(rtiles + 1, s);       // first triangle of each tile, and their number
    int kt = c.kbegin("corner_values", (double)M * (108 + 8 + 4 + 4) + (double)nD * 8 * 4);
    {
        // (no index here needs this bound; no tree of that size, 41 GB of nodes, has been meshed)
        if (nD >= (1ll << 28)) {
            set_last_error("a mesh from %lld finest nodes: 2^28 or more are not taken", (long long)nD);
            throw Error{PRGPU_ERR_LIMIT, {0}};
        }
        const i64 gfirst = (lo - 1) / 8, ng = nD / 8;
        ensure_group_rows(c);
        k_group_corners<false><<<group_blocks(ng), 32 * FC_WARPS, group_shared(D), s>>>(ea, c.gn_rows, gfirst, ng, c.iso,
                                                                                       cell_v, lo);
        CK_LAUNCH();
    }
    c.kend(kt);
    kt = c.kbegin("cells", (double)nD * (8 * 4 + 1));
    k_finest_cells<<<(unsigned)rtiles, CELL_BLOCK, 0, s>>>(cell_v, nD, cat, rtri);
    CK_LAUNCH();
    exclusive_scan<int, i64>(rtri, rfirst, rtiles, rfirst + rtiles, s);
    c.kend(kt);
    // ---- face marks and subdivision roots
    int* fflag = dalloc<int>(6 * M, s);
    CK(cudaMemsetAsync(fflag, 0, (size_t)(6 * M) * sizeof(int), s));
    kt = c.kbegin("mark_faces", (double)nD * (1 + 108) + (double)M * 24);
    k_mark_faces<<<grid_for(nD, 128, 1ll << 30), 128, 0, s>>>(nd, D, lo, M, cat, fflag);
    CK_LAUNCH();
    c.kend(kt);
    const i64 nCoarse = lo;   // nodes at depth < D
    dfree(c.d_has_tri, s);
    dfree(c.d_has_int, s);
    c.n_coarse = nCoarse;
    int* has_tri = c.d_has_tri = dalloc<int>(nCoarse, s);
    int* has_int = c.d_has_int = dalloc<int>(nCoarse, s);
    int* is_root = dalloc<int>(nCoarse, s);
    CK(cudaMemsetAsync(has_tri, 0, nCoarse * sizeof(int), s));
    CK(cudaMemsetAsync(has_int, 0, nCoarse * sizeof(int), s));
    CK(cudaMemsetAsync(is_root, 0, nCoarse * sizeof(int), s));
    if (nCoarse > 1) {
        const int kc = c.kbegin("coarse_leaves", (double)nCoarse * (4 + 108 + 8 + 3 * 4 + 8 * 4) + (double)M * 4);
        float* leaf_v = dalloc<float>(8 * nCoarse, s);
        const i64 ng = (lo - 1) / 8;
        k_group_corners<true><<<group_blocks(ng), 32 * FC_WARPS, group_shared(D), s>>>(ea, c.gn_rows, 0, ng, c.iso, leaf_v, 0);
        CK_LAUNCH();
        k_coarse_leaves<<<grid_for(nCoarse - 1, 128, 1ll << 30), 128, 0, s>>>(nd, 1, nCoarse, leaf_v, fflag, has_tri,
                                                                             has_int, is_root);
        CK_LAUNCH();
        c.kend(kc);
        dfree(leaf_v, s);
    }
    dfree(fflag, s);
    int kg = c.kbegin("mesh_lists", 0.0);
    // subdivision roots in node order, compacted on the device; the host reads only
    // the index of the first root of every depth
    int2* droot_list = nullptr;
    int nr = 0;
    RootLayout layout{};
    i64 tot[4] = {0, 0, 0, 0}, nbig = 0, nlarge = 0;
    int nbatches = 1;
    {
        int* rpos = dalloc<int>(nCoarse + 1, s);
        exclusive_scan<int, int>(is_root, rpos, nCoarse, rpos + nCoarse, s);
        DepthStarts ds{};
        for (int d = 0; d <= D; ++d) ds.base[d] = c.base[d];
        int* dfirst = dalloc<int>(D + 1, s);
        k_depth_firsts<<<1, 32, 0, s>>>(rpos, ds, D, dfirst);
        CK_LAUNCH();
        int hfirst[17];
        CK(cudaMemcpyAsync(hfirst, dfirst, (D + 1) * sizeof(int), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        dfree(dfirst, s);
        nr = hfirst[D];   // roots are coarse nodes (depth < D)
        droot_list = dalloc<int2>(std::max(nr, 1), s);
        k_root_list<<<grid_for(nCoarse, 256), 256, 0, s>>>(nd, is_root, rpos, nCoarse, droot_list);
        CK_LAUNCH();
        dfree(rpos, s);
        c.roots_per_depth.assign(D + 1, 0);
        int nb = 0;
        for (int d = 0; d <= D; ++d) {
            const int cnt = d < D ? hfirst[d + 1] - hfirst[d] : 0;
            c.roots_per_depth[d] = cnt;
            const int S = 1 << (D - d), E = std::min(S, BR), nbk = S / E;
            const int ns = (D - d >= 6) ? S / (4 * BR) : 0;
            layout.first[d] = hfirst[d];
            layout.per[0][d] = (i64)nbk * nbk * nbk;
            layout.per[1][d] = 3 * nbk;
            layout.per[2][d] = (i64)ns * ns * ns;
            layout.per[3][d] = 3 * ns;
            for (int q = 0; q < 4; ++q) {
                layout.off[q][d] = tot[q];
                tot[q] += (i64)cnt * layout.per[q][d];
            }
            if (D - d >= 6) nlarge = tot[0];   // bricks of leaves with lattice edge >= 64 (super-bricks) come first
            if (D - d >= 4) nbig = tot[0];     // then those of edge >= 16
            if (d < 3) nb += cnt;
            else if (cnt > 0) layout.batch[d] = ++nb;
        }
        nbatches = nb + 1;
    }
    dfree(is_root, s);
    c.subdivide_roots = nr;
    c.kend(kg);
    // ---- virtual cells: every subdivided leaf cut into bricks, bounded and culled
    // before evaluation
    i64 total_cells = 0, vtiles = 0;
    c.total_bricks = 0;
    c.live_bricks = 0;
    c.foreign_corners = 0;
    c.foreign_slow = 0;
    VRoot* droots = nullptr;
    unsigned char* vcat = nullptr;
    i64* vfirst = nullptr;
    int* bflag = nullptr;
    float* lat_brick = nullptr;
    LiveBrick* live = nullptr;
    unsigned long long* dcount = nullptr;   // foreign corners, window layout overflows, foreign corners evaluated
    i64 fcap = 0;
    LiveIndex lx{};
    VArgs va;
    va.e = ea;
    va.iso = c.iso;
    va.nroots = nr;
    if (nr > 0) {
        kg = c.kbegin("mesh_lists", 0.0);
        droots = dalloc<VRoot>(nr, s);
        bflag = dalloc<int>(M, s);
        // prefix tables: bricks, brick rows, super-bricks, super rows (nr + 1 entries each)
        i64* dpre = dalloc<i64>(4 * ((i64)nr + 1), s);
        k_make_roots<<<grid_for(nr, 256), 256, 0, s>>>(droot_list, nr, D, layout, droots, dpre);
        CK_LAUNCH();
        CK(cudaMemsetAsync(bflag, 0, M * sizeof(int), s));
        k_batch_flags<<<grid_for(nr, 256), 256, 0, s>>>(droots, nr, bflag);
        CK_LAUNCH();
        va.roots = droots;
        va.batch_root_flag = bflag;
        const i64 nbricks = tot[0], nsuper = tot[2], nsrows = tot[3];
        // Leaves of edge 2 (depth D - 1, the last roots) are not bounded but evaluated: the bound proves at most
        // 9 % of them (4 M points at maxDepth 11, 1M torus, an open plane; below 1 % of those of noisy spheres, a
        // filled volume, outliers and random normals) and, with its tables, costs 8 ns a brick where the
        // evaluation takes 2.6.
        const i64 nbound = layout.off[0][D - 1], nrows = layout.off[1][D - 1];
        const int nrbound = layout.first[D - 1];
        i64* dbpre = dpre;
        i64* drpre = dpre + nr + 1;
        i64* dsrpre = dpre + 3 * (nr + 1);
        float* rows = dalloc<float>(nrows * PROW * (D + 1), s);
        int* up = dalloc<int>((i64)nr * BR_LEVELS, s);
        float* anc = dalloc<float>((i64)nrbound * ANC_STRIDE, s);
        const i64 below0 = c.base[std::max(D - BELOW, 0)];
        float2* below = dalloc<float2>(BELOW * (lo - below0), s);
        float2* bsum = dalloc<float2>(D + 1, s);
        BrickIndex bix{dbpre, drpre, nr, rows, up, anc, below, below0, bsum, {}};
        for (int d = 0; d <= D; ++d) {
            bix.dl.first[d] = layout.first[d];
            bix.dl.lg[d] = std::max(D - d - 3, 0);          // bricks per edge 2^(D-d) / min(2^(D-d), 8)
            bix.dl.slg[d] = std::max(D - d - 5, 0);         // super-bricks per edge 2^(D-d) / 32 (D-d >= 6)
            bix.dl.boff[d] = layout.off[0][d];
            bix.dl.soff[d] = layout.off[2][d];
            bix.dl.roff[d] = layout.off[1][d];
            bix.dl.sroff[d] = layout.off[3][d];
        }
        c.kend(kg);
        const int kr = c.kbegin("brick_rows", (double)nrows * PROW * (D + 1) * 4);
        if (nrows > 0) {
            k_brick_rows<<<grid_for(nrows * (D + 1), 128), 128, 0, s>>>(va, bix.dl, nrows, 0, c.d_has_tri, rows);
            CK_LAUNCH();
        }
        float* srows = nullptr;
        if (nsrows > 0) {
            srows = dalloc<float>(nsrows * PROW * (D + 1), s);
            k_brick_rows<<<grid_for(nsrows * (D + 1), 128), 128, 0, s>>>(va, bix.dl, nsrows, 1, c.d_has_tri, srows);
            CK_LAUNCH();
        }
        k_root_up<<<grid_for(nr, 256), 256, 0, s>>>(nd, droots, nr, up);
        CK_LAUNCH();
        if (nrbound > 0) {
            k_brick_xl<<<grid_for((i64)nrbound * 32, 32 * XL_WARPS), 32 * XL_WARPS, 0, s>>>(va, nrbound, c.d_has_tri, up, anc);
            CK_LAUNCH();
        }
        for (int d = D - 1; d >= std::max(D - BELOW, 0); --d) {
            k_x_below<<<grid_for(c.count[d], 256, 1ll << 30), 256, 0, s>>>(nd, c.x, c.base[d], c.base[d + 1], below0, D - d,
                                                                           below);
            CK_LAUNCH();
        }
        k_basis_sums<<<D + 1, 256, 0, s>>>(lb, D, bsum);
        CK_LAUNCH();
        c.kend(kr);
        unsigned char* culled = dalloc<unsigned char>(nbricks, s);
        signed char* bsign = dalloc<signed char>(nbricks, s);
        int* root_of = dalloc<int>(nCoarse, s);
        CK(cudaMemsetAsync(root_of, 0xff, nCoarse * sizeof(int), s));
        k_root_of<<<grid_for(nr, 256), 256, 0, s>>>(droots, nr, root_of);
        CK_LAUNCH();
        // compulsory: every brick row and the leaves' ancestor polynomial (super-bricks: their
        // rows) once, the sign written and read, the culled flag written
        int* nopen = nullptr;
        i64* open = nullptr;
        if (nsuper > 0) {
            nopen = dalloc<int>(1, s);
            open = dalloc<i64>(nsuper, s);
            CK(cudaMemsetAsync(nopen, 0, sizeof(int), s));
            const int ksb = c.kbegin("super_bound", (double)nsrows * PROW * (D + 1) * 4 + (double)nr * ANC_STRIDE * 4 +
                                                        (double)nlarge);
            k_super_bound<<<grid_for(nsuper * 32, BB_BLOCK, (i64)c.sms * 256), BB_BLOCK, 0, s>>>(va, bix, dsrpre, srows,
                                                                                                nsuper, bsign, nopen, open);
            CK_LAUNCH();
            c.kend(ksb);
            if (c.profile) {   // statistics only
                c.super_bricks = nsuper;
                c.super_decided = nsuper - read_scalar(nopen, s);
            }
        }
        const int kb = c.kbegin("brick_bound", (double)nrows * PROW * (D + 1) * 4 +
                                                   (double)nrbound * ANC_STRIDE * 4 + (double)nbound * 3);
        if (nbig > 0) {
            k_brick_bound<<<grid_for(nbig * 32, BB_BLOCK, (i64)c.sms * 256), BB_BLOCK, 0, s>>>(
                va, bix, nopen, open, nlarge, nbig, c.d_has_tri, bsign);
            CK_LAUNCH();
        }
        c.kend(kb);
        const int kb2 = c.kbegin("brick_bound_small", (double)(nbound - nbig) * 3);
        CK(cudaMemsetAsync(bsign + nbound, 0, nbricks - nbound, s));
        if (nbound > nbig) {
            k_brick_bound<<<grid_for((nbound - nbig) * 32, BB_BLOCK, (i64)c.sms * 256), BB_BLOCK, 0, s>>>(
                va, bix, nullptr, nullptr, nbig, nbound, c.d_has_tri, bsign);
            CK_LAUNCH();
        }
        k_brick_cull<<<grid_for(nbricks, 256), 256, 0, s>>>(va, bix, root_of, bsign, nbricks, culled);
        CK_LAUNCH();
        c.kend(kb2);
        dfree(bsign, s);
        dfree(nopen, s);
        dfree(open, s);
        dfree(below, s);
        dfree(bsum, s);
        dfree(srows, s);
        dfree(anc, s);
        kg = c.kbegin("mesh_lists", 0.0);
        int* bf = dalloc<int>(nbricks, s);
        int* bp = dalloc<int>(nbricks + 1, s);
        k_live_flags<<<grid_for(nbricks, 256), 256, 0, s>>>(culled, nbricks, bf);
        CK_LAUNCH();
        exclusive_scan<int, int>(bf, bp, nbricks, bp + nbricks, s);
        dfree(bf, s);
        // live bricks of edge 8, and of edges 8 and 4, and in all: those before the first brick of depths
        // D - 2 and D - 1, and before the end
        int hl[3];
        const i64 at[3] = {layout.off[0][std::max(D - 2, 0)], layout.off[0][D - 1], nbricks};
        for (int q = 0; q < 3; ++q) CK(cudaMemcpyAsync(&hl[q], bp + at[q], sizeof(int), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        const i64 nlive = hl[2];
        c.total_bricks = nbricks;
        c.live_bricks = nlive;
        c.kend(kg);
        if (nlive > 0) {
            kg = c.kbegin("mesh_lists", 0.0);
            live = dalloc<LiveBrick>(nlive, s);
            lx = LiveIndex{live, hl[0], hl[1] - hl[0], hl[2] - hl[1]};
            k_live_bricks<<<grid_for(nbricks, 256), 256, 0, s>>>(va, bix, culled, bp, nbricks, live);
            CK_LAUNCH();
            total_cells = lx.cells();
            lat_brick = dalloc<float>(lx.lattices(), s);
            dcount = dalloc<unsigned long long>(4, s);
            CK(cudaMemsetAsync(dcount, 0, 4 * sizeof(unsigned long long), s));
            // corners owned by another leaf: at most the lower-face corners of the live bricks
            fcap = lx.lattices() - lx.cells();
            ForeignCorner* foreign = dalloc<ForeignCorner>(fcap, s);
            c.kend(kg);
            // compulsory: the corner values written (bricks of edge 8: 729 each)
            const int ke = c.kbegin("brick_eval", (double)lx.n8 * BR_CORNERS * 4);
            if (lx.n8 > 0) {
                k_brick_eval<8, 96><<<grid_for(lx.n8, 1, 1ll << 30), 96, 0, s>>>(
                    va, bix, root_of, lx, 0, lx.n8, lat_brick, dcount, foreign, fcap);
                CK_LAUNCH();
            }
            c.kend(ke);
            const int ks = c.kbegin("brick_eval_small", (double)(125 * lx.n4 + 27 * lx.n2) * 4);
            if (lx.n4 > 0) {
                k_brick_eval<4, 32><<<grid_for(lx.n4, 1, 1ll << 30), 32, 0, s>>>(
                    va, bix, root_of, lx, lx.n8, lx.n4, lat_brick, dcount, foreign, fcap);
                CK_LAUNCH();
            }
            if (lx.n2 > 0) {
                k_edge2_eval<<<grid_for(lx.n2, 3 * E2_WARPS, 1ll << 30), 32 * E2_WARPS, edge2_shared(D), s>>>(
                    va, bix, root_of, lx, lx.n8 + lx.n4, lx.n2, lat_brick, dcount, foreign, fcap);
                CK_LAUNCH();
            }
            c.kend(ks);
            const int kf = c.kbegin("foreign_fill", 0.0);
            const i64 hook = foreign_span_hook();
            if (fcap < FF_LISTED && !hook) {
                k_foreign_fill<false><<<grid_for(fcap, 128, (i64)c.sms * 512), 128, 0, s>>>(va, bix, lx, culled, bp, foreign, 0,
                                                                                           fcap, lat_brick, nullptr, dcount);
                CK_LAUNCH();
            } else {
                const i64 span = std::min(fcap, hook ? hook : FF_SPAN);
                unsigned* list = dalloc<unsigned>(span, s);
                for (i64 at = 0; at < fcap; at += span) {
                    if (at) CK(cudaMemsetAsync(dcount + 3, 0, sizeof(unsigned long long), s));
                    const i64 end = std::min(fcap, at + span);
                    k_foreign_fill<true><<<grid_for(end - at, 256, (i64)c.sms * 128), 256, 0, s>>>(
                        va, bix, lx, culled, bp, foreign, at, end, lat_brick, list, dcount);
                    CK_LAUNCH();
                    k_foreign_eval<<<grid_for(end - at, 64, (i64)c.sms * 256), 64, 0, s>>>(va, bix, lx, foreign, at, list,
                                                                                           lat_brick, dcount);
                    CK_LAUNCH();
                }
                dfree(list, s);
            }
            c.kend(kf);
            dfree(foreign, s);
        }
        dfree(bp, s);
        dfree(culled, s);
        dfree(root_of, s);
        dfree(dpre, s);
        dfree(rows, s);
        dfree(up, s);
        if (total_cells > 0) {
            vcat = dalloc<unsigned char>(total_cells, s);
            vtiles = (total_cells + CELL_TILE - 1) / CELL_TILE;
            int* vtri = dalloc<int>(vtiles, s);
            vfirst = dalloc<i64>(vtiles + 1, s);
            const int kc2 = c.kbegin("virtual_cells", (double)total_cells * (8 * 4 + 5));
            k_virtual_cells<<<(unsigned)vtiles, CELL_BLOCK, 0, s>>>(lx, lat_brick, total_cells, vcat, vtri);
            CK_LAUNCH();
            exclusive_scan<int, i64>(vtri, vfirst, vtiles, vfirst + vtiles, s);
            dfree(vtri, s);
            c.kend(kc2);
        }
    }
    // the triangles of both kinds, and the checks and counts of the evaluation, in one read
    i64 ntri_real = 0, ntri_virt = 0;
    unsigned long long hc[3] = {0, 0, 0};
    CK(cudaMemcpyAsync(&ntri_real, rfirst + rtiles, sizeof(i64), cudaMemcpyDeviceToHost, s));
    if (vfirst) CK(cudaMemcpyAsync(&ntri_virt, vfirst + vtiles, sizeof(i64), cudaMemcpyDeviceToHost, s));
    if (dcount) CK(cudaMemcpyAsync(hc, dcount, sizeof hc, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    dfree(dcount, s);
    if (hc[1]) {
        set_last_error("brick window layout overflow in %llu bricks", hc[1]);
        throw Error{PRGPU_ERR_LIMIT, {0}};
    }
    if ((i64)hc[0] > fcap) {
        set_last_error("foreign corner list overflow (%llu > %lld)", hc[0], (long long)fcap);
        throw Error{PRGPU_ERR_LIMIT, {0}};
    }
    c.foreign_corners = (i64)hc[0];
    c.foreign_slow = (i64)hc[2];
    c.virtual_cells = total_cells;
    // ---- emission, sort, vertex ids
    const i64 ntri_all = ntri_real + ntri_virt;
    const i64 nem = 3 * ntri_all;
    if (nem > 0x7fffffffLL) {
        set_last_error("mesh of %lld triangles exceeds 32-bit indexing", (long long)ntri_all);
        throw Error{PRGPU_ERR_LIMIT, {0}};
    }
    int local_bits = 0;
    {
        const double lat_edges = 3.0 * std::pow((double)((1 << D) + 1), 3.0);
        while ((double)(1ull << local_bits) < lat_edges) ++local_bits;
    }
    int batch_bits = 0;
    while (!c.params.weld && (1 << batch_bits) < nbatches) ++batch_bits;
    c.mesh_v.clear();
    c.mesh_f.clear();
    c.batch_tri.assign(1, ntri_real);
    c.batch_tri.push_back(ntri_virt);
    if (nem > 0) {
        EmitArgs em;
        em.D = D;
        em.local_bits = local_bits;
        em.weld = c.params.weld ? 1 : 0;
        em.tri_offset = 0;
        em.keys = dalloc<u64>(nem, s);
        em.pos = dalloc<float>(3 * nem, s);
        const int kem = c.kbegin("emit", (double)nem * (8 + 12));
        if (ntri_real > 0) {
            k_emit_real<<<(unsigned)rtiles, CELL_BLOCK, 0, s>>>(nd, em, lo, nD, cat, rfirst, cell_v);
            CK_LAUNCH();
        }
        if (ntri_virt > 0) {
            EmitArgs ev = em;
            ev.tri_offset = ntri_real;
            k_emit_virtual<<<(unsigned)vtiles, CELL_BLOCK, 0, s>>>(va, ev, lx, lat_brick, total_cells, vcat, vfirst);
            CK_LAUNCH();
        }
        c.kend(kem);
        u64* ktmp = dalloc<u64>(nem, s);
        uint32_t *slot = dalloc<uint32_t>(nem, s), *stmp = dalloc<uint32_t>(nem, s);
        const int ks = c.kbegin("edge_sort", (double)nem * 12 * 2);
        radix_sort_pairs(em.keys, slot, ktmp, stmp, nem, local_bits + batch_bits, s);
        c.kend(ks);
        dfree(ktmp, s);
        dfree(stmp, s);
        const int kvi = c.kbegin("vertex_ids", (double)nem * (8 * 2 + 4 + 4 + 12));
        int* hf = dalloc<int>(nem, s);
        int* hp = dalloc<int>(nem + 1, s);
        k_key_heads<<<grid_for(nem, 256), 256, 0, s>>>(em.keys, nem, hf);
        CK_LAUNCH();
        exclusive_scan<int, int>(hf, hp, nem, hp + nem, s);
        const i64 nvert = read_scalar(hp + nem, s);
        int32_t* tri_vid = dalloc<int32_t>(nem, s);
        float* vpos = dalloc<float>(3 * std::max<i64>(nvert, 1), s);
        k_vertex_ids<<<grid_for(nem, 256), 256, 0, s>>>(em.keys, slot, nem, hp, em.pos, c.scale,
                                                        make_float3(c.center[0], c.center[1], c.center[2]),
                                                        tri_vid, vpos);
        CK_LAUNCH();
        c.kend(kvi);
        const int kd = c.kbegin("mesh_d2h", (double)(3 * nvert + nem) * 4);
        c.mesh_v.resize(3 * nvert);
        c.mesh_f.resize(nem);
        CK(cudaMemcpyAsync(c.mesh_v.data(), vpos, 3 * nvert * sizeof(float), cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(c.mesh_f.data(), tri_vid, nem * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
        c.kend(kd);
        CK(cudaStreamSynchronize(s));
        dfree(hf, s); dfree(hp, s); dfree(tri_vid, s); dfree(vpos, s);
        dfree(em.keys, s); dfree(slot, s); dfree(em.pos, s);
    }
    dfree(rtri, s);
    dfree(rfirst, s);
    dfree(droots, s); dfree(droot_list, s);
    dfree(vcat, s); dfree(vfirst, s); dfree(bflag, s);
    dfree(lat_brick, s); dfree(live, s);
    dfree(cell_v, s);
    dfree(x27, s);
    dfree(lb, s);
    dfree(cat, s);
}

}  // namespace prgpu
