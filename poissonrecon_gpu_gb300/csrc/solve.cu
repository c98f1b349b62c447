// Per-depth Laplacian solve.  Replaces LaplacianIteration (main.cu:1223-1332)
// and solverCG_DeviceToDevice / gpuConjugateGradient (CG_CUDA.cuh:186-509).
//
// The reference assembles a CSR matrix per depth and runs one cooperative CG
// kernel per depth, one depth after the other.  Here the matrix is never
// stored: same-depth inner products are translation invariant, so row i of L_d
// is the depth's 27 stencil coefficients applied through the node's neighbour
// table (the reference's |L_ij| <= 1e-6 drop rule is applied to the stencil).
// The depths are independent systems (each starts from x0 = 0 and never sees
// the others), so ONE persistent cooperative launch solves all of them at
// once: the co-resident blocks are partitioned between the depths in
// proportion to their row counts, and each partition runs its own CG with its
// own grid sums.  Their waits have an iteration limit; on expiry the
// kernel records PRGPU_ERR_TIMEOUT and returns.
//
// Matrix-vector product by sibling groups: the 8 children of a node are
// contiguous, and their 27-neighbourhoods together form the 4x4x4 block of
// cells around them -- the children of the parent's 27 neighbours.  So the
// product reads, per group, the 27 first-child indices of the parent's
// neighbours (a table built once per solve, 13.5 bytes per row instead of the
// 108-byte neighbour rows) and the 64 values of r in the block, staged in
// shared memory.  A missing neighbour reads 0, and adding a zero product
// leaves the sum unchanged, so the product is the same as with the neighbour
// table.  The product is s = A r; the direction's product follows as
// q = A p = s + beta q_prev (p = r + beta p_prev), so each cell is gathered once
// per iteration (one vector) rather than forming p at every group that reads it.
#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include "cg_common.cuh"
#include "context.h"
#include "prims.cuh"

namespace prgpu {


struct CgArgs {
    int mode;               // prgpu_solve_mode
    float tol2;             // reference mode: float(tol)*float(tol)
    double rel2;            // relative mode: tol^2
    int max_iter;
    i64 M;
    const int* neigh;       // 27 x M
    const int* gnr;         // GN_ROW per sibling group: first child of each neighbour of its parent, or -1
    const float* b;
    float* x;
    float* r;
    float* p;               // search direction
    float* q;               // A p
    PartState* state;
    u64* slots;             // grid_sum's slots: one per block, one per depth (results), one never written
    int nslots;
    int* err;
    long long spin_limit;   // bounded waits (WaitLimits)
    int extra;
    int refine;             // relative mode: FP64 true-residual check and refinement
};

// per sibling group: first child of each of the parent's 27 neighbours (-1: none or a leaf)
__global__ void k_group_table(NodeArrays nd, i64 ngroups, int* __restrict__ gn) {
    const i64 M = nd.M;
    for (i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x; e < ngroups * 27; e += (i64)gridDim.x * blockDim.x) {
        const i64 g = e % ngroups;
        const int jp = (int)(e / ngroups);
        const int P = nd.parent[1 + 8 * g];
        const int pn = nd.neigh[(i64)jp * M + P];
        gn[e] = (pn == -1) ? -1 : nd.child0[pn];
    }
}

// the group table row by row (GN_ROW per group; the pad entry -1)
__global__ void k_group_rows(const int* __restrict__ gn, i64 ngroups, int* __restrict__ rows) {
    for (i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x; e < ngroups * GN_ROW; e += (i64)gridDim.x * blockDim.x) {
        const i64 g = e / GN_ROW;
        const int jp = (int)(e % GN_ROW);
        rows[e] = (jp < 27) ? gn[(i64)jp * ngroups + g] : -1;
    }
}

constexpr int CG_TILE_GROUPS = CG_BLOCK / 8;   // sibling groups per tile, one thread per row
constexpr int CG_WARP_TILES = 2;               // tiles of 4 groups a warp stages at once
constexpr int CG_BLOCK_ROWS = CG_BLOCK * CG_WARP_TILES;   // rows of a block's warps at once, consecutive

// 5 blocks per SM (48 registers): the partitions' warps wait on gathers and grid reductions, and
// 40 warps per SM hide more of that latency than 32 (measured: 2.41 -> 1.90 ms on the 1M-point
// torus at maxDepth 10; 6 blocks spill more and are slower again)
__global__ void __launch_bounds__(CG_BLOCK, 5) k_cg_all(CgArgs a, const CgDepth* __restrict__ deps,
                                                     const int* __restrict__ block_depth) {
    __shared__ float sp[(CG_BLOCK / 32) * CG_WARP_TILES * CG_TILE_WORDS];
    __shared__ int sgn[(CG_BLOCK / 32) * CG_WARP_TILES * 4 * GN_ROW];
    __shared__ float sst[27];
    __shared__ GridSumShared<1> gsm;
    const int d = block_depth[blockIdx.x];
    const CgDepth& dp = deps[d];
    if (threadIdx.x < 27) sst[threadIdx.x] = dp.st[threadIdx.x];
    const float cls[4] = {dp.cls[0], dp.cls[1], dp.cls[2], dp.cls[3]};
    __syncthreads();
    PartState* ps = &a.state[d];
    const int rank = blockIdx.x - dp.first_block;
    const i64 stride = (i64)dp.nblocks * blockDim.x;
    const i64 start = (i64)rank * blockDim.x + threadIdx.x;
    unsigned epoch = 0;
    const GridSum gs{a.slots, a.nslots, dp.first_block, dp.nblocks, rank, (int)gridDim.x + d, a.err, a.spin_limit, a.extra};

    // reduce a per-thread value over the partition; every thread gets the sum
    auto preduce = [&](auto v, bool data, bool& ok) -> double {
        const decltype(v) s[1] = {v};
        double t[1] = {0.0};
        ok = grid_sum(gs, ++epoch, data, s, gsm, t);
        return t[0];
    };

    // x = 0, r = b  (the host-side initialisation of CG_CUDA.cuh:435-439)
    FSum loc;
    for (i64 t = start; t < dp.n; t += stride) {
        const i64 i = dp.lo + t;
        const float bi = a.b[i];
        a.x[i] = 0.f;
        a.r[i] = bi;
        loc.add(bi * bi);
    }
    bool ok = true;
    const double bb = preduce(loc, true, ok);   // ||b||^2 in double (relative mode)
    float r1 = (float)bb;
    float r0 = 0.f;
    int k = 1;
    int refines = 0;
    double rr_true = -1.0;
    bool restart = true;
    // The product gathers r only: s = A r, then q = A p = s + beta q and p = r + beta p
    // are formed row by row by the row's own thread (in place: no other thread reads a
    // row's p or q during the pass)
    while (ok) {
        const bool go = (a.mode == PRGPU_SOLVE_REFERENCE) ? (r1 > a.tol2) : ((double)r1 > a.rel2 * bb);
        if (!go || k > a.max_iter) {
            if (!a.refine || a.mode != PRGPU_SOLVE_RELATIVE || k > a.max_iter) break;
            // the recurrence says converged: recompute r = b - A x with FP64 accumulation (x was
            // written after its r.r was published, so its rows are made visible first)
            preduce(0.0, true, ok);
            if (!ok) break;
            double tsum = 0.0;
            for (i64 t = start; t < dp.n; t += stride) {
                const i64 i = dp.lo + t;
                double acc = (double)a.b[i];
#pragma unroll
                for (int j = 0; j < 27; ++j) {
                    const int nb = a.neigh[(i64)j * a.M + i];
                    if (nb != -1) acc = fma(-(double)sst[j], (double)a.x[nb], acc);
                }
                a.r[i] = (float)acc;
                tsum = fma(acc, acc, tsum);
            }
            rr_true = preduce(tsum, true, ok);
            if (!ok || rr_true <= a.rel2 * bb || refines >= 2) break;
            // restart CG from the current x on the true residual
            ++refines;
            r1 = (float)rr_true;
            restart = true;
            continue;
        }
        const bool first = restart;
        restart = false;
        const float beta = first ? 0.f : r1 / r0;
        // own row i with s_i = (A r)_i: p_i = r_i + beta p_i, q_i = s_i + beta q_i; partial p.q
        auto own_row = [&](i64 i, float ri, float si) {
            float pi = ri, qi = si;
            if (!first) {
                pi = fmaf(beta, a.p[i], ri);
                qi = fmaf(beta, a.q[i], si);
            }
            a.p[i] = pi;
            a.q[i] = qi;
            loc.add(pi * qi);
        };
        loc = FSum();
        if (d == 0) {   // one row, one block
            for (i64 t = start; t < dp.n; t += stride) {
                const i64 i = dp.lo + t;
                float o = 0.f;
#pragma unroll
                for (int j = 0; j < 27; ++j) {
                    const int nb = a.neigh[(i64)j * a.M + i];
                    if (nb != -1 && sst[j] != 0.f) o = fmaf(sst[j], a.r[nb], o);
                }
                own_row(i, a.r[i], o);
            }
        } else {
            // one warp per CG_WARP_TILES tiles of 4 groups (32 rows each); warps run independently.
            // The tiles' group-table rows are one contiguous run, read coalesced into shared
            // memory; then every lane has 2 * CG_WARP_TILES * 8 independent gathers in flight.
            const i64 gfirst = (dp.lo - 1) >> 3, ng = dp.n >> 3;
            const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
            const int ch = lane & 7, gl = lane >> 3;
            const int sx = (ch >> 2) & 1, sy = (ch >> 1) & 1, sz = ch & 1;
            float* wsp = sp + wib * (CG_WARP_TILES * CG_TILE_WORDS);
            int* wgn = sgn + wib * (CG_WARP_TILES * 4 * GN_ROW);
            const i64 wstride = (i64)dp.nblocks * (CG_BLOCK / 32) * CG_WARP_TILES;
            for (i64 tile = ((i64)rank * (CG_BLOCK / 32) + wib) * CG_WARP_TILES; tile * 4 < ng; tile += wstride) {
                __syncwarp();
                {
                    // (read once per iteration and marked to leave L2 first, so that r, p and q stay: 1.82
                    // -> 1.68 ms on the 1M torus, whose vectors and table together exceed L2)
                    const i64 row0 = (gfirst + tile * 4) * GN_ROW;
                    const i64 nvalid = min((i64)CG_WARP_TILES * 4, ng - tile * 4) * GN_ROW;
#pragma unroll
                    for (int k = 0; k < (CG_WARP_TILES * 4 * GN_ROW + 31) / 32; ++k) {
                        const int idx = lane + 32 * k;
                        if (idx < CG_WARP_TILES * 4 * GN_ROW) wgn[idx] = (idx < nvalid) ? __ldcs(a.gnr + row0 + idx) : -1;
                    }
                }
                __syncwarp();
                // the 4x4x4 block of each group: cell (bx,by,bz) is child ((bx+1)&1, ...) of the
                // parent's neighbour ((bx+1)>>1, ...) in 0..2 per axis
                int cn[CG_WARP_TILES * 8];
#pragma unroll
                for (int m = 0; m < CG_WARP_TILES * 8; ++m) {
                    const int e = lane + 32 * m;
                    const int cell = e & 63, bx = cell >> 4, by = (cell >> 2) & 3, bz = cell & 3;
                    const int jp = 9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1) + ((bz + 1) >> 1);
                    cn[m] = wgn[(e >> 6) * GN_ROW + jp];
                }
#pragma unroll
                for (int m = 0; m < CG_WARP_TILES * 8; ++m) {
                    const int e = lane + 32 * m;
                    const int cell = e & 63, bx = cell >> 4, by = (cell >> 2) & 3, bz = cell & 3;
                    wsp[(e >> 8) * CG_TILE_WORDS + cg_block_base((e >> 6) & 3) + cell] = (cn[m] != -1)
                                 ? a.r[cn[m] + ((((bx + 1) & 1) << 2) | (((by + 1) & 1) << 1) | ((bz + 1) & 1))]
                                 : 0.f;
                }
                __syncwarp();
#pragma unroll
                for (int tt = 0; tt < CG_WARP_TILES; ++tt) {
                    const i64 g = (tile + tt) * 4 + gl;
                    if (g < ng) {
                        const float* blk = wsp + tt * CG_TILE_WORDS + cg_block_base(gl);
                        float o = 0.f;
                        if (dp.sym) {
#pragma unroll
                            for (int j = 0; j < 27; ++j)
                                o = fmaf(cls[stencil_class(j)],
                                         blk[(sx + j / 9) * 16 + (sy + (j / 3) % 3) * 4 + (sz + j % 3)], o);
                        } else {
#pragma unroll
                            for (int j = 0; j < 27; ++j)
                                o = fmaf(sst[j], blk[(sx + j / 9) * 16 + (sy + (j / 3) % 3) * 4 + (sz + j % 3)], o);
                        }
                        own_row(dp.lo + 8 * g + ch, blk[(sx + 1) * 16 + (sy + 1) * 4 + (sz + 1)], o);
                    }
                }
            }
        }
        // p.q carries no data: the update takes the rows whose p and q this block's product wrote
        // (CG_BLOCK_ROWS at a time), and r only after every block has read it
        const double pq = preduce(loc, false, ok);
        if (!ok) break;
        const float al = (float)((double)r1 / pq);
        const float nal = -al;
        loc = FSum();
        const i64 ustride = (i64)dp.nblocks * CG_BLOCK_ROWS;
        // four rows per thread per step, loads first (independent requests in flight)
        auto row4 = [&](i64 t, int u) { return t + (u & 1) * CG_BLOCK + (u >> 1) * ustride; };
        for (i64 t = (i64)rank * CG_BLOCK_ROWS + threadIdx.x; t < dp.n; t += 2 * ustride) {
            float qv[4], rv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool in = row4(t, u) < dp.n;
                const i64 i = dp.lo + row4(t, u);
                qv[u] = in ? a.q[i] : 0.f;
                rv[u] = in ? a.r[i] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (row4(t, u) < dp.n) {
                    const float ri = fmaf(nal, qv[u], rv[u]);
                    a.r[dp.lo + row4(t, u)] = ri;
                    loc.add(ri * ri);
                }
        }
        {
            // x (read by nobody else) while r.r travels
            const FSum s[1] = {loc};
            grid_publish(gs, ++epoch, true, s, gsm);
            for (i64 t = (i64)rank * CG_BLOCK_ROWS + threadIdx.x; t < dp.n; t += 2 * ustride) {
                float pv[4], xv[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const bool in = row4(t, u) < dp.n;
                    const i64 i = dp.lo + row4(t, u);
                    pv[u] = in ? a.p[i] : 0.f;
                    xv[u] = in ? a.x[i] : 0.f;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (row4(t, u) < dp.n) a.x[dp.lo + row4(t, u)] = fmaf(al, pv[u], xv[u]);
            }
            double rr[1] = {0.0};
            ok = grid_collect(gs, epoch, true, gsm, rr);
            r0 = r1;
            r1 = (float)rr[0];
        }
        ++k;
    }
    if (rank == 0 && threadIdx.x == 0) {
        ps->iters = k - 1;
        ps->rr = r1;
        ps->bb = bb;
        ps->rr_true = rr_true;
        ps->refines = refines;
        ps->status = ok ? 0 : PRGPU_ERR_TIMEOUT;
    }
}

// the group table row by row, built once per octree
void ensure_group_rows(Ctx& c) {
    if (c.gn_rows) return;
    ensure_group_table(c);
    const i64 ngroups = (c.nodes.M - 1) / 8;
    c.gn_rows = dalloc<int>(std::max<i64>(ngroups * GN_ROW, 1), c.stream);
    if (ngroups > 0) {
        k_group_rows<<<grid_for(ngroups * GN_ROW, 256), 256, 0, c.stream>>>(c.gn, ngroups, c.gn_rows);
        CK_LAUNCH();
    }
}

// the sibling-group table of the current octree, built once
void ensure_group_table(Ctx& c) {
    if (c.gn) return;
    const i64 ngroups = (c.nodes.M - 1) / 8;
    c.gn = dalloc<int>(std::max<i64>(ngroups * 27, 1), c.stream);
    if (ngroups > 0) {
        k_group_table<<<grid_for(ngroups * 27, 256), 256, 0, c.stream>>>(c.nodes, ngroups, c.gn);
        CK_LAUNCH();
    }
}

// ---------------------------------------------------------------------------
// Cascadic solve (params.cascadic; not the reference's): the depths are solved
// coarse to fine and depth d's right-hand side first loses the coarser depths'
// solution,
//   b'_i = b_i - sum_{e < d} sum_{j in N27(ancestor_e(i))} <grad B_i, grad B_j> x_j,
// the coarser nodes being the 27 neighbours of i's ancestor at each depth e (the
// truncation the reference's divergence uses).  The 3-D inner product has the
// same-depth stencil's form, dd_x t_y t_z + t_x dd_y t_z + t_x t_y dd_z, over
// the cross-depth 1-D tables (k_cascade_tables), so the sum over the 3x3x3
// neighbours factors axis by axis (z, then y, then x).  In double, with explicit fma, in this order:
//   zt[ox][oy] = fma(t_z0, X[ox][oy][0], fma(t_z1, X[ox][oy][1], t_z2 * X[ox][oy][2])), zd likewise
//   ytt = sum_oy t_y zt, ydt = sum_oy dd_y zt, ytd = sum_oy t_y zd   (the same nesting)
//   acc = fma(dd_x[ox], ytt, fma(t_x[ox], ydt + ytd, acc))          for ox = 0, 1, 2
// for e = 0.., X = x of the neighbour (0 where it is missing), read from a double
// copy of x.
// ---------------------------------------------------------------------------
constexpr int CASCADE_MAX_DEPTH = 16;
// prgpu_create accepts maxDepth 2..15, so the per-ancestor arrays below always fit
static_assert(PRGPU_MAX_DEPTH < CASCADE_MAX_DEPTH, "the cascadic arrays need a slot per depth below maxDepth");

struct CascadeArgs {
    int d, D;
    i64 lo, n, M;
    const u64* key;
    const int* parent;
    const int* neigh;       // 27 x M
    const double2* tab;
    i64 off[CASCADE_MAX_DEPTH];   // start of the (d, e) table, e < d
    const double* xd;       // x in double, rows of the depths < d
    const float* b;
    float* rhs;
};

__device__ __forceinline__ double dot3(double a0, double a1, double a2, double x0, double x1, double x2) {
    return fma(a0, x0, fma(a1, x1, a2 * x2));
}

// Two lanes per sibling group, one per z half: the 8 siblings share every ancestor, so the z sums are
// formed once per (group, z), the y sums once per (group, z, y), and only the x sums per node: 36 FP64
// operations per node and ancestor instead of 90.  Bound by the FP64 pipe and, at the coarse depths, by
// the chain through the ancestors.  All nine depths of a 200k torus at depth 9: 1.50 -> 0.76 ms.
constexpr int CASCADE_BLOCK = 64;
__global__ void __launch_bounds__(CASCADE_BLOCK) k_cascade_rhs(CascadeArgs a) {
    const int d = a.d, sh0 = 3 * (a.D - d);
    for (i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x; t < a.n / 4; t += (i64)gridDim.x * blockDim.x) {
        const i64 i = a.lo + 8 * (t >> 1);   // the group's first node, at the low end of each axis
        const int zb = (int)(t & 1);
        const u64 key = a.key[i] >> sh0;
        int p[3] = {0, 0, 0};
        for (int l = d - 1; l >= 0; --l) {
            p[0] = (p[0] << 1) | (int)((key >> (3 * l + 2)) & 1);
            p[1] = (p[1] << 1) | (int)((key >> (3 * l + 1)) & 1);
            p[2] = (p[2] << 1) | (int)((key >> (3 * l)) & 1);
        }
        int anc[CASCADE_MAX_DEPTH];
        int q = (int)i;
        for (int e = d - 1; e >= 0; --e) {
            q = a.parent[q];
            anc[e] = q;
        }
        double acc[2][2] = {};   // [x][y]
        for (int e = 0; e < d; ++e) {
            const int k = d - e;
            const int mask = (1 << k) - 1;
            const double2* T = a.tab + a.off[e];
            const int px = p[0] & mask, py = p[1] & mask, pz = (p[2] & mask) + zb;
            const int A = anc[e];
            double tz[3], dz[3];
#pragma unroll
            for (int o = 0; o < 3; ++o) {
                const double2 v = T[((i64)o << k) + pz];
                tz[o] = v.x;
                dz[o] = v.y;
            }
            double2 ty[2][3];
#pragma unroll
            for (int o = 0; o < 3; ++o) {
                ty[0][o] = T[((i64)o << k) + py];
                ty[1][o] = T[((i64)o << k) + py + 1];
            }
#pragma unroll
            for (int ox = 0; ox < 3; ++ox) {
                double zt[3], zd[3];
#pragma unroll
                for (int oy = 0; oy < 3; ++oy) {
                    double X[3];
#pragma unroll
                    for (int oz = 0; oz < 3; ++oz) {
                        const int nb = a.neigh[(i64)(9 * ox + 3 * oy + oz) * a.M + A];
                        X[oz] = nb >= 0 ? a.xd[nb] : 0.0;
                    }
                    zt[oy] = dot3(tz[0], tz[1], tz[2], X[0], X[1], X[2]);
                    zd[oy] = dot3(dz[0], dz[1], dz[2], X[0], X[1], X[2]);
                }
                const double2 tx[2] = {T[((i64)ox << k) + px], T[((i64)ox << k) + px + 1]};
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const double ytt = dot3(ty[y][0].x, ty[y][1].x, ty[y][2].x, zt[0], zt[1], zt[2]);
                    const double ydt = dot3(ty[y][0].y, ty[y][1].y, ty[y][2].y, zt[0], zt[1], zt[2]);
                    const double ytd = dot3(ty[y][0].x, ty[y][1].x, ty[y][2].x, zd[0], zd[1], zd[2]);
#pragma unroll
                    for (int x = 0; x < 2; ++x) acc[x][y] = fma(tx[x].y, ytt, fma(tx[x].x, ydt + ytd, acc[x][y]));
                }
            }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                const i64 o = i + 4 * x + 2 * y + zb;
                a.rhs[o] = (float)((double)a.b[o] - acc[x][y]);
            }
    }
}

__global__ void k_rows_to_double(const float* __restrict__ x, i64 n, double* __restrict__ xd) {
    for (i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (i64)gridDim.x * blockDim.x)
        xd[t] = (double)x[t];
}

// depth d's rows of rhs: the divergence less the coarser depths' current solution
void cascade_rhs(Ctx& c, int d, float* rhs) {
    cudaStream_t s = c.stream;
    const i64 lo = c.base[d], n = c.count[d];
    if (n == 0) return;
    if (d == 0) {
        CK(cudaMemcpyAsync(rhs + lo, c.divergence + lo, n * sizeof(float), cudaMemcpyDeviceToDevice, s));
        return;
    }
    if (c.D >= CASCADE_MAX_DEPTH) {
        set_last_error("cascadic solve supports maxDepth < %d", CASCADE_MAX_DEPTH);
        throw Error{PRGPU_ERR_LIMIT, {0}};
    }
    ensure_cascade_tables(c);
    // the coarser rows of x in double (rows base[0] .. base[d])
    const i64 nc = c.base[d];
    double* xd = dalloc<double>(nc, s);
    k_rows_to_double<<<grid_for(nc, 256), 256, 0, s>>>(c.x, nc, xd);
    CK_LAUNCH();
    CascadeArgs a;
    a.d = d;
    a.D = c.D;
    a.lo = lo;
    a.n = n;
    a.M = c.nodes.M;
    a.key = c.nodes.key;
    a.parent = c.nodes.parent;
    a.neigh = c.nodes.neigh;
    a.tab = c.cascade_tab;
    for (int e = 0; e < CASCADE_MAX_DEPTH; ++e) a.off[e] = e < d ? c.cascade_off[(size_t)d * (c.D + 1) + e] : 0;
    a.xd = xd;
    a.b = c.divergence;
    a.rhs = rhs;
    // compulsory: key, parent, b and rhs of each node; the coarser depths' neighbour rows and x
    // (double)
    double bytes = (double)n * 20;
    for (int e = 0; e < d; ++e) bytes += (double)c.count[e] * (27 * 4 + 8);
    const int kt = c.kbegin("cascade_rhs", bytes);
    k_cascade_rhs<<<grid_for(n / 4, CASCADE_BLOCK, 1ll << 30), CASCADE_BLOCK, 0, s>>>(a);
    CK_LAUNCH();
    c.kend(kt);
    dfree(xd, s);
}

void stage_solve(Ctx& c) {
    if (c.params.learned) {
        stage_solve_learned(c);
        return;
    }
    if (!c.params.cascadic) {
        stage_solve_depths(c, 0, c.D, c.params.solve_mode);
        return;
    }
    cudaStream_t s = c.stream;
    const i64 M = c.nodes.M;
    if (!c.x || c.x_rows != M) {
        dfree(c.x, s);
        c.x = dalloc<float>(M, s);
        c.x_rows = M;
        CK(cudaMemsetAsync(c.x, 0, M * sizeof(float), s));
    }
    float* rhs = dalloc<float>(M, s);
    for (int d = 0; d <= c.D; ++d) {
        cascade_rhs(c, d, rhs);
        stage_solve_depths(c, d, d, c.params.solve_mode, rhs);
    }
    dfree(rhs, s);
}

// co-resident blocks split between the depths d0..d1: one block for a depth of at most
// 4*256 rows, the rest in proportion to the rows; the depths outside d0..d1 get none
void partition_depths(const Ctx& c, int d0, int d1, int G, std::vector<CgDepth>& deps, std::vector<int>& block_depth) {
    const int D = c.D;
    deps.assign(D + 1, CgDepth());
    std::vector<int> nb(D + 1, 0);
    i64 big_rows = 0;
    const i64 small_rows = 4 * CG_BLOCK;
    int fixed = 0;
    for (int d = d0; d <= d1; ++d) {
        nb[d] = 1;
        if (c.count[d] <= small_rows) ++fixed;
        else big_rows += c.count[d];
    }
    int avail = std::max(0, G - fixed);
    for (int d = d0; d <= d1; ++d) {
        if (c.count[d] > small_rows) {
            i64 want = (i64)((double)avail * (double)c.count[d] / (double)std::max<i64>(big_rows, 1));
            i64 cap = (c.count[d] + CG_BLOCK - 1) / CG_BLOCK;
            nb[d] = (int)std::max<i64>(1, std::min(want, cap));
        }
    }
    int total = 0;
    for (int d = 0; d <= D; ++d) total += nb[d];
    while (total > G) {   // trim the largest partitions
        int dm = (int)(std::max_element(nb.begin(), nb.end()) - nb.begin());
        if (nb[dm] <= 1) break;
        --nb[dm];
        --total;
    }
    if (total > G) {
        set_last_error("solver needs %d co-resident blocks, device offers %d", total, G);
        throw Error{PRGPU_ERR_LIMIT, {0}};
    }
    block_depth.clear();
    for (int d = 0; d <= D; ++d) {
        deps[d].lo = c.base[d];
        deps[d].n = c.count[d];
        deps[d].first_block = (int)block_depth.size();
        deps[d].nblocks = nb[d];
        for (int j = 0; j < 27; ++j) deps[d].st[j] = c.stencil[27 * d + j];
        deps[d].sym = 1;
        for (int j = 0; j < 27; ++j) {
            const int k = stencil_class(j);
            const float rep = c.stencil[27 * d + (k == 0 ? 13 : k == 1 ? 4 : k == 2 ? 1 : 0)];
            if (c.stencil[27 * d + j] != rep) deps[d].sym = 0;
            deps[d].cls[k] = rep;
        }
        for (int k = 0; k < nb[d]; ++k) block_depth.push_back(d);
    }
}

// depths d0..d1 with the given mode (right-hand side: rhs, or the divergence);
// the other depths' rows of x are left as they are
void stage_solve_depths(Ctx& c, int d0, int d1, int mode, const float* rhs) {
    cudaStream_t s = c.stream;
    const int D = c.D;
    const i64 M = c.nodes.M;
    if (d0 == 0 && d1 == D) {   // every row is written
        dfree(c.x, s);
        c.x = dalloc<float>(M, s);
        c.x_rows = M;
    } else if (!c.x || c.x_rows != M) {   // the other depths start at 0
        dfree(c.x, s);
        c.x = dalloc<float>(M, s);
        c.x_rows = M;
        CK(cudaMemsetAsync(c.x, 0, M * sizeof(float), s));
    }
    float* r = dalloc<float>(M, s);
    float* p = dalloc<float>(M, s);
    float* q = dalloc<float>(M, s);
    // sibling-group table for the matrix-vector products
    ensure_group_rows(c);
    // co-resident capacity
    int dev = c.device, sms = 0, per_sm = 0;
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cg_all, CG_BLOCK, 0));
    if (per_sm < 1) per_sm = 1;
    const int G = sms * per_sm;
    c.solver_blocks = G;
    std::vector<CgDepth> deps;
    std::vector<int> block_depth;
    partition_depths(c, d0, d1, G, deps, block_depth);
    CgDepth* ddeps = dalloc<CgDepth>(D + 1, s);
    int* dbd = dalloc<int>((i64)block_depth.size(), s);
    PartState* st = dalloc<PartState>(D + 1, s);
    const int nslots = (int)block_depth.size() + D + 2;
    u64* slots = dalloc<u64>(grid_sum_words(nslots, 1), s);
    CK(cudaMemsetAsync(slots, 0, grid_sum_words(nslots, 1) * sizeof(u64), s));
    int* err = dalloc<int>(1, s);
    CK(cudaMemcpyAsync(ddeps, deps.data(), (D + 1) * sizeof(CgDepth), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(dbd, block_depth.data(), block_depth.size() * sizeof(int), cudaMemcpyHostToDevice, s));
    CK(cudaMemsetAsync(st, 0, (D + 1) * sizeof(PartState), s));
    CK(cudaMemsetAsync(err, 0, sizeof(int), s));
    CgArgs a;
    a.mode = mode;
    const float tolf = (float)c.params.cg_tol;
    a.tol2 = tolf * tolf;
    a.rel2 = c.params.cg_tol * c.params.cg_tol;
    a.max_iter = c.params.cg_max_iter;
    a.M = M;
    a.neigh = c.nodes.neigh;
    a.gnr = c.gn_rows;
    a.b = rhs ? rhs : c.divergence;
    a.x = c.x;
    a.r = r;
    a.p = p;
    a.q = q;
    a.state = st;
    a.slots = slots;
    a.nslots = nslots;
    a.err = err;
    const WaitLimits wl = wait_limits();
    a.spin_limit = wl.spin_limit;
    a.extra = wl.extra;
    a.refine = c.params.refine;
    void* kargs[] = {(void*)&a, (void*)&ddeps, (void*)&dbd};
    const int kt = c.kbegin("cg", 0.0);
    CK(cudaLaunchCooperativeKernel((void*)k_cg_all, dim3((unsigned)block_depth.size()), dim3(CG_BLOCK), kargs, 0, s));
    ++g_kernel_launches;
    c.kend(kt);
    std::vector<PartState> hs(D + 1);
    int herr = 0;
    CK(cudaMemcpyAsync(hs.data(), st, (D + 1) * sizeof(PartState), cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if ((int)c.cg_iters.size() != D + 1 || (d0 == 0 && d1 == D)) {
        c.cg_iters.assign(D + 1, 0);
        c.cg_rr.assign(D + 1, 0.f);
    }
    c.cg_fallback.assign(D + 1, -1);
    c.cg_true_rel.resize(D + 1, 0.0);
    c.cg_fp64_rel.resize(D + 1, -1.0);
    c.cg_refines.resize(D + 1, 0);
    for (int d = d0; d <= d1; ++d) {
        c.cg_iters[d] = hs[d].iters;
        c.cg_rr[d] = hs[d].rr;
        c.cg_true_rel[d] = hs[d].bb > 0 ? std::sqrt((double)hs[d].rr / hs[d].bb) : 0.0;
        c.cg_fp64_rel[d] = (hs[d].rr_true >= 0 && hs[d].bb > 0) ? std::sqrt(hs[d].rr_true / hs[d].bb) : -1.0;
        c.cg_refines[d] = hs[d].refines;
    }
    if (kt >= 0) {
        // compulsory per row and iteration: the group table (27 indices per 8 rows); r read
        // once by the product, p and q read and written; then p/q/x/r read and x/r written
        // (11 words)
        double bytes = 0;
        for (int d = d0; d <= d1; ++d) bytes += (double)hs[d].iters * (double)c.count[d] * (13.5 + 11 * 4);
        c.kpending[kt].bytes = bytes;
    }
    dfree(r, s); dfree(p, s); dfree(q, s);
    dfree(ddeps, s); dfree(dbd, s); dfree(st, s); dfree(slots, s); dfree(err, s);
    if (herr) {
        set_last_error("solver barrier timed out");
        throw Error{PRGPU_ERR_TIMEOUT, {0}};
    }
}

// ---------------------------------------------------------------------------
// CSR conjugate gradients with the reference's interface (CG_CUDA.cuh:344-509)
// ---------------------------------------------------------------------------
struct CsrArgs {
    int n;
    const int* rowptr;
    const int* col;
    const float* val;
    const float* b;
    float* x;
    float* r;
    float* p;
    float* q;
    float tol2;
    int max_iter;
    PartState* state;
    u64* slots;             // grid_sum's slots
    int* err;
    long long spin_limit;
    int extra;
};

// Two products, the same q bit for bit (a row's entries in order, one FMA each).
//
// Rows of few entries, or few rows: a thread per row walks its own entries.
//
// Rows of many entries (csr_stream): the product is bound by the matrix, 8 bytes an entry, once per
// iteration.  A thread per row reads a warp's lines a row apart, an eighth of each request used; on the
// 27-point stencil of 915 K rows (195 MB) an iteration took 84 us against 29 us of matrix bytes.  So a
// warp takes 32 consecutive rows, whose entries are one run of the arrays, in pieces of at most
// CSR_CHUNK entries: columns and values come into shared memory by asynchronous copies, the next piece
// while this one is summed, and each lane walks its own row there.  p is gathered in that walk, where
// the 32 lanes are at the same place of 32 rows (near columns, one or two lines a request), and not in
// the order of the entries (ten).  Pieces end where the 32 rows end: with a fixed size a piece holds
// parts of few rows and most lanes idle.  Two pieces of 7 KB for each of 15 warps fill an SM's shared
// memory, one block per SM.  Measured: 47 us a product (DRAM 3.2 TB/s and as much again from L2, which
// serves the gathers), 67 us an iteration.
constexpr int CSR_CHUNK = 896;
constexpr int CSR_BLOCK = 480;
constexpr int CSR_U = 9;                               // gathers in flight per lane
constexpr int CSR_WARPS = CSR_BLOCK / 32;
struct CsrWarpShared {
    int col[2][CSR_CHUNK];
    float val[2][CSR_CHUNK];
};
constexpr int CSR_DSMEM = CSR_WARPS * (int)sizeof(CsrWarpShared);

// entries [s, e) into a stage, at s & 3 when 'wide' (both arrays 16-byte aligned), else at 0
__device__ __forceinline__ void csr_fetch(const CsrArgs& a, int s, int e, bool wide, int* col, float* val) {
    const int lane = threadIdx.x & 31;
    const unsigned sc = (unsigned)__cvta_generic_to_shared(col), sv = (unsigned)__cvta_generic_to_shared(val);
    if (wide) {
        const int s0 = s & ~3;
        for (int k = 4 * lane; k < e - s0; k += 128) {
            const int bytes = 4 * min(e - s0 - k, 4);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sc + 4 * k), "l"(a.col + s0 + k), "r"(bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sv + 4 * k), "l"(a.val + s0 + k), "r"(bytes) : "memory");
        }
    } else {
        for (int k = lane; k < e - s; k += 32) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sc + 4 * k), "l"(a.col + s + k) : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sv + 4 * k), "l"(a.val + s + k) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

struct CsrRows {                                       // 32 rows: this lane's row and its entries
    int row, e0, e1;
    int end;                                           // the last entry + 1
    bool run;                                          // the offsets do not decrease
};
// the loads only; csr_rows_close makes them a group
__device__ __forceinline__ CsrRows csr_rows_load(const CsrArgs& a, i64 g) {
    CsrRows r;
    r.row = (int)min(32 * g + (threadIdx.x & 31), (i64)a.n);
    r.e0 = r.e1 = 0;
    if (r.row < a.n) {
        r.e0 = a.rowptr[r.row];
        r.e1 = a.rowptr[r.row + 1];
    }
    return r;
}
__device__ __forceinline__ void csr_rows_close(const CsrArgs& a, CsrRows& r) {
    r.run = __all_sync(0xffffffffu, r.e0 <= r.e1);
    const unsigned m = __ballot_sync(0xffffffffu, r.row < a.n);
    r.end = m ? __shfl_sync(0xffffffffu, r.e1, 31 - __clz(m)) : 0;
}

// the 32-row groups first, first + step, ... of q = A p, one warp.  Returns the lane's part of p.q
__device__ __forceinline__ double csr_stream(const CsrArgs& a, int first, int step, bool wide, CsrWarpShared& sm) {
    const int lane = threadIdx.x & 31;
    double loc = 0.0;
    const i64 ngroup = ((i64)a.n + 31) / 32;
    i64 g = first;
    if (g >= ngroup) return loc;
    CsrRows cur = csr_rows_load(a, g), nxt = csr_rows_load(a, g + step), far = csr_rows_load(a, g + 2 * (i64)step);
    csr_rows_close(a, cur);
    csr_rows_close(a, nxt);
    auto piece_end = [&](int from, const CsrRows& r) {
        return (int)min((i64)r.end, (i64)from - (wide ? from & 3 : 0) + CSR_CHUNK);
    };
    int s = __shfl_sync(0xffffffffu, cur.e0, 0);       // the current piece [s, e)
    int e = cur.run ? piece_end(s, cur) : s;
    __syncwarp();                                      // the previous product's readers are done
    csr_fetch(a, s, e, wide, sm.col[0], sm.val[0]);
    float o = 0.f, po = cur.row < a.n ? a.p[cur.row] : 0.f;
    for (int st = 0;; st ^= 1) {
        // the next piece: of this group, or the next group's first
        const bool last = e >= cur.end || !cur.run;
        const bool more = !last || g + step < ngroup;
        int s2 = e, e2 = e;
        if (last && more) s2 = e2 = __shfl_sync(0xffffffffu, nxt.e0, 0);
        if (more && (last ? nxt.run : true)) e2 = piece_end(s2, last ? nxt : cur);
        csr_fetch(a, s2, e2, wide, sm.col[st ^ 1], sm.val[st ^ 1]);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const int base = wide ? s & ~3 : s;            // entry k lies at k - base
        const int* col = sm.col[st];
        const float* sv = sm.val[st];
        const int t1 = min(cur.e1, e) - base;
        for (int t = max(cur.e0, s) - base; t < t1; t += CSR_U) {
            float pv[CSR_U], vv[CSR_U];
#pragma unroll
            for (int u = 0; u < CSR_U; ++u) pv[u] = t + u < t1 ? a.p[col[t + u]] : 0.f;
#pragma unroll
            for (int u = 0; u < CSR_U; ++u) vv[u] = t + u < t1 ? sv[t + u] : 0.f;
#pragma unroll
            for (int u = 0; u < CSR_U; ++u)
                if (t + u < t1) o = fmaf(vv[u], pv[u], o);
        }
        if (last) {
            if (cur.row < a.n) {
                // offsets that decrease: each row by itself, without entries when its end lies before its start
                if (!cur.run) {
                    o = 0.f;
                    for (int k = cur.e0; k < cur.e1; ++k) o = fmaf(a.val[k], a.p[a.col[k]], o);
                }
                a.q[cur.row] = o;
                loc += (double)(po * o);
            }
            if (!more) break;
            o = 0.f;
            g += step;
            cur = nxt;
            po = cur.row < a.n ? a.p[cur.row] : 0.f;
            nxt = far;
            csr_rows_close(a, nxt);
            far = csr_rows_load(a, g + 2 * (i64)step);
        }
        s = s2;
        e = e2;
        __syncwarp();                                  // this piece's readers are done
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    return loc;
}

// Whether the streamed product is the faster one for this system, from 32 consecutive rows per warp spread over the
// matrix: at least 3 in 4 of them have to fit (votes of 1 and -3), which they do when
//  * the entries at one place of the 32 rows (eight places are looked at) mostly lie within CSR_NEAR columns: matrix
//    pieces fill an SM's shared memory, so p is gathered through the 40 KB of L1 that are left, and where these do not
//    hold it a thread per row, with most of 256 KB and twice the warps, is the faster;
//  * within CSR_NEAR_TIGHT for rows of more than CSR_LONG_NNZ entries on average, and when 16 of the rows or more start
//    in one bank (rows of 64 entries: 32 lanes in one);
//  * their lanes' shares are alike, unless the longest row is an eighth of a piece at most: a piece holds parts of few
//    long rows, so most lanes idle when those are longer than the others.
// us an iteration, a thread per row against streamed, 1 M rows: 27 entries within 1,024 columns 91 and 65, within
// 8,192 106 and 106, within 32,768 140 and 188, anywhere 173 and 216; 64 entries within 8,192 columns 508 and 546, 125
// entries 425 and 553; rows of 1 to 319 entries 586 and 842; 81 entries a row on average, all in every fourth row,
// 388 and 484.  With 500 K rows, 27 entries: 57 and 40, 67 and 52, 80 and 97, 104 and 116.
constexpr int CSR_STREAM_NNZ = 16, CSR_LONG_NNZ = 88, CSR_STREAM_NNZ_MAX = 128, CSR_STREAM_ROWS = 1 << 17;
constexpr int CSR_NEAR = 5120, CSR_NEAR_TIGHT = 1280;
constexpr int CSR_LOOK_BLOCKS = 304;
__host__ __device__ constexpr bool csr_stream_length(i64 nz, i64 n) {
    return nz / n >= CSR_STREAM_NNZ && nz / n <= CSR_STREAM_NNZ_MAX;
}
__global__ void __launch_bounds__(CG_BLOCK) k_csr_look(CsrArgs a, int* __restrict__ vote) {
    const i64 nwarps = (i64)gridDim.x * (CG_BLOCK / 32), warp = (i64)blockIdx.x * (CG_BLOCK / 32) + (threadIdx.x >> 5);
    const i64 nz = (i64)a.rowptr[a.n] - a.rowptr[0];
    const CsrRows r = csr_rows_load(a, warp * (((i64)a.n + 31) / 32) / nwarps);
    const int len = min(max(r.e1 - r.e0, 0), 1 << 24), step = len >> 3;
    const int crowd = __reduce_max_sync(0xffffffffu, __popc(__match_any_sync(0xffffffffu, r.e0 & 31)));
    const bool longer = nz / a.n > CSR_LONG_NNZ;
    const int within = crowd < 16 && !longer ? CSR_NEAR : CSR_NEAR_TIGHT;
    int c[8], near = 0, seen = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) c[k] = step > 0 || k < len ? a.col[r.e0 + (step > 0 ? k * step : k)] : -1;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int hi = __reduce_max_sync(0xffffffffu, c[k]), lo = __reduce_min_sync(0xffffffffu, c[k] < 0 ? INT_MAX : c[k]);
        if (hi < 0) continue;                          // no row has this place
        ++seen;
        near += hi - lo < within;
    }
    const unsigned total = __reduce_add_sync(0xffffffffu, (unsigned)len), most = __reduce_max_sync(0xffffffffu, (unsigned)len);
    const bool even = most <= CSR_CHUNK / 8 || 32 * (u64)most <= (longer ? total + total / 4 : 3 * (u64)total);
    const bool fits = 4 * near >= 3 * seen && even && csr_stream_length(nz, a.n);
    if ((threadIdx.x & 31) == 0) atomicAdd(vote, fits ? 1 : -3);
}

// f over this thread's rows, four at a time: load (row, slot) for all four first
template <class L, class F>
__device__ __forceinline__ void csr_each(i64 start, i64 stride, i64 n, L load, F use) {
    for (i64 i = start; i < n; i += 4 * stride) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < n) load(i + u * stride, u);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < n) use(i + u * stride, u);
    }
}

template <bool STREAM>
__global__ void __launch_bounds__(STREAM ? CSR_BLOCK : CG_BLOCK, STREAM ? 1 : 4) k_cg_csr(CsrArgs a) {
    extern __shared__ __align__(16) unsigned char csr_dsm[];
    __shared__ GridSumShared<1> gsm;
    const i64 stride = (i64)gridDim.x * blockDim.x;
    const i64 start = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const int w = threadIdx.x >> 5;
    unsigned epoch = 0;
    const GridSum gs{a.slots, (int)gridDim.x + 2, 0, (int)gridDim.x, (int)blockIdx.x, (int)gridDim.x, a.err, a.spin_limit, a.extra};
    auto preduce = [&](double v, bool data, bool& ok) -> double {
        const double s[1] = {v};
        double t[1] = {0.0};
        ok = grid_sum(gs, ++epoch, data, s, gsm, t);
        return t[0];
    };
    float l0[4], l1[4];
    double loc = 0;
    for (i64 i = start; i < a.n; i += stride) {
        a.x[i] = 0.f;
        a.r[i] = a.b[i];
        loc += (double)(a.b[i] * a.b[i]);
    }
    bool ok = true;
    float r1 = (float)preduce(loc, true, ok), r0 = 0.f;
    int k = 1;
    while (ok && r1 > a.tol2 && k <= a.max_iter) {
        const float beta = k > 1 ? r1 / r0 : 0.f;
        csr_each(start, stride, a.n,
                 [&](i64 i, int u) { l0[u] = a.r[i]; l1[u] = k > 1 ? a.p[i] : 0.f; },
                 [&](i64 i, int u) { a.p[i] = k > 1 ? fmaf(beta, l1[u], l0[u]) : l0[u]; });
        preduce(0.0, true, ok);   // p is complete
        if (!ok) break;
        loc = 0;
        if constexpr (STREAM) {
            const bool wide = ((reinterpret_cast<u64>(a.col) | reinterpret_cast<u64>(a.val)) & 15) == 0;
            loc = csr_stream(a, blockIdx.x * CSR_WARPS + w, gridDim.x * CSR_WARPS, wide,
                             reinterpret_cast<CsrWarpShared*>(csr_dsm)[w]);
        } else {
            for (i64 i = start; i < a.n; i += stride) {
                float o = 0.f;
                for (int e = a.rowptr[i]; e < a.rowptr[i + 1]; ++e) o = fmaf(a.val[e], a.p[a.col[e]], o);
                a.q[i] = o;
                loc += (double)(a.p[i] * o);
            }
        }
        const double pq = preduce(loc, STREAM, ok);   // (a thread per row updates the rows of its q)
        if (!ok) break;
        const float al = (float)((double)r1 / pq), nal = -al;
        loc = 0;
        csr_each(start, stride, a.n,
                 [&](i64 i, int u) { l0[u] = a.q[i]; l1[u] = a.r[i]; },
                 [&](i64 i, int u) {
                     const float ri = fmaf(nal, l0[u], l1[u]);
                     a.r[i] = ri;
                     loc += (double)(ri * ri);
                 });
        // r is read and written by its own thread only, and so is p until it is complete again: r.r
        // carries no data, and x is updated while it travels
        const double s[1] = {loc};
        double rr[1] = {0.0};
        grid_publish(gs, ++epoch, false, s, gsm);
        csr_each(start, stride, a.n,
                 [&](i64 i, int u) { l0[u] = a.p[i]; l1[u] = a.x[i]; },
                 [&](i64 i, int u) { a.x[i] = fmaf(al, l0[u], l1[u]); });
        ok = grid_collect(gs, epoch, false, gsm, rr);
        r0 = r1;
        r1 = (float)rr[0];
        ++k;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.state->iters = k - 1;
        a.state->rr = r1;
    }
}

int cg_csr_impl(int n, int nz, const int* rowptr, const int* col, const float* val, const float* rhs, float* x, float tol,
                int max_iter, int* iters, float* ms) {
    cudaStream_t s = 0;
    int dev = 0, sms = 0, per_sm = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    float *r = nullptr, *p = nullptr, *q = nullptr;
    PartState* st = nullptr;
    u64* slots = nullptr;
    int* err = nullptr;
    CK(cudaMalloc(&r, sizeof(float) * std::max(n, 1)));
    CK(cudaMalloc(&p, sizeof(float) * std::max(n, 1)));
    CK(cudaMalloc(&q, sizeof(float) * std::max(n, 1)));
    CK(cudaMalloc(&st, sizeof(PartState)));
    CK(cudaMalloc(&err, sizeof(int)));
    CK(cudaMemset(st, 0, sizeof(PartState)));
    CK(cudaMemset(err, 0, sizeof(int)));
    CsrArgs a;
    a.n = n; a.rowptr = rowptr; a.col = col; a.val = val; a.b = rhs; a.x = x; a.r = r; a.p = p; a.q = q;
    a.tol2 = tol * tol;
    a.max_iter = max_iter;
    a.state = st;
    a.err = err;
    const WaitLimits wl = wait_limits();
    a.spin_limit = wl.spin_limit;
    a.extra = wl.extra;
    cudaEvent_t e0, e1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    // A system whose size and number of entries allow the streamed product is looked at on the device (k_csr_look, which
    // also sees a wrong nz: a few us and a read); a thread per row takes what is declined there and the rest.  Below
    // CSR_STREAM_ROWS rows neither is the faster for all: 98,304 rows of 27 entries 23 us an iteration and 20, of 48 entries
    // 36 and 41.
    bool stream = n >= CSR_STREAM_ROWS && csr_stream_length(nz, n);
    if (stream) {
        k_csr_look<<<CSR_LOOK_BLOCKS, CG_BLOCK, 0, s>>>(a, &st->status);
        CK_LAUNCH();
        int vote = 0;
        CK(cudaMemcpy(&vote, &st->status, sizeof vote, cudaMemcpyDeviceToHost));
        stream = vote >= 0;
    }
    const int block = stream ? CSR_BLOCK : CG_BLOCK, dsmem = stream ? CSR_DSMEM : 0;
    void (*kernel)(CsrArgs) = stream ? k_cg_csr<true> : k_cg_csr<false>;
    if (stream) CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CSR_DSMEM));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, dsmem));
    const i64 want = ((i64)n + block - 1) / block;
    const int G = (int)std::max<i64>(1, std::min<i64>((i64)sms * std::max(per_sm, 1), want));
    const i64 words = grid_sum_words(G + 2, 1);
    CK(cudaMalloc(&slots, sizeof(u64) * words));
    CK(cudaMemset(slots, 0, sizeof(u64) * words));
    a.slots = slots;
    void* kargs[] = {(void*)&a};
    CK(cudaEventRecord(e0, s));
    CK(cudaLaunchCooperativeKernel((void*)kernel, dim3(G), dim3(block), kargs, dsmem, s));
    ++g_kernel_launches;
    CK(cudaEventRecord(e1, s));
    CK(cudaEventSynchronize(e1));
    float t = 0;
    CK(cudaEventElapsedTime(&t, e0, e1));
    PartState hs;
    int herr = 0;
    CK(cudaMemcpy(&hs, st, sizeof hs, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(&herr, err, sizeof herr, cudaMemcpyDeviceToHost));
    cudaFree(r); cudaFree(p); cudaFree(q); cudaFree(st); cudaFree(slots); cudaFree(err);
    cudaEventDestroy(e0); cudaEventDestroy(e1);
    if (iters) *iters = hs.iters;
    if (ms) *ms = t;
    if (herr) {
        set_last_error("CG barrier timed out");
        return PRGPU_ERR_TIMEOUT;
    }
    return hs.iters >= max_iter && hs.rr > a.tol2 ? PRGPU_ERR_NOT_CONVERGED : PRGPU_OK;
}

}  // namespace prgpu
