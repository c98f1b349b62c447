// Right-hand side: vector-field splat at the finest depth and divergence at
// every depth.  Replaces computeVectorField (main.cu:913-964),
// computeEncodedFinerNodesDivergence (main.cu:1007-1060) and the per-node host
// loop of the coarse divergence (main.cu:3399-3458).
#include "context.h"
#include "prims.cuh"

namespace prgpu {

// BinaryNode<float>::CenterAndWidth for a finest-depth function index
__device__ __forceinline__ float finest_center(int off, int D) {
    float w = (float)(1.0 / (double)(1 << D));
    return (float)((0.5 + (double)off) * (double)w);
}

// The splat weight is (F/F(0)) scaled to the finest width, shifted to the sample and evaluated at the node
// centre (main.cu:913-964), a product of one value per axis.  A sample meets the 27 nodes around its leaf,
// so along an axis only three centres: nine values per sample, where evaluating them per (node, sample)
// pair takes 81, each with the shifted polynomial's arithmetic.  Per sample: its normal (and a pad), then the
// values of the centres one cell below, at and above its leaf along x, y and z (and three pads): 64 bytes a
// sample for the stage, 1.9 GB for 30 M.
constexpr int SW_STRIDE = 16;
__global__ void k_sample_weights(NodeArrays nd, int D, CPoly f, const float* __restrict__ pts, const float* __restrict__ nrm,
                                 const int* __restrict__ point_node, i64 n, float4* __restrict__ out, int stable) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        int c[3];
        key_coords(nd.key[point_node[i]], D, D, c);
        float w[9];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const float p = pts[3 * i + ax];
            CPoly s;
            if (!stable) cpoly_shift<2>(f, p, s);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const int k = c[ax] + t - 1;
                // stable: F/F(0) at (centre - p) 2^D = (k + 1/2) - p 2^D, one rounding
                w[3 * ax + t] = stable ? bspline_unit(fmaf(-p, (float)(1 << D), (float)k + 0.5f))
                                       : cpoly_value<2>(s, finest_center(k, D));
            }
        }
        float4* o = out + i * (SW_STRIDE / 4);
        o[0] = make_float4(nrm[3 * i], nrm[3 * i + 1], nrm[3 * i + 2], 0.f);
        o[1] = make_float4(w[0], w[1], w[2], w[3]);
        o[2] = make_float4(w[4], w[5], w[6], w[7]);
        o[3] = make_float4(w[8], 0.f, 0.f, 0.f);
    }
}

// One lane per finest slot, neighbours and their points in the reference's order (main.cu:913-964).  A warp
// takes 4 sibling groups: the 27-neighbourhoods of a group's 8 nodes are the 4x4x4 block of the
// children of the parent's 27 neighbours (the group table), whose point ranges are staged once per
// group, with a bit per cell that holds any (a surface fills few of the 64).  Each lane walks the set bits
// of its own 3x3x3, which lie in neighbour order, and a cell's samples in one flat loop, so that the lanes
// stay together, the next sample loaded while this one is added.  Bound by the latency of the sample
// gathers.  1M torus: 0.72 ms with the weights evaluated per pair and all 27 cells visited, 0.63 with the
// weights per sample, 0.36 with the empty cells skipped; 4M displaced sphere 2.8, 2.53 and 1.58.
// VEC false sums the products of the three values alone, one float per node (the density of a depth's nodes).
constexpr int SPLAT_BLOCK = 128;
template <bool VEC>
__global__ void __launch_bounds__(SPLAT_BLOCK) k_splat(NodeArrays nd, const int* __restrict__ gn, i64 ngroups_all,
                                                       i64 gfirst, i64 ng, i64 lo, const float4* __restrict__ sw,
                                                       float* __restrict__ field) {
    __shared__ int2 rng[SPLAT_BLOCK / 32][4][64];   // (first point, count) of each block cell
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
    for (i64 tile = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile * 4 < ng; tile += nwarps) {
        __syncwarp();
        unsigned long long held = 0;   // the cells of this lane's group that hold points, a bit each
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int e = lane + 32 * m;
            const i64 g = tile * 4 + (e >> 6);
            const int cell = e & 63, bx = cell >> 4, by = (cell >> 2) & 3, bz = cell & 3;
            int2 r = make_int2(0, 0);
            if (g < ng) {
                const int jp = 9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1) + ((bz + 1) >> 1);
                const int cn = gn[(i64)jp * ngroups_all + gfirst + g];
                if (cn != -1) {
                    const int node = cn + ((((bx + 1) & 1) << 2) | (((by + 1) & 1) << 1) | ((bz + 1) & 1));
                    r = make_int2(nd.pidx[node], nd.pnum[node]);
                }
            }
            rng[w][e >> 6][cell] = r;
            const unsigned b = __ballot_sync(0xffffffffu, r.y > 0);
            if ((lane >> 3) == (m >> 1)) held |= (unsigned long long)b << (32 * (m & 1));
        }
        __syncwarp();
        const i64 g = tile * 4 + (lane >> 3);
        if (g >= ng) continue;
        const int s = lane & 7, sx = s >> 2, sy = (s >> 1) & 1, sz = s & 1;
        const i64 i = lo + 8 * g + s;
        const int2* br = rng[w][lane >> 3];
        // the node's 27 cells are a 3x3x3 of the 4x4x4, in the same order as their bits
        held &= 0x077707770777ull << (sx * 16 + sy * 4 + sz);
        float v0 = 0.f, v1 = 0.f, v2 = 0.f;
        const float* q = nullptr;  // the next sample
        int left = 0;              // samples of the current cell from it on
        int ox = 0, oy = 0, oz = 0;
        struct Sample { float4 n; float wx, wy, wz; };
        auto next = [&]() {        // the next pair's sample
            if (left == 0) {
                const int cell = __ffsll(held) - 1;
                held &= held - 1;
                const int2 r = br[cell];
                q = reinterpret_cast<const float*>(sw) + (i64)r.x * SW_STRIDE;
                left = r.y;
                // the node lies one cell below the sample's leaf (value 0) when the neighbour is above it (2)
                ox = 4 + 2 + sx - (cell >> 4);
                oy = 7 + 2 + sy - ((cell >> 2) & 3);
                oz = 10 + 2 + sz - (cell & 3);
            }
            Sample r;
            if (VEC) r.n = *reinterpret_cast<const float4*>(q);
            r.wx = q[ox];
            r.wy = q[oy];
            r.wz = q[oz];
            q += SW_STRIDE;
            --left;
            return r;
        };
        if (held != 0) {
            Sample a = next();
            for (;;) {
                const bool more = left != 0 || held != 0;
                Sample b = a;
                if (more) b = next();
                const float wgt = a.wx * a.wy * a.wz;
                if (VEC) {
                    v0 = fmaf(wgt, a.n.x, v0);
                    v1 = fmaf(wgt, a.n.y, v1);
                    v2 = fmaf(wgt, a.n.z, v2);
                } else {
                    v0 += wgt;
                }
                if (!more) break;
                a = b;
            }
        }
        const i64 o = i - lo;
        if (VEC) {
            field[3 * o] = v0;
            field[3 * o + 1] = v1;
            field[3 * o + 2] = v2;
        } else {
            field[o] = v0;
        }
    }
}

// finest-slot coordinates, packed for the divergence gathers
__global__ void k_finest_coords(const u64* __restrict__ key, i64 lo, i64 n, int D, short4* __restrict__ out) {
    for (i64 o = (i64)blockIdx.x * blockDim.x + threadIdx.x; o < n; o += (i64)gridDim.x * blockDim.x) {
        int xyz[3];
        key_coords(key[lo + o], D, D, xyz);
        out[o] = make_short4((short)xyz[0], (short)xyz[1], (short)xyz[2], 0);
    }
}

struct DivArgs {
    int D;
    i64 M;
    const float* vfield;
    const short4* fc;          // finest coordinates
    const float* rows;         // compact inner-product rows
    const i64* row_start;      // per depth (device)
};

// one divergence term: float dot product of V_o with the three table values,
// ordered as DotProduct with the reference's fused multiply-adds (main.cu:966-972)
__device__ __forceinline__ float div_term(const DivArgs& a, const float* r0, const float* r1, const float* r2,
                                          const int t0[3], i64 o) {
    const short4 c = a.fc[o];
    const float u0 = r0[c.x - t0[0]], u1 = r1[c.y - t0[1]], u2 = r2[c.z - t0[2]];
    const float vx = a.vfield[3 * o], vy = a.vfield[3 * o + 1], vz = a.vfield[3 * o + 2];
    float t = vx * u0;
    t = fmaf(vy, u1, t);
    t = fmaf(vz, u2, t);
    return t;
}

__device__ __forceinline__ void node_rows(const DivArgs& a, u64 key, int d, const float*& r0, const float*& r1,
                                          const float*& r2, int t0[3]) {
    int xyz[3];
    key_coords(key, d, a.D, xyz);
    const i64 W = 3ll << (a.D - d);
    const i64 rs = a.row_start[d];
    r0 = a.rows + rs + xyz[0] * W;
    r1 = a.rows + rs + xyz[1] * W;
    r2 = a.rows + rs + xyz[2] * W;
    for (int q = 0; q < 3; ++q) t0[q] = (xyz[q] - 1) * (1 << (a.D - d));
}

// The value of a double sum of floats added one after the other, rounded to float at the end, without
// the FP64 pipe (2 operations a cycle and SM: a conversion and an addition per term were most of the two
// finest depths' divergence).  The terms go into three floats by error-free additions: h + l + m differs
// from the exact sum S by at most n^3 u^3 T (u = 2^-24, T the sum of the terms' magnitudes), the double
// sum by at most n 2^-53 T, both together below 2^-44 T for n <= 216.  Where every value within that of
// h + l + m rounds to the same float, that is the double sum's rounding too.  Ties of that rounding (two
// terms of one exponent make one in two cases) are settled by exactness: when T has less than 2^29 times
// the smallest non-zero term's power of two, every partial sum is a multiple of that term's last place
// below 2^53 of it, so the double sum is exact and so are h + l + m and its value in double.  Elsewhere
// ('sure' false: about one node in a million, and sums that are not finite) the caller adds in double.
struct FloatSum3 {
    float h = 0.f, l = 0.f, m = 0.f, T = 0.f;
    unsigned least = 0xffffffffu;   // bits of the smallest non-zero magnitude, less one
    __device__ __forceinline__ void add(float t) {
        const float s = h + t, a = s - h, e = (h - (s - a)) + (t - a);
        const float q = l + e, b = q - l;
        m += (l - (q - b)) + (e - b);
        h = s;
        l = q;
        T += fabsf(t);
        least = min(least, (__float_as_uint(t) & 0x7fffffffu) - 1u);
    }
    __device__ __forceinline__ float rounded(bool& sure) const {
        const double v = (double)h + ((double)l + (double)m), d = (double)T * 5.684341886080802e-14;   // 2^-44
        // exponents of T and the smallest term (a subnormal counts as exponent 1), T finite
        const int eT = (int)(__float_as_uint(T) >> 23), en = max((int)((least + 1u) >> 23), 1);
        const float f = (float)(v - d);
        if (f == (float)(v + d)) {
            sure = true;
            return f;
        }
        sure = eT < 255 && eT - en <= 28;
        return (float)v;
    }
};

// Depth D - 1 by sibling groups: the 27 neighbours of a group's 8 nodes are the 4x4x4 block of the children
// of the parent's 27 neighbours (the group table), and each block cell's finest descendants are its 8
// children (or none), consecutive finest slots whose V is 96 aligned bytes.  A lane takes a node and adds
// its at most 216 terms in neighbour order, each neighbour's children in order.  The row entry of a
// child along an axis is 2 j + bit of the node's 6 (j the neighbour's offset 0..2), so no coordinates are
// read.  1M torus: 0.98 ms with a thread per node, its 27 neighbour loops unrolled (half the issue slots
// waiting for instructions, four loads a term) and a double addition per term.
__device__ __forceinline__ float div_child_term(float vx, float vy, float vz, float u0, float u1, float u2) {
    float t = vx * u0;
    t = fmaf(vy, u1, t);
    return fmaf(vz, u2, t);
}
constexpr int DIV_PARENT_WARPS = 4;
__global__ void __launch_bounds__(32 * DIV_PARENT_WARPS) k_div_parents(NodeArrays nd, DivArgs a, const int* __restrict__ gn,
                                                                       i64 ngroups_all, i64 gfirst, i64 ng, i64 lo,
                                                                       i64 finest, float* __restrict__ out) {
    __shared__ int s_slot[DIV_PARENT_WARPS][4][64];   // first finest slot of each block cell, -1: none
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ch = lane & 7, sx = ch >> 2, sy = (ch >> 1) & 1, sz = ch & 1;
    const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
    for (i64 tile = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile * 4 < ng; tile += nwarps) {
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int e = lane + 32 * q;
            const i64 g = tile * 4 + (e >> 6);
            const int cell = e & 63, bx = cell >> 4, by = (cell >> 2) & 3, bz = cell & 3;
            int s0 = -1;
            if (g < ng) {
                const int c0 = gn[(i64)(9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1) + ((bz + 1) >> 1)) * ngroups_all + gfirst + g];
                if (c0 != -1) {
                    const int f = nd.child0[c0 + ((((bx + 1) & 1) << 2) | (((by + 1) & 1) << 1) | ((bz + 1) & 1))];
                    if (f != -1) s0 = (int)(f - finest);
                }
            }
            s_slot[w][e >> 6][cell] = s0;
        }
        __syncwarp();
        const i64 g = tile * 4 + (lane >> 3);
        if (g >= ng) continue;
        const i64 i = lo + 8 * g + ch;
        const float *r0, *r1, *r2;
        int t0[3];
        node_rows(a, nd.key[i], a.D - 1, r0, r1, r2, t0);
        float u2[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) u2[k] = r2[k];
        const int* blk = s_slot[w][lane >> 3];
        // f for each term, in order
        auto each = [&](auto f) {
#pragma unroll 1
            for (int jxy = 0; jxy < 9; ++jxy) {
                const int jx = jxy / 3, jy = jxy % 3;
                const float u0a = r0[2 * jx], u0b = r0[2 * jx + 1], u1a = r1[2 * jy], u1b = r1[2 * jy + 1];
#pragma unroll
                for (int jz = 0; jz < 3; ++jz) {
                    const int s0 = blk[(sx + jx) * 16 + (sy + jy) * 4 + sz + jz];
                    if (s0 < 0) continue;
                    const float4* V = reinterpret_cast<const float4*>(a.vfield + 3 * (i64)s0);
                    float vv[24];
#pragma unroll
                    for (int k = 0; k < 6; ++k) {
                        const float4 q = V[k];
                        vv[4 * k] = q.x; vv[4 * k + 1] = q.y; vv[4 * k + 2] = q.z; vv[4 * k + 3] = q.w;
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        f(div_child_term(vv[3 * k], vv[3 * k + 1], vv[3 * k + 2], (k >> 2) ? u0b : u0a,
                                         ((k >> 1) & 1) ? u1b : u1a, u2[2 * jz + (k & 1)]));
                }
            }
        };
        FloatSum3 s;
        each([&](float t) { s.add(t); });
        bool sure;
        float val = s.rounded(sure);
        if (!sure) {
            double d = 0.0;
            each([&](float t) { d += (double)t; });
            val = (float)d;
        }
        out[i] = val;
    }
}

// finest depth by sibling groups: the 27 neighbours of the 8 children of a node
// are the 4x4x4 block of the children of the parent's 27 neighbours (the solve's
// group table).  One warp stages the V of the blocks of 4 groups in shared
// memory; each row then adds its 27 terms in neighbour order.  Every finest node
// has exactly one finest descendant (itself), and the neighbour at offset
// j = (jx,jy,jz) reads the row entries jx, jy, jz of the node's 3-entry rows.
__global__ void __launch_bounds__(256) k_div_finest(NodeArrays nd, DivArgs a, const int* __restrict__ gn,
                                                    i64 ngroups_all, i64 gfirst, i64 ng, i64 lo,
                                                    float* __restrict__ out) {
    __shared__ float4 cells[8][4 * 64];   // per warp: V of the 4x4x4 block of 4 groups, w = 1 if the cell exists
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int ch = lane & 7, gl = lane >> 3;
    const int sx = ch >> 2, sy = (ch >> 1) & 1, sz = ch & 1;
    const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
    float4* blk = cells[wib];
    for (i64 tile = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; tile * 4 < ng; tile += nwarps) {
        __syncwarp();
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int e = lane + 32 * m;
            const i64 g = tile * 4 + (e >> 6);
            const int cell = e & 63, bx = cell >> 4, by = (cell >> 2) & 3, bz = cell & 3;
            float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
            if (g < ng) {
                const int jp = 9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1) + ((bz + 1) >> 1);
                const int cn = gn[(i64)jp * ngroups_all + gfirst + g];
                if (cn != -1) {
                    const i64 o = cn + ((((bx + 1) & 1) << 2) | (((by + 1) & 1) << 1) | ((bz + 1) & 1)) - lo;
                    val = make_float4(a.vfield[3 * o], a.vfield[3 * o + 1], a.vfield[3 * o + 2], 1.f);
                }
            }
            blk[e] = val;
        }
        __syncwarp();
        const i64 g = tile * 4 + gl;
        if (g < ng) {
            const i64 i = lo + 8 * g + ch;
            int xyz[3];
            key_coords(nd.key[i], a.D, a.D, xyz);
            const float* rr = a.rows + a.row_start[a.D];
            float R[3][3];
#pragma unroll
            for (int ax = 0; ax < 3; ++ax)
#pragma unroll
                for (int t = 0; t < 3; ++t) R[ax][t] = rr[xyz[ax] * 3 + t];
            const float4* b = blk + gl * 64;
            FloatSum3 s;
#pragma unroll
            for (int j = 0; j < 27; ++j) {
                const int jx = j / 9, jy = (j / 3) % 3, jz = j % 3;
                const float4 c = b[(sx + jx) * 16 + (sy + jy) * 4 + (sz + jz)];
                if (c.w != 0.f) s.add(div_child_term(c.x, c.y, c.z, R[0][jx], R[1][jy], R[2][jz]));   // else no neighbour
            }
            bool sure;
            float val = s.rounded(sure);
            if (!sure) {
                double d = 0.0;
#pragma unroll 1
                for (int jxy = 0; jxy < 9; ++jxy) {
                    const int jx = jxy / 3, jy = jxy % 3;
#pragma unroll
                    for (int jz = 0; jz < 3; ++jz) {
                        const float4 c = b[(sx + jx) * 16 + (sy + jy) * 4 + (sz + jz)];
                        if (c.w != 0.f)
                            d += (double)div_child_term(c.x, c.y, c.z, rr[xyz[0] * 3 + jx], rr[xyz[1] * 3 + jy], R[2][jz]);
                    }
                }
                val = (float)d;
            }
            out[i] = val;
        }
    }
}

// the root (all finest nodes are its terms): the node's terms, in neighbour order,
// are cut into chunks of DIV_CHUNK; one warp sums a chunk and the chunk sums are
// added per node in FP64 in a fixed order (k_div_sum: deterministic).  Within a chunk each
// lane keeps a compensated float pair (hi + lo, Neumaier's summation), whose
// error is at most 2u|sum| + O(n u^2) sum|term| -- FP64 accuracy for these
// lengths without FP64 arithmetic per term.
constexpr int DIV_CHUNK = 2048;
constexpr int DIV_WARPS = 8;

__device__ __forceinline__ i64 node_terms(const NodeArrays& nd, i64 M, i64 i) {
    i64 T = 0;
    for (int j = 0; j < 27; ++j) {
        const int nb = nd.neigh[(i64)j * M + i];
        if (nb != -1) T += nd.dnum[nb];
    }
    return T;
}

__global__ void k_div_count(NodeArrays nd, i64 n, int* __restrict__ nchunks) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
        nchunks[i] = (int)((node_terms(nd, nd.M, i) + DIV_CHUNK - 1) / DIV_CHUNK);
}

__global__ void k_div_items(const int* __restrict__ nchunks, const int* __restrict__ first, i64 n,
                            int* __restrict__ item_node) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
        for (int c = 0; c < nchunks[i]; ++c) item_node[first[i] + c] = (int)i;
}

__global__ void __launch_bounds__(DIV_WARPS * 32) k_div_chunks(NodeArrays nd, DivArgs a, const int* __restrict__ item_node,
                                                               const int* __restrict__ first, i64 nitems,
                                                               double* __restrict__ partial) {
    __shared__ int pre[DIV_WARPS][28];
    __shared__ int sidx[DIV_WARPS][27];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const i64 warp = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
    for (i64 it = warp; it < nitems; it += nwarps) {
        const i64 i = item_node[it];
        const int chunk = (int)(it - first[i]);
        // prefix of the neighbours' finest-descendant counts, in neighbour order
        int cnt = 0, sx = 0;
        if (lane < 27) {
            const int nb = nd.neigh[(i64)lane * a.M + i];
            if (nb != -1) { cnt = nd.dnum[nb]; sx = nd.didx[nb]; }
        }
        int inc = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        __syncwarp();
        if (lane < 27) { pre[w][lane] = inc - cnt; sidx[w][lane] = sx; }
        if (lane == 26) pre[w][27] = inc;
        __syncwarp();
        const float *r0, *r1, *r2;
        int t0[3];
        node_rows(a, nd.key[i], nd.depth[i], r0, r1, r2, t0);
        const int total = pre[w][27];
        const int lo = chunk * DIV_CHUNK, hi = min(total, lo + DIV_CHUNK);
        float sh = 0.f, sl = 0.f;
        int j = 0;
        while (pre[w][j + 1] <= lo) ++j;
        // neighbour by neighbour: each is a contiguous range of finest slots
        for (; j < 27 && pre[w][j] < hi; ++j) {
            const int a0 = max(lo, pre[w][j]), a1 = min(hi, pre[w][j + 1]);
            const i64 base = (i64)sidx[w][j] - pre[w][j];
            int t = a0 + lane;
            // four terms per step: their loads are issued together
            for (; t + 96 < a1; t += 128) {
                float tv[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) tv[q] = div_term(a, r0, r1, r2, t0, base + t + 32 * q);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float s = sh + tv[q];
                    sl += (fabsf(sh) >= fabsf(tv[q])) ? (sh - s) + tv[q] : (tv[q] - s) + sh;
                    sh = s;
                }
            }
            for (; t + 32 < a1; t += 64) {
                const float t1 = div_term(a, r0, r1, r2, t0, base + t);
                const float t2 = div_term(a, r0, r1, r2, t0, base + t + 32);
                float s = sh + t1;
                sl += (fabsf(sh) >= fabsf(t1)) ? (sh - s) + t1 : (t1 - s) + sh;
                sh = s;
                s = sh + t2;
                sl += (fabsf(sh) >= fabsf(t2)) ? (sh - s) + t2 : (t2 - s) + sh;
                sh = s;
            }
            if (t < a1) {
                const float term = div_term(a, r0, r1, r2, t0, base + t);
                const float s = sh + term;
                sl += (fabsf(sh) >= fabsf(term)) ? (sh - s) + term : (term - s) + sh;
                sh = s;
            }
        }
        double val = (double)sh + (double)sl;
        for (int o = 16; o; o >>= 1) val += __shfl_xor_sync(0xffffffffu, val, o);
        if (lane == 0) partial[it] = val;
        __syncwarp();
    }
}

// Depths 1..D-2 by sibling groups.  The 27-neighbourhoods of the 8 children of a
// node are the 4x4x4 block of the children of the parent's 27 neighbours (the
// group table), and in x-major block order every child meets its own neighbours
// in neighbour order.  A group's terms are the finest descendants of the block's
// cells, concatenated in block order and cut into chunks of DIV_CHUNK finest
// nodes; one warp reads each finest node of a chunk once and adds its term to
// every child whose neighbourhood holds the cell (1, 2, 4 or 8 children), each
// child in its own compensated pair.  The term is the one k_div_chunks forms:
// child b on an axis reads the row of coordinate 2P+b at offset c - (2P+b-1)S,
// which is the row of 2P at offset (c - (2P-1)S) + 2bS.
__device__ __forceinline__ void neu_add(float& sh, float& sl, float t) {
    const float s = sh + t;
    sl += (fabsf(sh) >= fabsf(t)) ? (sh - s) + t : (t - s) + sh;
    sh = s;
}

__device__ __forceinline__ int group_cell_node(const int* __restrict__ gn, i64 ngroups_all, i64 g, int cell) {
    const int bx = cell >> 4, by = (cell >> 2) & 3, bz = cell & 3;
    const int jp = 9 * ((bx + 1) >> 1) + 3 * ((by + 1) >> 1) + ((bz + 1) >> 1);
    const int cn = gn[(i64)jp * ngroups_all + g];
    return cn == -1 ? -1 : cn + ((((bx + 1) & 1) << 2) | (((by + 1) & 1) << 1) | ((bz + 1) & 1));
}

__global__ void k_div_group_count(NodeArrays nd, const int* __restrict__ gn, i64 ngroups_all, i64 ng,
                                  int* __restrict__ nchunks) {
    for (i64 g = (i64)blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += (i64)gridDim.x * blockDim.x) {
        i64 T = 0;
        for (int cell = 0; cell < 64; ++cell) {
            const int n = group_cell_node(gn, ngroups_all, g, cell);
            if (n != -1) T += nd.dnum[n];
        }
        nchunks[g] = (int)((T + DIV_CHUNK - 1) / DIV_CHUNK);
    }
}

__global__ void __launch_bounds__(DIV_WARPS * 32) k_div_groups(NodeArrays nd, DivArgs a, const int* __restrict__ gn,
                                                               i64 ngroups_all, const int* __restrict__ item_group,
                                                               const int* __restrict__ first, i64 nitems,
                                                               double* __restrict__ partial) {
    __shared__ int pre[DIV_WARPS][65];
    __shared__ int sidx[DIV_WARPS][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const i64 warp = ((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
    for (i64 it = warp; it < nitems; it += nwarps) {
        const i64 g = item_group[it];
        const int chunk = (int)(it - first[g]);
        // prefix of the block cells' finest-descendant counts, two cells per lane
        int cnt[2], sx[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int n = group_cell_node(gn, ngroups_all, g, 2 * lane + q);
            cnt[q] = n == -1 ? 0 : nd.dnum[n];
            sx[q] = n == -1 ? 0 : nd.didx[n];
        }
        const int pair = cnt[0] + cnt[1];
        int inc = pair;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        __syncwarp();
        pre[w][2 * lane] = inc - pair;
        pre[w][2 * lane + 1] = inc - pair + cnt[0];
        sidx[w][2 * lane] = sx[0];
        sidx[w][2 * lane + 1] = sx[1];
        if (lane == 31) pre[w][64] = inc;
        __syncwarp();
        // child 0 of the group has the even coordinates 2P
        const i64 i0 = 1 + 8 * g;
        const int d = nd.depth[i0];
        int xyz[3];
        key_coords(nd.key[i0], d, a.D, xyz);
        const int S = 1 << (a.D - d), W = 3 * S;
        const float* R[3];
        int t0[3];
        const i64 rs = a.row_start[d];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            R[ax] = a.rows + rs + (i64)xyz[ax] * W;
            t0[ax] = (xyz[ax] - 1) * S;
        }
        const int total = pre[w][64];
        const int lo = chunk * DIV_CHUNK, hi = min(total, lo + DIV_CHUNK);
        float sh[8], sl[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) { sh[s] = 0.f; sl[s] = 0.f; }
        // lanes run over the chunk across cell boundaries; each lane tracks its
        // cell (empty cells are skipped by the prefix)
        int j = 0;
        while (j < 63 && pre[w][j + 1] <= lo + lane) ++j;
        for (int t = lo + lane; t < hi; t += 32) {
            while (pre[w][j + 1] <= t) ++j;
            const i64 o = (i64)sidx[w][j] - pre[w][j] + t;
            const int bx = j >> 4, by = (j >> 2) & 3, bz = j & 3;
            // which children hold this cell, per axis: b = 0 for block 0..2, b = 1 for 1..3
            const bool x0 = bx <= 2, x1 = bx >= 1, y0 = by <= 2, y1 = by >= 1, z0 = bz <= 2, z1 = bz >= 1;
            const short4 c = a.fc[o];
            const float vx = a.vfield[3 * o], vy = a.vfield[3 * o + 1], vz = a.vfield[3 * o + 2];
            const int ox = c.x - t0[0], oy = c.y - t0[1], oz = c.z - t0[2];
            const float ux0 = x0 ? R[0][ox] : 0.f, ux1 = x1 ? R[0][ox + 2 * S] : 0.f;
            const float uy0 = y0 ? R[1][oy] : 0.f, uy1 = y1 ? R[1][oy + 2 * S] : 0.f;
            const float uz0 = z0 ? R[2][oz] : 0.f, uz1 = z1 ? R[2][oz + 2 * S] : 0.f;
            const float px[2] = {vx * ux0, vx * ux1};
            const float uy[2] = {uy0, uy1}, uz[2] = {uz0, uz1};
            const bool hx[2] = {x0, x1}, hy[2] = {y0, y1}, hz[2] = {z0, z1};
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const int bsx = s >> 2, bsy = (s >> 1) & 1, bsz = s & 1;
                if (hx[bsx] && hy[bsy] && hz[bsz]) {
                    float term = fmaf(vy, uy[bsy], px[bsx]);
                    term = fmaf(vz, uz[bsz], term);
                    neu_add(sh[s], sl[s], term);
                }
            }
        }
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            double val = (double)sh[s] + (double)sl[s];
            for (int o = 16; o; o >>= 1) val += __shfl_xor_sync(0xffffffffu, val, o);
            if (lane == 0) partial[it * 8 + s] = val;
        }
        __syncwarp();
    }
}

// one warp per node: the node's chunk partials (per entity of `per` nodes, node
// s of the entity at offset s) summed lane-strided in FP64 and then by a fixed
// butterfly, so the result does not depend on the schedule
__global__ void k_div_sum(const int* __restrict__ nchunks, const int* __restrict__ first,
                          const double* __restrict__ partial, i64 lo, i64 hi, int per, float* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const i64 nwarps = ((i64)gridDim.x * blockDim.x) >> 5;
    for (i64 i = lo + (((i64)blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < hi; i += nwarps) {
        const i64 g = (i - lo) / per;
        const int s = (int)((i - lo) % per), n = nchunks[g];
        const i64 f = first[g];
        double v = 0.0;
        for (int q = lane; q < n; q += 32) v += partial[(f + q) * per + s];
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) out[i] = (float)v;
    }
}

// the same sum of sibling-group partials (node i is child (i-1) % per of group
// (i-1) / per) for nodes with few chunks: one thread per node, in chunk order
__global__ void k_div_sum_thread(const int* __restrict__ nchunks, const int* __restrict__ first,
                                 const double* __restrict__ partial, i64 lo, i64 hi, int per, float* __restrict__ out) {
    for (i64 i = lo + (i64)blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += (i64)gridDim.x * blockDim.x) {
        const i64 g = (i - 1) / per;
        const int s = (int)((i - 1) % per), n = nchunks[g];
        const i64 f = first[g];
        double v = 0.0;
        for (int q = 0; q < n; ++q) v += partial[(f + q) * per + s];
        out[i] = (float)v;
    }
}

// ---- density weights (params.density_weights; not in the reference)
// Kazhdan's weighting of non-uniform samples: at the kernel depth k, node o
// collects w_o = sum over the points p around it of B_o(p) (B_o the depth-k basis
// function of o, a product of its three axis functions); a point's density is
// W(s) = sum over the 27 depth-k nodes around it of B_o(s) w_o, and its weight
// 1/W(s), scaled to mean 1, multiplies its normal and its share of the iso-value.
// Both sums take a sample's basis values along an axis at three centres only, so these nine are evaluated once
// per sample (the splat's entries, without a normal); the first sum is then the splat's walk over the depth-k
// groups.  200k torus at depth 9, the whole weighting: 0.34 -> 0.14 ms.
__global__ void k_density_samples(NodeArrays nd, i64 n, const int* __restrict__ point_node, int k, int D,
                                  const CPoly* __restrict__ basis, const float* __restrict__ pts,
                                  int* __restrict__ ancestor, float4* __restrict__ out) {
    const int off = (1 << k) - 1;
    for (i64 s = (i64)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (i64)gridDim.x * blockDim.x) {
        int node = point_node[s];
        for (int d = D; d > k; --d) node = nd.parent[node];
        ancestor[s] = node;
        int c[3];
        key_coords(nd.key[node], k, D, c);
        float w[9];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const float p = pts[3 * s + ax];
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const int o = c[ax] + t - 1;   // outside the domain no node has the value
                w[3 * ax + t] = o >= 0 && o < (1 << k) ? cpoly_value<3>(basis[off + o], p) : 0.f;
            }
        }
        float4* q = out + s * (SW_STRIDE / 4);
        q[1] = make_float4(w[0], w[1], w[2], w[3]);
        q[2] = make_float4(w[4], w[5], w[6], w[7]);
        q[3] = make_float4(w[8], 0.f, 0.f, 0.f);
    }
}

__global__ void k_density_points(const int* __restrict__ neigh, i64 M, i64 n, const int* __restrict__ ancestor, i64 lo_k,
                                 const float4* __restrict__ sw, const float* __restrict__ w, float* __restrict__ inv,
                                 double* __restrict__ sum) {
    double loc = 0.0;
    for (i64 s = (i64)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (i64)gridDim.x * blockDim.x) {
        const i64 node = ancestor[s];
        const float4* q = sw + s * (SW_STRIDE / 4);
        const float4 a = q[1], b = q[2];
        const float wx[3] = {a.x, a.y, a.z}, wy[3] = {a.w, b.x, b.y}, wz[3] = {b.z, b.w, q[3].x};
        float W = 0.f;
#pragma unroll
        for (int j = 0; j < 27; ++j) {
            const int nb = neigh[(i64)j * M + node];
            if (nb != -1) W += wx[j / 9] * wy[(j / 3) % 3] * wz[j % 3] * w[nb - lo_k];
        }
        const float iw = W > 0.f ? 1.0f / W : 0.f;
        inv[s] = iw;
        loc += (double)iw;
    }
    for (int o = 16; o; o >>= 1) loc += __shfl_xor_sync(0xffffffffu, loc, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(sum, loc);
}

__global__ void k_weight_normals(i64 n, const double* __restrict__ sum, const float* __restrict__ nrm,
                                 float* __restrict__ weight, float* __restrict__ wnrm) {
    const float scale = (float)((double)n / *sum);
    for (i64 s = (i64)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (i64)gridDim.x * blockDim.x) {
        const float a = weight[s] * scale;
        weight[s] = a;
        wnrm[3 * s] = a * nrm[3 * s];
        wnrm[3 * s + 1] = a * nrm[3 * s + 1];
        wnrm[3 * s + 2] = a * nrm[3 * s + 2];
    }
}

static void density_weights(Ctx& c) {
    cudaStream_t s = c.stream;
    const int D = c.D, k = std::max(D - 2, 1);
    const i64 lo_k = c.base[k], hi_k = c.base[k + 1];
    float* w = dalloc<float>(hi_k - lo_k, s);
    double* sum = dalloc<double>(1, s);
    CK(cudaMemsetAsync(sum, 0, sizeof(double), s));
    dfree(c.point_weight, s);
    dfree(c.wnrm, s);
    c.point_weight = dalloc<float>(c.N, s);
    c.wnrm = dalloc<float>(3 * c.N, s);
    const int kt = c.kbegin("density_weights", (double)c.N * (12 + 12 + 4 + 12) + (double)(hi_k - lo_k) * 120);
    ensure_group_table(c);
    const i64 ngroups_all = (c.nodes.M - 1) / 8, gfirst = (lo_k - 1) / 8, ng = (hi_k - lo_k) / 8;
    float4* sw = dalloc<float4>(c.N * (SW_STRIDE / 4), s);
    int* ancestor = dalloc<int>(c.N, s);
    k_density_samples<<<grid_for(c.N, 128, 1ll << 30), 128, 0, s>>>(c.nodes, c.N, c.point_node, k, D, c.basis, c.pts,
                                                                    ancestor, sw);
    CK_LAUNCH();
    k_splat<false><<<grid_for(ng * 8, SPLAT_BLOCK, 1ll << 30), SPLAT_BLOCK, 0, s>>>(c.nodes, c.gn, ngroups_all, gfirst, ng,
                                                                                    lo_k, sw, w);
    CK_LAUNCH();
    k_density_points<<<grid_for(c.N, 128, (i64)c.sms * 32), 128, 0, s>>>(c.nodes.neigh, c.nodes.M, c.N, ancestor, lo_k, sw,
                                                                         w, c.point_weight, sum);
    CK_LAUNCH();
    dfree(ancestor, s);
    dfree(sw, s);
    k_weight_normals<<<grid_for(c.N, 256), 256, 0, s>>>(c.N, sum, c.nrm, c.point_weight, c.wnrm);
    CK_LAUNCH();
    c.kend(kt);
    dfree(w, s);
    dfree(sum, s);
}

void stage_splat(Ctx& c) {
    cudaStream_t s = c.stream;
    const int D = c.D;
    const i64 lo = c.base[D], hi = c.base[D + 1];
    dfree(c.vfield, s);
    c.vfield = dalloc<float>(3 * (hi - lo), s);
    const float* nrm = c.nrm;
    if (c.params.density_weights) {
        density_weights(c);
        nrm = c.wnrm;
    } else {
        dfree(c.point_weight, s);
        dfree(c.wnrm, s);
    }
    // compulsory: points+normals once, finest keys and neighbour tables, V written
    const int kt = c.kbegin("splat", (double)c.N * 24 + (double)(hi - lo) * (8 + 108 + 12));
    ensure_group_table(c);
    {
        const i64 ngroups_all = (c.nodes.M - 1) / 8, gfirst = (lo - 1) / 8, ng = (hi - lo) / 8;
        float4* sw = dalloc<float4>(c.N * (SW_STRIDE / 4), s);
        k_sample_weights<<<grid_for(c.N, 128, 1ll << 30), 128, 0, s>>>(c.nodes, D, c.basis_maxdepth, c.pts, nrm,
                                                                       c.point_node, c.N, sw, c.params.stable_basis);
        CK_LAUNCH();
        k_splat<true><<<grid_for(ng * 8, SPLAT_BLOCK, 1ll << 30), SPLAT_BLOCK, 0, s>>>(c.nodes, c.gn, ngroups_all, gfirst,
                                                                                       ng, lo, sw, c.vfield);
        CK_LAUNCH();
        dfree(sw, s);
    }
    c.kend(kt);
}

void stage_divergence(Ctx& c) {
    cudaStream_t s = c.stream;
    const int D = c.D;
    const i64 M = c.nodes.M, lo = c.base[D], nD = c.count[D];
    dfree(c.divergence, s);
    c.divergence = dalloc<float>(M, s);
    short4* fc = dalloc<short4>(nD, s);
    k_finest_coords<<<grid_for(nD, 256), 256, 0, s>>>(c.nodes.key, lo, nD, D, fc);
    CK_LAUNCH();
    i64* rs = dalloc<i64>(D + 2, s);
    CK(cudaMemcpyAsync(rs, c.ddot_row_start.data(), (D + 2) * sizeof(i64), cudaMemcpyHostToDevice, s));
    DivArgs a;
    a.D = D;
    a.M = M;
    a.vfield = c.vfield;
    a.fc = fc;
    a.rows = c.ddot_div;
    a.row_start = rs;
    // depths D and D-1: at most 27 and 216 terms per node
    const int split = D >= 1 ? D - 1 : 0;
    // compulsory: every node's key, depth, neighbours and b; V and coordinates of the finest slots
    const int kt = c.kbegin("divergence", (double)M * (8 + 1 + 108 + 4) + (double)nD * (12 + 8));
    // depth D - 1 by sibling groups (a depth-1 group hangs off the root; depth 0 has no group), depth D too
    const int ktg = c.kbegin("group_table", 0.0);
    ensure_group_table(c);
    c.kend(ktg);
    const int kt1 = c.kbegin("divergence_d1", 0.0);
    if (split >= 1) {
        const i64 ngroups_all = (M - 1) / 8, plo = c.base[split], png = (c.base[D] - plo) / 8;
        k_div_parents<<<grid_for(png * 8, 32 * DIV_PARENT_WARPS, 1ll << 30), 32 * DIV_PARENT_WARPS, 0, s>>>(
            c.nodes, a, c.gn, ngroups_all, (plo - 1) / 8, png, plo, lo, c.divergence);
        CK_LAUNCH();
    }
    c.kend(kt1);
    const int kt2 = c.kbegin("divergence_d", 0.0);
    {
        const i64 ngroups_all = (M - 1) / 8, gfirst = (lo - 1) / 8, ng = nD / 8;
        k_div_finest<<<grid_for(ng * 8, 256, (i64)c.sms * 8 * 8), 256, 0, s>>>(c.nodes, a, c.gn, ngroups_all, gfirst,
                                                                               ng, lo, c.divergence);
        CK_LAUNCH();
    }
    c.kend(kt2);
    const i64 nc = c.base[split];   // nodes at depths < D-1
    if (nc > 0) {
        // the root: its terms in chunks; depths 1..D-2: sibling groups in chunks
        const i64 ngroups_all = (M - 1) / 8, ngc = (nc - 1) / 8;
        int* nch = dalloc<int>(1 + ngc, s);
        int* first = dalloc<int>(1 + 1 + ngc + 1, s);
        int* gfirst = first + 2;
        k_div_count<<<1, 32, 0, s>>>(c.nodes, 1, nch);
        CK_LAUNCH();
        exclusive_scan<int, int>(nch, first, 1, first + 1, s);
        if (ngc > 0) {
            k_div_group_count<<<grid_for(ngc, 256), 256, 0, s>>>(c.nodes, c.gn, ngroups_all, ngc, nch + 1);
            CK_LAUNCH();
            exclusive_scan<int, int>(nch + 1, gfirst, ngc, gfirst + ngc, s);
        }
        int hroot = 0, hgroups = 0;
        CK(cudaMemcpyAsync(&hroot, first + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
        if (ngc > 0) CK(cudaMemcpyAsync(&hgroups, gfirst + ngc, sizeof(int), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        const i64 nroot = hroot, ngitems = hgroups;
        int* item_node = dalloc<int>(std::max<i64>(nroot + ngitems, 1), s);
        double* partial = dalloc<double>(std::max<i64>(nroot + 8 * ngitems, 1), s);
        const int ktr = c.kbegin("divergence_root", 0.0);
        if (nroot > 0) {
            k_div_items<<<1, 32, 0, s>>>(nch, first, 1, item_node);
            CK_LAUNCH();
            k_div_chunks<<<grid_for(nroot * 32, DIV_WARPS * 32, (i64)c.sms * 8), DIV_WARPS * 32, 0, s>>>(
                c.nodes, a, item_node, first, nroot, partial);
            CK_LAUNCH();
        }
        k_div_sum<<<1, 32, 0, s>>>(nch, first, partial, 0, 1, 1, c.divergence);
        CK_LAUNCH();
        c.kend(ktr);
        if (ngc > 0) {
            int* item_group = item_node + nroot;
            double* gpartial = partial + nroot;
            k_div_items<<<grid_for(ngc, 256), 256, 0, s>>>(nch + 1, gfirst, ngc, item_group);
            CK_LAUNCH();
            if (ngitems > 0) {
                const int kt3 = c.kbegin("divergence_groups", 0.0);
                k_div_groups<<<grid_for(ngitems * 32, DIV_WARPS * 32, (i64)c.sms * 256), DIV_WARPS * 32, 0, s>>>(
                    c.nodes, a, c.gn, ngroups_all, item_group, gfirst, ngitems, gpartial);
                CK_LAUNCH();
                c.kend(kt3);
            }
            // depths 1..3 (up to 584 nodes, thousands of chunks each at depths 1-2): a warp per
            // node; deeper nodes have few chunks: a thread per node
            const i64 wide = std::min<i64>(nc, c.base[std::min(4, D)]);
            k_div_sum<<<grid_for((wide - 1) * 32, 256), 256, 0, s>>>(nch + 1, gfirst, gpartial, 1, wide, 8,
                                                                     c.divergence);
            CK_LAUNCH();
            if (nc > wide) {
                k_div_sum_thread<<<grid_for(nc - wide, 256), 256, 0, s>>>(nch + 1, gfirst, gpartial, wide, nc, 8,
                                                                           c.divergence);
            }
            CK_LAUNCH();
        }
        dfree(nch, s);
        dfree(first, s);
        dfree(item_node, s);
        dfree(partial, s);
    }
    c.kend(kt);
    dfree(fc, s);
    dfree(rs, s);
}

}  // namespace prgpu
