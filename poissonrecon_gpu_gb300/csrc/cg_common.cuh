// Definitions shared by the plain (solve.cu) and the flexible (flexcg.cu)
// persistent CG kernels: per-depth partition state, the per-depth stencil
// description, compensated partial sums, and sums over warps and grids.
#pragma once
#include "common.cuh"

namespace prgpu {

constexpr int CG_BLOCK = 256;

struct PartState {          // one per depth, in global memory, zero-initialised
    int iters;
    float rr;
    int status;
    int refines;            // true-residual refinements taken
    double bb;              // b.b (FP64 reduction)
    double rr_true;         // |b - Ax|^2 with FP64 accumulation (-1: not computed)
};

struct CgDepth {
    i64 lo, n;              // global row range
    int first_block, nblocks;
    float st[27];
    // The Laplacian stencil is symmetric under the reflections and permutations of the
    // axes (a product of symmetric 1-D tables), so entry j depends only on how many of
    // its offsets are nonzero: cls[0] centre, [1] faces, [2] edges, [3] corners.  sym = 1
    // when the float entries are exactly so; the matrix-vector product then keeps the
    // four values in registers (the same values in the same FMA order).
    float cls[4];
    int sym;
};

// Shared-memory layout of a tile of 4 sibling groups' 4x4x4 blocks in the matrix-vector
// product.  For each stencil entry the lanes of a warp read the 8 children of 4 groups,
// at cell offsets {0,1,4,5,16,17,20,21} plus a constant from the group's block start;
// group gl's block starts 0, 2, 8 or 10 words past a multiple of 32, so the 32 reads fall
// in 32 distinct banks (with blocks 64 words apart, 4 groups hit the same banks).
constexpr int CG_TILE_WORDS = 272;
__host__ __device__ constexpr int cg_block_base(int gl) { return gl * 66 + (gl >> 1) * 4; }

__host__ __device__ constexpr int stencil_class(int j) {
    return (j / 9 != 1) + ((j / 3) % 3 != 1) + (j % 3 != 1);
}

// ---------------------------------------------------------------------------
// Sums over a warp without the FP64 pipe.  It does 2 additions a cycle and SM at a latency of over 60
// cycles, so a butterfly of doubles in each warp of a block, five blocks an SM, costs microseconds per
// reduction; a solve does two reductions an iteration.  Here the lanes' values are aligned to the
// largest exponent as 58-bit integers (one REDUX), split in limbs of 24 bits that 32 lanes cannot
// overflow, and added by three more REDUX.  What alignment drops is below 2^-57 of the largest value's
// power of two per lane, 2^-52 of it in all: two roundings of a double addition at most.  The sum is then
// rounded once to a double.  Values that are not finite or whose sum may not be (exponent field from
// 0x7fa), and tiny ones (below 64), take the butterfly.  Every lane gets the result.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum_butterfly(double v) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// the sum of the lanes' x (|x| < 2^58) times 2^q, rounded to nearest; q + 1086 within 64..2046
__device__ __forceinline__ double warp_sum_aligned(i64 x, int q) {
    const int lo = __reduce_add_sync(0xffffffffu, (int)(x & 0xffffff));
    const int mid = __reduce_add_sync(0xffffffffu, (int)((x >> 24) & 0xffffff));
    const int hi = __reduce_add_sync(0xffffffffu, (int)(x >> 48));
    const i64 S = ((i64)hi << 48) + ((i64)mid << 24) + (i64)lo;
    if (S == 0) return 0.0;
    u64 u = S < 0 ? (u64)(-S) : (u64)S;
    const int lz = __clzll((i64)u);
    u <<= lz;
    // the carry of the rounding moves into the exponent, as it should
    const u64 bits = ((u64)(1023 + 63 - lz + q) << 52) + ((u >> 11) & 0xfffffffffffffull) + ((u >> 10) & 1ull);
    return __longlong_as_double((i64)(bits | (S < 0 ? 0x8000000000000000ull : 0ull)));
}
__device__ __forceinline__ double warp_sum(double v) {
    const u64 b = (u64)__double_as_longlong(v);
    const int e = (int)(b >> 52) & 0x7ff;
    const int emax = __reduce_max_sync(0xffffffffu, e);
    if (emax < 64 || emax >= 0x7fa) {
        if (!__any_sync(0xffffffffu, v != 0.0)) return 0.0;
        return warp_sum_butterfly(v);
    }
    const u64 m = e ? ((b & 0xfffffffffffffull) | 0x10000000000000ull) : 0ull;
    const i64 x = (i64)((m << 5) >> min(emax - e, 63));
    return warp_sum_aligned((i64)b < 0 ? -x : x, emax - 1080);
}

// per-thread partial dot product: a compensated float pair (Neumaier), exact to
// about 2u|sum| + n u^2 sum|term| -- FP64 accuracy for a thread's few dozen rows
// without FP64 arithmetic per row
struct FSum {
    float h = 0.f, l = 0.f;
    __device__ __forceinline__ void add(float v) {
        const float t = h + v;
        l += (fabsf(h) >= fabsf(v)) ? (h - t) + v : (v - t) + h;
        h = t;
    }
    __device__ __forceinline__ double value() const { return (double)h + (double)l; }
};
// the pairs' 24-bit mantissas aligned to the largest exponent with 33 bits below: below 2^-56 of the largest
// float's power of two is dropped per float, 2^-50 of it in all 64
__device__ __forceinline__ double warp_sum(const FSum& v) {
    const unsigned bh = __float_as_uint(v.h), bl = __float_as_uint(v.l);
    const int eh = (int)(bh >> 23) & 255, el = (int)(bl >> 23) & 255;
    const int emax = max(__reduce_max_sync(0xffffffffu, max(eh, el)), 1);
    if (emax == 255) return warp_sum_butterfly(v.value());
    auto fixed = [&](unsigned b, int e) {
        const u64 m = (b & 0x7fffffu) | (e ? 0x800000u : 0u);
        const i64 x = (i64)((m << 33) >> min(emax - max(e, 1), 63));
        return (b >> 31) ? -x : x;
    };
    return warp_sum_aligned(fixed(bh, eh) + fixed(bl, el), emax - 183);
}

// ---------------------------------------------------------------------------
// Sum of NV values over the blocks of a partition of co-resident blocks, which is also the partition's
// barrier: what a block wrote before the sum is visible to every block after it.
//
// An iteration of a small system is mostly this latency.  A block publishes its partial together with
// the sum's number (epoch) and every block reads all partials at once: publish and read, two trips to
// L2, where an arrival counter, a last block that sums and a generation word that the others poll take
// five.  A 64-bit word holds the epoch and half of the double, so a reader knows from the words
// themselves that both halves belong to this sum, without a flag behind the data.  Two sets of slots
// alternate: a block publishes epoch e + 2 only after every block published e + 1, hence after every
// block read e.  Partitions of more than GS_ALL blocks would poll nblocks^2 slots, so there rank 0 sums
// the partials and publishes the result (63 blocks: 6.3 K cycles a sum against 8.7 K with rank 0; 184 and
// 503 blocks beside others on their SMs: 14 K against 10-11 K).  Sums run in a fixed order, independent of arrival.
//
// data = false: the sum does not have to make the blocks' writes visible to each other, so it takes no
// fences (about a microsecond each with stores in flight).  It still orders the blocks' reads before the
// others' later writes: what a block publishes depends on every value it read.
//
// Waits poll at most spin_limit times; on expiry (or when another block gave up) the error flag is
// set and false returned.  extra = 1 (a test hook) waits for one block more than the partition has:
// that slot, behind the last block's, is never written.
// ---------------------------------------------------------------------------
constexpr int GS_ALL = 64;              // largest partition whose blocks read every partial
struct GridSum {
    u64* slots;                         // grid_sum_words words, zeroed before the launch
    int cap;                            // slots per set: launched blocks, partitions' results, one never written
    int first, nblocks, rank;           // this partition
    int result;                         // slot of the partition's result
    int* err;
    long long spin_limit;
    int extra;
};
__host__ __device__ constexpr i64 grid_sum_words(int cap, int nv) { return 4ll * cap * nv; }

__device__ __forceinline__ void gs_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void gs_publish(u64* w, double v, unsigned epoch) {
    const u64 e = (u64)epoch << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(e | (unsigned)__double2loint(v)),
                 "l"(e | (unsigned)__double2hiint(v))
                 : "memory");
}
// one slot of NV values, published with this epoch; false when the wait gave up
template <int NV>
__device__ __forceinline__ bool gs_read(const GridSum& g, const u64* w, unsigned epoch, double* v) {
    long long spins = 0;
    for (;;) {
        u64 a[NV], b[NV];
        bool all = true;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                         : "=l"(a[j]), "=l"(b[j])
                         : "l"(w + 2 * j)
                         : "memory");
            all &= (unsigned)(a[j] >> 32) == epoch && (unsigned)(b[j] >> 32) == epoch;
        }
        if (all) {
#pragma unroll
            for (int j = 0; j < NV; ++j) v[j] = __hiloint2double((int)(unsigned)b[j], (int)(unsigned)a[j]);
            return true;
        }
        ++spins;
        if (spins > g.spin_limit || ((spins & 15) == 0 && *(volatile int*)g.err)) {
            atomicExch(g.err, PRGPU_ERR_TIMEOUT);
            return false;
        }
        __nanosleep(20);
    }
}

// shared memory of a block's grid_sum calls, by the parity of the epoch
template <int NV>
struct GridSumShared {
    double part[2][NV][32];             // the block's warps
    double all[2][NV][32];              // the warps that read slots
};

// The sum in two calls, so that work that needs neither its result nor other blocks' data runs while
// the partials travel.  grid_publish: v (per thread) summed over the block and published.  grid_collect:
// every thread gets the partition's sums in out.  The block has a multiple of 32 threads.
template <int NV, class V>
__device__ __forceinline__ void grid_publish(const GridSum& g, unsigned epoch, bool data, const V (&v)[NV],
                                             GridSumShared<NV>& sm) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, par = epoch & 1;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const double s = warp_sum(v[j]);
        if (lane == 0) sm.part[par][j][w] = s;
    }
    __syncthreads();
    if (g.nblocks + g.extra > 1 && w == 0) {
        double s[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) s[j] = warp_sum(lane < nw ? sm.part[par][j][lane] : 0.0);
        if (lane == 0) {
            u64* set = g.slots + par * (2ll * g.cap * NV);
            if (data) gs_fence();
#pragma unroll
            for (int j = 0; j < NV; ++j) gs_publish(set + 2ll * NV * (g.first + g.rank) + 2 * j, s[j], epoch);
        }
    }
}
template <int NV>
__device__ __forceinline__ bool grid_collect(const GridSum& g, unsigned epoch, bool data, GridSumShared<NV>& sm,
                                             double (&out)[NV]) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5, par = epoch & 1;
    u64* set = g.slots + par * (2ll * g.cap * NV);
    auto slot = [&](int k) { return set + 2ll * NV * k; };
    const int ne = g.nblocks + g.extra;
    if (ne == 1) {   // the sums of one block: every warp adds the warps' values
#pragma unroll
        for (int j = 0; j < NV; ++j) out[j] = warp_sum(lane < nw ? sm.part[par][j][lane] : 0.0);
        return true;
    }
    bool ok = true;
    const bool sums = ne <= GS_ALL || g.rank == 0;
    const int rw = sums ? min(nw, (ne + 31) >> 5) : 1;   // warps that read
    if (w < rw) {
        double u[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) u[j] = 0.0;
        if (sums) {
            for (int k = tid; k < ne && ok; k += blockDim.x) {
                double t[NV];
                ok = gs_read<NV>(g, slot(k < g.nblocks ? g.first + k : g.cap - 1), epoch, t);
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    if (ok) u[j] = (k == tid) ? t[j] : u[j] + t[j];
            }
        } else if (lane == 0) {
            ok = gs_read<NV>(g, slot(g.result), epoch, u);
        }
        if (data) gs_fence();
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const double s = sums ? warp_sum(u[j]) : u[j];
            if (lane == 0) sm.all[par][j][w] = s;
        }
    }
    ok = __syncthreads_and(ok);
    if (!ok) return false;
#pragma unroll
    for (int j = 0; j < NV; ++j) out[j] = sums ? warp_sum(lane < rw ? sm.all[par][j][lane] : 0.0) : sm.all[par][j][0];
    if (ne > GS_ALL && g.rank == 0 && tid == 0) {
        if (data) gs_fence();
#pragma unroll
        for (int j = 0; j < NV; ++j) gs_publish(slot(g.result) + 2 * j, out[j], epoch);
    }
    return true;
}
template <int NV, class V>
__device__ __forceinline__ bool grid_sum(const GridSum& g, unsigned epoch, bool data, const V (&v)[NV],
                                         GridSumShared<NV>& sm, double (&out)[NV]) {
    grid_publish(g, epoch, data, v, sm);
    return grid_collect(g, epoch, data, sm, out);
}

}  // namespace prgpu
