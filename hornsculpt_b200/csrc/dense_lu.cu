// Batched dense complex LU with partial pivoting, triangular solves and the
// FP64 refinement residual (cuda_solver.cu:1485-1581). The plain form
// factors in FP64; the mixed form factors an FP32 copy and refines in FP64
// (the reference factors in FP32 with cuSOLVER getrf/getrs).
//
// Matrices are column-major N x N complex (interleaved reals), one per
// frequency of the batch (blockIdx.y / blockIdx.z). Right-looking blocked LU in
// two levels: 32-wide panels in the registers of a thread-block cluster update
// the rest of their outer block, whose U rows are then solved at once and the
// trailing matrix updated once, in FP64 by the FP64 matrix instruction, in FP32
// by the tensor cores (3xTF32).
#include "device_once.hpp"
#include "device_types.cuh"
#include "kernel_timer.hpp"

#include <cooperative_groups.h>

#include <algorithm>
#include <stdexcept>
#include <string>
#include <vector>

namespace hsb {
namespace {

constexpr int kPanel = 32;

void check(cudaError_t e, const char *what) {
    if (e != cudaSuccess)
        throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

// complex element type of a real type
template <class R> struct Cx;
template <> struct Cx<double> {
    using type = double2;
};
template <> struct Cx<float> {
    using type = float2;
};
template <class R> using C2 = typename Cx<R>::type;
template <class R> __device__ __forceinline__ C2<R> mk(R x, R y) {
    C2<R> v;
    v.x = x;
    v.y = y;
    return v;
}
template <class R> __device__ __forceinline__ C2<R> ld2(const R *p) { return *reinterpret_cast<const C2<R> *>(p); }
template <class R> __device__ __forceinline__ void st2(R *p, C2<R> v) { *reinterpret_cast<C2<R> *>(p) = v; }
template <class R> __device__ __forceinline__ C2<R> cmul(C2<R> a, C2<R> b) {
    return mk<R>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// v -= a * b
template <class R> __device__ __forceinline__ void csub(C2<R> &v, C2<R> a, C2<R> b) {
    v.x -= a.x * b.x - a.y * b.y;
    v.y -= a.x * b.y + a.y * b.x;
}
template <> __device__ __forceinline__ void csub<double>(double2 &v, double2 a, double2 b) {  // four FP64 instructions, not six
    v.x = fma(a.y, b.y, fma(-a.x, b.x, v.x));
    v.y = fma(-a.y, b.x, fma(-a.x, b.y, v.y));
}

// Panel factorisation of columns [k0, k0+jb) over rows [k0, N) of one matrix.
template <class R>
__global__ void __launch_bounds__(512) panelKernel(R *LU, uint32_t N, uint32_t k0, uint32_t jb, int *pivots,
                                                   int *info) {
    R *M = LU + size_t(blockIdx.x) * N * N * 2;
    int *piv = pivots + size_t(blockIdx.x) * N;
    __shared__ R sVal[16];
    __shared__ int sIdx[16];
    __shared__ C2<R> sRow[kPanel];
    __shared__ int sPivot;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (uint32_t j = 0; j < jb; ++j) {
        const uint32_t c = k0 + j;
        // argmax |re|+|im| over rows [c, N), first index on ties
        R best = -1;
        int bestRow = int(c);
        for (uint32_t i = c + threadIdx.x; i < N; i += blockDim.x) {
            const C2<R> v = ld2(M + 2 * (size_t(c) * N + i));
            const R a = fabs(v.x) + fabs(v.y);
            if (a > best) {
                best = a;
                bestRow = int(i);
            }
        }
        for (int off = 16; off > 0; off >>= 1) {
            const R ob = __shfl_down_sync(0xffffffffu, best, off);
            const int oi = __shfl_down_sync(0xffffffffu, bestRow, off);
            if (ob > best || (ob == best && oi < bestRow)) {
                best = ob;
                bestRow = oi;
            }
        }
        if (lane == 0) {
            sVal[warp] = best;
            sIdx[warp] = bestRow;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            R b = sVal[0];
            int bi = sIdx[0];
            for (int w = 1; w < warps; ++w)
                if (sVal[w] > b || (sVal[w] == b && sIdx[w] < bi)) {
                    b = sVal[w];
                    bi = sIdx[w];
                }
            sPivot = bi;
            piv[c] = bi;
            if (!(b > 0) && *info == 0)
                atomicCAS(info, 0, int(c) + 1);
        }
        __syncthreads();
        const int p = sPivot;
        if (threadIdx.x < jb && p != int(c)) {
            R *a = M + 2 * (size_t(k0 + threadIdx.x) * N + c);
            R *b = M + 2 * (size_t(k0 + threadIdx.x) * N + p);
            const C2<R> va = ld2(a), vb = ld2(b);
            st2(a, vb);
            st2(b, va);
        }
        __syncthreads();
        if (threadIdx.x < jb)
            sRow[threadIdx.x] = ld2(M + 2 * (size_t(k0 + threadIdx.x) * N + c));
        __syncthreads();
        const C2<R> d = sRow[j];
        const R den = d.x * d.x + d.y * d.y;
        const C2<R> inv = den > 0 ? mk<R>(d.x / den, -d.y / den) : mk<R>(0, 0);
        for (uint32_t i = c + 1 + threadIdx.x; i < N; i += blockDim.x) {
            R *col = M + 2 * (size_t(c) * N + i);
            const C2<R> l = cmul<R>(ld2(col), inv);
            st2(col, l);
            for (uint32_t q = j + 1; q < jb; ++q) {
                R *e = M + 2 * (size_t(k0 + q) * N + i);
                C2<R> v = ld2(e);
                csub<R>(v, l, sRow[q]);
                st2(e, v);
            }
        }
        __syncthreads();
    }
}

// Panel factorisation for tall panels, spread over a thread-block cluster:
// CTA r of the cluster owns panel rows [r * rowsPerBlock, ...). The first
// `cap` of them live in shared memory, one per thread; the rest (at most
// kGlobalSlots per thread) stay in place in global memory and are eliminated
// there by their thread. Pivot choice, tie rule and interchange sequence are
// those of panelRegKernel. Per column: each warp's best candidate goes to its
// CTA's shared memory (double-buffered by column parity); one cluster barrier;
// every warp reduces the candidates of all CTAs through distributed shared
// memory; one warp per CTA copies the pivot row from the CTA that holds it
// (distributed shared memory, or global memory for a row kept there); each
// CTA eliminates its own rows. Rows that are pivots never change again, so
// reading them remotely needs no further barrier. Write-back: a row kept in
// global memory moves only when it is a pivot, to one of the first jb
// positions, whose own rows are in CTA 0's shared memory; such rows are copied
// first, and after a cluster barrier the shared-memory rows are written to
// their final positions. A final cluster barrier keeps every CTA's shared
// memory alive until all remote reads are done.
template <class R> constexpr uint32_t kClusterRows = sizeof(R) == 8 ? 384 : 768;
constexpr int kGlobalSlots = 4;

template <class R> struct ClusterPanelShared {
    R best[32];
    int idx[32];
    R ctaBest[2];  // this CTA's candidate per column parity
    int ctaIdx[2];
    C2<R> pivot[kPanel];
    int sel[kPanel];
    int mapRow[2 * kPanel], mapPos[2 * kPanel];
    int mapCount;
};

template <class R>
__global__ void __launch_bounds__(1024) panelClusterKernel(R *LU, uint32_t N, uint32_t k0, uint32_t jb,
                                                           uint32_t rowsPerBlock, uint32_t cap, int *pivots,
                                                           int *info) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char rawSmem[];
    __shared__ ClusterPanelShared<R> sh;
    C2<R> *P = reinterpret_cast<C2<R> *>(rawSmem);  // [jb][cap]
    const uint32_t rank = cluster.block_rank(), C = cluster.num_blocks();
    const uint32_t rows = N - k0, rowBegin = rank * rowsPerBlock;
    const uint32_t myRows = rowBegin < rows ? min(rowsPerBlock, rows - rowBegin) : 0u;
    R *M = LU + size_t(blockIdx.y) * N * N * 2;
    int *piv = pivots + size_t(blockIdx.y) * N;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = int(blockDim.x >> 5);
    const uint32_t i = threadIdx.x;
    // slot 0: shared-memory row i; slot s >= 1: global row cap + (s - 1) * blockDim + i
    const auto local = [&](int s) { return s == 0 ? i : cap + uint32_t(s - 1) * blockDim.x + i; };
    const auto owns = [&](int s) { return s == 0 ? (i < cap && i < myRows) : local(s) < myRows; };
    const auto column = [&](uint32_t q) { return M + 2 * (size_t(k0 + q) * N + k0); };  // panel column q
    constexpr int kLoad = sizeof(R) == 8 ? 4 : 8;
    if (owns(0))
        for (uint32_t q0 = 0; q0 < jb; q0 += kLoad) {
            C2<R> v[kLoad];
#pragma unroll
            for (int t = 0; t < kLoad; ++t)
                if (q0 + t < jb)
                    v[t] = ld2(column(q0 + t) + 2 * (rowBegin + i));
#pragma unroll
            for (int t = 0; t < kLoad; ++t)
                if (q0 + t < jb)
                    P[size_t(q0 + t) * cap + i] = v[t];
        }
    const auto magnitude = [](C2<R> z) {
        const R a = fabs(z.x) + fabs(z.y);
        return a >= R(0) ? a : R(0);  // a NaN row competes as zero, so a pivot row always exists
    };
    bool taken[1 + kGlobalSlots];
    R best = R(-1);
    int bestRow = int(rows);
#pragma unroll
    for (int s = 0; s <= kGlobalSlots; ++s) {
        taken[s] = !owns(s);
        if (!taken[s]) {
            const uint32_t g = rowBegin + local(s);
            const R m = magnitude(s == 0 ? P[i] : ld2(column(0) + 2 * g));
            if (m > best || (m == best && int(g) < bestRow)) {
                best = m;
                bestRow = int(g);
            }
        }
    }
    for (uint32_t j = 0; j < jb; ++j) {
        const int buf = j & 1;
        for (int off = 16; off > 0; off >>= 1) {
            const R ob = __shfl_xor_sync(0xffffffffu, best, off);
            const int oi = __shfl_xor_sync(0xffffffffu, bestRow, off);
            if (ob > best || (ob == best && oi < bestRow)) {
                best = ob;
                bestRow = oi;
            }
        }
        if (lane == 0) {
            sh.best[warp] = best;
            sh.idx[warp] = bestRow;
        }
        __syncthreads();
        if (warp == 0) {  // this CTA's candidate
            R b = lane < W ? sh.best[lane] : R(-1);
            int r = lane < W ? sh.idx[lane] : int(rows);
            for (int off = 16; off > 0; off >>= 1) {
                const R ob = __shfl_xor_sync(0xffffffffu, b, off);
                const int oi = __shfl_xor_sync(0xffffffffu, r, off);
                if (ob > b || (ob == b && oi < r)) {
                    b = ob;
                    r = oi;
                }
            }
            if (lane == 0) {
                sh.ctaBest[buf] = b;
                sh.ctaIdx[buf] = r;
            }
        }
        cluster.sync();
        // the candidates of all CTAs, one per lane, read through distributed shared memory
        R pb = R(-1);
        int p = int(rows);
        if (uint32_t(lane) < C) {
            const ClusterPanelShared<R> *other = cluster.map_shared_rank(&sh, lane);
            pb = other->ctaBest[buf];
            p = other->ctaIdx[buf];
        }
        for (int off = 16; off > 0; off >>= 1) {
            const R ob = __shfl_xor_sync(0xffffffffu, pb, off);
            const int oi = __shfl_xor_sync(0xffffffffu, p, off);
            if (ob > pb || (ob == pb && oi < p)) {
                pb = ob;
                p = oi;
            }
        }
        if (warp == 0) {
            // copy the pivot row (columns j.. of panel row p) from the CTA that holds it
            const uint32_t owner = uint32_t(p) / rowsPerBlock, at = uint32_t(p) % rowsPerBlock;
            if (uint32_t(lane) >= j && uint32_t(lane) < jb) {
                if (at < cap)
                    sh.pivot[lane] = cluster.map_shared_rank(P, int(owner))[size_t(lane) * cap + at];
                else
                    sh.pivot[lane] = ld2(column(lane) + 2 * uint32_t(p));
            }
            if (rank == 0 && lane == 0) {
                sh.sel[j] = p;
                if (!(pb > 0) && *info == 0)
                    atomicCAS(info, 0, int(k0 + j) + 1);
            }
        }
        __syncthreads();
        const C2<R> d = sh.pivot[j];
        const R den = d.x * d.x + d.y * d.y;
        const R rden = den > 0 ? R(1) / den : R(0);
        const C2<R> inv = mk<R>(d.x * rden, -d.y * rden);
        best = -1;
        bestRow = int(rows);
#pragma unroll
        for (int s = 0; s <= kGlobalSlots; ++s) {
            if (taken[s])
                continue;
            const uint32_t g = rowBegin + local(s);
            if (int(g) == p) {
                taken[s] = true;
                continue;
            }
            C2<R> next = mk<R>(0, 0);
            if (s == 0) {
                const C2<R> l = cmul<R>(P[size_t(j) * cap + i], inv);
                P[size_t(j) * cap + i] = l;
                for (uint32_t q0 = j + 1; q0 < jb; q0 += kLoad) {
                    C2<R> v[kLoad];
#pragma unroll
                    for (int t = 0; t < kLoad; ++t)
                        if (q0 + t < jb)
                            v[t] = P[size_t(q0 + t) * cap + i];
#pragma unroll
                    for (int t = 0; t < kLoad; ++t)
                        if (q0 + t < jb) {
                            csub<R>(v[t], l, sh.pivot[q0 + t]);
                            P[size_t(q0 + t) * cap + i] = v[t];
                        }
                    if (q0 == j + 1)
                        next = v[0];
                }
            } else {
                const C2<R> l = cmul<R>(ld2(column(j) + 2 * g), inv);
                st2(column(j) + 2 * g, l);
                for (uint32_t q0 = j + 1; q0 < jb; q0 += kLoad) {
                    C2<R> v[kLoad];
#pragma unroll
                    for (int t = 0; t < kLoad; ++t)
                        if (q0 + t < jb)
                            v[t] = ld2(column(q0 + t) + 2 * g);
#pragma unroll
                    for (int t = 0; t < kLoad; ++t)
                        if (q0 + t < jb) {
                            csub<R>(v[t], l, sh.pivot[q0 + t]);
                            st2(column(q0 + t) + 2 * g, v[t]);
                        }
                    if (q0 == j + 1)
                        next = v[0];
                }
            }
            if (j + 1 < jb) {
                const R m = magnitude(next);
                if (m > best || (m == best && int(g) < bestRow)) {
                    best = m;
                    bestRow = int(g);
                }
            }
        }
    }
    cluster.sync();
    // Interchange sequence and the final position of every row that moved, by warp 0 of
    // rank 0: the (row, position) pairs of the moved rows live in lane registers, two per
    // lane (at most 2 * jb), and each lookup is one ballot.
    if (rank == 0 && warp == 0) {
        int rowA = -1, posA = 0, rowB = -1, posB = 0;  // slots lane and lane + 32
        int n = 0;
        const auto whereOf = [&](int row) {  // current position of a row
            const unsigned a = __ballot_sync(0xffffffffu, rowA == row), b = __ballot_sync(0xffffffffu, rowB == row);
            if (a)
                return __shfl_sync(0xffffffffu, posA, __ffs(a) - 1);
            if (b)
                return __shfl_sync(0xffffffffu, posB, __ffs(b) - 1);
            return row;
        };
        const auto rowAt = [&](int pos) {  // row currently at a position
            const unsigned a = __ballot_sync(0xffffffffu, rowA >= 0 && posA == pos);
            const unsigned b = __ballot_sync(0xffffffffu, rowB >= 0 && posB == pos);
            if (a)
                return __shfl_sync(0xffffffffu, rowA, __ffs(a) - 1);
            if (b)
                return __shfl_sync(0xffffffffu, rowB, __ffs(b) - 1);
            return pos;
        };
        const auto setWhere = [&](int row, int pos) {
            const unsigned a = __ballot_sync(0xffffffffu, rowA == row), b = __ballot_sync(0xffffffffu, rowB == row);
            if (a) {
                if (lane == __ffs(a) - 1)
                    posA = pos;
            } else if (b) {
                if (lane == __ffs(b) - 1)
                    posB = pos;
            } else {
                if (n < 32 && lane == n) {
                    rowA = row;
                    posA = pos;
                } else if (n >= 32 && lane == n - 32) {
                    rowB = row;
                    posB = pos;
                }
                ++n;
            }
        };
        for (uint32_t j = 0; j < jb; ++j) {
            const int r = sh.sel[j], pj = whereOf(r), rj = rowAt(int(j));
            if (lane == 0)
                piv[k0 + j] = int(k0) + pj;
            setWhere(r, int(j));
            setWhere(rj, pj);
        }
        const unsigned a = __ballot_sync(0xffffffffu, rowA >= 0 && rowA != posA);
        const unsigned b = __ballot_sync(0xffffffffu, rowB >= 0 && rowB != posB);
        const unsigned below = (1u << lane) - 1u;
        if (a >> lane & 1u) {
            sh.mapRow[__popc(a & below)] = rowA;
            sh.mapPos[__popc(a & below)] = posA;
        }
        if (b >> lane & 1u) {
            sh.mapRow[__popc(a) + __popc(b & below)] = rowB;
            sh.mapPos[__popc(a) + __popc(b & below)] = posB;
        }
        if (lane == 0)
            sh.mapCount = __popc(a) + __popc(b);
    }
    cluster.sync();
    if (rank != 0) {  // a local copy of rank 0's map
        const ClusterPanelShared<R> *root = cluster.map_shared_rank(&sh, 0);
        for (uint32_t q = threadIdx.x; q < 2 * kPanel; q += blockDim.x) {
            sh.mapRow[q] = root->mapRow[q];
            sh.mapPos[q] = root->mapPos[q];
        }
        if (threadIdx.x == 0)
            sh.mapCount = root->mapCount;
    }
    __syncthreads();
    const int moved = sh.mapCount;
    const auto finalPosition = [&](uint32_t g) {
        uint32_t pos = g;
        for (int q = 0; q < moved; ++q)
            if (sh.mapRow[q] == int(g))
                pos = uint32_t(sh.mapPos[q]);
        return pos;
    };
    // pivots kept in global memory move to their positions (< jb; those rows are in CTA 0's shared memory)
#pragma unroll
    for (int s = 1; s <= kGlobalSlots; ++s)
        if (owns(s)) {
            const uint32_t g = rowBegin + local(s), pos = finalPosition(g);
            if (pos != g)
                for (uint32_t q = 0; q < jb; ++q)
                    st2(column(q) + 2 * pos, ld2(column(q) + 2 * g));
        }
    cluster.sync();
    if (owns(0)) {
        const uint32_t g = rowBegin + i, pos = finalPosition(g);
        for (uint32_t q = 0; q < jb; ++q)
            st2(column(q) + 2 * pos, P[size_t(q) * cap + i]);
    }
    cluster.sync();  // keep rank 0's map alive until every CTA has read it
}

// Panel factorisation in registers: the panel's rows are spread over a cluster
// of at most kMaxCluster CTAs (one for small matrices), one row per thread, two
// in FP32 where one does not reach (panelShape). Pivot rule: largest
// |re| + |im|, the lowest row on ties, a NaN row competes as zero; rows stay in
// place until the end, where the selection order becomes the LAPACK
// interchange sequence.
//
// Bound: the chain of 32 columns, each a maximum over all rows, the pivot row's
// way to every thread and the elimination. So:
//   * The panel is factored in two halves of 16 columns. A row's 16 values stay
//     in registers and the elimination reads nothing but the pivot row
//     (elimination in shared memory moved every remaining entry twice per
//     column). Before the right half, its 16 pivot rows are solved with the
//     left half's multipliers and every other row gets the left half's update
//     in one pass. Each entry sees the operations of a 32-column right-looking
//     elimination in the same order.
//   * A column costs one block barrier and one cluster barrier: warps find their
//     best row with integer reductions on the magnitude's bits (while the other
//     columns' updates are still in flight), and its lane publishes the row;
//     after the block barrier every warp finds the CTA's winner, and the warps
//     push it to the CTAs of the cluster; after the cluster barrier each CTA has
//     all candidates in its own shared memory. Candidate slots alternate with
//     the column's parity: a slot is written again only after the barrier of
//     the next column, which its readers have passed.
//   * Register indices must be constants, and 16 unrolled columns are too long
//     for the instruction cache, so the loop body handles kPanelUnroll columns
//     and rotates the rows by that many: at column j of a half, a[r][c] holds
//     its column j + c for c < 16 - j, and the finished columns after them.
// The pushes of a column precede its cluster barrier and nothing is read
// remotely after the last one, so a CTA may exit on its own.
//
// Measured, all panels of a solve, against panels in shared memory (one CTA or
// cluster) and 32-column register panels of one CTA. FP64: N = 258 0.56 -> 0.32
// ms, N = 642 x 32 1.78 -> 1.00, N = 2562 x 2 8.9 -> 4.6, N = 6380 28.1 -> 13.6.
// FP32: N = 642 x 32 1.00 -> 0.82, N = 4023 x 3 13.2 -> 6.4, N = 6380 22.3 ->
// 11.0. Of a column's 1.7 us at 15 CTAs about 0.7 are the push and the cluster
// barrier, 0.3 the reductions within the CTA, 0.3 the candidate, 0.2 the updates.
constexpr int kHalf = 16;
constexpr int kPanelUnroll = 2;
constexpr uint32_t kPanelThreads = 512;  // at most
constexpr int kPanelWarps = int(kPanelThreads / 32);
constexpr uint32_t kMaxCluster = 16;
// Row moves of one panel: entry q < 32 the panel row that goes to position q,
// entry 32 + r the position of panel row r when it is no pivot row and moves (else -1).
constexpr int kMoves = 2 * kPanel;

// Order-preserving key of a magnitude (non-negative), zero for "no row".
struct PivotKey {
    unsigned hi = 0, lo = 0;
};
__device__ __forceinline__ PivotKey pivotKey(double m) {
    return {unsigned(__double2hiint(m)) + 1u, unsigned(__double2loint(m))};
}
__device__ __forceinline__ PivotKey pivotKey(float m) { return {__float_as_uint(m) + 1u, 0u}; }
__device__ __forceinline__ bool zeroKey(PivotKey k) { return k.hi <= 1u && k.lo == 0u; }

// The largest key of the warp and the lowest row that has it; true in the lanes that hold it.
template <class R> __device__ __forceinline__ bool warpPivot(PivotKey &key, int &row) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, key.hi);
    bool mine = key.hi == hi;
    unsigned lo = 0;
    if constexpr (sizeof(R) == 8) {
        lo = __reduce_max_sync(0xffffffffu, mine ? key.lo : 0u);
        mine = mine && key.lo == lo;
    }
    const int lowest = __reduce_min_sync(0xffffffffu, mine ? row : 0x7fffffff);
    mine = mine && row == lowest;
    key = {hi, lo};
    row = lowest;
    return mine;
}

template <class R> struct PanelShared {
    __align__(16) C2<R> warpRow[2][kPanelWarps][kHalf];  // per warp: its candidate's remaining columns
    __align__(16) C2<R> ctaRow[2][kMaxCluster][kHalf];   // per CTA of the cluster, pushed by it
    __align__(16) C2<R> own[kHalf][kPanel];              // left pivot rows of this CTA: multipliers, right half
    __align__(16) C2<R> top[kHalf][kPanel];              // all left pivot rows, then their solved right half
    int4 warpKey[2][kPanelWarps];
    int4 ctaKey[2][kMaxCluster];  // (hi, lo, row, 0)
    int sel[kPanel], position[kPanel];
};

template <class R, int RT>
__global__ void __launch_bounds__(kPanelThreads, 1) panelRegKernel(R *LU, uint32_t N, uint32_t k0, uint32_t jb,
                                                                   uint32_t perBlock, int *pivots, int *moves,
                                                                   int *info) {
    namespace cg = cooperative_groups;
    constexpr int U = kPanelUnroll;
    static_assert(kHalf % U == 0 && kPanel == 2 * kHalf, "the column groups must tile the halves");
    extern __shared__ __align__(16) unsigned char rawSmem[];
    C2<R> *left = reinterpret_cast<C2<R> *>(rawSmem);  // [kHalf][perBlock]: the finished left half
    __shared__ PanelShared<R> sh;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), C = cluster.num_blocks();
    // a CTA's shared memory may be written by the others only once it runs: arrive
    // here, wait before the first push
    if (C > 1)
        cluster.barrier_arrive();
    const uint32_t rows = N - k0, rowBegin = rank * perBlock;
    const uint32_t myRows = rowBegin < rows ? min(perBlock, rows - rowBegin) : 0u;
    R *M = LU + size_t(blockIdx.y) * N * N * 2 + 2 * (size_t(k0) * N + k0);  // entry (0, 0) of the panel
    const size_t stride = size_t(N) * 2;
    const uint32_t threads = blockDim.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = int(threads >> 5);
    const C2<R> zero = mk<R>(0, 0);
    int row[RT], taken[RT];  // panel row (-1: none); its pivot index, -1 for none, kPanel without a row
#pragma unroll
    for (int r = 0; r < RT; ++r) {
        const uint32_t local = threadIdx.x + r * threads;
        row[r] = local < myRows ? int(rowBegin + local) : -1;  // never equal to a pivot of another CTA
        taken[r] = local < myRows ? -1 : kPanel;
    }
    const auto magnitude = [](C2<R> z) {
        const R m = fabs(z.x) + fabs(z.y);
        return m >= R(0) ? m : R(0);
    };
    C2<R> a[RT][kHalf];
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
        const int h0 = h * kHalf, width = min(kHalf, int(jb) - h0);
        if (width <= 0)
            break;
#pragma unroll
        for (int c = 0; c < kHalf; ++c)
#pragma unroll
            for (int r = 0; r < RT; ++r)
                a[r][c] = taken[r] != kPanel && c < width ? ld2(M + (h0 + c) * stride + 2 * row[r]) : zero;
        if (h == 0 && C > 1)
            cluster.barrier_wait();
        if (h == 1) {  // the left half's update: solved values for its pivot rows, 16 products for the others
#pragma unroll 1
            for (int j = 0; j < kHalf; ++j) {
                C2<R> l[RT];
#pragma unroll
                for (int r = 0; r < RT; ++r)
                    l[r] = taken[r] < 0 ? left[size_t(j) * perBlock + threadIdx.x + r * threads] : zero;
#pragma unroll
                for (int c = 0; c < kHalf; ++c) {
                    const C2<R> u = sh.top[j][kHalf + c];
#pragma unroll
                    for (int r = 0; r < RT; ++r)
                        csub<R>(a[r][c], l[r], u);
                }
            }
#pragma unroll
            for (int r = 0; r < RT; ++r)
                if (taken[r] >= 0 && taken[r] < kPanel)
#pragma unroll
                    for (int c = 0; c < kHalf; ++c)
                        a[r][c] = sh.top[taken[r]][kHalf + c];
        }
        // this warp's best row for the entries at index c; the row's lane returns true
        const auto candidate = [&](int c, PivotKey &key, int &bestRow, int &slot) {
            R best = R(-1);
            bestRow = 0x7fffffff;
            slot = -1;
#pragma unroll
            for (int r = 0; r < RT; ++r)
                if (taken[r] < 0) {
                    const R m = magnitude(a[r][c]);
                    if (m > best) {  // rows ascend with r: ties keep the lower row
                        best = m;
                        bestRow = row[r];
                        slot = r;
                    }
                }
            key = slot >= 0 ? pivotKey(best) : PivotKey{};
            return warpPivot<R>(key, bestRow) && slot >= 0;
        };
        PivotKey key;
        int bestRow, slot;
        bool mine = candidate(0, key, bestRow, slot);
#pragma unroll 1
        for (int j0 = 0; j0 < kHalf; j0 += U) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                // column j of the half sits at index u of the rotated rows
                const int j = j0 + u, remaining = kHalf - j, buf = j & 1;
                if (j >= width)
                    break;  // the same for the whole cluster
                if (mine) {
#pragma unroll
                    for (int c = 0; c < kHalf; ++c) {
                        if (c >= remaining)
                            break;
                        C2<R> v = a[0][(u + c) % kHalf];
#pragma unroll
                        for (int r = 1; r < RT; ++r)
                            if (slot == r)
                                v = a[r][(u + c) % kHalf];
                        sh.warpRow[buf][warp][c] = v;
                    }
                }
                if (lane == 0)
                    sh.warpKey[buf][warp] = make_int4(int(key.hi), int(key.lo), bestRow, 0);
                __syncthreads();
                int4 found = lane < warps ? sh.warpKey[buf][lane] : make_int4(0, 0, 0x7fffffff, 0);
                key = {unsigned(found.x), unsigned(found.y)};
                int p = found.z;
                int winner = __ffs(__ballot_sync(0xffffffffu, warpPivot<R>(key, p))) - 1;
                const C2<R> *pivotRow = sh.warpRow[buf][winner];
                if (C > 1) {
                    for (uint32_t to = warp; to < C; to += warps) {
                        PanelShared<R> *other = cluster.map_shared_rank(&sh, int(to));
                        if (lane < kHalf)
                            other->ctaRow[buf][rank][lane] = pivotRow[lane];
                        else if (lane == kHalf)
                            other->ctaKey[buf][rank] = make_int4(int(key.hi), int(key.lo), p, 0);
                    }
                    cluster.sync();
                    found = uint32_t(lane) < C ? sh.ctaKey[buf][lane] : make_int4(0, 0, 0x7fffffff, 0);
                    key = {unsigned(found.x), unsigned(found.y)};
                    p = found.z;
                    winner = __ffs(__ballot_sync(0xffffffffu, warpPivot<R>(key, p))) - 1;
                    pivotRow = sh.ctaRow[buf][winner];
                }
                if (threadIdx.x == 0) {
                    sh.sel[h0 + j] = p;
                    if (rank == 0 && zeroKey(key) && *info == 0)
                        atomicCAS(info, 0, int(k0) + h0 + j + 1);
                }
                const C2<R> d = pivotRow[0];
                const R den = d.x * d.x + d.y * d.y;
                const R rden = den > R(0) ? R(1) / den : R(0);
                const C2<R> inv = mk<R>(d.x * rden, -d.y * rden);
                C2<R> l[RT];
#pragma unroll
                for (int r = 0; r < RT; ++r) {
                    if (row[r] == p)
                        taken[r] = h0 + j;
                    const C2<R> m = cmul<R>(a[r][u], inv);
                    l[r] = taken[r] >= 0 ? zero : m;  // a pivot row keeps its values
                    a[r][u] = taken[r] >= 0 ? a[r][u] : m;
                }
                // the next column first: its candidate's reductions overlap the other columns' updates
                if (remaining > 1)
#pragma unroll
                    for (int r = 0; r < RT; ++r)
                        csub<R>(a[r][(u + 1) % kHalf], l[r], pivotRow[1]);
                mine = candidate((u + 1) % kHalf, key, bestRow, slot);
#pragma unroll
                for (int c = 2; c < kHalf; ++c) {
                    if (c >= remaining)  // finished columns
                        break;
                    const C2<R> pv = pivotRow[c];
#pragma unroll
                    for (int r = 0; r < RT; ++r)
                        csub<R>(a[r][(u + c) % kHalf], l[r], pv);
                }
            }
            // rotate every row left by U
#pragma unroll
            for (int r = 0; r < RT; ++r) {
                C2<R> t[U];
#pragma unroll
                for (int c = 0; c < U; ++c)
                    t[c] = a[r][c];
#pragma unroll
                for (int c = 0; c + U < kHalf; ++c)
                    a[r][c] = a[r][c + U];
#pragma unroll
                for (int c = 0; c < U; ++c)
                    a[r][kHalf - U + c] = t[c];
            }
        }
        if (h == 0 && int(jb) > kHalf) {
            // put the left half aside; its pivot rows, with their right half, to every CTA
#pragma unroll
            for (int r = 0; r < RT; ++r)
                if (taken[r] != kPanel) {
#pragma unroll
                    for (int c = 0; c < kHalf; ++c)
                        left[size_t(c) * perBlock + threadIdx.x + r * threads] = a[r][c];
                    if (taken[r] >= 0)
#pragma unroll
                        for (int c = 0; c < kHalf; ++c) {
                            sh.own[taken[r]][c] = a[r][c];
                            sh.own[taken[r]][kHalf + c] =
                                kHalf + c < int(jb) ? ld2(M + (kHalf + c) * stride + 2 * row[r]) : zero;
                        }
                }
            cluster.sync();
            for (uint32_t e = threadIdx.x; e < uint32_t(kHalf * kPanel); e += threads) {
                const uint32_t q = e / kPanel, c = e % kPanel;
                sh.top[q][c] = cluster.map_shared_rank(&sh, int(uint32_t(sh.sel[q]) / perBlock))->own[q][c];
            }
            __syncthreads();
            if (warp < kHalf / 2) {  // U12 = L11^-1 A12: a half warp per column, lane = pivot row
                const int i = lane & (kHalf - 1), c = kHalf + 2 * warp + (lane >> 4);
                C2<R> x = sh.top[i][c];
#pragma unroll
                for (int j = 0; j + 1 < kHalf; ++j) {
                    const int from = (lane & kHalf) | j;
                    const C2<R> xj = mk<R>(__shfl_sync(0xffffffffu, x.x, from), __shfl_sync(0xffffffffu, x.y, from));
                    if (i > j)
                        csub<R>(x, sh.top[i][j], xj);
                }
                __syncwarp();
                sh.top[i][c] = x;
            }
            __syncthreads();
        }
    }
    __syncthreads();
    // Selection order -> interchanges (row k0 + j swapped with row piv[k0 + j]) and final positions:
    // lane q holds the row now at position q and the position of panel row q.
    if (warp == 0) {
        int at = lane, where = lane;
        bool selected = false;
        for (int j = 0; j < int(jb); ++j) {
            const int s = sh.sel[j], here = __shfl_sync(0xffffffffu, at, j);
            const int from = __shfl_sync(0xffffffffu, where, s & 31);
            const int pj = s < kPanel ? from : s;
            if (rank == 0 && lane == 0)
                pivots[size_t(blockIdx.y) * N + k0 + j] = int(k0) + pj;
            if (lane == pj)
                at = here;
            if (lane == j)
                at = s;
            if (lane == here)
                where = pj;
            if (lane == s) {
                where = j;
                selected = true;
            }
        }
        sh.position[lane] = where;
        if (rank == 0) {
            int *mv = moves + size_t(blockIdx.y) * kMoves;
            mv[lane] = lane < int(jb) ? sh.sel[lane] : -1;
            mv[kPanel + lane] = selected || where == lane ? -1 : where;
        }
    }
    __syncthreads();
    const int h0 = int(jb) > kHalf ? kHalf : 0;
#pragma unroll
    for (int r = 0; r < RT; ++r) {
        if (taken[r] == kPanel)
            continue;
        const int pos = taken[r] >= 0 ? taken[r] : row[r] < kPanel ? sh.position[row[r]] : row[r];
        R *out = M + 2 * pos;
        if (h0)
#pragma unroll
            for (int c = 0; c < kHalf; ++c)
                st2(out + c * stride, left[size_t(c) * perBlock + threadIdx.x + r * threads]);
#pragma unroll
        for (int c = 0; c < kHalf; ++c)
            if (h0 + c < int(jb))
                st2(out + (h0 + c) * stride, a[r][c]);
    }
}

// Moves of one panel for the panels that do not come from panelRegKernel: from
// the interchange sequence, one warp per matrix (see kMoves).
__global__ void panelMovesKernel(const int *pivots, uint32_t N, uint32_t k0, uint32_t jb, int *moves) {
    __shared__ int rowAt[kMoves], position[kMoves];  // the rows and positions the interchanges touch
    const int *piv = pivots + size_t(blockIdx.x) * N;
    int *mv = moves + size_t(blockIdx.x) * kMoves;
    const int lane = threadIdx.x;
    // slots 0..31 are positions 0..31, slot 32 + j the position of interchange j's partner if it is below them
    rowAt[lane] = lane;
    position[lane] = lane;
    const int partner = lane < int(jb) ? piv[k0 + lane] - int(k0) : -1;
    rowAt[kPanel + lane] = position[kPanel + lane] = partner >= kPanel ? partner : -1;
    mv[lane] = mv[kPanel + lane] = -1;
    __syncwarp();
    if (lane == 0)
        for (int j = 0; j < int(jb); ++j) {
            const int q = piv[k0 + j] - int(k0);
            int slot = q;
            if (q >= kPanel) {  // the first slot of that position carries its row
                slot = kPanel;
                while (position[slot] != q)
                    ++slot;
            }
            const int t = rowAt[j];
            rowAt[j] = rowAt[slot];
            rowAt[slot] = t;
        }
    __syncwarp();
    if (lane < int(jb))
        mv[lane] = rowAt[lane];
    __syncwarp();
    // rows of the first 32 that ended below: a position's first slot holds its row
    const int slot = kPanel + lane, at = position[slot];
    bool first = at >= 0;
    for (int q = kPanel; q < slot; ++q)
        first = first && position[q] != at;
    if (first && rowAt[slot] < kPanel)
        mv[kPanel + rowAt[slot]] = at;
}

// Row interchanges of the panel applied to the columns outside it: a warp takes
// kSwapColumns columns, reads the (at most 64) entries that move and writes them
// to their places. All reads are in flight together; following the
// interchanges one after the other took a memory latency for each
// (N = 6380: 1.74 -> 1.31 ms over a factorisation's 200 panels).
constexpr int kSwapColumns = 4;
template <class R>
__global__ void __launch_bounds__(256) swapKernel(R *LU, uint32_t N, uint32_t k0, uint32_t jb, const int *moves) {
    const int lane = threadIdx.x & 31;
    const int *mv = moves + size_t(blockIdx.y) * kMoves;
    const int from = mv[lane], to = mv[kPanel + lane];  // row `from` to position lane, row lane to position `to`
    const bool in = from >= 0 && from != lane, out = to >= 0;
    const uint32_t first = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kSwapColumns;
    R *M = LU + size_t(blockIdx.y) * N * N * 2 + 2 * (size_t(first) * N + k0);
    C2<R> vIn[kSwapColumns], vOut[kSwapColumns];
    bool active[kSwapColumns];
#pragma unroll
    for (int c = 0; c < kSwapColumns; ++c) {
        const uint32_t col = first + c;
        active[c] = col < N && (col < k0 || col >= k0 + jb);
        if (active[c] && in)
            vIn[c] = ld2(M + 2 * (size_t(c) * N + from));
        if (active[c] && out)
            vOut[c] = ld2(M + 2 * (size_t(c) * N + lane));
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < kSwapColumns; ++c) {
        if (active[c] && in)
            st2(M + 2 * (size_t(c) * N + lane), vIn[c]);
        if (active[c] && out)
            st2(M + 2 * (size_t(c) * N + to), vOut[c]);
    }
}

// U12 = L11^{-1} A12 (unit lower L11 of the panel) for columns
// [k0 + jb, cEnd), 32 per CTA: L11 and the 32x32 tile of A12 are staged in
// shared memory with coalesced column reads; a warp solves one column at a
// time (lane = row, L11 row in registers, the solved unknown broadcast by
// shuffle).
template <class R>
__global__ void __launch_bounds__(256) trsmKernel(R *LU, uint32_t N, uint32_t k0, uint32_t jb, uint32_t cEnd) {
    __shared__ C2<R> L[kPanel][kPanel + 1];
    __shared__ C2<R> X[kPanel][kPanel + 1];  // [column][row]
    R *M = LU + size_t(blockIdx.y) * N * N * 2;
    const uint32_t c0 = k0 + jb + blockIdx.x * kPanel;
    const uint32_t cols = min(uint32_t(kPanel), cEnd - c0);
    for (uint32_t e = threadIdx.x; e < jb * jb; e += blockDim.x) {
        const uint32_t r = e % jb, c = e / jb;
        L[r][c] = ld2(M + 2 * (size_t(k0 + c) * N + k0 + r));
    }
    for (uint32_t e = threadIdx.x; e < cols * jb; e += blockDim.x) {
        const uint32_t r = e % jb, c = e / jb;
        X[c][r] = ld2(M + 2 * (size_t(c0 + c) * N + k0 + r));
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    C2<R> row[kPanel];
#pragma unroll
    for (int m = 0; m < kPanel; ++m)
        row[m] = (lane < int(jb) && m < int(jb)) ? L[lane][m] : mk<R>(0, 0);
    for (uint32_t c = warp; c < cols; c += blockDim.x >> 5) {
        C2<R> v = lane < int(jb) ? X[c][lane] : mk<R>(0, 0);
#pragma unroll
        for (int m = 0; m < kPanel; ++m) {
            const C2<R> xm = mk<R>(__shfl_sync(0xffffffffu, v.x, m), __shfl_sync(0xffffffffu, v.y, m));
            if (lane > m)
                csub<R>(v, row[m], xm);
        }
        if (lane < int(jb))
            X[c][lane] = v;
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < cols * jb; e += blockDim.x) {
        const uint32_t r = e % jb, c = e / jb;
        st2(M + 2 * (size_t(c0 + c) * N + k0 + r), X[c][r]);
    }
}

// FP32: A22 -= L21 * U12 with 64x64 output tiles, K = jb <= 32, over rows
// [k0 + jb, N) and columns [k0 + jb, cEnd).
template <class R>
__global__ void __launch_bounds__(256) gemmKernel(R *LU, uint32_t N, uint32_t k0, uint32_t jb, uint32_t cEnd) {
    extern __shared__ __align__(16) unsigned char rawSmem[];
    C2<R> *sA = reinterpret_cast<C2<R> *>(rawSmem);  // [kPanel][64]  L21 tile, k-major
    C2<R> *sB = sA + kPanel * 64;                      // [kPanel][64]  U12 tile, k-major
    R *M = LU + size_t(blockIdx.z) * N * N * 2;
    const uint32_t r0 = k0 + jb + blockIdx.x * 64, c0 = k0 + jb + blockIdx.y * 64;
    for (uint32_t e = threadIdx.x; e < jb * 64; e += blockDim.x) {
        const uint32_t kk = e / 64, x = e % 64;
        const uint32_t r = r0 + x, c = c0 + x;
        sA[kk * 64 + x] = r < N ? ld2(M + 2 * (size_t(k0 + kk) * N + r)) : mk<R>(0, 0);
        sB[kk * 64 + x] = c < cEnd ? ld2(M + 2 * (size_t(c) * N + k0 + kk)) : mk<R>(0, 0);
    }
    __syncthreads();
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    C2<R> acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            acc[i][j] = mk<R>(0, 0);
    for (uint32_t kk = 0; kk < jb; ++kk) {
        C2<R> a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            a[i] = sA[kk * 64 + tx + 16 * i];
            b[i] = sB[kk * 64 + ty + 16 * i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[i][j].x += a[i].x * b[j].x - a[i].y * b[j].y;
                acc[i][j].y += a[i].x * b[j].y + a[i].y * b[j].x;
            }
    }
    // the 16 outputs are read first (independent loads in flight), then written
    C2<R> old[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t r = r0 + tx + 16 * i, c = c0 + ty + 16 * j;
            old[i][j] = (r < N && c < cEnd) ? ld2(M + 2 * (size_t(c) * N + r)) : mk<R>(0, 0);
        }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t r = r0 + tx + 16 * i, c = c0 + ty + 16 * j;
            if (r < N && c < cEnd)
                st2(M + 2 * (size_t(c) * N + r), mk<R>(old[i][j].x - acc[i][j].x, old[i][j].y - acc[i][j].y));
        }
}

// ---------------------------------------------------------------------------
// FP64 update C -= L U (complex, K = kPanel or kOuter64 columns of L) on the
// FP64 matrix instruction (mma.sync m8n8k4; tcgen05 has no FP64 kind).
//
// Bound: at K = 96 a 64 x 64 tile is 1.57 M fused operations against 128 KB of
// C and 192 KB of operands, so the FP64 pipe (24.6 k cycles per tile on one SM)
// leads the memory by more than a factor of two; at K = 32 they tie, which is why
// the factorisation has two levels. A warp owns 4 x 4 (or 2 x 2) blocks of 8 x 8
// outputs, real and imaginary accumulators in registers. Operands come in stages
// of 16 columns by cp.async into two buffers, as complex pairs: one 16-byte load
// gives a fragment's real and imaginary part, and 8 loads feed 64 matrix
// instructions. Leading dimensions of 2 (L) and 4 (U)
// modulo 8 entries make both fragment reads free of bank conflicts. Three CTAs
// per SM: a tile's reads and writes of C overlap the others' products (two left
// the matrix pipe at 51 %). The products are summed from zero and taken from C
// at the end: accumulators that start from C round every product at C's size,
// which raised the solve residual of the 12.8k horn from 5e-15 to 2.8e-14.
//
// Tile 64 x 64, or 32 x 32 where 64 x 64 tiles would leave SMs idle.
// Measured, all updates of a factorisation, against one level of K = 32 updates
// with FP64 fused multiply-adds: N = 6380 65.2 -> 24.5 ms (outer block 64: 28.0;
// two CTAs per SM: 39.2), N = 2562 x 2 9.2 -> 3.9, N = 642 x 32 2.56 -> 1.04,
// N = 258 0.137 -> 0.077
// ---------------------------------------------------------------------------
constexpr int kStageK = 16;
constexpr int kOuter64 = 96;  // outer block width of the FP64 factorisation

__device__ __forceinline__ void mma884(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
// 16 bytes from global to shared memory, zeros when `valid` is false
__device__ __forceinline__ void copyEntry(double2 *dst, const double *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))),
                 "l"(src), "r"(valid ? 16 : 0));
}

template <int TILE>
constexpr size_t kGemm64Smem = 2 * (kStageK * (TILE + 2) + TILE * (kStageK + 4)) * sizeof(double2);  // 73 KB at 64

// Rows [r0, N), columns [c0, cEnd), inner columns [k0, k0 + K): C(r, c) -= sum_k M(r, k) M(k, c). K is a
// multiple of kStageK.
template <int TILE>
__global__ void __launch_bounds__(128, TILE == 64 ? 3 : 4) gemm64Kernel(double *LU, uint32_t N, uint32_t k0, uint32_t K,
                                                                       uint32_t r0, uint32_t c0, uint32_t cEnd) {
    constexpr int LDA = TILE + 2, LDB = kStageK + 4, W = TILE / 16;  // W x W blocks of 8 x 8 per warp
    extern __shared__ __align__(16) unsigned char rawSmem[];
    double2 *const sA = reinterpret_cast<double2 *>(rawSmem);  // two buffers [k][row]
    double2 *const sB = sA + 2 * kStageK * LDA;                // two buffers [column][k]
    double *M = LU + size_t(blockIdx.z) * N * N * 2;
    const uint32_t row0 = r0 + blockIdx.x * TILE, col0 = c0 + blockIdx.y * TILE;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wr = (warp & 1) * (TILE / 2), wc = (warp >> 1) * (TILE / 2);  // the warp's corner in the tile
    const auto stage = [&](int buffer, uint32_t k) {
        for (int e = threadIdx.x; e < kStageK * TILE; e += 128) {
            const int kk = e / TILE, x = e % TILE;
            const bool inside = row0 + x < N;
            copyEntry(sA + buffer * kStageK * LDA + kk * LDA + x, M + 2 * (size_t(k + kk) * N + (inside ? row0 + x : 0)), inside);
        }
        for (int e = threadIdx.x; e < kStageK * TILE; e += 128) {
            const int c = e / kStageK, kk = e % kStageK;
            const bool inside = col0 + c < cEnd;
            copyEntry(sB + buffer * TILE * LDB + c * LDB + kk, M + 2 * (size_t(inside ? col0 + c : 0) * N + k + kk), inside);
        }
        asm volatile("cp.async.commit_group;");
    };
    stage(0, k0);
    // sums of the products (from zero: started from C, which is larger, every product would be rounded at C's
    // size). Block (i, j) holds rows wr + 8i + lane / 4, columns wc + 8j + 2 (lane % 4) + {0, 1}.
    double re[W][W][2], im[W][W][2];
    const uint32_t row = row0 + wr + lane / 4, col = col0 + wc + 2 * (lane % 4);
#pragma unroll
    for (int i = 0; i < W; ++i)
#pragma unroll
        for (int j = 0; j < W; ++j)
            re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0;
    const int stages = int(K) / kStageK;
    for (int s = 0; s < stages; ++s) {
        if (s + 1 < stages) {
            stage((s + 1) & 1, k0 + (s + 1) * kStageK);
            asm volatile("cp.async.wait_group 1;");
        } else
            asm volatile("cp.async.wait_group 0;");
        __syncthreads();
        const double2 *A = sA + (s & 1) * kStageK * LDA + (lane % 4) * LDA + wr + lane / 4;
        const double2 *B = sB + (s & 1) * TILE * LDB + (wc + lane / 4) * LDB + lane % 4;
#pragma unroll
        for (int kk = 0; kk < kStageK; kk += 4) {
            double2 a[W], b[W];
#pragma unroll
            for (int i = 0; i < W; ++i) {
                a[i] = A[kk * LDA + 8 * i];
                b[i] = B[8 * i * LDB + kk];
            }
            // four sweeps over the blocks: consecutive instructions have different accumulators
#pragma unroll
            for (int i = 0; i < W; ++i)
#pragma unroll
                for (int j = 0; j < W; ++j)
                    mma884(re[i][j], a[i].x, b[j].x);
#pragma unroll
            for (int i = 0; i < W; ++i)
#pragma unroll
                for (int j = 0; j < W; ++j)
                    mma884(im[i][j], a[i].x, b[j].y);
#pragma unroll
            for (int i = 0; i < W; ++i)
#pragma unroll
                for (int j = 0; j < W; ++j)
                    mma884(re[i][j], -a[i].y, b[j].y);
#pragma unroll
            for (int i = 0; i < W; ++i)
#pragma unroll
                for (int j = 0; j < W; ++j)
                    mma884(im[i][j], a[i].y, b[j].x);
        }
        __syncthreads();
    }
    // a column block's entries of C are read together, then written
#pragma unroll
    for (int j = 0; j < W; ++j) {
        double2 old[W][2];
#pragma unroll
        for (int i = 0; i < W; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t r = row + 8 * i, c = col + 8 * j + h;
                old[i][h] = r < N && c < cEnd ? ld2(M + 2 * (size_t(c) * N + r)) : make_double2(0, 0);
            }
#pragma unroll
        for (int i = 0; i < W; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t r = row + 8 * i, c = col + 8 * j + h;
                if (r < N && c < cEnd)
                    st2(M + 2 * (size_t(c) * N + r), make_double2(old[i][h].x - re[i][j][h], old[i][h].y - im[i][j][h]));
            }
    }
}

// ---------------------------------------------------------------------------
// FP32 trailing update of the two-level factorisation on the tensor cores
// (tcgen05): A22 -= L21 * U12 with K = kOuter = 128 complex columns, as a real
// GEMM of the split complex operands, output real parts and imaginary parts
// side by side:
//   [C_re, C_im] = [L_re, L_im] * [[U_re, U_im]; [-U_im, U_re]].
// Operands are multiplied as hi*hi + hi*lo + lo*hi (3xTF32: TF32 hi part plus
// TF32 remainder) with FP32 accumulation, which keeps FP32 accuracy.
//
// packKernel converts L21 and U12 once per outer block into operand tiles
// that are already in the tensor cores' shared-memory layout (K-major,
// unswizzled canonical layout: 8-row x 16-byte core matrices, row groups 128 B
// apart (SBO), 16-byte K chunks (rows/8)*128 B apart (LBO)), hi then lo, one
// tile per 128 rows (A) or 64 complex columns (B, 128 operand rows) and per
// stage of 16 complex K columns. trailingTensorKernel then owns 128 complex
// rows x 64 complex columns of A22 (an M = 128, N = 128 real accumulator in
// tensor memory) and runs three roles:
//   * warp 0 copies the stage tiles into a ring of kTcStages shared-memory
//     buffers with bulk asynchronous copies that complete on the buffer's
//     `full` mbarrier;
//   * warp 1 issues the stage's MMAs from one thread and commits them to the
//     buffer's `empty` mbarrier, which lets warp 0 refill it; after the last
//     stage it commits to `done`;
//   * every thread loads its 32 outputs of A22 at the start (the loads overlap
//     the main loop), waits for `done`, reads its accumulator row (32 lanes x
//     32 columns, real and imaginary parts) from tensor memory and writes the
//     updated outputs (a warp writes 32 consecutive rows of a column).
// Every wait is bounded by a clock budget; a timeout leaves kTensorTimeout in
// the LU status word and skips the update.
// ---------------------------------------------------------------------------
constexpr int kOuter = 128;                            // outer block width of the two-level factorisation
constexpr int kTcRows = 128, kTcCols = 64, kTcK = 16;  // complex rows, complex columns, complex K per stage
constexpr int kTcStages = 3, kTcThreads = 256;
constexpr int kTcSteps = kOuter / kTcK;                // stages per update
constexpr int kTcTile = 2 * kTcRows * (2 * kTcK);      // floats of one operand tile, hi + lo (A and B alike)
constexpr size_t kTcSmem = size_t(kTcStages) * 2 * kTcTile * sizeof(float);  // 192 KB: one CTA per SM
constexpr int kTensorTimeout = -1;
constexpr long long kWaitCycles = 4000000000ll;  // about two seconds

static_assert(2 * kTcCols == kTcRows, "A and B operand tiles have the same shape");
static_assert(kOuter % kTcK == 0 && kOuter % kPanel == 0, "outer block must hold whole stages and panels");
static_assert(kTcSmem > 114 * 1024 && kTcSmem <= 227 * 1024, "one CTA per SM keeps tensor-memory allocation uncontended");

// floats of the packed operand tiles of one matrix (the first outer block has the most)
size_t packFloats(uint32_t N) {
    if (N <= uint32_t(kOuter))
        return 0;
    const size_t rest = N - kOuter;
    return ((rest + kTcRows - 1) / kTcRows + (rest + kTcCols - 1) / kTcCols) * kTcSteps * size_t(kTcTile);
}

__device__ __forceinline__ uint32_t smemAddr(const void *p) { return uint32_t(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ float tf32Round(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// offset (floats) of element (row r, k) in a K-major core-matrix tile of `rows` rows
__device__ __forceinline__ int coreOffset(int r, int k, int rows) {
    return ((k >> 2) * (rows >> 3) + (r >> 3)) * 32 + (r & 7) * 4 + (k & 3);
}

// UMMA shared-memory matrix descriptor: start, LBO, SBO (16-byte units), version 1, no swizzle
__device__ __forceinline__ uint64_t matrixDescriptor(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return uint64_t((addr >> 4) & 0x3FFF) | (uint64_t((lbo >> 4) & 0x3FFF) << 16) |
           (uint64_t((sbo >> 4) & 0x3FFF) << 32) | (uint64_t(1) << 46);
}

// Bounded wait for the phase of `parity` on an mbarrier; false on timeout.
__device__ __forceinline__ bool waitPhase(uint32_t bar, uint32_t parity) {
    const long long start = clock64();
    uint32_t done = 0;
    while (!done) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity));
        if (!done && clock64() - start > kWaitCycles)
            return false;
    }
    return true;
}

// Operand tiles of one outer block: per matrix the A tiles of L21 [row tile][stage], then the B tiles
// of U12 [column tile][stage]. Grid: (row tiles + column tiles, stages, matrices).
__global__ void __launch_bounds__(256) packKernel(const float *LU, uint32_t N, uint32_t K0, float *pack,
                                                  size_t packStride) {
    const uint32_t begin = K0 + kOuter, rest = N - begin;
    const uint32_t rowTiles = (rest + kTcRows - 1) / kTcRows, t = blockIdx.x, c = blockIdx.y;
    const float *M = LU + size_t(blockIdx.z) * N * N * 2;
    float *hi = pack + blockIdx.z * packStride + (size_t(t) * kTcSteps + c) * kTcTile, *lo = hi + kTcTile / 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t kc = K0 + c * kTcK;
    // a warp fills whole core matrices: lane = (row & 7) * 4 + (k & 3), 32 stores to 128 contiguous bytes
    if (t < rowTiles) {  // A: row i takes (L_re, L_im) at k and k + 16
        const uint32_t r0 = begin + t * kTcRows;
        float2 v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int cm = warp + 8 * q, i = (cm % 16) * 8 + (lane >> 2), k = (cm / 16) * 4 + (lane & 3);
            v[q] = r0 + i < N ? *reinterpret_cast<const float2 *>(M + 2 * (size_t(kc + k) * N + r0 + i))
                              : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int cm = warp + 8 * q, i = (cm % 16) * 8 + (lane >> 2), k = (cm / 16) * 4 + (lane & 3);
            const float hr = tf32Round(v[q].x), hm = tf32Round(v[q].y);
            hi[coreOffset(i, k, kTcRows)] = hr;
            lo[coreOffset(i, k, kTcRows)] = tf32Round(v[q].x - hr);
            hi[coreOffset(i, k + kTcK, kTcRows)] = hm;
            lo[coreOffset(i, k + kTcK, kTcRows)] = tf32Round(v[q].y - hm);
        }
    } else {  // B: operand row j takes (U_re, -U_im), row j + 64 takes (U_im, U_re)
        const uint32_t c0 = begin + (t - rowTiles) * kTcCols;
        float2 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int cm = warp + 8 * q, j = (cm % 8) * 8 + (lane >> 2), k = (cm / 8) * 4 + (lane & 3);
            v[q] = c0 + j < N ? *reinterpret_cast<const float2 *>(M + 2 * (size_t(c0 + j) * N + kc + k))
                              : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int cm = warp + 8 * q, j = (cm % 8) * 8 + (lane >> 2), k = (cm / 8) * 4 + (lane & 3);
            const float parts[4] = {v[q].x, -v[q].y, v[q].y, v[q].x};  // (j, k), (j, k+16), (j+64, k), (j+64, k+16)
            const int rows[4] = {j, j, j + kTcCols, j + kTcCols}, ks[4] = {k, k + kTcK, k, k + kTcK};
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const float h = tf32Round(parts[p]);
                hi[coreOffset(rows[p], ks[p], kTcRows)] = h;
                lo[coreOffset(rows[p], ks[p], kTcRows)] = tf32Round(parts[p] - h);
            }
        }
    }
}

__global__ void __launch_bounds__(kTcThreads, 1) trailingTensorKernel(float *LU, uint32_t N, uint32_t K0,
                                                                      const float *pack, size_t packStride,
                                                                      int *info) {
    extern __shared__ __align__(1024) float ring[];  // kTcStages x {A hi, A lo, B hi, B lo}
    __shared__ __align__(8) uint64_t full[kTcStages], empty[kTcStages], done;
    __shared__ uint32_t tmemBase;
    constexpr int NB = 2 * kTcCols;  // real accumulator columns
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t begin = K0 + kOuter, rest = N - begin;
    const uint32_t rowTiles = (rest + kTcRows - 1) / kTcRows;
    const uint32_t r0 = begin + blockIdx.x * kTcRows, c0 = begin + blockIdx.y * kTcCols;
    float *M = LU + size_t(blockIdx.z) * N * N * 2;
    const float *tilesA = pack + blockIdx.z * packStride + size_t(blockIdx.x) * kTcSteps * kTcTile;
    const float *tilesB = pack + blockIdx.z * packStride + (size_t(rowTiles) + blockIdx.y) * kTcSteps * kTcTile;
    // this thread's outputs: row 32 (warp % 4) + lane, columns 32 (warp / 4) .. + 31
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t row = r0 + quarter * 32 + lane, col0 = c0 + half * 32;
    float2 old[32];
#pragma unroll
    for (int j = 0; j < 32; ++j)
        old[j] = (row < N && col0 + j < N) ? *reinterpret_cast<const float2 *>(M + 2 * (size_t(col0 + j) * N + row))
                                           : make_float2(0.f, 0.f);
    if (tid == 0) {
        for (int s = 0; s < kTcStages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smemAddr(&full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smemAddr(&empty[s])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smemAddr(&done)));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemBase)),
                     "r"(NB));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        asm volatile("tcgen05.fence::before_thread_sync;");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmemBase;
    bool ok = true;
    int issued = 0;
    if (warp == 0) {  // producer
        for (int c = 0; c < kTcSteps; ++c) {
            const int s = c % kTcStages;
            if (c >= kTcStages) {  // the MMAs of stage c - kTcStages have read this buffer
                ok = __all_sync(0xffffffffu, waitPhase(smemAddr(&empty[s]), uint32_t((c - kTcStages) / kTcStages) & 1u));
                if (!ok)
                    break;
            }
            if (lane == 0) {
                const uint32_t dst = smemAddr(ring + size_t(s) * 2 * kTcTile), bar = smemAddr(&full[s]);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                             "r"(uint32_t(2 * kTcTile * sizeof(float))));
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                    "l"(tilesA + size_t(c) * kTcTile), "r"(uint32_t(kTcTile * sizeof(float))), "r"(bar)
                    : "memory");
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        dst + uint32_t(kTcTile * sizeof(float))),
                    "l"(tilesB + size_t(c) * kTcTile), "r"(uint32_t(kTcTile * sizeof(float))), "r"(bar)
                    : "memory");
            }
            issued = c + 1;
        }
    } else if (warp == 1) {  // MMA issue
        // D: F32; A, B: TF32, K-major; N = NB (>> 3), M = 128 (>> 4)
        constexpr uint32_t idesc =
            (1u << 4) | (2u << 7) | (2u << 10) | (uint32_t(NB >> 3) << 17) | (uint32_t(kTcRows >> 4) << 24);
        constexpr uint32_t lbo = (kTcRows / 8) * 128, sbo = 128;
        for (int c = 0; c < kTcSteps; ++c) {
            const int s = c % kTcStages;
            ok = __all_sync(0xffffffffu, waitPhase(smemAddr(&full[s]), uint32_t(c / kTcStages) & 1u));
            if (!ok)
                break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            if (lane == 0) {
                const uint32_t aHi = smemAddr(ring + size_t(s) * 2 * kTcTile), aLo = aHi + kTcTile * 2;
                const uint32_t bHi = aHi + kTcTile * 4, bLo = bHi + kTcTile * 2;
                const uint32_t As[3] = {aHi, aHi, aLo}, Bs[3] = {bHi, bLo, bHi};
#pragma unroll
                for (int pass = 0; pass < 3; ++pass)
#pragma unroll
                    for (int step = 0; step < 2 * kTcK / 8; ++step) {
                        const uint64_t da = matrixDescriptor(As[pass] + uint32_t(2 * step) * lbo, lbo, sbo);
                        const uint64_t db = matrixDescriptor(Bs[pass] + uint32_t(2 * step) * lbo, lbo, sbo);
                        const uint32_t accumulate = (c | pass | step) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
                            "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
                    }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                    smemAddr(&empty[s])));
                if (c == kTcSteps - 1)  // completes when every MMA of the CTA has
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                        smemAddr(&done)));
            }
            __syncwarp();
        }
    }
    const bool accumulated = __syncthreads_and(ok && waitPhase(smemAddr(&done), 0));
    if (!accumulated) {
        if (tid == 0)
            atomicCAS(info, 0, kTensorTimeout);
        if (warp == 0)  // let the last copies into each buffer land before the CTA exits
            for (int c = issued > kTcStages ? issued - kTcStages : 0; c < issued; ++c)
                waitPhase(smemAddr(&full[c % kTcStages]), uint32_t(c / kTcStages) & 1u);
    }
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (accumulated) {
        uint32_t re[32], im[32];
        const uint32_t lanes = uint32_t(quarter * 32) << 16;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(re[0]), "=r"(re[1]), "=r"(re[2]), "=r"(re[3]), "=r"(re[4]), "=r"(re[5]), "=r"(re[6]), "=r"(re[7]),
              "=r"(re[8]), "=r"(re[9]), "=r"(re[10]), "=r"(re[11]), "=r"(re[12]), "=r"(re[13]), "=r"(re[14]),
              "=r"(re[15]), "=r"(re[16]), "=r"(re[17]), "=r"(re[18]), "=r"(re[19]), "=r"(re[20]), "=r"(re[21]),
              "=r"(re[22]), "=r"(re[23]), "=r"(re[24]), "=r"(re[25]), "=r"(re[26]), "=r"(re[27]), "=r"(re[28]),
              "=r"(re[29]), "=r"(re[30]), "=r"(re[31])
            : "r"(tmem + lanes + uint32_t(half * 32)));
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(im[0]), "=r"(im[1]), "=r"(im[2]), "=r"(im[3]), "=r"(im[4]), "=r"(im[5]), "=r"(im[6]), "=r"(im[7]),
              "=r"(im[8]), "=r"(im[9]), "=r"(im[10]), "=r"(im[11]), "=r"(im[12]), "=r"(im[13]), "=r"(im[14]),
              "=r"(im[15]), "=r"(im[16]), "=r"(im[17]), "=r"(im[18]), "=r"(im[19]), "=r"(im[20]), "=r"(im[21]),
              "=r"(im[22]), "=r"(im[23]), "=r"(im[24]), "=r"(im[25]), "=r"(im[26]), "=r"(im[27]), "=r"(im[28]),
              "=r"(im[29]), "=r"(im[30]), "=r"(im[31])
            : "r"(tmem + lanes + uint32_t(kTcCols + half * 32)));
        asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (row < N && col0 + j < N)
                *reinterpret_cast<float2 *>(M + 2 * (size_t(col0 + j) * N + row)) =
                    make_float2(old[j].x - __uint_as_float(re[j]), old[j].y - __uint_as_float(im[j]));
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 2)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NB));
}

// U12 = L11^{-1} A12 for the outer block (L11: the OUTER x OUTER unit lower
// triangle at (K0, K0)), over the trailing columns [K0 + OUTER, N). L11 is
// staged in shared memory column by column (coalesced); a warp solves one
// column at a time with lane l holding rows l, l + 32, ... in registers and the
// solved unknown broadcast by shuffle. FP32 at OUTER = 128, FP64 at 96.
constexpr int kTrsmColumns = 64, kTrsmThreads = 512;
template <class R> constexpr int kOuterOf = sizeof(R) == 4 ? kOuter : kOuter64;
template <class R> constexpr size_t kTrsmSmem = size_t(kOuterOf<R>) * kOuterOf<R> * sizeof(C2<R>);  // 128 KB, 144 KB

template <class R>
__global__ void __launch_bounds__(kTrsmThreads, 1) trsmBlockKernel(R *LU, uint32_t N, uint32_t K0, uint32_t columns) {
    constexpr int OUTER = kOuterOf<R>, S = OUTER / 32;
    extern __shared__ __align__(16) unsigned char rawSmem[];
    C2<R> *Lc = reinterpret_cast<C2<R> *>(rawSmem);  // [column m][row]
    R *M = LU + size_t(blockIdx.y) * N * N * 2;
    for (uint32_t e = threadIdx.x; e < uint32_t(OUTER * OUTER); e += blockDim.x) {
        const uint32_t r = e % OUTER, m = e / OUTER;
        Lc[e] = ld2(M + 2 * (size_t(K0 + m) * N + K0 + r));
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t c0 = K0 + OUTER + blockIdx.x * columns;
    for (uint32_t c = c0 + warp; c < min(N, c0 + columns); c += blockDim.x / 32) {
        C2<R> *col = reinterpret_cast<C2<R> *>(M + 2 * (size_t(c) * N + K0));
        C2<R> v[S];
#pragma unroll
        for (int s = 0; s < S; ++s)
            v[s] = col[lane + 32 * s];
#pragma unroll
        for (int sb = 0; sb < S; ++sb)
#pragma unroll 8
            for (int mm = 0; mm < 32; ++mm) {
                const int m = 32 * sb + mm;
                const C2<R> x = mk<R>(__shfl_sync(0xffffffffu, v[sb].x, mm), __shfl_sync(0xffffffffu, v[sb].y, mm));
#pragma unroll
                for (int s = sb; s < S; ++s)
                    if (lane + 32 * s > m)
                        csub<R>(v[s], Lc[m * OUTER + lane + 32 * s], x);
            }
#pragma unroll
        for (int s = 0; s < S; ++s)
            col[lane + 32 * s] = v[s];
    }
}

// Blocked triangular solves. The row interchanges of a factorisation are
// composed once into a permutation (permutationKernel, stored after the
// interchanges), so a solve starts with a parallel gather of the right-hand
// side into a work vector. In FP32 (a preconditioner) the 32 x 32 diagonal blocks
// of both triangles are inverted once per factorisation (diagonalInverseKernel,
// stored after the permutations); FP64 solves by substitution. Forward and backward substitution then run in blocks of
// kTriBlock unknowns, one launch per block: CTA 0 brings the next block's rows
// up to date with the block solved last and solves the next diagonal block; the
// other CTAs apply the block solved last to every remaining row. The backward
// sweep writes each solved block to the output vector.
//
// Bound: the chain of blocks. Everything CTA 0 needs is in flight from its
// first instruction (the diagonal block by cp.async, 32 column loads per
// thread), a 32 x 32 sub-block is one matrix-vector product with its inverse
// (FP32) or 32 shuffled steps from shared memory with the reciprocal diagonal
// (FP64), and partial sums stay in the thread that owns their row and columns until their
// sub-block is next. Measured per solve against shuffled sub-blocks loaded when
// their turn came (one CTA per system up to N = 1024): FP32 N = 6380 3.2 -> 1.0
// ms, N = 4023 x 3 2.1 -> 0.65, N = 642 x 32 0.25 -> 0.125; FP64 N = 6380
// 4.2 -> 1.7, N = 2562 x 2 1.7 -> 0.71, N = 258 0.117 -> 0.073 (before the
// steps overlapped, see triStepKernel).
constexpr uint32_t kTriBlock = 128, kSub = 32;
constexpr uint32_t kTriThreads = 512;                  // 128 rows x 4 column groups
constexpr uint32_t kTriGroups = kTriThreads / kTriBlock;
constexpr uint32_t kTriSubs = kTriBlock / kSub;
// shared memory of CTA 0: the sub-blocks of one triangle of the diagonal block (inverses on the diagonal)
template <class R> constexpr size_t kTriSmem = size_t(kTriSubs * (kTriSubs + 1) / 2) * kSub * kSub * sizeof(C2<R>);

// Complex entries of the inverses of one triangle of one matrix, and where they start in the pivot buffer.
__host__ __device__ inline size_t inverseEntries(uint32_t N) { return size_t((N + kSub - 1) / kSub) * kSub * kSub; }
__host__ __device__ inline size_t inverseOffset(uint32_t N, uint32_t B) {  // in ints, 16-byte aligned
    return (size_t(B) * (2 * size_t(N) + kMoves) + 3) / 4 * 4;
}
template <class R> __host__ __device__ const C2<R> *inverses(const int *pivots, uint32_t N, uint32_t B, uint32_t f, bool lower) {
    return reinterpret_cast<const C2<R> *>(pivots + inverseOffset(N, B)) + (2 * size_t(f) + (lower ? 0 : 1)) * inverseEntries(N);
}

// FP32: inverses of the 32 x 32 diagonal blocks (blockIdx.x) of both triangles
// (blockIdx.z) of each matrix: lane c solves for column c of the inverse,
// rows stored contiguously. Rows past N are those of the identity.
template <class R>
__global__ void __launch_bounds__(32) diagonalInverseKernel(const R *LU, uint32_t N, int *pivots, uint32_t B) {
    __shared__ C2<R> D[kSub][kSub + 1];  // [row][column]
    const uint32_t f = blockIdx.y, k = blockIdx.x * kSub;
    const bool lower = blockIdx.z == 0;
    const int lane = threadIdx.x;
    const R *M = LU + size_t(f) * N * N * 2;
    for (int c = 0; c < int(kSub); ++c)
        D[lane][c] = k + lane < N && k + c < N ? ld2(M + 2 * (size_t(k + c) * N + k + lane)) : mk<R>(lane == c ? 1 : 0, 0);
    __syncwarp();
    if (!lower) {  // reciprocal diagonal
        const C2<R> d = D[lane][lane];
        const R den = d.x * d.x + d.y * d.y;
        D[lane][lane] = mk<R>(d.x / den, -d.y / den);
        __syncwarp();
    }
    C2<R> x[kSub];
#pragma unroll
    for (int q = 0; q < int(kSub); ++q) {
        const int i = lower ? q : int(kSub) - 1 - q;
        C2<R> v = mk<R>(i == lane ? 1 : 0, 0);
#pragma unroll
        for (int p = 0; p < q; ++p)
            csub<R>(v, D[i][lower ? p : int(kSub) - 1 - p], x[p]);
        x[q] = lower ? v : cmul<R>(v, D[i][i]);
    }
    C2<R> *out = const_cast<C2<R> *>(inverses<R>(pivots, N, B, f, lower)) + size_t(blockIdx.x) * kSub * kSub;
#pragma unroll
    for (int q = 0; q < int(kSub); ++q)
        out[(lower ? q : int(kSub) - 1 - q) * kSub + lane] = x[q];
}

__global__ void permutationKernel(const int *pivots, uint32_t N, int *perm) {
    extern __shared__ int p[];  // [N] the permutation, [N] the interchange sequence
    int *piv = p + N;
    for (uint32_t i = threadIdx.x; i < N; i += blockDim.x) {
        p[i] = int(i);
        piv[i] = pivots[size_t(blockIdx.x) * N + i];
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (uint32_t c = 0; c < N; ++c) {
            const int q = piv[c];
            if (q != int(c)) {
                const int t = p[c];
                p[c] = p[q];
                p[q] = t;
            }
        }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < N; i += blockDim.x)
        perm[size_t(blockIdx.x) * N + i] = p[i];
}

// work[f][e][i] = x[f][e][perm[f][i]]
template <class R> __global__ void gatherRhsKernel(const R *x, const int *perm, uint32_t N, uint32_t E, R *work) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, e = blockIdx.y, f = blockIdx.z;
    if (i >= N)
        return;
    const size_t v = (size_t(f) * E + e) * N;
    st2(work + 2 * (v + i), ld2(x + 2 * (v + perm[size_t(f) * N + i])));
}

// v + a * b, and v = sum of the products of one thread
template <class R> __device__ __forceinline__ void cadd(C2<R> &v, C2<R> a, C2<R> b) {
    v.x = fma(-a.y, b.y, fma(a.x, b.x, v.x));
    v.y = fma(a.y, b.x, fma(a.x, b.y, v.y));
}
// one complex value from global to shared memory without a register
template <class R> __device__ __forceinline__ void copyAsync(C2<R> *dst, const R *src) {
    const uint32_t to = uint32_t(__cvta_generic_to_shared(dst));
    if constexpr (sizeof(R) == 8)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src));
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to), "l"(src));
}

// A step reads its matrix entries, which no step writes, before it waits for the
// vectors of the step before it: the launch and these loads, more than half of
// a step, then overlap the steps ahead of it. Every thread waits before it ends,
// so the end of the last step is the end of all. N = 6380: FP32 solve 1.03 ->
// 0.44 ms, FP64 1.74 -> 1.11 ms; N = 642 x 32 systems FP32 0.13 -> 0.08 ms. The
// factorisation's kernels, which can load nothing ahead, gained nothing from it
// (N = 6380 FP32 and FP64 0.5 ms slower: waiting blocks hold the SMs a cluster needs).
__device__ __forceinline__ void chainRelease() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void chainWait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// One step of a sweep. Known block: unknowns [c0, c0 + cw) (cw = 0 on the first step); next block
// [n0, n0 + nw). Forward (Lower): unit lower triangle, updated rows [n0 + nw, N). Backward: upper
// triangle with its diagonal, updated rows [0, n0).
template <class R, bool Lower>
__global__ void __launch_bounds__(kTriThreads) triStepKernel(const R *LU, const int *pivots, uint32_t N, uint32_t E,
                                                             R *work, R *out, uint32_t c0, uint32_t cw, uint32_t n0,
                                                             uint32_t nw) {
    extern __shared__ __align__(16) unsigned char rawSmem[];
    __shared__ C2<R> y[kTriBlock];
    __shared__ C2<R> part[kTriGroups][kTriBlock];
    const uint32_t e = blockIdx.y, f = blockIdx.z, tid = threadIdx.x;
    const uint32_t i = tid % kTriBlock, g = tid / kTriBlock;  // this thread's row and column group
    const R *M = LU + size_t(f) * N * N * 2;
    R *w = work + (size_t(f) * E + e) * N * 2;
    const C2<R> zero = mk<R>(0, 0);
    chainRelease();
    const bool solver = blockIdx.x == 0;
    const uint32_t r = solver ? n0 + i : (Lower ? n0 + nw : 0) + (blockIdx.x - 1) * kTriBlock + i;
    const bool mine = solver ? i < nw : r < (Lower ? N : n0);
    // sub-block (p, q) of the diagonal block, p >= q forward, p <= q backward, in steps of the sweep:
    // step index s = p forward, last - p backward
    C2<R> *const D = reinterpret_cast<C2<R> *>(rawSmem);
    const uint32_t subs = (nw + kSub - 1) / kSub;
    const auto subBlock = [&](uint32_t row, uint32_t column) {  // by sweep order, column <= row
        return D + (row * (row + 1) / 2 + column) * kSub * kSub;
    };
    const auto subAt = [&](uint32_t s) { return Lower ? s : subs - 1 - s; };  // sub-block solved in step s
    if (solver) {
        [[maybe_unused]] const C2<R> *inverse =
            sizeof(R) == 4 ? inverses<R>(pivots, N, gridDim.z, f, Lower) + size_t(n0 / kSub) * kSub * kSub : nullptr;
        for (uint32_t a = 0; a < subs; ++a)
            for (uint32_t b = 0; b <= a; ++b) {
                C2<R> *block = subBlock(a, b);
                if (a == b && sizeof(R) == 8) {  // the triangle itself; identity past the end
                    for (uint32_t x = tid; x < kSub * kSub; x += kTriThreads) {
                        const uint32_t row = kSub * subAt(a) + x % kSub, column = kSub * subAt(a) + x / kSub;
                        if (row < nw && column < nw)
                            copyAsync<R>(block + x, M + 2 * (size_t(n0 + column) * N + n0 + row));
                        else
                            block[x] = mk<R>(row == column ? 1 : 0, 0);
                    }
                    continue;
                }
                if (a == b) {  // the inverse, [row][column]
                    for (uint32_t x = tid; x < kSub * kSub; x += kTriThreads)
                        copyAsync<R>(block + x, reinterpret_cast<const R *>(inverse + size_t(subAt(a)) * kSub * kSub + x));
                    continue;
                }
                for (uint32_t x = tid; x < kSub * kSub; x += kTriThreads) {  // [column][row]
                    const uint32_t row = kSub * subAt(a) + x % kSub, column = kSub * subAt(b) + x / kSub;
                    if (row < nw && column < nw)
                        copyAsync<R>(block + x, M + 2 * (size_t(n0 + column) * N + n0 + row));
                    else
                        block[x] = zero;
                }
            }
        asm volatile("cp.async.commit_group;");
    }
    // this row's products with the block solved last: 32 column loads in flight (FP64: 16)
    C2<R> acc = zero;
    if (cw) {
        constexpr uint32_t kLoads = sizeof(R) == 8 ? kSub / 2 : kSub;
        C2<R> a[kLoads];
        const uint32_t first = kSub * g;
#pragma unroll
        for (uint32_t h = 0; h < kSub; h += kLoads) {
#pragma unroll
            for (uint32_t c = 0; c < kLoads; ++c)
                a[c] = mine && first + h + c < cw ? ld2(M + 2 * (size_t(c0 + first + h + c) * N + r)) : zero;
            if (h == 0) {
                chainWait();
                for (uint32_t x = tid; x < kTriBlock; x += kTriThreads)
                    y[x] = x < cw ? ld2(w + 2 * (c0 + x)) : zero;
                __syncthreads();
            }
#pragma unroll
            for (uint32_t c = 0; c < kLoads; ++c)
                cadd<R>(acc, a[c], y[first + h + c]);
        }
    } else
        chainWait();
    if (!solver) {
        part[g][i] = acc;
        __syncthreads();
        if (g == 0 && mine) {
            C2<R> t = ld2(w + 2 * r);
#pragma unroll
            for (uint32_t q = 0; q < kTriGroups; ++q) {
                t.x -= part[q][i].x;
                t.y -= part[q][i].y;
            }
            st2(w + 2 * r, t);
        }
        return;
    }
    // The next block: its right-hand side in y, solved in place sub-block by sub-block.
    __syncthreads();  // y has been read
    if (tid < kTriBlock)
        y[tid] = tid < nw ? ld2(w + 2 * (n0 + tid)) : zero;
    asm volatile("cp.async.wait_group 0;");
    for (uint32_t s = 0; s < subs; ++s) {
        const uint32_t sub = subAt(s);
        if (i / kSub == sub)
            part[g][i] = acc;
        __syncthreads();
        if constexpr (sizeof(R) == 8) {  // substitution, lane = row, by the first warp
            if (tid < kSub) {
                const uint32_t at = kSub * sub + tid;
                C2<R> t = y[at];
#pragma unroll
                for (uint32_t q = 0; q < kTriGroups; ++q) {
                    t.x -= part[q][at].x;
                    t.y -= part[q][at].y;
                }
                const C2<R> *column = subBlock(s, s) + tid;
                const C2<R> d = Lower ? mk<R>(1, 0) : column[tid * kSub];
                const R den = d.x * d.x + d.y * d.y;
                const C2<R> reciprocal = mk<R>(d.x / den, -d.y / den);
#pragma unroll 8
                for (uint32_t q = 0; q < kSub; ++q) {
                    const uint32_t m = Lower ? q : kSub - 1 - q;
                    const C2<R> l = column[m * kSub];
                    if (!Lower && tid == m)
                        t = cmul<R>(t, reciprocal);
                    const C2<R> x = mk<R>(__shfl_sync(0xffffffffu, t.x, m), __shfl_sync(0xffffffffu, t.y, m));
                    if (Lower ? tid > m : tid < m)
                        csub<R>(t, l, x);
                }
                y[at] = t;
            }
            __syncthreads();
        } else {
            // x = inverse * (y - partial sums): 16 threads per row, two columns each
            const uint32_t row = tid / 16, c = 2 * (tid % 16);
            const C2<R> *block = subBlock(s, s) + row * kSub + c;
            C2<R> x = zero;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint32_t at = kSub * sub + c + h;
                C2<R> t = y[at];
#pragma unroll
                for (uint32_t q = 0; q < kTriGroups; ++q) {
                    t.x -= part[q][at].x;
                    t.y -= part[q][at].y;
                }
                cadd<R>(x, block[h], t);
            }
#pragma unroll
            for (int h = 8; h >= 1; h >>= 1) {
                x.x += __shfl_xor_sync(0xffffffffu, x.x, h);
                x.y += __shfl_xor_sync(0xffffffffu, x.y, h);
            }
            __syncthreads();  // y of this sub-block has been read
            if (c == 0)
                y[kSub * sub + row] = x;
            __syncthreads();
        }
        // its products into the rows still to be solved: 8 columns per thread
        const uint32_t ahead = Lower ? i / kSub : subs - 1 - i / kSub;  // this row's step
        if (i < kSub * subs && ahead > s) {
            const C2<R> *product = subBlock(ahead, s) + i % kSub;
#pragma unroll
            for (uint32_t q = 0; q < kSub / kTriGroups; ++q) {
                const uint32_t column = g * (kSub / kTriGroups) + q;
                cadd<R>(acc, product[column * kSub], y[kSub * sub + column]);
            }
        }
    }
    if (tid < nw) {
        st2(w + 2 * (n0 + tid), y[tid]);
        if (!Lower)
            st2(out + 2 * ((size_t(f) * E + e) * N + n0 + tid), y[tid]);
    }
}

// r = b - A x per row (FP64 accumulation), plus mass-scaled squares for the
// norms. A CTA takes 32 rows; its 8 warps take every 8th column, and the 8
// partial sums are added in a fixed order (deterministic).
__global__ void __launch_bounds__(256) residualKernel(const double *A, const double *b, const double *x,
                                                      const double *mass, uint32_t N, uint32_t E, double *correction,
                                                      double *squares) {
    __shared__ double2 part[8][32];
    const uint32_t lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const uint32_t a = blockIdx.x * 32 + lane;
    const uint32_t e = blockIdx.y, f = blockIdx.z;
    const double *M = A + size_t(f) * N * N * 2;
    const double *xv = x + (size_t(f) * E + e) * N * 2;
    double re = 0, im = 0;
    if (a < N)
        for (uint32_t c = g; c < N; c += 8) {
            const double2 m = ld2(M + 2 * (size_t(c) * N + a));
            const double2 v = ld2(xv + 2 * c);
            re += m.x * v.x - m.y * v.y;
            im += m.x * v.y + m.y * v.x;
        }
    part[g][lane] = mk<double>(re, im);
    __syncthreads();
    if (g != 0 || a >= N)
        return;
    re = 0;
    im = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        re += part[w][lane].x;
        im += part[w][lane].y;
    }
    const size_t idx = (size_t(f) * E + e) * N + a;
    const double2 bb = ld2(b + 2 * idx);
    re = bb.x - re;
    im = bb.y - im;
    st2(correction + 2 * idx, mk<double>(re, im));
    const double s = mass[a];
    squares[2 * idx] = (re * s) * (re * s) + (im * s) * (im * s);
    squares[2 * idx + 1] = (bb.x * s) * (bb.x * s) + (bb.y * s) * (bb.y * s);
}

// Deterministic per-vector sums of the squares -> norms[2] per (f, e).
__global__ void normKernel(const double *squares, uint32_t N, double *norms) {
    __shared__ double red[2][256];
    const size_t v = blockIdx.x;
    double r = 0, b = 0;
    for (uint32_t a = threadIdx.x; a < N; a += blockDim.x) {
        r += squares[2 * (v * N + a)];
        b += squares[2 * (v * N + a) + 1];
    }
    red[0][threadIdx.x] = r;
    red[1][threadIdx.x] = b;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < unsigned(s)) {
            red[0][threadIdx.x] += red[0][threadIdx.x + s];
            red[1][threadIdx.x] += red[1][threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        norms[2 * v] = sqrt(red[0][0]);
        norms[2 * v + 1] = sqrt(red[1][0]);
    }
}

__global__ void addKernel(double *x, const double *c, size_t count) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < count)
        x[i] += c[i];
}
__global__ void addFromFloatKernel(double *x, const float *c, size_t count) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < count)
        x[i] += double(c[i]);
}
__global__ void toFloatKernel(const double *in, float *out, size_t count) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < count)
        out[i] = float(in[i]);
}

template <class R> constexpr size_t panelRegSmem(uint32_t perBlock) { return size_t(kHalf) * perBlock * sizeof(C2<R>); }
template <class R> constexpr size_t kClusterSmem = size_t(kPanel) * kClusterRows<R> * sizeof(C2<R>);

cudaLaunchConfig_t clusterConfig(uint32_t C, uint32_t B, uint32_t threads, size_t smem, cudaStream_t stream,
                                 cudaLaunchAttribute &attr) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(C, B);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = C;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Shape of a panelRegKernel launch. Small CTAs shorten every step of a column
// (256 threads against 512: 11.0 against 11.7 ms FP32 and 13.6 against 14.8 ms
// FP64 at N = 6380, 0.82 against 0.89 at N = 642 x 32), as long as a cluster
// holds the panel and the batch's CTAs fit the device at once. For 257 to 512 rows
// that means two CTAs and a cluster barrier where one of 512 threads would do:
// FP64 equal within 1 % (N = 258: 0.319 against 0.317 ms, N = 505: 0.729 against
// 0.725), FP32 1 to 6 % slower (0.269 against 0.266, 0.605 against 0.570).
struct PanelShape {
    uint32_t threads, rowsPerThread;
};
template <class R> PanelShape panelShape(uint32_t rows, uint32_t B, uint32_t limit) {
    const uint32_t sms = uint32_t(smCount());
    PanelShape shape{256, 1};
    const auto ctas = [&]() { return (rows + shape.threads * shape.rowsPerThread - 1) / (shape.threads * shape.rowsPerThread); };
    if (ctas() > limit || B * ctas() > sms)
        shape.threads = 512;
    if (sizeof(R) == 4 && (ctas() > limit || B * ctas() > sms))
        shape.rowsPerThread = 2;
    return shape;
}
template <class R> uint32_t panelRegRows(uint32_t limit) { return limit * kPanelThreads * (sizeof(R) == 4 ? 2u : 1u); }

// Largest cluster the panel kernels may use on this device: 16 CTAs (opt-in)
// when the device can schedule such clusters with full shared memory, else the
// portable 8, else one CTA.
template <class R> uint32_t clusterLimitNow() {
    const auto fits = [](auto kernel, uint32_t c, uint32_t threads, size_t smem) {
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = clusterConfig(c, 1, threads, smem, nullptr, attr);
        int clusters = 0;
        const bool ok =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) == cudaSuccess &&
            (c <= 8 || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
            cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0;
        if (!ok)
            cudaGetLastError();
        return ok;
    };
    for (uint32_t c : {kMaxCluster, 8u, 1u}) {
        bool ok = fits(panelRegKernel<R, 1>, c, kPanelThreads, panelRegSmem<R>(kPanelThreads)) &&
                  (c == 1 || fits(panelClusterKernel<R>, c, 1024, kClusterSmem<R>));
        if constexpr (sizeof(R) == 4)
            ok = ok && fits(panelRegKernel<R, 2>, c, kPanelThreads, panelRegSmem<R>(2 * kPanelThreads));
        if (ok)
            return c;
    }
    throw std::runtime_error("LU panel kernel does not fit this device.");
}
template <class R> uint32_t clusterLimit() {
    static PerDeviceValue<uint32_t> limit;
    return limit.get([]() { return clusterLimitNow<R>(); });
}

// C -= L U of the FP64 factorisation over rows and columns from `from` on, up to column cEnd.
void launchGemm64(double *LU, uint32_t N, uint32_t B, uint32_t k0, uint32_t K, uint32_t cEnd, cudaStream_t stream) {
    const uint32_t from = k0 + K, rows = N - from, cols = cEnd - from;
    const auto tiles = [&](uint32_t t) { return dim3((rows + t - 1) / t, (cols + t - 1) / t, B); };
    const dim3 wide = tiles(64);
    if (size_t(wide.x) * wide.y * B >= size_t(smCount()))
        gemm64Kernel<64><<<wide, 128, kGemm64Smem<64>, stream>>>(LU, N, k0, K, from, from, cEnd);
    else
        gemm64Kernel<32><<<tiles(32), 128, kGemm64Smem<32>, stream>>>(LU, N, k0, K, from, from, cEnd);
}

// Columns per CTA of trsmBlockKernel: kTrsmColumns, or one per warp where that would leave most SMs idle.
template <class R> uint32_t trsmColumns(uint32_t rest, uint32_t B) {
    const uint32_t wide = uint32_t(kTrsmColumns);
    return size_t((rest + wide - 1) / wide) * B >= size_t(smCount()) ? wide : kTrsmThreads / 32;
}

// Right-looking LU with partial pivoting, 32-wide panels, two levels: panels
// update only the rest of their outer block (FP32: kOuter columns, FP64:
// kOuter64), then the outer block's U12 is solved (trsmBlockKernel) and the
// trailing matrix is updated once with K = the block's width, in FP32 on the
// tensor cores (trailingTensorKernel), in FP64 by gemm64Kernel.
template <class R> void factor(R *LU, uint32_t N, uint32_t B, int *pivots, int *info, cudaStream_t stream,
                               KernelTimer *timer, float *pack) {
    check(cudaMemsetAsync(info, 0, sizeof(int), stream), "LU info reset");
    const size_t gemmSmem = 2 * kPanel * 64 * sizeof(C2<R>);
    int *moves = pivots + 2 * size_t(B) * N;
    static PerDeviceOnce attributes;
    attributes.run([&]() {
        check(cudaFuncSetAttribute(trsmBlockKernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTrsmSmem<R>)),
              "block trsm smem attribute");
        if constexpr (sizeof(R) == 4) {
            check(cudaFuncSetAttribute(gemmKernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(gemmSmem)),
                  "gemm smem attribute");
            check(cudaFuncSetAttribute(trailingTensorKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTcSmem)),
                  "tensor update smem attribute");
        } else {
            check(cudaFuncSetAttribute(gemm64Kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(kGemm64Smem<64>)),
                  "gemm smem attribute");
        }
    });
    constexpr uint32_t outer = uint32_t(kOuterOf<R>);
    for (uint32_t K0 = 0; K0 < N; K0 += outer) {
        const uint32_t end = std::min(N, K0 + outer);
        for (uint32_t k0 = K0; k0 < end; k0 += kPanel) {
            const uint32_t jb = std::min(uint32_t(kPanel), end - k0);
            {
                TimedScope s(timer, "lu_panel", stream);
                const uint32_t rows = N - k0, limit = clusterLimit<R>();
                if (rows <= panelRegRows<R>(limit)) {  // rows in registers
                    const PanelShape shape = panelShape<R>(rows, B, limit);
                    const uint32_t perCta = shape.threads * shape.rowsPerThread;
                    const uint32_t C = (rows + perCta - 1) / perCta, perBlock = (rows + C - 1) / C;
                    cudaLaunchAttribute attr;
                    const cudaLaunchConfig_t cfg =
                        clusterConfig(C, B, shape.threads, panelRegSmem<R>(perBlock), stream, attr);
                    if constexpr (sizeof(R) == 4) {
                        const auto kernel = shape.rowsPerThread == 2 ? panelRegKernel<R, 2> : panelRegKernel<R, 1>;
                        check(cudaLaunchKernelEx(&cfg, kernel, LU, N, k0, jb, perBlock, pivots, moves, info),
                              "panel launch");
                    } else
                        check(cudaLaunchKernelEx(&cfg, panelRegKernel<R, 1>, LU, N, k0, jb, perBlock, pivots, moves,
                                                 info),
                              "panel launch");
                } else {
                    const uint32_t perBlock = (rows + limit - 1) / limit, cap = std::min(perBlock, kClusterRows<R>);
                    if (limit > 1 && rows <= limit * (kClusterRows<R> + kGlobalSlots * 1024u)) {
                        cudaLaunchAttribute attr;
                        const cudaLaunchConfig_t cfg =
                            clusterConfig(limit, B, 1024, size_t(jb) * cap * sizeof(C2<R>), stream, attr);
                        check(cudaLaunchKernelEx(&cfg, panelClusterKernel<R>, LU, N, k0, jb, perBlock, cap, pivots, info),
                              "cluster panel launch");
                    } else
                        panelKernel<R><<<B, 512, 0, stream>>>(LU, N, k0, jb, pivots, info);
                    panelMovesKernel<<<B, 32, 0, stream>>>(pivots, N, k0, jb, moves);
                }
            }
            {
                TimedScope s(timer, "lu_swap", stream);
                constexpr uint32_t columns = 8 * kSwapColumns;
                swapKernel<R><<<dim3((N + columns - 1) / columns, B), 256, 0, stream>>>(LU, N, k0, jb, moves);
            }
            const uint32_t cols = end - k0 - jb;  // columns of the outer block right of the panel
            if (cols) {
                {
                    TimedScope s(timer, "lu_trsm", stream);
                    trsmKernel<R><<<dim3((cols + kPanel - 1) / kPanel, B), 256, 0, stream>>>(LU, N, k0, jb, end);
                }
                TimedScope s(timer, "lu_gemm", stream);
                if constexpr (sizeof(R) == 4) {
                    const uint32_t rows = N - k0 - jb;
                    gemmKernel<R><<<dim3((rows + 63) / 64, (cols + 63) / 64, B), 256, gemmSmem, stream>>>(LU, N, k0, jb,
                                                                                                          end);
                } else
                    launchGemm64(LU, N, B, k0, jb, end, stream);
            }
            check(cudaGetLastError(), "LU launch");
        }
        if (end == N)
            break;
        const uint32_t rest = N - end;
        {
            TimedScope s(timer, "lu_trsm_outer", stream);
            const uint32_t columns = trsmColumns<R>(rest, B);
            trsmBlockKernel<R><<<dim3((rest + columns - 1) / columns, B), kTrsmThreads, kTrsmSmem<R>, stream>>>(
                LU, N, K0, columns);
        }
        if constexpr (sizeof(R) == 4) {
            const uint32_t rowTiles = (rest + kTcRows - 1) / kTcRows, colTiles = (rest + kTcCols - 1) / kTcCols;
            const size_t packStride = packFloats(N);
            {
                TimedScope s(timer, "lu_pack", stream);
                packKernel<<<dim3(rowTiles + colTiles, kTcSteps, B), 256, 0, stream>>>(LU, N, K0, pack, packStride);
            }
            TimedScope s(timer, "lu_gemm_tensor", stream);
            trailingTensorKernel<<<dim3(rowTiles, colTiles, B), kTcThreads, kTcSmem, stream>>>(LU, N, K0, pack,
                                                                                                packStride, info);
        } else {
            TimedScope s(timer, "lu_gemm", stream);
            launchGemm64(LU, N, B, K0, outer, N, stream);
        }
        check(cudaGetLastError(), "LU outer update launch");
    }
}

// A step that may start while the one before it runs (chainWait). The first follows gatherRhsKernel,
// a plain launch, so the factors are complete before any step starts.
template <class... P, class... A>
void launchStep(void (*kernel)(P...), dim3 grid, size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kTriThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    check(cudaLaunchKernelEx(&cfg, kernel, P(args)...), "triangular solve launch");
}

template <class R> void solve(const R *LU, const int *pivots, uint32_t N, uint32_t B, uint32_t E, R *x,
                              void *scratch, cudaStream_t stream, KernelTimer *timer) {
    TimedScope s(timer, "lu_solve", stream);
    static PerDeviceOnce attributes;
    attributes.run([]() {
        check(cudaFuncSetAttribute(triStepKernel<R, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTriSmem<R>)),
              "solve smem attribute");
        check(cudaFuncSetAttribute(triStepKernel<R, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTriSmem<R>)),
              "solve smem attribute");
    });
    const int *perm = pivots + size_t(B) * N;
    R *work = static_cast<R *>(scratch);
    gatherRhsKernel<R><<<dim3((N + 255) / 256, E, B), 256, 0, stream>>>(x, perm, N, E, work);
    const uint32_t blocks = (N + kTriBlock - 1) / kTriBlock;
    const auto grid = [&](uint32_t rows) { return dim3(1 + (rows + kTriBlock - 1) / kTriBlock, E, B); };
    // forward: block b is solved in step b with the rows updated by block b - 1
    for (uint32_t b = 0; b < blocks; ++b) {
        const uint32_t n0 = b * kTriBlock, nw = std::min(kTriBlock, N - n0);
        const uint32_t c0 = b ? n0 - kTriBlock : 0, cw = b ? kTriBlock : 0;
        launchStep(triStepKernel<R, true>, grid(b ? N - n0 - nw : 0), kTriSmem<R>, stream, LU, pivots, N, E, work, x, c0,
                   cw, n0, nw);
    }
    // backward: from the last block up
    for (uint32_t q = 0; q < blocks; ++q) {
        const uint32_t b = blocks - 1 - q;
        const uint32_t n0 = b * kTriBlock, nw = std::min(kTriBlock, N - n0);
        const uint32_t c0 = q ? n0 + kTriBlock : 0, cw = q ? std::min(kTriBlock, N - c0) : 0;
        launchStep(triStepKernel<R, false>, grid(q ? n0 : 0), kTriSmem<R>, stream, LU, pivots, N, E, work, x, c0, cw, n0,
                   nw);
    }
    check(cudaGetLastError(), "triangular solve launch");
}

// What the solves need of a factorisation: the composed permutations and, in FP32, the inverted diagonal blocks.
template <class R> void prepareSolves(const R *LU, int *pivots, uint32_t N, uint32_t B, cudaStream_t stream) {
    const size_t smem = 2 * size_t(N) * sizeof(int);
    if (smem > 48 * 1024)  // one kernel for both precisions, so one limit
        allowSharedMemory(permutationKernel);
    permutationKernel<<<B, 256, smem, stream>>>(pivots, N, pivots + size_t(B) * N);
    if constexpr (sizeof(R) == 4)
        diagonalInverseKernel<R><<<dim3((N + kSub - 1) / kSub, B, 2), 32, 0, stream>>>(LU, N, pivots, B);
    check(cudaGetLastError(), "solve preparation launch");
}

}  // namespace

void luFactorBatch(double *LU, uint32_t N, uint32_t B, int *pivots, int *info, cudaStream_t stream,
                   KernelTimer *timer) {
    factor<double>(LU, N, B, pivots, info, stream, timer, nullptr);
    prepareSolves<double>(LU, pivots, N, B, stream);
}
void luFactorBatch(float *LU, uint32_t N, uint32_t B, int *pivots, int *info, cudaStream_t stream,
                   KernelTimer *timer, float *pack) {
    factor<float>(LU, N, B, pivots, info, stream, timer, pack);
    prepareSolves<float>(LU, pivots, N, B, stream);
}
void luSolveBatch(const double *LU, const int *pivots, uint32_t N, uint32_t B, uint32_t E, double *x,
                  void *scratch, cudaStream_t stream, KernelTimer *timer) {
    solve<double>(LU, pivots, N, B, E, x, scratch, stream, timer);
}
void luSolveBatch(const float *LU, const int *pivots, uint32_t N, uint32_t B, uint32_t E, float *x,
                  void *scratch, cudaStream_t stream, KernelTimer *timer) {
    solve<float>(LU, pivots, N, B, E, x, scratch, stream, timer);
}

void residualBatch(const double *A, const double *b, const double *x, const double *mass, uint32_t N, uint32_t B,
                   uint32_t E, double *correction, double *norms, cudaStream_t stream, KernelTimer *timer) {
    double *squares = norms + 2 * size_t(B) * E;  // scratch after the norms
    {
        TimedScope s(timer, "residual", stream);
        residualKernel<<<dim3((N + 31) / 32, E, B), 256, 0, stream>>>(A, b, x, mass, N, E, correction, squares);
    }
    {
        TimedScope s(timer, "residual_norm", stream);
        normKernel<<<unsigned(B * E), 256, 0, stream>>>(squares, N, norms);
    }
    check(cudaGetLastError(), "residual launch");
}

void addCorrectionBatch(double *x, const double *correction, size_t count, cudaStream_t stream) {
    addKernel<<<unsigned((count + 255) / 256), 256, 0, stream>>>(x, correction, count);
    check(cudaGetLastError(), "refinement update launch");
}
void addCorrectionBatch(double *x, const float *correction, size_t count, cudaStream_t stream) {
    addFromFloatKernel<<<unsigned((count + 255) / 256), 256, 0, stream>>>(x, correction, count);
    check(cudaGetLastError(), "refinement update launch");
}
void roundToFloat(const double *in, float *out, size_t count, cudaStream_t stream) {
    toFloatKernel<<<unsigned((count + 255) / 256), 256, 0, stream>>>(in, out, count);
    check(cudaGetLastError(), "FP32 rounding launch");
}

namespace {
// Device memory of the LU test hook, freed on every exit path.
struct HookBuffer {
    void *p = nullptr;
    explicit HookBuffer(size_t bytes) { check(cudaMalloc(&p, std::max<size_t>(bytes, 16)), "LU hook allocation"); }
    ~HookBuffer() { cudaFree(p); }
    HookBuffer(const HookBuffer &) = delete;
    HookBuffer &operator=(const HookBuffer &) = delete;
};
}  // namespace

void debugLuFactor(bool fp32, uint32_t N, uint32_t B, const double *matrices, double *factors, int *pivots,
                   int *info) {
    const size_t reals = size_t(B) * N * N * 2;
    cudaStream_t stream = nullptr;
    check(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "LU hook stream");
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() { cudaStreamDestroy(s); }
    } guard{stream};
    HookBuffer lu(reals * (fp32 ? sizeof(float) : sizeof(double))), piv(luWorkspaceBytes(N, B)), status(sizeof(int));
    if (fp32) {
        HookBuffer pack(luPackBytes(N, B));
        std::vector<float> host(matrices, matrices + reals);
        check(cudaMemcpyAsync(lu.p, host.data(), reals * sizeof(float), cudaMemcpyHostToDevice, stream), "LU hook upload");
        luFactorBatch(static_cast<float *>(lu.p), N, B, static_cast<int *>(piv.p), static_cast<int *>(status.p), stream,
                      nullptr, static_cast<float *>(pack.p));
        check(cudaMemcpyAsync(host.data(), lu.p, reals * sizeof(float), cudaMemcpyDeviceToHost, stream), "LU hook download");
        check(cudaMemcpyAsync(pivots, piv.p, size_t(B) * N * sizeof(int), cudaMemcpyDeviceToHost, stream), "LU hook pivots");
        check(cudaMemcpyAsync(info, status.p, sizeof(int), cudaMemcpyDeviceToHost, stream), "LU hook status");
        check(cudaStreamSynchronize(stream), "LU hook");
        std::copy(host.begin(), host.end(), factors);
        return;
    }
    check(cudaMemcpyAsync(lu.p, matrices, reals * sizeof(double), cudaMemcpyHostToDevice, stream), "LU hook upload");
    luFactorBatch(static_cast<double *>(lu.p), N, B, static_cast<int *>(piv.p), static_cast<int *>(status.p), stream,
                  nullptr);
    check(cudaMemcpyAsync(factors, lu.p, reals * sizeof(double), cudaMemcpyDeviceToHost, stream), "LU hook download");
    check(cudaMemcpyAsync(pivots, piv.p, size_t(B) * N * sizeof(int), cudaMemcpyDeviceToHost, stream), "LU hook pivots");
    check(cudaMemcpyAsync(info, status.p, sizeof(int), cudaMemcpyDeviceToHost, stream), "LU hook status");
    check(cudaStreamSynchronize(stream), "LU hook");
}

size_t luWorkspaceBytes(uint32_t N, uint32_t B) {
    return inverseOffset(N, B) * sizeof(int) + size_t(B) * 2 * inverseEntries(N) * sizeof(float2);
}
size_t luPackBytes(uint32_t N, uint32_t B) { return size_t(B) * packFloats(N) * sizeof(float); }

}  // namespace hsb
