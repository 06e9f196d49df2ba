// FP64 Burton-Miller Galerkin assembly for sm_100a (the plain form).
//
// Method: modules/bem/cuda/cuda_solver.cu:266-540 with the FP64 sample of
// panel_integrals.cuh:166-198 — regular disjoint pairs with the qualified
// Dunavant 4/6/8 rule (or an accepted whole-panel 8/14 rule), touching pairs
// with Sauter-Schwab sectors, near pairs with their plan patches, plus half
// the P1 mass, rows equilibrated by the reciprocal lumped mass.
//
// B200 layout: a batch of frequencies runs in one launch (blockIdx.y). Each
// unordered regular or near pair is integrated once and yields both ordered
// blocks, because the reverse direction's double-layer kernel is the forward
// adjoint kernel at the same points. Pair blocks are written to per-pair
// records (no atomics) and reduced to the matrix by two deterministic
// gathers (trial vertex, then test vertex), so results are bit-reproducible.
#include "autotune.hpp"
#include "device_once.hpp"
#include "device_types.cuh"
#include "green_math.cuh"
#include "host_mesh.hpp"
#include "kernel_timer.hpp"
#include "near_tiles.cuh"

#include <algorithm>
#include <stdexcept>
#include <string>
#include <type_traits>

namespace hsb {
namespace {

constexpr double kInvFourPi = 0.07957747154594766788;
constexpr size_t kGatherColumnSmem = 200 * 1024;  // fused column gather: 3T complex FP64 entries

// Rule points (b0, b1, b2, w) of the four regular bins, in bin order
// (offsets 0, 6, 18, 34).
constexpr int kRulePoints = 98;
__constant__ double cRule[kRulePoints * 4];
__constant__ double cRuleSquares[kRulePoints * 3];  // b1^2, b1 b2, b2^2
__constant__ double cGauss20[40];

template <int NP> __device__ constexpr int ruleOffset() {
    return NP == 6 ? 0 : NP == 12 ? 6 : NP == 16 ? 18 : 34;
}

void cudaCheck(cudaError_t e, const char *what) {
    if (e != cudaSuccess)
        throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

__device__ __forceinline__ void flagError(int *error, int code) { atomicExch(error, code); }

// First entry of bin `bin` of frequency f (exactly packed bins when offsets are given).
__device__ __forceinline__ size_t binStart(const uint64_t *offsets, size_t capacity, int f, int bin) {
    return offsets ? size_t(offsets[f * kBins + bin]) : (size_t(f) * kBins + bin) * capacity;
}

// Moment accumulators of one ordered pair: MG = sum g bt bs, MP = sum P bt bs,
// MQ = sum Q bt bs (3x3 complex each) where, for delta = x_test - y_trial,
// g = w exp(-ikr)/(4 pi r), P = g (1+ikr) (delta.n_trial)/r^2 (double layer),
// Q = -g (1+ikr) (delta.n_test)/r^2 (adjoint double layer).
struct PairMoments {
    double g[18], p[18], q[18];
};

// Record entry o (0..11 forward block (test t, trial s); 12..23 reverse
// block (test s, trial t)) of an unordered pair from its moments. Forward:
// A_ij = -MP_ij + i k (n_t.n_s) MG_ij + alpha G (curl_ti . curl_sj),
// b_i = sum_j (-MG_ij + (i/k) MQ_ij); reverse swaps P and Q and transposes.
template <class Real>
__device__ __forceinline__ void pairRecordValue(int o, const Real *MG, const Real *MP, const Real *MQ,
                                                const DPanel &t, const DPanel &s, double k, double invk,
                                                double &re, double &im) {
    const double nn = t.n[0] * s.n[0] + t.n[1] * s.n[1] + t.n[2] * s.n[2];
    const bool reverse = o >= 12;
    const int e = reverse ? o - 12 : o;
    const Real *X = reverse ? MQ : MP;  // double-layer moments of this direction
    const Real *Y = reverse ? MP : MQ;  // adjoint moments of this direction
    if (e < 9) {
        // forward element (i, j); reverse element (row j of s, col i of t) = moments (i, j)
        const int row = e / 3, col = e % 3;
        const int i = reverse ? col : row, j = reverse ? row : col;
        const int m = 2 * (3 * i + j);
        double gre = 0, gim = 0;
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            gre += MG[2 * c];
            gim += MG[2 * c + 1];
        }
        const double curl = t.curl[3 * i] * s.curl[3 * j] + t.curl[3 * i + 1] * s.curl[3 * j + 1] +
                            t.curl[3 * i + 2] * s.curl[3 * j + 2];
        re = -X[m] - k * nn * MG[m + 1] + gim * curl * invk;
        im = -X[m + 1] + k * nn * MG[m] - gre * curl * invk;
    } else {
        const int a = e - 9;  // local row of this direction's test panel
        double sg_re = 0, sg_im = 0, sy_re = 0, sy_im = 0;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const int m = reverse ? 2 * (3 * b + a) : 2 * (3 * a + b);
            sg_re += MG[m];
            sg_im += MG[m + 1];
            sy_re += Y[m];
            sy_im += Y[m + 1];
        }
        re = -sg_re - sy_im * invk;
        im = -sg_im + sy_re * invk;
    }
}

// Both records of an unordered pair from its moments M = {MG, MP, MQ} (the
// formulas of pairRecordValue). ps = plane stride in complex values; whether a
// value was infinite or NaN is returned.
__device__ __forceinline__ bool storePairRecords(const double (&M)[54], const DPanel &t, const DPanel &s, double k,
                                                 double invk, double2 *fwd, double2 *rev, size_t ps) {
    const double *MG = M, *MP = M + 18, *MQ = M + 36;
    const double knn = k * (t.n[0] * s.n[0] + t.n[1] * s.n[1] + t.n[2] * s.n[2]);
    double gre = 0, gim = 0;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        gre += MG[2 * c];
        gim += MG[2 * c + 1];
    }
    gre *= invk;
    gim *= invk;
    unsigned largest = 0;  // of the high words: 0x7ff..... only for infinities and NaN
    const auto value = [&](double re, double im) {
        largest = max(largest, max(unsigned(__double2hiint(re)) & 0x7fffffffu, unsigned(__double2hiint(im)) & 0x7fffffffu));
        return make_double2(re, im);
    };
    // element (i, j): test vertex i, trial vertex j; X = MP forward, MQ reverse
    const auto element = [&](int i, int j, const double *X) {
        const double curl = t.curl[3 * i] * s.curl[3 * j] + t.curl[3 * i + 1] * s.curl[3 * j + 1] +
                            t.curl[3 * i + 2] * s.curl[3 * j + 2];
        const int m = 2 * (3 * i + j);
        return value(fma(gim, curl, fma(-knn, MG[m + 1], -X[m])), fma(-gre, curl, fma(knn, MG[m], -X[m + 1])));
    };
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        #pragma unroll
        for (int i = 0; i < 3; ++i) {
            fwd[j * ps + i] = element(i, j, MP);
            rev[i * ps + j] = element(i, j, MQ);
        }
    }
    // right-hand side moments of vertex a: sums over the other panel's vertices
    const auto moment = [&](int a, int own, int other, const double *Y) {
        double gr = 0, gi = 0, yr = 0, yi = 0;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const int m = own * a + other * b;
            gr += MG[m];
            gi += MG[m + 1];
            yr += Y[m];
            yi += Y[m + 1];
        }
        return value(fma(-yi, invk, -gr), fma(yr, invk, -gi));
    };
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        fwd[3 * ps + a] = moment(a, 6, 2, MQ);
        rev[3 * ps + a] = moment(a, 2, 6, MP);
    }
    return largest >= 0x7ff00000u;
}

// ---------------------------------------------------------------------------
// Regular pairs of the plain form: SPLIT threads per unordered pair, each
// owning every SPLIT-th test point with all its trial points.
//
// Bound: the FP64 pipe (64 fma per SM and clock), so the kernel is built to
// spend few FP64 instructions per sample and to keep the pipe fed from one
// thread's own unrolled samples. Per sample it accumulates moments against
// {1, b1, b2} of the trial barycentrics (b0 = 1 - b1 - b2 is taken once per
// test point) of g and of u = g (1 + ikr) / r^2, with u's second moments:
// the double-layer factor (x - y).n_trial is constant over the trial panel
// and (x - y).n_test affine in b1, b2, so both layers follow from u's moments
// once per test point. The 27 complex moments of the pair stay in registers
// and the records are written straight from them, without shared-memory
// exchanges or barriers between the steps of a pair. 128 threads at two CTAs
// per SM: 255 registers per thread. Measured (1280 triangles, 32 frequencies):
// 12 points 12.5 -> 7.25 ms, 6 points 11.0 -> 4.5 ms against one thread per
// test point with the contraction in shared memory; ncu: FP64 pipe 66 % and
// 61 % active, the rest fixed latencies that two warps per scheduler do not
// cover.
//
// SPLIT = 1 for the 6- and 12-point rules, whose pairs number in the
// millions on every mesh. The 16- and 64-point rules serve few pairs on small
// meshes (256 and 4096 samples each); there 8 and 32 threads share a pair and
// add their moments by shuffles.
// ---------------------------------------------------------------------------
constexpr int kPlainThreads = 128;

template <int NP> __device__ constexpr int plainSplit() { return NP == 64 ? 32 : NP == 16 ? 8 : 1; }

template <int NP>
__global__ void __launch_bounds__(kPlainThreads, 2) regularPairsKernel(const DPanel *__restrict__ panels, uint32_t T,
                                                          const double *__restrict__ ks,
                                                          const uint2 *__restrict__ bins,
                                                          const uint32_t *__restrict__ binCounts, size_t binCapacity,
                                                          const uint64_t *__restrict__ binOffsets, int bin,
                                                          double *__restrict__ records, SlotMap map, int *error) {
    constexpr int RO = ruleOffset<NP>(), SPLIT = plainSplit<NP>(), UNROLL = NP == 6 ? 6 : 4;
    const int f = blockIdx.y;
    const double k = ks[f], invk = 1.0 / k;
    const uint32_t count = binCounts[f * kBins + bin];
    const uint2 *list = bins + binStart(binOffsets, binCapacity, f, bin);
    double *rec = records + size_t(f) * map.planeSlots * kRecordDoubles;
    const uint32_t part = threadIdx.x % SPLIT;
    DistanceCheck distance;
    bool nonFinite = false, escaped = false;
    constexpr uint32_t PPC = kPlainThreads / SPLIT;
    for (uint32_t base = blockIdx.x * PPC; base < count; base += gridDim.x * PPC) {
        const uint32_t p = base + threadIdx.x / SPLIT;
        if (SPLIT == 1 && p >= count)
            break;
        // threads that share pairs stay together for the shuffles: a group past the end repeats the last pair
        const uint2 pr = list[SPLIT == 1 ? p : min(p, count - 1)];
        const DPanel &A = panels[pr.x], &S = panels[pr.y];
        const double se1[3] = {S.e1[0], S.e1[1], S.e1[2]}, se2[3] = {S.e2[0], S.e2[1], S.e2[2]};
        double M[54];
#pragma unroll
        for (int c = 0; c < 54; ++c)
            M[c] = 0;
#pragma unroll 1
        for (int x = int(part); x < NP; x += SPLIT) {
            const double bx1 = cRule[4 * (RO + x) + 1], bx2 = cRule[4 * (RO + x) + 2];
            // test point x relative to the trial panel's first vertex
            const double P0 = (A.v0[0] - S.v0[0]) + (A.e1[0] * bx1 + A.e2[0] * bx2);
            const double P1 = (A.v0[1] - S.v0[1]) + (A.e1[1] * bx1 + A.e2[1] * bx2);
            const double P2 = (A.v0[2] - S.v0[2]) + (A.e1[2] * bx1 + A.e2[2] * bx2);
            double g[6], u[12];  // g against 1, b1, b2; u against 1, b1, b2, b1^2, b1 b2, b2^2
#pragma unroll
            for (int c = 0; c < 6; ++c)
                g[c] = 0;
#pragma unroll
            for (int c = 0; c < 12; ++c)
                u[c] = 0;
#pragma unroll UNROLL
            for (int y = 0; y < NP; ++y) {
                const double b1 = cRule[4 * (RO + y) + 1], b2 = cRule[4 * (RO + y) + 2];
                const double *bb = cRuleSquares + 3 * (RO + y);
                const double dx = fma(-b2, se2[0], fma(-b1, se1[0], P0));
                const double dy = fma(-b2, se2[1], fma(-b1, se1[1], P1));
                const double dz = fma(-b2, se2[2], fma(-b1, se1[2], P2));
                const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
                distance.add(r2);
                const double rinv = reciprocalRoot(r2);
                const double kr = k * (r2 * rinv);
                double sn, cs;
                sinCos(kr, sn, cs);
                const double sc = cRule[4 * (RO + y) + 3] * rinv;
                const double gr = cs * sc, gi = -sn * sc;
                const double rinv2 = rinv * rinv;
                const double ur = fma(-gi, kr, gr) * rinv2, ui = fma(gr, kr, gi) * rinv2;
                g[0] += gr;
                g[1] += gi;
                g[2] = fma(gr, b1, g[2]);
                g[3] = fma(gi, b1, g[3]);
                g[4] = fma(gr, b2, g[4]);
                g[5] = fma(gi, b2, g[5]);
                u[0] += ur;
                u[1] += ui;
                u[2] = fma(ur, b1, u[2]);
                u[3] = fma(ui, b1, u[3]);
                u[4] = fma(ur, b2, u[4]);
                u[5] = fma(ui, b2, u[5]);
                u[6] = fma(ur, bb[0], u[6]);
                u[7] = fma(ui, bb[0], u[7]);
                u[8] = fma(ur, bb[1], u[8]);
                u[9] = fma(ui, bb[1], u[9]);
                u[10] = fma(ur, bb[2], u[10]);
                u[11] = fma(ui, bb[2], u[11]);
            }
            const double wx = cRule[4 * (RO + x) + 3];
            const double row[3] = {wx, wx * bx1, wx * bx2};
            // (x - y).n_trial: constant over the trial panel; -(x - y).n_test = q0 + t1 b1 + t2 b2
            const double ps = P0 * S.n[0] + P1 * S.n[1] + P2 * S.n[2];
            const double q0 = -(P0 * A.n[0] + P1 * A.n[1] + P2 * A.n[2]);
            const double t1 = se1[0] * A.n[0] + se1[1] * A.n[1] + se1[2] * A.n[2];
            const double t2 = se2[0] * A.n[0] + se2[1] * A.n[1] + se2[2] * A.n[2];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double rp = row[i] * ps;
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    M[6 * i + c] = fma(row[i], g[c], M[6 * i + c]);
                    M[18 + 6 * i + c] = fma(rp, u[c], M[18 + 6 * i + c]);
                }
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const double q[3] = {fma(t2, u[4 + c], fma(t1, u[2 + c], q0 * u[c])),
                                     fma(t2, u[8 + c], fma(t1, u[6 + c], q0 * u[2 + c])),
                                     fma(t2, u[10 + c], fma(t1, u[8 + c], q0 * u[4 + c]))};
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j)
                        M[36 + 6 * i + 2 * j + c] = fma(row[i], q[j], M[36 + 6 * i + 2 * j + c]);
            }
        }
        if (SPLIT > 1) {
#pragma unroll
            for (int h = SPLIT / 2; h >= 1; h >>= 1)
#pragma unroll
                for (int c = 0; c < 54; ++c)
                    M[c] += __shfl_xor_sync(0xffffffffu, M[c], h);
            if (part != 0 || p >= count)
                continue;
        }
        // from (1, b1, b2) to (b0, b1, b2) on both sides, and the panels' Jacobians
        const double w4 = 4.0 * A.area * S.area * kInvFourPi;
#pragma unroll
        for (int kind = 0; kind < 3; ++kind) {
            double *m = M + 18 * kind;
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    m[6 * i + c] -= m[6 * i + 2 + c] + m[6 * i + 4 + c];
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                m[c] = (m[c] - (m[6 + c] + m[12 + c])) * w4;
                m[6 + c] *= w4;
                m[12 + c] *= w4;
            }
        }
        const size_t fwd = mapSlot(map, T, pr.x, pr.y), rev = mapSlot(map, T, pr.y, pr.x);
        if (fwd == kNoSlot || rev == kNoSlot)
            escaped = true;
        else
            nonFinite |= storePairRecords(M, A, S, k, invk, reinterpret_cast<double2 *>(rec) + 3 * fwd,
                                          reinterpret_cast<double2 *>(rec) + 3 * rev, map.planeSlots * 3);
    }
    if (distance.bad())
        flagError(error, kErrDistance);
    if (nonFinite)
        flagError(error, kErrNonFinite);
    if (escaped)
        flagError(error, kErrEscapedPlan);
}

// ---------------------------------------------------------------------------
// Mixed form: the Green-kernel sample with FP32 arithmetic. The displacement
// and the phase k*r stay in FP64 (the phase reduced modulo 2 pi before the
// FP32 sine/cosine), because rounding r or k*r to FP32 leaves an
// O(eps_fp32 * k*r) phase error that no quadrature refinement removes
// (panel_integrals.cuh:91-142 keeps FP64 for k*r > 1 for the same reason).
// Returns g, P and Q (see PairMoments) as (re, im) pairs.
// ---------------------------------------------------------------------------
constexpr double kTwoPiHi = 6.283185307179586, kTwoPiLo = 2.4492935982947064e-16, kInvTwoPi = 0.15915494309189535;

__device__ __forceinline__ void mixedValues(double dx, double dy, double dz, float w, double k, const float *ns,
                                            const float *nt, float (&val)[6], bool &bad) {
    const float fx = float(dx), fy = float(dy), fz = float(dz);
    const float r2 = fx * fx + fy * fy + fz * fz;
    bad |= !(r2 > 0.f) || !isfinite(r2);
    const float rinv = rsqrtf(r2);
    // r in FP64 from one Newton step on the FP32 reciprocal root
    const double r2d = dx * dx + dy * dy + dz * dz;
    double y = double(rinv);
    y = y * (1.5 - 0.5 * r2d * y * y);
    const double ph = k * (r2d * y);
    const double turns = (ph * kInvTwoPi + 6755399441055744.0) - 6755399441055744.0;  // round to nearest
    const double th = fma(-turns, kTwoPiLo, fma(-turns, kTwoPiHi, ph));
    float sn, cs;
    __sincosf(float(th), &sn, &cs);  // th in [-pi, pi]: hardware sin/cos, absolute error about 4e-7
    const float kr = float(ph);
    const float sc = w * rinv;
    const float gr = cs * sc, gi = -sn * sc;
    const float rr = gr - gi * kr, ri = gi + gr * kr;
    const float rinv2 = rinv * rinv;
    const float ps = (fx * ns[0] + fy * ns[1] + fz * ns[2]) * rinv2;
    const float qt = -(fx * nt[0] + fy * nt[1] + fz * nt[2]) * rinv2;
    val[0] = gr;
    val[1] = gi;
    val[2] = rr * ps;
    val[3] = ri * ps;
    val[4] = rr * qt;
    val[5] = ri * qt;
}

// Regular pairs in the mixed form: one unordered pair per thread, NP x NP
// samples, trial bases contracted per test point, no FP64 per sample.
//
// Phase. Rounding r or k*r to FP32 leaves an O(eps_fp32 * k*r) phase error
// that no quadrature refinement removes (panel_integrals.cuh:91-142 keeps
// FP64 for k*r > 1 for that reason). Here the pair's centre distance r0 and
// its phase k*r0 are FP64 (reduced modulo 2 pi once per pair) and each sample
// adds k*(r - r0) = k*Delta/(r + r0) with Delta = r^2 - r0^2. With c the
// centre displacement, p the test point's offset and e(y) = E1 b1 + E2 b2 the
// trial point's offset (trial edges E1, E2), Delta = (2c + p).p
// - 2 (c + p).e(y) + |e(y)|^2, a quadratic in the trial barycentrics whose
// coefficients are formed once per pair and test point; its terms are
// O(r0 * h), so the FP32 phase error is O(eps * k * h), independent of k*r0.
// r^2 = r0^2 + Delta. sin/cos of the phase reduced to [-pi, pi] use the
// hardware approximation (absolute error about 4e-7).
// Amplitude. FP32 throughout (relative error ~eps_fp32, as for the
// reference's mixed sample); the double-layer projection (x - y).n_trial is
// constant over the trial panel and the adjoint one affine in b1, b2.
// Rule table per point: b0, b1, b2, w, b1^2, 2 b1 b2, b2^2, 0.
__constant__ float cRuleF[kRulePoints * 8];

// Record stores of a warp's 32 unordered pairs, one plane and direction at a
// time. A record plane entry is three complex values (48 B in FP64, 24 B in
// FP32), so a lane writing its own pair's values would touch 32 different
// sectors with every store and each sector two to four times. Here the lanes
// put their values in shared memory and write them out in memory order: the
// classification lists pairs in tiles of 8 test x 4 trial panels, so runs of 8
// (forward) and 4 (reverse) entries are contiguous and most sectors are
// written whole, once. On meshes whose record planes stay near the caches the
// second-level cache merges the partial sectors and the detour costs more than
// it saves, so DirectStore is the other form (launchRegular chooses).
template <class V> struct PlaneStore {
    V *stage;     // 96 entries of the warp
    V *dst[3];    // this lane's targets in plane 0 (null: no record)
    int src[3];   // and their places in `stage`
    // base: this lane's entry in plane 0, null without a pair; reverse: the order of the reverse slots
    __device__ __forceinline__ PlaneStore(V *warpStage, V *base, bool reverse) : stage(warpStage) {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int q = lane + 32 * c, t = q / 3, row = q % 3;
            const int pair = reverse ? (t & 3) * 8 + (t >> 2) : t;
            V *p = reinterpret_cast<V *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(base), pair));
            dst[c] = p ? p + row : nullptr;
            src[c] = 3 * pair + row;
        }
    }
    __device__ __forceinline__ void put(size_t offset, V v0, V v1, V v2) const {
        const int lane = threadIdx.x & 31;
        __syncwarp();  // the previous plane has been read
        stage[3 * lane] = v0;
        stage[3 * lane + 1] = v1;
        stage[3 * lane + 2] = v2;
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 3; ++c)
            if (dst[c])
                dst[c][offset] = stage[src[c]];
    }
};

// The same interface for a lane that writes its own pair's entries.
template <class V> struct DirectStore {
    V *base;
    __device__ __forceinline__ DirectStore(V *, V *entry, bool) : base(entry) {}
    __device__ __forceinline__ void put(size_t offset, V v0, V v1, V v2) const {
        base[offset] = v0;
        base[offset + 1] = v1;
        base[offset + 2] = v2;
    }
};

// Both records of an unordered regular pair (forward: test A, trial S;
// reverse: test S, trial A) from its FP32 moments (the layout and formulas of
// pairRecordValue). ps = plane stride in complex values; whether a value was
// infinite or NaN is returned.
template <class Store>
__device__ __forceinline__ bool storePairRecords(const float (&M)[54], const MixedPanel *__restrict__ pa,
                                                 const MixedPanel *__restrict__ pb, float k, float invk,
                                                 const Store &fwd, const Store &rev, size_t ps) {
    const float *MG = M, *MP = M + 18, *MQ = M + 36;
    const float4 na = pa->n, nb = pb->n;
    const float knn = k * (na.x * nb.x + na.y * nb.y + na.z * nb.z);
    float gre = 0.f, gim = 0.f;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        gre += MG[2 * c];
        gim += MG[2 * c + 1];
    }
    gre *= invk;
    gim *= invk;
    const float4 ca[3] = {pa->curl[0], pa->curl[1], pa->curl[2]}, cs[3] = {pb->curl[0], pb->curl[1], pb->curl[2]};
    float check = 0.f;
    const auto value = [&](float re, float im) {
        check += fabsf(re) + fabsf(im);
        return make_float2(re, im);
    };
    // element (i, j): A's local vertex i, S's local vertex j; X = MP forward, MQ reverse
    const auto element = [&](int i, int j, const float *X) {
        const float curl = ca[i].x * cs[j].x + ca[i].y * cs[j].y + ca[i].z * cs[j].z;
        const int m = 2 * (3 * i + j);
        return value(fmaf(gim, curl, fmaf(-knn, MG[m + 1], -X[m])), fmaf(-gre, curl, fmaf(knn, MG[m], -X[m + 1])));
    };
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        fwd.put(j * ps, element(0, j, MP), element(1, j, MP), element(2, j, MP));
        rev.put(j * ps, element(j, 0, MQ), element(j, 1, MQ), element(j, 2, MQ));
    }
    // right-hand side moments of vertex a: sums over the other panel's vertices
    const auto moment = [&](int a, int own, int other, const float *Y) {
        float gr = 0.f, gi = 0.f, yr = 0.f, yi = 0.f;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const int m = own * a + other * b;
            gr += MG[m];
            gi += MG[m + 1];
            yr += Y[m];
            yi += Y[m + 1];
        }
        return value(fmaf(-yi, invk, -gr), fmaf(yr, invk, -gi));
    };
    fwd.put(3 * ps, moment(0, 6, 2, MQ), moment(1, 6, 2, MQ), moment(2, 6, 2, MQ));
    rev.put(3 * ps, moment(0, 2, 6, MP), moment(1, 2, 6, MP), moment(2, 2, 6, MP));
    return !isfinite(check);
}

// Instruction issue bounds the sample loop (issue slots 79 % taken by the
// 12-point rule, 68 % by the 6-point one, whose pairs also wait for their
// panels). The real and imaginary accumulations therefore go out as one packed
// instruction, each half rounded as fmaf rounds it, and three CTAs an SM
// have the registers to hold the moments without spills:
// 12-point rule, 1280 panels at 32 frequencies 3.03 -> 2.72 ms, 8042 panels at
// three 9.2 -> 8.3 ms; staged 6-point rule at 12,756 panels 10.4 -> 9.4 ms.
// The direct 6-point rule waits on stores and keeps four CTAs (1.82 against
// 1.89 ms).
struct Packed {
    unsigned long long bits;
};
__device__ __forceinline__ Packed packed(float lo, float hi) {
    Packed p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p.bits) : "f"(lo), "f"(hi));
    return p;
}
__device__ __forceinline__ float2 unpacked(Packed p) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(p.bits));
    return v;
}
__device__ __forceinline__ Packed fma2(Packed a, Packed b, Packed c) {
    Packed r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.bits) : "l"(a.bits), "l"(b.bits), "l"(c.bits));
    return r;
}

template <int NP, bool Staged>
__global__ void __launch_bounds__(128, NP == 6 && !Staged ? 4 : 3) regularMixedKernel(const MixedPanel *__restrict__ mpanels,
                                                             const Bounds *__restrict__ bounds, uint32_t T,
                                                             const double *__restrict__ ks,
                                                             const uint2 *__restrict__ bins,
                                                             const uint32_t *__restrict__ binCounts, size_t binCapacity,
                                                             const uint64_t *__restrict__ binOffsets, int bin,
                                                             float *__restrict__ records, int *error) {
    constexpr int RO = ruleOffset<NP>();
    constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52: adding and subtracting rounds to an integer
    constexpr double kTwoPi = 6.283185307179586, kTwoPiLo = 2.4492935982947064e-16, kInvTwoPi = 0.15915494309189535;
    constexpr float kRoundF = 12582912.f;  // 1.5 * 2^23, the same for FP32
    constexpr float kTwoPiHiF = 6.28318548f, kTwoPiLoF = -1.74845553e-7f, kInvTwoPiF = 0.159154943f;
    const int f = blockIdx.y;
    const double k = ks[f];
    const float kf = float(k), invkf = float(1.0 / k);
    const uint32_t count = binCounts[f * kBins + bin];
    const uint2 *list = bins + binStart(binOffsets, binCapacity, f, bin);
    float2 *rec = reinterpret_cast<float2 *>(records + size_t(f) * T * T * kRecordDoubles);
    __shared__ float2 stage[4][Staged ? 96 : 1];
    float2 *const warpStage = stage[threadIdx.x / 32];
    using Store = std::conditional_t<Staged, PlaneStore<float2>, DirectStore<float2>>;
    bool bad = false, nonFinite = false;
    // staged: a warp takes 32 consecutive pairs, and lanes past the end repeat the last pair and store nothing
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; Staged ? (p & ~31u) < count : p < count;
         p += gridDim.x * blockDim.x) {
        const uint2 pr = list[Staged ? min(p, count - 1) : p];
        const MixedPanel &A = mpanels[pr.x], &S = mpanels[pr.y];
        const V3 ca = bounds[pr.x].center, cb = bounds[pr.y].center;
        // centre displacement, distance and phase (reduced to [-pi, pi]) in FP64
        const double cx = ca.x - cb.x, cy = ca.y - cb.y, cz = ca.z - cb.z;
        const double r0sqd = cx * cx + cy * cy + cz * cz, r0 = sqrt(r0sqd);
        const double ph0 = k * r0;
        const double turns = (ph0 * kInvTwoPi + kRound) - kRound;
        const float theta0 = float(fma(-turns, kTwoPiLo, fma(-turns, kTwoPi, ph0)));
        const float c[3] = {float(cx), float(cy), float(cz)};
        const float r0f = float(r0), r0sq = float(r0sqd);
        // test first vertex minus trial first vertex, about the centres
        const float4 aOff = A.offset, sOff = S.offset, aE1 = A.e1, aE2 = A.e2, sE1 = S.e1, sE2 = S.e2, aN = A.n,
                     sN = S.n;
        const float o0[3] = {aOff.x - sOff.x, aOff.y - sOff.y, aOff.z - sOff.z};
        const float ae1[3] = {aE1.x, aE1.y, aE1.z}, ae2[3] = {aE2.x, aE2.y, aE2.z};
        const float se1[3] = {sE1.x, sE1.y, sE1.z}, se2[3] = {sE2.x, sE2.y, sE2.z};
        const float ns[3] = {sN.x, sN.y, sN.z}, nt[3] = {aN.x, aN.y, aN.z};
        // |e(y)|^2 coefficients and trial edges against the test normal
        const float E11 = sE1.w, E12 = sN.w, E22 = sE2.w;
        const float t1 = se1[0] * nt[0] + se1[1] * nt[1] + se1[2] * nt[2];
        const float t2 = se2[0] * nt[0] + se2[1] * nt[1] + se2[2] * nt[2];
        const float w4 = 4.f * aOff.w * sOff.w * float(kInvFourPi);
        Packed moments[27];  // (re, im), three 3 x 3 blocks
#pragma unroll
        for (int i = 0; i < 27; ++i)
            moments[i] = packed(0.f, 0.f);
        float r2min = 3.4e38f;
#pragma unroll 1
        for (int x = 0; x < NP; ++x) {
            const float bx1 = cRuleF[8 * (RO + x) + 1], bx2 = cRuleF[8 * (RO + x) + 2];
            // P: test point minus the trial panel's first vertex, about the centres; CP = c + P
            float P[3], CP[3], C2P[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                P[i] = fmaf(ae1[i], bx1, fmaf(ae2[i], bx2, o0[i]));
                CP[i] = c[i] + P[i];
                C2P[i] = c[i] + CP[i];
            }
            const float psx = CP[0] * ns[0] + CP[1] * ns[1] + CP[2] * ns[2];
            const float qtx = -(CP[0] * nt[0] + CP[1] * nt[1] + CP[2] * nt[2]);
            // Delta = Ax + a1 b1 + a2 b2 + E11 b1^2 + 2 E12 b1 b2 + E22 b2^2
            const float Ax = C2P[0] * P[0] + C2P[1] * P[1] + C2P[2] * P[2];
            const float a1 = -2.f * (CP[0] * se1[0] + CP[1] * se1[1] + CP[2] * se1[2]);
            const float a2 = -2.f * (CP[0] * se2[0] + CP[1] * se2[1] + CP[2] * se2[2]);
            const float wx = cRuleF[8 * (RO + x) + 3] * w4;
            Packed G[3], U[3], Q[3];
#pragma unroll
            for (int i = 0; i < 3; ++i)
                G[i] = U[i] = Q[i] = packed(0.f, 0.f);
#pragma unroll(NP <= 16 ? NP : 4)
            for (int y = 0; y < NP; ++y) {
                const float *ry = cRuleF + 8 * (RO + y);
                const float b0 = ry[0], b1 = ry[1], b2 = ry[2];
                const float delta = fmaf(E22, ry[6], fmaf(E12, ry[5], fmaf(E11, ry[4], fmaf(a2, b2, fmaf(a1, b1, Ax)))));
                const float r2 = r0sq + delta;
                r2min = fminf(r2min, r2);
                const float rinv = rsqrtf(r2);
                const float r = r2 * rinv;
                const float theta = fmaf(kf, __fdividef(delta, r + r0f), theta0);
                const float qn = fmaf(theta, kInvTwoPiF, kRoundF) - kRoundF;
                float sn, cs;
                __sincosf(fmaf(-qn, kTwoPiLoF, fmaf(-qn, kTwoPiHiF, theta)), &sn, &cs);
                const float kr = kf * r;
                const float sc = (wx * ry[3]) * rinv;
                const float gr = cs * sc, gi = -sn * sc;
                const float rr = fmaf(-gi, kr, gr), ri = fmaf(gr, kr, gi);
                const float rinv2 = rinv * rinv;
                const float ur = rr * rinv2, ui = ri * rinv2;
                const float qt = fmaf(t1, b1, fmaf(t2, b2, qtx));
                const float qr = ur * qt, qi = ui * qt;
                const Packed g = packed(gr, gi), u = packed(ur, ui), q = packed(qr, qi);
                const Packed bs[3] = {packed(b0, b0), packed(b1, b1), packed(b2, b2)};
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    G[j] = fma2(g, bs[j], G[j]);
                    U[j] = fma2(u, bs[j], U[j]);
                    Q[j] = fma2(q, bs[j], Q[j]);
                }
            }
            const float bt[3] = {cRuleF[8 * (RO + x)], bx1, bx2};
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const float bp = bt[i] * psx;
                const Packed b = packed(bt[i], bt[i]), s = packed(bp, bp);
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    moments[3 * i + j] = fma2(b, G[j], moments[3 * i + j]);
                    moments[9 + 3 * i + j] = fma2(s, U[j], moments[9 + 3 * i + j]);
                    moments[18 + 3 * i + j] = fma2(b, Q[j], moments[18 + 3 * i + j]);
                }
            }
        }
        float M[54];
#pragma unroll
        for (int i = 0; i < 27; ++i) {
            const float2 v = unpacked(moments[i]);
            M[2 * i] = v.x;
            M[2 * i + 1] = v.y;
        }
        bad |= !(r2min > 0.f);
        nonFinite |= storePairRecords(
            M, &A, &S, kf, invkf,
            Store(warpStage, !Staged || p < count ? rec + (size_t(pr.y) * T + pr.x) * 3 : nullptr, false),
            Store(warpStage, !Staged || p < count ? rec + (size_t(pr.x) * T + pr.y) * 3 : nullptr, true),
            size_t(T) * T * 3);
    }
    if (bad)
        flagError(error, kErrDistance);
    if (nonFinite)
        flagError(error, kErrNonFinite);
}

// Number of 8 x 4 pair tiles before block q of trial panels j = 4q .. 4q + 3
// (block q holds q / 2 + 1 tiles of 8 test panels i = 8p .. 8p + 7, i < j).
__host__ __device__ inline uint64_t tilesBefore(uint64_t q) {
    const uint64_t m = q / 2;
    return q % 2 ? (m + 1) * (m + 1) : m * (m + 1);
}

// Sorts unordered regular pairs of each frequency into rule bins. Pairs are
// enumerated in tiles of 8 test x 4 trial panels, one tile per warp, so a
// warp's pairs (kept in lane order by the appends) write both
// orientations of their records in runs of whole sectors: 8 consecutive slots
// per trial panel forward, 4 per test panel in reverse. A thread decodes its
// pair, reads the pair code and both panels' bounds once, then classifies it
// at every frequency of the batch.
// The appends bound it: with one atomic per warp and bin, all to a few
// addresses, they were nearly all of its time. The CTA's warps therefore share
// one append per bin. 12,800 panels, both passes: 3.6 -> 1.9 ms.
constexpr int kClassifyThreads = 256;
__global__ void __launch_bounds__(kClassifyThreads)
    classifyPairsKernel(const uint8_t *__restrict__ pairCode, const Bounds *__restrict__ bounds, uint32_t T,
                        const double *__restrict__ ks, uint32_t B, double tol, uint32_t minDegree, uint2 *bins,
                        uint32_t *binCounts, size_t binCapacity, const uint64_t *binOffsets, bool countOnly,
                        int *error) {
    static_assert(kClassifyThreads / 32 * kBins == 32);
    __shared__ uint32_t starts[32];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t threads = 32 * tilesBefore((uint64_t(T) + 3) / 4);
    for (uint64_t base = uint64_t(blockIdx.x) * blockDim.x; base < threads; base += uint64_t(gridDim.x) * blockDim.x) {
        const uint64_t tile = (base + threadIdx.x) / 32;  // the same for the whole warp
        uint32_t i = 0, j = 0;
        uint8_t code = kPairTouching;  // no bin
        Bounds bi{}, bj{};
        if (tile < threads / 32) {
            uint64_t m = uint64_t((sqrt(4.0 * double(tile) + 1.0) - 1.0) * 0.5);
            while (m * (m + 1) > tile)
                --m;
            while ((m + 1) * (m + 2) <= tile)
                ++m;
            const uint64_t q = tile >= (m + 1) * (m + 1) ? 2 * m + 1 : 2 * m;
            const uint64_t p = tile - tilesBefore(q);
            i = uint32_t(8 * p + (lane & 7));
            j = uint32_t(4 * q + (lane >> 3));
        }
        if (j < T && i < j) {
            code = pairCode[uint64_t(j) * (j - 1) / 2 + i];
            if (code == kPairRegular) {
                bi = bounds[i];
                bj = bounds[j];
            }
        }
        for (uint32_t f = 0; f < B; ++f) {
            int bin = -1;
            if (code == kPairWhole8)
                bin = 2;
            else if (code == kPairWhole14)
                bin = 3;
            else if (code == kPairRegular) {
                const unsigned d = qualifiedDegree(bi, bj, ks[f], tol, minDegree);
                if (d == 4)
                    bin = 0;
                else if (d == 6)
                    bin = 1;
                else if (d == 8)
                    bin = 2;
                else
                    flagError(error, kErrEscapedPlan);
            }
            unsigned mask = 0, mine = 0;  // lanes of this lane's bin; lane b < kBins: count of bin b
#pragma unroll
            for (int b = 0; b < kBins; ++b) {
                const unsigned m = __ballot_sync(0xffffffffu, bin == b);
                if (bin == b)
                    mask = m;
                if (lane == unsigned(b))
                    mine = unsigned(__popc(m));
            }
            __syncwarp();  // the warp's other lanes have read the places of the frequency before
            if (lane < kBins)
                starts[warp * kBins + lane] = mine;
            __syncthreads();
            if (warp == 0) {  // lane = warp * kBins + bin: scan over the warps, one append per bin
                const uint32_t own = starts[lane];
                uint32_t sum = own;
#pragma unroll
                for (int d = kBins; d < 32; d *= 2) {
                    const uint32_t up = __shfl_up_sync(0xffffffffu, sum, d);
                    if (lane >= unsigned(d))
                        sum += up;
                }
                uint32_t start = 0;
                if (lane >= 32 - kBins && sum)
                    start = atomicAdd(&binCounts[f * kBins + lane % kBins], sum);
                start = __shfl_sync(0xffffffffu, start, 32 - kBins + lane % kBins);
                starts[lane] = start + sum - own;
            }
            __syncthreads();
            if (bin >= 0 && !countOnly)
                bins[binStart(binOffsets, binCapacity, int(f), bin) + starts[warp * kBins + bin] +
                     __popc(mask & ((1u << lane) - 1))] = make_uint2(i, j);
        }
    }
}

// Exclusive scan of the bin counts of all frequencies into bin offsets (a few
// dozen entries, one thread); the counts start again from zero for the fill pass.
__global__ void binOffsetsKernel(uint32_t *binCounts, uint64_t *binOffsets, uint32_t n) {
    uint64_t sum = 0;
    for (uint32_t q = 0; q < n; ++q) {
        binOffsets[q] = sum;
        sum += binCounts[q];
        binCounts[q] = 0;
    }
}

// The classification of classifyPairsKernel for a list of unordered pairs
// (i < j): the fast-multipole near field, whose records are only those of the
// near support pairs. Appends warp-aggregated like the full enumeration.
__global__ void classifyListKernel(const uint2 *__restrict__ list, uint64_t count, const uint8_t *__restrict__ pairCode,
                                   const Bounds *__restrict__ bounds, const double *__restrict__ ks, uint32_t B,
                                   double tol, uint32_t minDegree, uint2 *bins, uint32_t *binCounts,
                                   size_t binCapacity, int *error) {
    const unsigned lane = threadIdx.x & 31;
    const uint64_t padded = (count + 31) / 32 * 32;
    for (uint64_t q = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < padded; q += uint64_t(gridDim.x) * blockDim.x) {
        uint8_t code = kPairTouching;
        uint2 pr = make_uint2(0, 0);
        Bounds bi{}, bj{};
        if (q < count) {
            pr = list[q];
            code = pairCode[uint64_t(pr.y) * (pr.y - 1) / 2 + pr.x];
            if (code == kPairRegular) {
                bi = bounds[pr.x];
                bj = bounds[pr.y];
            }
        }
        for (uint32_t f = 0; f < B; ++f) {
            int bin = -1;
            if (code == kPairWhole8)
                bin = 2;
            else if (code == kPairWhole14)
                bin = 3;
            else if (code == kPairRegular) {
                const unsigned d = qualifiedDegree(bi, bj, ks[f], tol, minDegree);
                bin = d == 4 ? 0 : d == 6 ? 1 : d == 8 ? 2 : -1;
                if (bin < 0)
                    flagError(error, kErrEscapedPlan);
            }
#pragma unroll
            for (int b = 0; b < kBins; ++b) {
                const unsigned mask = __ballot_sync(0xffffffffu, bin == b);
                if (!mask)
                    continue;
                uint32_t start = 0;
                if (lane == unsigned(__ffs(mask) - 1))
                    start = atomicAdd(&binCounts[f * kBins + b], uint32_t(__popc(mask)));
                start = __shfl_sync(0xffffffffu, start, __ffs(mask) - 1);
                if (bin == b)
                    bins[(size_t(f) * kBins + b) * binCapacity + start + __popc(mask & ((1u << lane) - 1))] = pr;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Touching pairs (cuda_solver.cu:382-429) of the plain form: one warp per
// ordered job, a lane takes every 32nd (sector, u, v, w) tuple and runs over
// its radial nodes.
//
// Bound: the FP64 pipe. The sector maps do not depend on the job, so the
// tuples come from a table (buildSingularTuples: canonical barycentrics,
// displacement coefficients, weight) instead of being mapped again for every
// job. Along the radius a tuple's displacement is r l and both bases are
// affine in r, so a radial node only adds cos, sin and (1 + ikr) e^-ikr to
// moments against powers of r times the node's weight (34 FP64 instructions,
// 21 of them the phase's sine and cosine); the layers, normals and bases
// follow once per tuple. Shared edges are merged in the displacement
// coefficients, so l keeps its relative accuracy where the points nearly meet.
// Measured (1280 triangles, 32 frequencies): 7.15 -> 3.15 ms against one CTA per
// job that mapped its tuples and contracted every sample. Four CTAs per SM (a
// few registers spilled) beat three (3.28 ms) and two (3.57 ms).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 4) singularKernel(const DPanel *__restrict__ panels, uint32_t T,
                                                         const TouchingJob *__restrict__ jobs, uint32_t jobCount,
                                                         const double *__restrict__ ks,
                                                         const double *__restrict__ table, uint32_t order,
                                                         double *__restrict__ records, SlotMap map, int *error) {
    const uint32_t jobIndex = blockIdx.x * 4 + (threadIdx.x >> 5);
    const unsigned lane = threadIdx.x & 31;
    if (jobIndex >= jobCount)
        return;  // warp-uniform
    const TouchingJob job = jobs[jobIndex];
    const int f = blockIdx.y;
    const double k = ks[f], invk = 1.0 / k;
    const DPanel &t = panels[job.test];
    const DPanel &s = panels[job.trial];
    const bool coincident = job.topology == kCoincident;
    // canonical edges from the first shared vertex
    double A1[3], A2[3], B1[3], B2[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double te1 = t.e1[i], te2 = t.e2[i], se1 = s.e1[i], se2 = s.e2[i];
        const auto corner = [](int v, double e1, double e2) { return v == 0 ? 0.0 : v == 1 ? e1 : e2; };
        const double ta = corner(job.permTest[0], te1, te2), sa = corner(job.permTrial[0], se1, se2);
        A1[i] = corner(job.permTest[1], te1, te2) - ta;
        A2[i] = corner(job.permTest[2], te1, te2) - ta;
        B1[i] = corner(job.permTrial[1], se1, se2) - sa;
        B2[i] = corner(job.permTrial[2], se1, se2) - sa;
    }
    const double w4 = 4.0 * t.area * s.area * kInvFourPi;
    const double knn = k * (t.n[0] * s.n[0] + t.n[1] * s.n[1] + t.n[2] * s.n[2]);
    const uint32_t per = order * order * order;
    const uint32_t count = sectorCount(job.topology) * per;
    const uint32_t first = job.topology == kSharedVertex ? 0u : job.topology == kSharedEdge ? 2u * per : 7u * per;
    const double2 *tuples = reinterpret_cast<const double2 *>(table) + 6 * size_t(first);
    const double2 *radial = reinterpret_cast<const double2 *>(table) + 6 * size_t(13 * per);
    double m[18], b[6], g[2] = {0, 0};
#pragma unroll
    for (int c = 0; c < 18; ++c)
        m[c] = 0;
#pragma unroll
    for (int c = 0; c < 6; ++c)
        b[c] = 0;
    DistanceCheck distance;
#pragma unroll 1
    for (uint32_t idx = lane; idx < count; idx += 32) {
        const double2 *q = tuples + 6 * size_t(idx);
        const double2 q3 = q[3], q4 = q[4], q5 = q[5];
        double l[3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            l[i] = fma(A1[i], q3.x, fma(A2[i], q3.y, fma(-B1[i], q4.x, -B2[i] * q4.y)));
        const double lr2 = fma(l[0], l[0], fma(l[1], l[1], l[2] * l[2]));
        distance.add(lr2);
        const double linv = reciprocalRoot(lr2);
        const double kl = k * (lr2 * linv);
        // sums over the radial nodes: cos, sin against r^2 w (1, r, r^2), the real and imaginary part of
        // (1 + ikr) e^-ikr against r w (1, r, r^2)
        double gc[3] = {0, 0, 0}, gs[3] = {0, 0, 0}, uc[3] = {0, 0, 0}, us[3] = {0, 0, 0};
#pragma unroll 4
        for (uint32_t ri = 0; ri < order; ++ri) {
            const double2 r0 = radial[3 * ri], r1 = radial[3 * ri + 1], r2 = radial[3 * ri + 2];
            const double kr = kl * r0.x, weight[4] = {r0.y, r1.x, r1.y, r2.x};  // r w .. r^4 w
            double sn, cs;
            sinCos(kr, sn, cs);
            const double ur = fma(sn, kr, cs), ui = fma(cs, kr, -sn);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                gc[c] = fma(cs, weight[c + 1], gc[c]);
                gs[c] = fma(sn, weight[c + 1], gs[c]);
                uc[c] = fma(ur, weight[c], uc[c]);
                us[c] = fma(ui, weight[c], us[c]);
            }
        }
        const double scale = q5.x * w4 * linv, layer = coincident ? 0.0 : scale * (linv * linv);
        const double ps = layer * (l[0] * s.n[0] + l[1] * s.n[1] + l[2] * s.n[2]);
        const double qt = -layer * invk * (l[0] * t.n[0] + l[1] * t.n[1] + l[2] * t.n[2]);
        const double skn = scale * knn;
        g[0] = fma(scale, gc[0], g[0]);
        g[1] = fma(-scale, gs[0], g[1]);
        // bases at radius r: (1, 0, 0) + r c (test) and (1, 0, 0) + r d (trial)
        const double2 q0 = q[0], q1 = q[1], q2 = q[2];
        const double ct[3] = {q0.x, q0.y, q1.x}, dt[3] = {q1.y, q2.x, q2.y};
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            double a[3];
#pragma unroll
            for (int c = 0; c < 3; ++c)
                a[c] = part ? fma(skn, gc[c], -ps * us[c]) : fma(skn, gs[c], -ps * uc[c]);
            const double e[3] = {fma(dt[0], a[2], a[1]), dt[1] * a[2], dt[2] * a[2]};
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    m[2 * (3 * i + j) + part] = fma(ct[i], e[j], m[2 * (3 * i + j) + part]);
            m[part] += a[0];
#pragma unroll
            for (int j = 0; j < 3; ++j)
                m[2 * j + part] = fma(dt[j], a[1], m[2 * j + part]);
            const double b0 = part ? fma(scale, gs[0], qt * uc[0]) : -fma(scale, gc[0], qt * us[0]);
            const double b1 = part ? fma(scale, gs[1], qt * uc[1]) : -fma(scale, gc[1], qt * us[1]);
            b[part] += b0;
#pragma unroll
            for (int i = 0; i < 3; ++i)
                b[2 * i + part] = fma(ct[i], b1, b[2 * i + part]);
        }
    }
    if (__any_sync(0xffffffffu, distance.bad()) && lane == 0)
        flagError(error, kErrDistance);
    // warp sums as a reduce-scatter (31 shuffles): lane l ends with the sum of value l
    double v[32];
#pragma unroll
    for (int c = 0; c < 18; ++c)
        v[c] = m[c];
#pragma unroll
    for (int c = 0; c < 6; ++c)
        v[18 + c] = b[c];
    v[24] = g[0];
    v[25] = g[1];
#pragma unroll
    for (int c = 26; c < 32; ++c)
        v[c] = 0;
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
        const bool upper = (lane & unsigned(h)) != 0;
#pragma unroll
        for (int c = 0; c < h; ++c) {
            const double send = upper ? v[c] : v[c + h], keep = upper ? v[c + h] : v[c];
            v[c] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    const double sum = v[0];  // value `lane`
    // lanes 0..11 write record entry `lane`: canonical index of each local vertex
    const auto canonical = [](const uint8_t *perm, int vertex) {
        return perm[0] == vertex ? 0 : perm[1] == vertex ? 1 : 2;
    };
    const int o = lane < 12 ? int(lane) : 0;
    const int i = o < 9 ? o / 3 : o - 9, j = o % 3;
    const int ci = canonical(job.permTest, i), cj = canonical(job.permTrial, j);
    const int src = o < 9 ? 2 * (3 * ci + cj) : 18 + 2 * ci;
    const double vre = __shfl_sync(0xffffffffu, sum, src), vim = __shfl_sync(0xffffffffu, sum, src + 1);
    const double g0 = __shfl_sync(0xffffffffu, sum, 24), g1 = __shfl_sync(0xffffffffu, sum, 25);
    if (lane < 12) {
        double re = vre, im = vim;
        if (o < 9) {
            const double curl = t.curl[3 * i] * s.curl[3 * j] + t.curl[3 * i + 1] * s.curl[3 * j + 1] +
                                t.curl[3 * i + 2] * s.curl[3 * j + 2];
            re += g1 * curl * invk;
            im -= g0 * curl * invk;
        } else if (coincident)
            im += t.area / (6.0 * k);
        if (!isfinite(re) || !isfinite(im))
            flagError(error, kErrNonFinite);
        const size_t slot = mapSlot(map, T, job.test, job.trial);
        if (slot == kNoSlot)
            flagError(error, kErrEscapedPlan);
        else
            *reinterpret_cast<double2 *>(records + size_t(f) * map.planeSlots * kRecordDoubles +
                                         mapOffset(map.planeSlots, slot, o)) = make_double2(re, im);
    }
}

// Mixed form of the touching pairs: one warp per ordered job, FP32 samples.
// The sector maps do not depend on the job, so the (sector, u, v, w) tuples
// come from a table built once per singular order in FP64
// (buildSingularTable): canonical-order barycentrics at radius 1, the
// weight, and coefficients (a1, a2, b1, b2) of the displacement
// l = A1 a1 + A2 a2 - B1 b1 - B2 b2 over the canonical edges A (test) and B
// (trial) from the first shared vertex. For shared edges and coincident
// panels the shared edges are merged and their coefficients are differences
// formed in FP64, so l keeps FP32 relative accuracy where the two points
// nearly meet. Touching pairs have k*r <= 2 k h, so the FP32 phase needs no
// FP64 help; it is reduced to [-pi, pi] for the hardware sin/cos (absolute
// error about 4e-7). Moments accumulate in canonical order and are permuted
// back to local order once per job.
__global__ void __launch_bounds__(128, 6) singularMixedKernel(const DPanel *__restrict__ panels, uint32_t T,
                                                           const TouchingJob *__restrict__ jobs, uint32_t jobCount,
                                                           const double *__restrict__ ks,
                                                           const float4 *__restrict__ table, uint32_t order,
                                                           float *__restrict__ records, int *error) {
    constexpr float kRoundF = 12582912.f, kTwoPiHiF = 6.28318548f, kTwoPiLoF = -1.74845553e-7f,
                    kInvTwoPiF = 0.159154943f;
    const uint32_t jobIndex = blockIdx.x * 4 + (threadIdx.x >> 5);
    const unsigned lane = threadIdx.x & 31;
    if (jobIndex >= jobCount)
        return;  // warp-uniform
    const TouchingJob job = jobs[jobIndex];
    const int f = blockIdx.y;
    const double k = ks[f], invk = 1.0 / k;
    const float kf = float(k), invkf = float(invk);
    const DPanel &t = panels[job.test];
    const DPanel &s = panels[job.trial];
    const bool coincident = job.topology == kCoincident;
    // canonical edges from the first shared vertex, in FP64 then rounded
    float A1[3], A2[3], B1[3], B2[3];
    {
        const int ta = job.permTest[0], tb = job.permTest[1], tc = job.permTest[2];
        const int sa = job.permTrial[0], sb = job.permTrial[1], sc = job.permTrial[2];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double te[3] = {0.0, t.e1[i], t.e2[i]}, se[3] = {0.0, s.e1[i], s.e2[i]};
            A1[i] = float(te[tb] - te[ta]);
            A2[i] = float(te[tc] - te[ta]);
            B1[i] = float(se[sb] - se[sa]);
            B2[i] = float(se[sc] - se[sa]);
        }
    }
    const float w4 = float(4.0 * t.area * s.area * kInvFourPi);
    const float tn[3] = {float(t.n[0]), float(t.n[1]), float(t.n[2])};
    const float sn3[3] = {float(s.n[0]), float(s.n[1]), float(s.n[2])};
    const float knn = kf * float(t.n[0] * s.n[0] + t.n[1] * s.n[1] + t.n[2] * s.n[2]);
    const uint32_t per = order * order * order;
    const uint32_t count = sectorCount(job.topology) * per;
    const uint32_t base = job.topology == kSharedVertex ? 0u : job.topology == kSharedEdge ? 2u * per : 7u * per;
    const float4 *tuples = table + 3 * size_t(base);
    const float4 *radial = table + 3 * size_t(13 * per);
    float m[18], b[6], g[2] = {0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 18; ++c)
        m[c] = 0.f;
#pragma unroll
    for (int c = 0; c < 6; ++c)
        b[c] = 0.f;
    bool bad = false;
    for (uint32_t idx = lane; idx < count; idx += 32) {
        const float4 q0 = tuples[3 * idx], q1 = tuples[3 * idx + 1], q2 = tuples[3 * idx + 2];
        const float pt[3] = {q0.x, q0.y, q0.z}, pq[3] = {q0.w, q1.x, q1.y};
        float l[3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            l[i] = fmaf(A1[i], q1.z, fmaf(A2[i], q1.w, fmaf(-B1[i], q2.x, -B2[i] * q2.y)));
        const float ps1 = coincident ? 0.f : l[0] * sn3[0] + l[1] * sn3[1] + l[2] * sn3[2];
        const float qt1 = coincident ? 0.f : -(l[0] * tn[0] + l[1] * tn[1] + l[2] * tn[2]);
        const float lr2 = l[0] * l[0] + l[1] * l[1] + l[2] * l[2];
        bad |= !(lr2 > 0.f) || !isfinite(lr2);
        const float linv = rsqrtf(lr2), llen = lr2 * linv;
        const float pw = q2.z * w4;
#pragma unroll 4
        for (uint32_t ri = 0; ri < order; ++ri) {
            const float4 rad = radial[ri];  // (r, r^3 w_r, 1/r, 1 - r)
            const float r = rad.x;
            // sample at radial fraction r: displacement r*l, distance r*|l|
            const float rinv = linv * rad.z, kr = kf * (llen * r);
            // phase reduced to [-pi, pi], hardware sin/cos (absolute error about 4e-7)
            const float qn = fmaf(kr, kInvTwoPiF, kRoundF) - kRoundF;
            float sn, cs;
            __sincosf(fmaf(-qn, kTwoPiLoF, fmaf(-qn, kTwoPiHiF, kr)), &sn, &cs);
            const float sc = pw * rad.y * rinv;
            const float gr = cs * sc, gi = -sn * sc;
            g[0] += gr;
            g[1] += gi;
            const float rr = fmaf(-gi, kr, gr), ri2 = fmaf(gr, kr, gi);
            // (r l).n / (r |l|)^2 = (l.n) / (r |l|^2)
            const float inv = rinv * linv;
            const float ps = ps1 * inv, qt = qt1 * inv;
            const float ar = fmaf(-rr, ps, -knn * gi), ai = fmaf(-ri2, ps, knn * gr);
            const float br = fmaf(-ri2 * qt, invkf, -gr), bi = fmaf(rr * qt, invkf, -gi);
            const float bt[3] = {fmaf(r, pt[0], rad.w), r * pt[1], r * pt[2]};
            const float bs[3] = {fmaf(r, pq[0], rad.w), r * pq[1], r * pq[2]};
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                b[2 * i] = fmaf(br, bt[i], b[2 * i]);
                b[2 * i + 1] = fmaf(bi, bt[i], b[2 * i + 1]);
                const float ari = ar * bt[i], aii = ai * bt[i];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    m[2 * (3 * i + j)] = fmaf(ari, bs[j], m[2 * (3 * i + j)]);
                    m[2 * (3 * i + j) + 1] = fmaf(aii, bs[j], m[2 * (3 * i + j) + 1]);
                }
            }
        }
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0)
        flagError(error, kErrDistance);
    // Warp sums of the 26 moment values as a reduce-scatter: after the pass at
    // distance h a lane keeps the h partial sums of the half its lane bit h
    // selects, so after five passes (31 shuffles instead of 26 x 5) lane l holds
    // the sum of value l.
    float v[32];
#pragma unroll
    for (int c = 0; c < 18; ++c)
        v[c] = m[c];
#pragma unroll
    for (int c = 0; c < 6; ++c)
        v[18 + c] = b[c];
    v[24] = g[0];
    v[25] = g[1];
#pragma unroll
    for (int c = 26; c < 32; ++c)
        v[c] = 0.f;
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
        const bool upper = (lane & unsigned(h)) != 0;
#pragma unroll
        for (int c = 0; c < h; ++c) {
            const float send = upper ? v[c] : v[c + h], keep = upper ? v[c + h] : v[c];
            v[c] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    const float sum = v[0];  // value `lane`
    // lanes 0..11 write record entry `lane`: canonical index of each local vertex
    int invT[3], invS[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        invT[job.permTest[c]] = c;
        invS[job.permTrial[c]] = c;
    }
    const int o = lane < 12 ? int(lane) : 0;
    const int i = o < 9 ? o / 3 : o - 9, j = o % 3;
    const int src = o < 9 ? 2 * (3 * invT[i] + invS[j]) : 18 + 2 * invT[i];
    const float vre = __shfl_sync(0xffffffffu, sum, src), vim = __shfl_sync(0xffffffffu, sum, src + 1);
    const float g0 = __shfl_sync(0xffffffffu, sum, 24), g1 = __shfl_sync(0xffffffffu, sum, 25);
    if (lane < 12) {
        double re, im;
        if (o < 9) {
            const double curl = t.curl[3 * i] * s.curl[3 * j] + t.curl[3 * i + 1] * s.curl[3 * j + 1] +
                                t.curl[3 * i + 2] * s.curl[3 * j + 2];
            re = double(vre) + double(g1) * curl * invk;
            im = double(vim) - double(g0) * curl * invk;
        } else {
            re = vre;
            im = double(vim) + (coincident ? t.area / (6.0 * k) : 0.0);
        }
        if (!isfinite(re) || !isfinite(im))
            flagError(error, kErrNonFinite);
        float *dst = records + size_t(f) * T * T * kRecordDoubles + recordOffset(T, size_t(job.trial) * T + job.test, o);
        *reinterpret_cast<float2 *>(dst) = make_float2(float(re), float(im));
    }
}

// ---------------------------------------------------------------------------
// Near pairs (cuda_solver.cu:430-518, near_projection.hpp:228-254): one CTA
// per unordered pair, both directions from the shared patch samples.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void nearSample(double (&acc)[54], const DPanel &t, const DPanel &s, const double *bt,
                                           const double *bs, double w, double k, bool &bad) {
    const double dx = (t.v0[0] - s.v0[0]) + ((t.e1[0] * bt[1] + t.e2[0] * bt[2]) - (s.e1[0] * bs[1] + s.e2[0] * bs[2]));
    const double dy = (t.v0[1] - s.v0[1]) + ((t.e1[1] * bt[1] + t.e2[1] * bt[2]) - (s.e1[1] * bs[1] + s.e2[1] * bs[2]));
    const double dz = (t.v0[2] - s.v0[2]) + ((t.e1[2] * bt[1] + t.e2[2] * bt[2]) - (s.e1[2] * bs[1] + s.e2[2] * bs[2]));
    const double r2 = dx * dx + dy * dy + dz * dz;
    bad |= !(r2 > 0) || !isfinite(r2);
    const double rinv = rsqrt(r2);
    const double r = r2 * rinv, kr = k * r;
    double sn, cs;
    sincos(kr, &sn, &cs);
    const double sc = w * rinv;
    const double gr = cs * sc, gi = -sn * sc;
    const double rr = gr - gi * kr, ri = gi + gr * kr;
    const double rinv2 = rinv * rinv;
    const double ps = (dx * s.n[0] + dy * s.n[1] + dz * s.n[2]) * rinv2;
    const double qt = -(dx * t.n[0] + dy * t.n[1] + dz * t.n[2]) * rinv2;
    const double val[6] = {gr, gi, rr * ps, ri * ps, rr * qt, ri * qt};
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double bij = bt[i] * bs[j];
#pragma unroll
            for (int kind = 0; kind < 3; ++kind) {
                acc[kind * 18 + 2 * (3 * i + j)] += val[2 * kind] * bij;
                acc[kind * 18 + 2 * (3 * i + j) + 1] += val[2 * kind + 1] * bij;
            }
        }
}

// Mixed-form near sample: FP64 displacement and phase, FP32 kernel values
// and accumulation.
__device__ __forceinline__ void nearSample(float (&acc)[54], const DPanel &t, const DPanel &s, const double *bt,
                                           const double *bs, double w, double k, bool &bad) {
    const double dx = (t.v0[0] - s.v0[0]) + ((t.e1[0] * bt[1] + t.e2[0] * bt[2]) - (s.e1[0] * bs[1] + s.e2[0] * bs[2]));
    const double dy = (t.v0[1] - s.v0[1]) + ((t.e1[1] * bt[1] + t.e2[1] * bt[2]) - (s.e1[1] * bs[1] + s.e2[1] * bs[2]));
    const double dz = (t.v0[2] - s.v0[2]) + ((t.e1[2] * bt[1] + t.e2[2] * bt[2]) - (s.e1[2] * bs[1] + s.e2[2] * bs[2]));
    const float ns[3] = {float(s.n[0]), float(s.n[1]), float(s.n[2])};
    const float nt[3] = {float(t.n[0]), float(t.n[1]), float(t.n[2])};
    float val[6];
    mixedValues(dx, dy, dz, float(w), k, ns, nt, val, bad);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const float bij = float(bt[i] * bs[j]);
#pragma unroll
            for (int kind = 0; kind < 3; ++kind) {
                acc[kind * 18 + 2 * (3 * i + j)] += val[2 * kind] * bij;
                acc[kind * 18 + 2 * (3 * i + j) + 1] += val[2 * kind + 1] * bij;
            }
        }
}

// Near pairs whose patches are all tensor patches: one warp per unordered
// pair. Lane (x, half) owns test point x of the patch rule and half of the
// trial points; trial bases are contracted in registers, test bases through
// shared memory by the 27 lanes that own a (kind, i, j) moment. Pairs with
// projected patches go to nearKernel.
//
// The plain form accumulates the moments of regularPairsKernel with the short
// root and sine/cosine; the mixed form keeps its sample and converts a patch
// point's barycentrics to FP32 once. Jobs come with the most patches first (the
// plan sorts them): patch counts range from one to hundreds, and in plan order
// long pairs that started last left two thirds of the warps idle. Measured:
// 8042 triangles x 3 frequencies (mixed) 16.8 -> 10.8 ms, 12 756 triangles plain
// 11.7 -> 6.3, mixed 7.5 -> 5.0, 1280 x 32 plain 1.91 -> 1.39. Eight CTAs per SM
// (mixed) and six (plain) are the most without spills. FP64 pipe 52 % (plain),
// conversion pipe 49 % (mixed) active.
template <bool Mixed>
__global__ void __launch_bounds__(64, Mixed ? 8 : 6) nearWarpKernel(const DPanel *__restrict__ panels, uint32_t T,
                                                      const NearPairJob *__restrict__ jobs, uint32_t jobCount,
                                                      const Patch *__restrict__ patches, const double *__restrict__ ks,
                                                      std::conditional_t<Mixed, float, double> *__restrict__ records,
                                                      SlotMap map, int *error) {
    using Acc = std::conditional_t<Mixed, float, double>;
    __shared__ Acc sS[2][64][18];     // per warp: trial-contracted values S(x)
    __shared__ double sB[2][64][3];   // per warp: mapped test barycentrics
    __shared__ __align__(16) double2 sE[2][64][2];  // per warp: trial points' offsets from the trial panel's first vertex
    // per warp and trial point: mapped barycentrics (mixed: b0, b1, b2 in FP32; plain: b1, b2, b1^2, b1 b2, b2^2)
    __shared__ __align__(16) std::conditional_t<Mixed, float4, double2> sY[2][64][Mixed ? 1 : 3];
    __shared__ double sM[2][54];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t pairIndex = blockIdx.x * 2 + warp;
    if (pairIndex >= jobCount)
        return;
    const NearPairJob job = jobs[pairIndex];
    const int f = blockIdx.y;
    const double k = ks[f], invk = 1.0 / k;
    const DPanel &t = panels[job.first];
    const DPanel &s = panels[job.second];
    const double w4 = 4.0 * t.area * s.area * kInvFourPi;
    bool bad = false;
    double own[2] = {0, 0};  // lanes 0..26: accumulated moment (kind, i, j) of this pair
    const double d0[3] = {t.v0[0] - s.v0[0], t.v0[1] - s.v0[1], t.v0[2] - s.v0[2]};
    [[maybe_unused]] const float nsF[3] = {float(s.n[0]), float(s.n[1]), float(s.n[2])};
    [[maybe_unused]] const float ntF[3] = {float(t.n[0]), float(t.n[1]), float(t.n[2])};
    // plain: -(x - y).n_test = q0 + t1 b1 + t2 b2 of the trial barycentrics
    [[maybe_unused]] double q0 = 0, t1 = 0, t2 = 0;
    if constexpr (!Mixed) {
        q0 = -(d0[0] * t.n[0] + d0[1] * t.n[1] + d0[2] * t.n[2]);
        t1 = s.e1[0] * t.n[0] + s.e1[1] * t.n[1] + s.e1[2] * t.n[2];
        t2 = s.e2[0] * t.n[0] + s.e2[1] * t.n[1] + s.e2[2] * t.n[2];
    }
    [[maybe_unused]] DistanceCheck distance;
    for (uint32_t q = 0; q < job.patchCount; ++q) {
        const Patch &patch = patches[job.firstPatch + q];
        const int n = patch.degree == 14 ? 64 : 16;
        const int ro = patch.degree == 14 ? 34 : 18;  // rule offsets of the 16- and 64-point bins
        // mapped rule points of this patch (test from patch.test, trial from patch.trial)
        for (int idx = lane; idx < n; idx += 32) {
            double by[3], e[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                sB[warp][idx][i] = cRule[4 * (ro + idx)] * patch.test[i] + cRule[4 * (ro + idx) + 1] * patch.test[3 + i] +
                                   cRule[4 * (ro + idx) + 2] * patch.test[6 + i];
                by[i] = cRule[4 * (ro + idx)] * patch.trial[i] + cRule[4 * (ro + idx) + 1] * patch.trial[3 + i] +
                        cRule[4 * (ro + idx) + 2] * patch.trial[6 + i];
            }
            // the trial point's offset from the trial panel's first vertex, once per patch point
#pragma unroll
            for (int c = 0; c < 3; ++c)
                e[c] = s.e1[c] * by[1] + s.e2[c] * by[2];
            sE[warp][idx][0] = make_double2(e[0], e[1]);
            sE[warp][idx][1] = make_double2(e[2], 0);
            if constexpr (Mixed)
                sY[warp][idx][0] = make_float4(float(by[0]), float(by[1]), float(by[2]), 0.f);
            else {
                sY[warp][idx][0] = make_double2(by[1], by[2]);
                sY[warp][idx][1] = make_double2(by[1] * by[1], by[1] * by[2]);
                sY[warp][idx][2] = make_double2(by[2] * by[2], 0);
            }
        }
        __syncwarp();
        const double wpatch = patch.areaFraction * w4;
        // lane -> test points x = lane (+32) ; for n = 16, lanes 16..31 take the second half of the trial points
        const int xCount = n == 16 ? 1 : 2;
        for (int xi = 0; xi < xCount; ++xi) {
            const int x = n == 16 ? (lane & 15) : lane + 32 * xi;
            const int y0 = n == 16 ? (lane >> 4) * 8 : 0, y1 = n == 16 ? y0 + 8 : n;
            const double *bt = sB[warp][x];
            const double Dx = d0[0] + (t.e1[0] * bt[1] + t.e2[0] * bt[2]);
            const double Dy = d0[1] + (t.e1[1] * bt[1] + t.e2[1] * bt[2]);
            const double Dz = d0[2] + (t.e1[2] * bt[1] + t.e2[2] * bt[2]);
            const double wx = cRule[4 * (ro + x) + 3] * wpatch;
            Acc S[18];
            if constexpr (Mixed) {
#pragma unroll
                for (int c = 0; c < 18; ++c)
                    S[c] = 0;
#pragma unroll 2
                for (int y = y0; y < y1; ++y) {
                    const float4 bs = sY[warp][y][0];
                    const double2 e0 = sE[warp][y][0];
                    const double dx = Dx - e0.x;
                    const double dy = Dy - e0.y;
                    const double dz = Dz - sE[warp][y][1].x;
                    float val[6];
                    mixedValues(dx, dy, dz, float(wx * cRule[4 * (ro + y) + 3]), k, nsF, ntF, val, bad);
                    const float b[3] = {bs.x, bs.y, bs.z};
#pragma unroll
                    for (int kind = 0; kind < 3; ++kind)
#pragma unroll
                        for (int j = 0; j < 3; ++j) {
                            S[kind * 6 + 2 * j] += val[2 * kind] * b[j];
                            S[kind * 6 + 2 * j + 1] += val[2 * kind + 1] * b[j];
                        }
                }
            } else {
                // moments of g against 1, b1, b2 and of u = g (1 + ikr) / r^2 up to second order, as in
                // regularPairsKernel
                double g[6], u[12];
#pragma unroll
                for (int c = 0; c < 6; ++c)
                    g[c] = 0;
#pragma unroll
                for (int c = 0; c < 12; ++c)
                    u[c] = 0;
#pragma unroll 2
                for (int y = y0; y < y1; ++y) {
                    const double2 e0 = sE[warp][y][0], b01 = sY[warp][y][0], b2nd = sY[warp][y][1];
                    const double b1 = b01.x, b2 = b01.y, b22 = sY[warp][y][2].x;
                    const double dx = Dx - e0.x, dy = Dy - e0.y, dz = Dz - sE[warp][y][1].x;
                    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
                    distance.add(r2);
                    const double rinv = reciprocalRoot(r2);
                    const double kr = k * (r2 * rinv);
                    double sn, cs;
                    sinCos(kr, sn, cs);
                    const double sc = cRule[4 * (ro + y) + 3] * rinv;
                    const double gr = cs * sc, gi = -sn * sc;
                    const double rinv2 = rinv * rinv;
                    const double ur = fma(-gi, kr, gr) * rinv2, ui = fma(gr, kr, gi) * rinv2;
                    g[0] += gr;
                    g[1] += gi;
                    g[2] = fma(gr, b1, g[2]);
                    g[3] = fma(gi, b1, g[3]);
                    g[4] = fma(gr, b2, g[4]);
                    g[5] = fma(gi, b2, g[5]);
                    u[0] += ur;
                    u[1] += ui;
                    u[2] = fma(ur, b1, u[2]);
                    u[3] = fma(ui, b1, u[3]);
                    u[4] = fma(ur, b2, u[4]);
                    u[5] = fma(ui, b2, u[5]);
                    u[6] = fma(ur, b2nd.x, u[6]);
                    u[7] = fma(ui, b2nd.x, u[7]);
                    u[8] = fma(ur, b2nd.y, u[8]);
                    u[9] = fma(ui, b2nd.y, u[9]);
                    u[10] = fma(ur, b22, u[10]);
                    u[11] = fma(ui, b22, u[11]);
                }
                // (x - y).n_trial is constant over the trial panel
                const double ps = wx * (Dx * s.n[0] + Dy * s.n[1] + Dz * s.n[2]);
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    S[2 + c] = wx * g[2 + c];
                    S[4 + c] = wx * g[4 + c];
                    S[c] = wx * (g[c] - (g[2 + c] + g[4 + c]));
                    S[8 + c] = ps * u[2 + c];
                    S[10 + c] = ps * u[4 + c];
                    S[6 + c] = ps * (u[c] - (u[2 + c] + u[4 + c]));
                    const double m0 = fma(t2, u[4 + c], fma(t1, u[2 + c], q0 * u[c]));
                    const double m1 = fma(t2, u[8 + c], fma(t1, u[6 + c], q0 * u[2 + c]));
                    const double m2 = fma(t2, u[10 + c], fma(t1, u[8 + c], q0 * u[4 + c]));
                    S[14 + c] = wx * m1;
                    S[16 + c] = wx * m2;
                    S[12 + c] = wx * (m0 - (m1 + m2));
                }
            }
            if (n == 16) {
#pragma unroll
                for (int c = 0; c < 18; ++c)
                    S[c] += __shfl_xor_sync(0xffffffffu, S[c], 16);
                if (lane < 16)
#pragma unroll
                    for (int c = 0; c < 18; ++c)
                        sS[warp][x][c] = S[c];
            } else {
#pragma unroll
                for (int c = 0; c < 18; ++c)
                    sS[warp][x][c] = S[c];
            }
        }
        __syncwarp();
        if (lane < 27) {
            const int kind = lane / 9, i = (lane % 9) / 3, j = lane % 3;
            double re = 0, im = 0;
            for (int x = 0; x < n; ++x) {
                re += sB[warp][x][i] * sS[warp][x][kind * 6 + 2 * j];
                im += sB[warp][x][i] * sS[warp][x][kind * 6 + 2 * j + 1];
            }
            own[0] += re;
            own[1] += im;
        }
        __syncwarp();
    }
    if (lane < 27) {
        const int kind = lane / 9, e = lane % 9;
        sM[warp][kind * 18 + 2 * e] = own[0];
        sM[warp][kind * 18 + 2 * e + 1] = own[1];
    }
    if constexpr (!Mixed)
        bad = distance.bad();
    if (__any_sync(0xffffffffu, bad) && lane == 0)
        flagError(error, kErrDistance);
    __syncwarp();
    if (lane < 24) {
        const int o = lane;
        double re, im;
        pairRecordValue(o, &sM[warp][0], &sM[warp][18], &sM[warp][36], t, s, k, invk, re, im);
        if (!isfinite(re) || !isfinite(im))
            flagError(error, kErrNonFinite);
        const size_t slot = o < 12 ? mapSlot(map, T, job.first, job.second) : mapSlot(map, T, job.second, job.first);
        const int e = o < 12 ? o : o - 12;
        if (slot != kNoSlot) {
            Acc *dst = records + size_t(f) * map.planeSlots * kRecordDoubles + mapOffset(map.planeSlots, slot, e);
            dst[0] = Acc(re);
            dst[1] = Acc(im);
        } else
            flagError(error, kErrEscapedPlan);
    }
}

// Block sums of N values, left in smem[0][0..N). Within a warp a
// reduce-scatter per group of 32 values: after the pass at distance h a lane
// keeps the h partial sums of the half its lane bit h selects, so after five
// passes (31 shuffles per group instead of 32 x 5) lane l holds the sum of
// value l of the group. The warps' sums are then added in warp order by the
// thread that owns each value.
template <int N>
__device__ __forceinline__ void blockReduce(double (&v)[N], double (*smem)[N]) {
    constexpr int G = (N + 31) / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int gi = 0; gi < G; ++gi) {
        double x[32];
#pragma unroll
        for (int c = 0; c < 32; ++c)
            x[c] = 32 * gi + c < N ? v[32 * gi + c] : 0.0;
#pragma unroll
        for (int h = 16; h >= 1; h >>= 1) {
            const bool upper = (lane & h) != 0;
#pragma unroll
            for (int c = 0; c < h; ++c) {
                const double send = upper ? x[c] : x[c + h], keep = upper ? x[c + h] : x[c];
                x[c] = keep + __shfl_xor_sync(0xffffffffu, send, h);
            }
        }
        if (32 * gi + lane < N)
            smem[warp][32 * gi + lane] = x[0];
    }
    __syncthreads();
    const int warps = blockDim.x >> 5;
    for (int c = threadIdx.x; c < N; c += blockDim.x) {
        double sum = smem[0][c];
        for (int w = 1; w < warps; ++w)
            sum += smem[w][c];
        smem[0][c] = sum;
    }
    __syncthreads();
}

template <bool Mixed>
__global__ void __launch_bounds__(128) nearKernel(const DPanel *__restrict__ panels, uint32_t T,
                                                  const NearPairJob *__restrict__ jobs,
                                                  const Patch *__restrict__ patches, const double *__restrict__ ks,
                                                  std::conditional_t<Mixed, float, double> *__restrict__ records,
                                                  SlotMap map, int *error) {
    using Acc = std::conditional_t<Mixed, float, double>;
    __shared__ double red[4][54];
    __shared__ double pts[2][64][3];
    const NearPairJob job = jobs[blockIdx.x];
    const int f = blockIdx.y;
    const double k = ks[f], invk = 1.0 / k;
    const DPanel &t = panels[job.first];
    const DPanel &s = panels[job.second];
    const double w4 = 4.0 * t.area * s.area * kInvFourPi;
    Acc acc[54];
#pragma unroll
    for (int c = 0; c < 54; ++c)
        acc[c] = 0;
    bool bad = false;
    FanPanel ft, fs;
    for (int i = 0; i < 3; ++i) {
        ft.v[i] = V3{t.v0[0] + (i == 1 ? t.e1[0] : i == 2 ? t.e2[0] : 0.0), t.v0[1] + (i == 1 ? t.e1[1] : i == 2 ? t.e2[1] : 0.0),
                     t.v0[2] + (i == 1 ? t.e1[2] : i == 2 ? t.e2[2] : 0.0)};
        fs.v[i] = V3{s.v0[0] + (i == 1 ? s.e1[0] : i == 2 ? s.e2[0] : 0.0), s.v0[1] + (i == 1 ? s.e1[1] : i == 2 ? s.e2[1] : 0.0),
                     s.v0[2] + (i == 1 ? s.e1[2] : i == 2 ? s.e2[2] : 0.0)};
    }
    ft.n = V3{t.n[0], t.n[1], t.n[2]};
    fs.n = V3{s.n[0], s.n[1], s.n[2]};
    ft.area = t.area;
    fs.area = s.area;
    for (uint32_t q = 0; q < job.patchCount; ++q) {
        const Patch &patch = patches[job.firstPatch + q];
        const int n = patch.degree == 14 ? 64 : 16;
        const int ro = patch.degree == 14 ? 34 : 18;  // rule offsets of the 16- and 64-point bins
        if (!patch.projection) {
            __syncthreads();
            for (int idx = threadIdx.x; idx < 2 * n; idx += blockDim.x) {
                const int side = idx / n, x = idx % n;
                const double *pv = side ? patch.trial : patch.test;
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    pts[side][x][i] = cRule[4 * (ro + x)] * pv[i] + cRule[4 * (ro + x) + 1] * pv[3 + i] +
                                      cRule[4 * (ro + x) + 2] * pv[6 + i];
            }
            __syncthreads();
            for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x) {
                const int x = idx / n, y = idx % n;
                const double w = cRule[4 * (ro + x) + 3] * cRule[4 * (ro + y) + 3] * patch.areaFraction * w4;
                nearSample(acc, t, s, pts[0][x], pts[1][y], w, k, bad);
            }
            continue;
        }
        const uint32_t order = 20 * patch.intervals;
        const uint32_t points = uint32_t(n) * 3 * order * order;
        for (uint32_t idx = threadIdx.x; idx < points; idx += blockDim.x) {
            uint32_t rest = idx;
            const uint32_t radial = rest % order;
            rest /= order;
            const uint32_t angular = rest % order;
            rest /= order;
            const uint32_t edge = rest % 3, outer = rest / 3;
            GaussPoint u{cGauss20[2 * (angular % 20)], cGauss20[2 * (angular % 20) + 1]};
            GaussPoint v{cGauss20[2 * (radial % 20)], cGauss20[2 * (radial % 20) + 1]};
            u.x = (angular / 20 + u.x) / patch.intervals;
            v.x = (radial / 20 + v.x) / patch.intervals;
            u.w /= patch.intervals;
            v.w /= patch.intervals;
            const double ob[3] = {cRule[4 * (ro + outer)], cRule[4 * (ro + outer) + 1], cRule[4 * (ro + outer) + 2]};
            const ProjOuter po = projOuter(ob, cRule[4 * (ro + outer) + 3], patch, ft, fs);
            const PairPoint pp = projPoint(po, projRay(po, projEdge(po, edge, fs), u), v);
            nearSample(acc, t, s, pp.t, pp.s, pp.w * w4, k, bad);
        }
    }
    if (bad)
        flagError(error, kErrDistance);
    __syncthreads();
    double accd[54];
#pragma unroll
    for (int c = 0; c < 54; ++c)
        accd[c] = acc[c];
    blockReduce<54>(accd, red);
    if (threadIdx.x < 24) {
        const int o = threadIdx.x;
        double re, im;
        pairRecordValue(o, &red[0][0], &red[0][18], &red[0][36], t, s, k, invk, re, im);
        if (!isfinite(re) || !isfinite(im))
            flagError(error, kErrNonFinite);
        const size_t slot = o < 12 ? mapSlot(map, T, job.first, job.second) : mapSlot(map, T, job.second, job.first);
        const int e = o < 12 ? o : o - 12;
        if (slot != kNoSlot) {
            Acc *dst = records + size_t(f) * map.planeSlots * kRecordDoubles + mapOffset(map.planeSlots, slot, e);
            dst[0] = Acc(re);
            dst[1] = Acc(im);
        } else
            flagError(error, kErrEscapedPlan);
    }
}

// ---------------------------------------------------------------------------
// Deterministic gathers: records -> per-(test panel, trial vertex) columns ->
// matrix entries, and records x flux -> right-hand side.
// ---------------------------------------------------------------------------
// Both gathers in one CTA per matrix column (trial vertex b, frequency f),
// for meshes whose 3T column entries fit in shared memory: first the
// per-(test panel, local row) sums over the trial panels at b (coalesced
// plane reads), then each row's sum over its incident panels plus the half
// mass, written as a contiguous column. Same summation order as
// gatherTrialKernel followed by gatherTestKernel.
// Three complex values of a record plane entry as three vector loads (entries
// are 6 values: 24 B in FP32, 48 B in FP64, so 8- and 16-byte aligned).
__device__ __forceinline__ void load6(const float *r, float (&v)[6]) {
    const float2 *q = reinterpret_cast<const float2 *>(r);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float2 x = q[c];
        v[2 * c] = x.x;
        v[2 * c + 1] = x.y;
    }
}
__device__ __forceinline__ void load6(const double *r, double (&v)[6]) {
    const double2 *q = reinterpret_cast<const double2 *>(r);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double2 x = q[c];
        v[2 * c] = x.x;
        v[2 * c + 1] = x.y;
    }
}

// One complex entry of a gathered column (6 T values a column: 8- or 16-byte aligned).
__device__ __forceinline__ void load2(const float *p, float (&v)[2]) {
    const float2 x = *reinterpret_cast<const float2 *>(p);
    v[0] = x.x;
    v[1] = x.y;
}
__device__ __forceinline__ void load2(const double *p, double (&v)[2]) {
    const double2 x = *reinterpret_cast<const double2 *>(p);
    v[0] = x.x;
    v[1] = x.y;
}

template <class Rec>
__global__ void __launch_bounds__(512, 2) gatherColumnKernel(const Rec *__restrict__ records,
                                                          const uint32_t *__restrict__ incOffsets,
                                                          const uint32_t *__restrict__ incPanel,
                                                          const uint8_t *__restrict__ incLocal,
                                                          const DPanel *__restrict__ panels,
                                                          const double *__restrict__ rowScale, uint32_t T, uint32_t N,
                                                          double *__restrict__ A) {
    extern __shared__ double2 column[];  // [3T]: entry (test panel t, local row la) of column b
    const uint32_t b = blockIdx.x;
    const int f = blockIdx.y;
    const Rec *rec = records + size_t(f) * T * T * kRecordDoubles;
    const uint32_t o0 = incOffsets[b], o1 = incOffsets[b + 1];
    for (uint32_t t = threadIdx.x; t < T; t += blockDim.x) {
        double acc[6] = {0, 0, 0, 0, 0, 0};
        // trial panels at b in chunks of 4: the record loads of a chunk are in flight together
        for (uint32_t o = o0; o < o1; o += 4) {
            Rec v[4][6];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (o + u < o1)
                    load6(rec + recordOffset(T, size_t(incPanel[o + u]) * T + t, incLocal[o + u]), v[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (o + u < o1)
#pragma unroll
                    for (int c = 0; c < 6; ++c)
                        acc[c] += double(v[u][c]);
        }
#pragma unroll
        for (int la = 0; la < 3; ++la)
            column[3 * t + la] = make_double2(acc[2 * la], acc[2 * la + 1]);
    }
    __syncthreads();
    for (uint32_t a = threadIdx.x; a < N; a += blockDim.x) {
        double re = 0, im = 0;
        const uint32_t a0 = incOffsets[a], a1 = incOffsets[a + 1];
        for (uint32_t o = a0; o < a1; o += 4) {
            uint32_t t[4], n[4][3];
            int la[4];
            double area[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (o + u < a1) {
                    t[u] = incPanel[o + u];
                    la[u] = incLocal[o + u];
                    const DPanel &p = panels[t[u]];
                    n[u][0] = p.nodes[0];
                    n[u][1] = p.nodes[1];
                    n[u][2] = p.nodes[2];
                    area[u] = p.area;
                }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (o + u < a1) {
                    const double2 v = column[3 * t[u] + la[u]];
                    re += v.x;
                    im += v.y;
                    if (n[u][0] == b || n[u][1] == b || n[u][2] == b)
                        re += area[u] * (a == b ? 2.0 : 1.0) / 24.0;
                }
        }
        const double sc = rowScale[a];
        double *dst = A + (size_t(f) * N * N + size_t(b) * N + a) * 2;
        dst[0] = re * sc;
        dst[1] = im * sc;
    }
}

template <class Rec>
__global__ void gatherTrialKernel(const Rec *__restrict__ records, const uint32_t *__restrict__ incOffsets,
                                  const uint32_t *__restrict__ incPanel, const uint8_t *__restrict__ incLocal,
                                  uint32_t T, uint32_t N, Rec *__restrict__ columns) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t b = blockIdx.y;
    const int f = blockIdx.z;
    if (t >= T)
        return;
    const Rec *rec = records + size_t(f) * T * T * kRecordDoubles;
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (uint32_t o = incOffsets[b]; o < incOffsets[b + 1]; ++o) {
        const uint32_t s = incPanel[o];
        const int lb = incLocal[o];
        // column lb of the (trial s, test t) block: 3 contiguous complex values
        Rec v[6];
        load6(rec + recordOffset(T, size_t(s) * T + t, lb), v);
#pragma unroll
        for (int c = 0; c < 6; ++c)
            acc[c] += double(v[c]);
    }
    Rec *dst = columns + (size_t(f) * N + b) * 6 * T + 6 * size_t(t);
#pragma unroll
    for (int c = 0; c < 6; ++c)
        dst[c] = Rec(acc[c]);
}

// Rows of the gathered columns: A[a, b] sums column b over the star of a. The
// incidence and panel reads of a star are those of every column, and one thread
// per entry spent most of its loads on them; a thread now takes row a of
// kTestColumns columns, whose record loads are in flight together.
// 12,800 panels, FP32 records: 2.2 -> 0.84 ms, FP64 2.7 -> 1.2 ms.
constexpr int kTestColumns = 4;
template <class Rec>
__global__ void __launch_bounds__(128) gatherTestKernel(const Rec *__restrict__ columns,
                                                        const DPanel *__restrict__ panels,
                                                        const uint32_t *__restrict__ incOffsets,
                                                        const uint32_t *__restrict__ incPanel,
                                                        const uint8_t *__restrict__ incLocal,
                                                        const double *__restrict__ rowScale, uint32_t T, uint32_t N,
                                                        double *__restrict__ A) {
    const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t b0 = blockIdx.y * kTestColumns;
    const int f = blockIdx.z;
    if (a >= N)
        return;
    const uint32_t count = min(uint32_t(kTestColumns), N - b0);
    const Rec *col = columns + (size_t(f) * N + b0) * 6 * T;
    double re[kTestColumns] = {}, im[kTestColumns] = {};
    const uint32_t end = incOffsets[a + 1];
    for (uint32_t o = incOffsets[a]; o < end; ++o) {
        const uint32_t t = incPanel[o];
        const size_t at = 6 * size_t(t) + 2 * incLocal[o];
        const DPanel &p = panels[t];
        const uint32_t n0 = p.nodes[0], n1 = p.nodes[1], n2 = p.nodes[2];
        const double area = p.area;
        Rec v[kTestColumns][2];
#pragma unroll
        for (int c = 0; c < kTestColumns; ++c)
            if (uint32_t(c) < count)
                load2(col + size_t(c) * 6 * T + at, v[c]);
#pragma unroll
        for (int c = 0; c < kTestColumns; ++c)
            if (uint32_t(c) < count) {
                const uint32_t b = b0 + c;
                re[c] += double(v[c][0]);
                im[c] += double(v[c][1]);
                if (n0 == b || n1 == b || n2 == b)
                    re[c] += area * (a == b ? 2.0 : 1.0) / 24.0;
            }
    }
    const double sc = rowScale[a];
    double2 *dst = reinterpret_cast<double2 *>(A) + size_t(f) * N * N + size_t(b0) * N + a;
#pragma unroll
    for (int c = 0; c < kTestColumns; ++c)
        if (uint32_t(c) < count)
            dst[size_t(c) * N] = make_double2(re[c] * sc, im[c] * sc);
}

// Per-panel right-hand-side partials: sum over trial panels s of the
// (s, t) moments times the flux of s. A CTA takes 32 test panels; its 8
// warps take every 8th trial panel, and the partial sums are added in a
// fixed order (deterministic).
template <class Rec>
__global__ void __launch_bounds__(256) rhsPanelKernel(const Rec *__restrict__ records, const double *__restrict__ flux,
                                                      uint32_t T, uint32_t E, double *__restrict__ panelRhs) {
    __shared__ double part[8][32][6];
    const uint32_t lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const uint32_t t = blockIdx.x * 32 + lane;
    const uint32_t e = blockIdx.y;
    const int f = blockIdx.z;
    const Rec *rec = records + size_t(f) * T * T * kRecordDoubles;
    const double *q = flux + (size_t(f) * E + e) * 2 * T;
    double acc[6] = {0, 0, 0, 0, 0, 0};
    if (t < T)
        for (uint32_t s = g; s < T; s += 8) {
            const double qr = q[2 * s], qi = q[2 * s + 1];
            if (qr == 0 && qi == 0)
                continue;
            Rec r[6];
            load6(rec + recordOffset(T, size_t(s) * T + t, 9), r);
#pragma unroll
            for (int la = 0; la < 3; ++la) {
                const double rr = r[2 * la], ri = r[2 * la + 1];
                acc[2 * la] += rr * qr - ri * qi;
                acc[2 * la + 1] += rr * qi + ri * qr;
            }
        }
#pragma unroll
    for (int c = 0; c < 6; ++c)
        part[g][lane][c] = acc[c];
    __syncthreads();
    if (g != 0 || t >= T)
        return;
    double *dst = panelRhs + (size_t(f) * E + e) * 6 * T + 6 * size_t(t);
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        double v = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w)
            v += part[w][lane][c];
        dst[c] = v;
    }
}

__global__ void rhsVertexKernel(const double *__restrict__ panelRhs, const uint32_t *__restrict__ incOffsets,
                                const uint32_t *__restrict__ incPanel, const uint8_t *__restrict__ incLocal,
                                const double *__restrict__ rowScale, uint32_t T, uint32_t N, uint32_t E,
                                double *__restrict__ rhs) {
    const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t e = blockIdx.y;
    const int f = blockIdx.z;
    if (a >= N)
        return;
    const double *src = panelRhs + (size_t(f) * E + e) * 6 * T;
    double re = 0, im = 0;
    for (uint32_t o = incOffsets[a]; o < incOffsets[a + 1]; ++o) {
        re += src[6 * size_t(incPanel[o]) + 2 * incLocal[o]];
        im += src[6 * size_t(incPanel[o]) + 2 * incLocal[o] + 1];
    }
    double *dst = rhs + ((size_t(f) * E + e) * N + a) * 2;
    dst[0] = re * rowScale[a];
    dst[1] = im * rowScale[a];
}

template <int NP>
void launchRegular(const AssemblyGeometry &g, const double *ks, uint32_t B, const AssemblyWorkspace &ws, int bin,
                   int *error, cudaStream_t stream, KernelTimer *timer, bool mixed, const SlotMap &map) {
    const char *names[kBins] = {"regular_q6", "regular_q12", "regular_q16", "regular_q64"};
    const char *mixedNames[kBins] = {"regular_mixed_q6", "regular_mixed_q12", "regular_mixed_q16",
                                     "regular_mixed_q64"};
    TimedScope scope(timer, mixed ? mixedNames[bin] : names[bin], stream);
    // Grid of the grid-stride pair loop in CTAs per SM: each pair is one
    // independent item, so the choice moves only the load balance and occupancy.
    static constexpr int kMixedCtas[] = {24, 12, 6, 48};  // 3 or 4 CTAs an SM are resident
    static constexpr int kPlainCtas[] = {8, 4, 16};
    const int candidates = mixed ? 4 : 3;
    const auto launch = [&](int c) {
        if (mixed) {
            const dim3 grid(unsigned(smCount() * kMixedCtas[c]), B);
            // The 6-point rule writes the most for its samples. Staged stores from 4096 triangles on: 8042
            // triangles 13.5 -> 10.6 ms, 12 756 triangles 12.1 -> 10.6 ms when they came in; equal at 3604,
            // slower at 1280 (1.89 against 2.14 ms), and slower for the 12-point rule at every size
            // (3.04 against 3.30 ms).
            const auto kernel = NP == 6 && g.T >= 4096 ? regularMixedKernel<NP, NP == 6> : regularMixedKernel<NP, false>;
            kernel<<<grid, 128, 0, stream>>>(g.mixedPanels, g.bounds, g.T, ks, ws.bins, ws.binCounts, ws.binCapacity,
                                             ws.binOffsets, bin, static_cast<float *>(ws.records), error);
        } else {
            const dim3 grid(unsigned(smCount() * kPlainCtas[c]), B);
            regularPairsKernel<NP><<<grid, kPlainThreads, 0, stream>>>(g.panels, g.T, ks, ws.bins, ws.binCounts,
                                                             ws.binCapacity, ws.binOffsets, bin,
                                                             static_cast<double *>(ws.records), map, error);
        }
        cudaCheck(cudaGetLastError(), "regular pair assembly launch");
    };
    // size class: the form, the rule, the batch and the mesh size to a power of two
    const std::string key = std::string(mixed ? "regular_mixed" : "regular_fp64") + "_q" + std::to_string(NP) +
                            "_B" + std::to_string(B) + "_T2^" + std::to_string(31 - __builtin_clz(g.T | 1u)) +
                            (map.row ? "_near" : "");
    Autotuner &tuner = Autotuner::instance();
    int c = tuner.choice(key);
    // tuned on first use, outside a capture and outside a profiled solve (whose
    // per-family times would count the candidates' launches)
    if (c < 0 && tuner.enabled() && !(timer && timer->enabled()) && !capturing(stream)) {
        tuner.tune(key, candidates, stream, launch);
        return;
    }
    launch(c < 0 ? 0 : c);
}

}  // namespace

namespace {
// Touching tuples of one singular order, in table order: visit(row, canonical
// point at radius 1, displacement coefficients {a1, a2, b1, b2} over the
// canonical edges with the shared ones merged, weight).
template <class Visit> void forEachSingularTuple(unsigned order, const Visit &visit) {
    const auto gauss = gaussLegendre01(order);
    const size_t per = size_t(order) * order * order;
    const uint32_t topologies[3] = {kSharedVertex, kSharedEdge, kCoincident};
    size_t row = 0;
    for (uint32_t topo : topologies)
        for (unsigned sector = 0; sector < sectorCount(topo); ++sector)
            for (size_t tuple = 0; tuple < per; ++tuple, ++row) {
                const size_t wi = tuple % order, vi = (tuple / order) % order, ui = tuple / (size_t(order) * order);
                const PairPoint p = sauterSchwab(topo, sector, 1.0, gauss[ui].x, gauss[vi].x, gauss[wi].x);
                double d[4] = {p.t[1], p.t[2], p.s[1], p.s[2]};
                if (topo == kSharedEdge || topo == kCoincident) {
                    d[0] -= d[2];
                    d[2] = 0;
                }
                if (topo == kCoincident) {
                    d[1] -= d[3];
                    d[3] = 0;
                }
                visit(row, p, d, p.w * gauss[ui].w * gauss[vi].w * gauss[wi].w);
            }
}
}  // namespace

std::vector<float> buildSingularTable(unsigned order) {
    const auto gauss = gaussLegendre01(order);
    const size_t per = size_t(order) * order * order;
    std::vector<float> out((13 * per) * 12 + order * 4, 0.f);
    forEachSingularTuple(order, [&](size_t row, const PairPoint &p, const double *d, double w) {
        const double v[11] = {p.t[0], p.t[1], p.t[2], p.s[0], p.s[1], p.s[2], d[0], d[1], d[2], d[3], w};
        for (int c = 0; c < 11; ++c)
            out[12 * row + c] = float(v[c]);
    });
    for (unsigned ri = 0; ri < order; ++ri) {
        const double r = gauss[ri].x;
        out[12 * 13 * per + 4 * ri] = float(r);
        out[12 * 13 * per + 4 * ri + 1] = float(r * r * r * gauss[ri].w);
        out[12 * 13 * per + 4 * ri + 2] = float(1.0 / r);
        out[12 * 13 * per + 4 * ri + 3] = float(1.0 - r);
    }
    return out;
}

std::vector<double> buildSingularTuples(unsigned order) {
    const auto gauss = gaussLegendre01(order);
    const size_t per = size_t(order) * order * order;
    std::vector<double> out((13 * per) * 12 + order * 6, 0.0);
    forEachSingularTuple(order, [&](size_t row, const PairPoint &p, const double *d, double w) {
        // radial slopes of the bases: at radius r they are (1, 0, 0) + r (slope)
        const double v[11] = {-(p.t[1] + p.t[2]), p.t[1], p.t[2], -(p.s[1] + p.s[2]), p.s[1], p.s[2],
                              d[0],               d[1],   d[2],   d[3],               w};
        std::copy(v, v + 11, &out[12 * row]);
    });
    for (unsigned ri = 0; ri < order; ++ri) {
        double *q = &out[12 * 13 * per + 6 * ri];
        const double r = q[0] = gauss[ri].x;
        q[1] = r * gauss[ri].w;
        for (int c = 2; c < 5; ++c)
            q[c] = q[c - 1] * r;
    }
    return out;
}

namespace {
void uploadRuleTablesNow(cudaStream_t stream) {
    double table[kRulePoints * 4];
    const unsigned degrees[kBins] = {4, 6, 8, 14};
    int o = 0;
    for (int b = 0; b < kBins; ++b) {
        const auto r = triangleRule(degrees[b]);
        for (const auto &p : r) {
            table[4 * o] = p.b[0];
            table[4 * o + 1] = p.b[1];
            table[4 * o + 2] = p.b[2];
            table[4 * o + 3] = p.w;
            ++o;
        }
    }
    cudaCheck(cudaMemcpyToSymbolAsync(cRule, table, sizeof(table), 0, cudaMemcpyHostToDevice, stream), "rule upload");
    double squares[kRulePoints * 3];
    for (int i = 0; i < kRulePoints; ++i) {
        const double b1 = table[4 * i + 1], b2 = table[4 * i + 2];
        squares[3 * i] = b1 * b1;
        squares[3 * i + 1] = b1 * b2;
        squares[3 * i + 2] = b2 * b2;
    }
    cudaCheck(cudaMemcpyToSymbolAsync(cRuleSquares, squares, sizeof(squares), 0, cudaMemcpyHostToDevice, stream),
              "rule upload");
    static float tableF[kRulePoints * 8];
    for (int i = 0; i < kRulePoints; ++i) {
        const double b1 = table[4 * i + 1], b2 = table[4 * i + 2];
        const double v[8] = {table[4 * i], b1, b2, table[4 * i + 3], b1 * b1, 2 * b1 * b2, b2 * b2, 0.0};
        for (int c = 0; c < 8; ++c)
            tableF[8 * i + c] = float(v[c]);
    }
    cudaCheck(cudaMemcpyToSymbolAsync(cRuleF, tableF, sizeof(tableF), 0, cudaMemcpyHostToDevice, stream),
              "rule upload");
    double g20[40];
    const auto g = gaussLegendre01(20);
    for (int i = 0; i < 20; ++i) {
        g20[2 * i] = g[i].x;
        g20[2 * i + 1] = g[i].w;
    }
    cudaCheck(cudaMemcpyToSymbolAsync(cGauss20, g20, sizeof(g20), 0, cudaMemcpyHostToDevice, stream), "gauss upload");
    cudaCheck(cudaStreamSynchronize(stream), "rule upload sync");
}
}  // namespace

// The rule tables in constant memory, once per device (each device has its own
// copy of the __constant__ arrays).
void uploadRuleTables(cudaStream_t stream) {
    static PerDeviceOnce once;
    once.run([&]() { uploadRuleTablesNow(stream); });
}

bool gatherUsesColumns(uint32_t T) { return size_t(3) * T * sizeof(double2) > kGatherColumnSmem; }

size_t recordBytes(uint32_t T, bool mixed) { return size_t(T) * T * kRecordDoubles * (mixed ? 4 : 8); }

size_t assemblyWorkspaceBytes(uint32_t T, uint32_t N, uint32_t E, uint32_t B, bool mixed) {
    const size_t pairs = size_t(T) * (T - 1) / 2;
    const size_t columns = gatherUsesColumns(T) ? size_t(N) * 6 * T * (mixed ? 4 : 8) : 0;
    const size_t bins = (T > kExactBinsT ? 1 : kBins) * pairs * sizeof(uint2);
    return size_t(B) * (recordBytes(T, mixed) + columns + size_t(E) * 6 * T * 8 + bins + kBins * (4 + 8));
}

namespace {
// Pair records of B frequencies: classification into rule bins (all
// unordered pairs, or the listed ones), then the regular, touching and near
// kernels, every record stored at its slot of `map`.
void computeRecords(const AssemblyGeometry &g, const double *ks, const double *singularTuples, uint32_t B,
                    const AssemblyWorkspace &ws, const SlotMap &map, const uint2 *pairList, uint64_t listCount,
                    int *error, cudaStream_t stream, KernelTimer *timer, bool mixed) {
    const uint64_t pairs = uint64_t(g.T) * (g.T - 1) / 2;
    double *recD = static_cast<double *>(ws.records);
    float *recF = static_cast<float *>(ws.records);
    cudaCheck(cudaMemsetAsync(ws.binCounts, 0, sizeof(uint32_t) * kBins * B, stream), "bin reset");
    if (pairList) {
        TimedScope scope(timer, "classify_pairs", stream);
        if (listCount) {
            const unsigned blocks = unsigned(std::min<uint64_t>((listCount + 255) / 256, uint64_t(smCount()) * 16));
            classifyListKernel<<<blocks, 256, 0, stream>>>(pairList, listCount, g.pairCode, g.bounds, ks, B,
                                                           g.nearTolerance, g.minimumDegree, ws.bins, ws.binCounts,
                                                           ws.binCapacity, error);
            cudaCheck(cudaGetLastError(), "pair list classification launch");
        }
    } else if (pairs) {
        TimedScope scope(timer, "classify_pairs", stream);
        const unsigned blocks = unsigned(std::min<uint64_t>((pairs + 255) / 256, uint64_t(smCount()) * 16));
        if (ws.binOffsets) {  // count, scan, fill
            classifyPairsKernel<<<blocks, kClassifyThreads, 0, stream>>>(g.pairCode, g.bounds, g.T, ks, B, g.nearTolerance,
                                                            g.minimumDegree, ws.bins, ws.binCounts, ws.binCapacity,
                                                            ws.binOffsets, true, error);
            binOffsetsKernel<<<1, 1, 0, stream>>>(ws.binCounts, ws.binOffsets, B * kBins);
        }
        classifyPairsKernel<<<blocks, kClassifyThreads, 0, stream>>>(g.pairCode, g.bounds, g.T, ks, B, g.nearTolerance,
                                                        g.minimumDegree, ws.bins, ws.binCounts, ws.binCapacity,
                                                        ws.binOffsets, false, error);
        cudaCheck(cudaGetLastError(), "pair classification launch");
    }
    launchRegular<6>(g, ks, B, ws, 0, error, stream, timer, mixed, map);
    launchRegular<12>(g, ks, B, ws, 1, error, stream, timer, mixed, map);
    launchRegular<16>(g, ks, B, ws, 2, error, stream, timer, mixed, map);
    launchRegular<64>(g, ks, B, ws, 3, error, stream, timer, mixed, map);
    if (g.touchingCount) {
        TimedScope scope(timer, mixed ? "singular_mixed" : "singular", stream);
        if (mixed)
            singularMixedKernel<<<dim3((g.touchingCount + 3) / 4, B), 128, 0, stream>>>(
                g.panels, g.T, g.touching, g.touchingCount, ks, g.singularTable, g.singularOrder, recF, error);
        else
            singularKernel<<<dim3((g.touchingCount + 3) / 4, B), 128, 0, stream>>>(
                g.panels, g.T, g.touching, g.touchingCount, ks, singularTuples, g.singularOrder, recD, map, error);
        cudaCheck(cudaGetLastError(), "singular assembly launch");
    }
    if (g.nearPairCount - g.projectedPairCount) {
        TimedScope scope(timer, "near", stream);
        const uint32_t tensorPairs = g.nearPairCount - g.projectedPairCount;
        const dim3 grid((tensorPairs + 1) / 2, B);
        if (mixed)
            nearWarpKernel<true><<<grid, 64, 0, stream>>>(g.panels, g.T, g.nearPairs, tensorPairs, g.patches, ks,
                                                          recF, map, error);
        else
            nearWarpKernel<false><<<grid, 64, 0, stream>>>(g.panels, g.T, g.nearPairs, tensorPairs, g.patches, ks,
                                                           recD, map, error);
        cudaCheck(cudaGetLastError(), "near assembly launch");
    }
    if (g.projectedPairCount) {
        TimedScope scope(timer, "near_projected", stream);
        const NearPairJob *projected = g.nearPairs + (g.nearPairCount - g.projectedPairCount);
        if (mixed)
            nearKernel<true><<<dim3(g.projectedPairCount, B), 128, 0, stream>>>(g.panels, g.T, projected, g.patches,
                                                                                ks, recF, map, error);
        else
            nearKernel<false><<<dim3(g.projectedPairCount, B), 128, 0, stream>>>(g.panels, g.T, projected, g.patches,
                                                                                 ks, recD, map, error);
        cudaCheck(cudaGetLastError(), "projected near assembly launch");
    }
}
}  // namespace

void assembleBatch(const AssemblyGeometry &g, const double *ks, const double *singularTuples, const double *flux,
                   uint32_t E, uint32_t B, const AssemblyWorkspace &ws, double *A, double *rhs, int *error,
                   cudaStream_t stream, KernelTimer *timer, bool mixed) {
    if (g.N > 65535 || B > 65535 || E > 65535)
        throw std::runtime_error("Dense assembly grid limits exceeded (more than 65535 vertices, frequencies or excitations).");
    SlotMap dense;
    dense.planeSlots = size_t(g.T) * g.T;
    computeRecords(g, ks, singularTuples, B, ws, dense, nullptr, 0, error, stream, timer, mixed);
    double *recD = static_cast<double *>(ws.records);
    float *recF = static_cast<float *>(ws.records);
    const size_t columnBytes = size_t(3) * g.T * sizeof(double2);
    if (!gatherUsesColumns(g.T)) {
        TimedScope scope(timer, "gather_column", stream);
        static PerDeviceOnce attributes;
        attributes.run([]() {
            cudaCheck(cudaFuncSetAttribute(gatherColumnKernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           int(kGatherColumnSmem)),
                      "gather smem attribute");
            cudaCheck(cudaFuncSetAttribute(gatherColumnKernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           int(kGatherColumnSmem)),
                      "gather smem attribute");
        });
        const dim3 grid(g.N, B);
        if (mixed)
            gatherColumnKernel<<<grid, 512, columnBytes, stream>>>(recF, g.incOffsets, g.incPanel, g.incLocal,
                                                                   g.panels, g.rowScale, g.T, g.N, A);
        else
            gatherColumnKernel<<<grid, 512, columnBytes, stream>>>(recD, g.incOffsets, g.incPanel, g.incLocal,
                                                                   g.panels, g.rowScale, g.T, g.N, A);
        cudaCheck(cudaGetLastError(), "column gather launch");
    } else {
        {
            TimedScope scope(timer, "gather_trial", stream);
            const dim3 grid((g.T + 127) / 128, g.N, B);
            if (mixed)
                gatherTrialKernel<<<grid, 128, 0, stream>>>(recF, g.incOffsets, g.incPanel, g.incLocal, g.T, g.N,
                                                            static_cast<float *>(ws.columns));
            else
                gatherTrialKernel<<<grid, 128, 0, stream>>>(recD, g.incOffsets, g.incPanel, g.incLocal, g.T, g.N,
                                                            static_cast<double *>(ws.columns));
            cudaCheck(cudaGetLastError(), "trial gather launch");
        }
        {
            TimedScope scope(timer, "gather_test", stream);
            const dim3 grid((g.N + 127) / 128, (g.N + kTestColumns - 1) / kTestColumns, B);
            if (mixed)
                gatherTestKernel<<<grid, 128, 0, stream>>>(static_cast<const float *>(ws.columns), g.panels,
                                                           g.incOffsets, g.incPanel, g.incLocal, g.rowScale, g.T, g.N,
                                                           A);
            else
                gatherTestKernel<<<grid, 128, 0, stream>>>(static_cast<const double *>(ws.columns), g.panels,
                                                           g.incOffsets, g.incPanel, g.incLocal, g.rowScale, g.T, g.N,
                                                           A);
            cudaCheck(cudaGetLastError(), "test gather launch");
        }
    }
    {
        TimedScope scope(timer, "rhs_panel", stream);
        const dim3 grid((g.T + 31) / 32, E, B);
        if (mixed)
            rhsPanelKernel<<<grid, 256, 0, stream>>>(recF, flux, g.T, E, ws.panelRhs);
        else
            rhsPanelKernel<<<grid, 256, 0, stream>>>(recD, flux, g.T, E, ws.panelRhs);
    }
    {
        TimedScope scope(timer, "rhs_vertex", stream);
        rhsVertexKernel<<<dim3((g.N + 127) / 128, E, B), 128, 0, stream>>>(ws.panelRhs, g.incOffsets, g.incPanel,
                                                                           g.incLocal, g.rowScale, g.T, g.N, E, rhs);
    }
    cudaCheck(cudaGetLastError(), "rhs gather launch");
}

// ---------------------------------------------------------------------------
// Fast-multipole near field: records of the near panel pairs only (SlotMap
// over a panel-pair CSR), reduced into the near support-pair CSR values and
// the near part of the right-hand side.
// ---------------------------------------------------------------------------
namespace {

// vals[e] for entry e = (i, j) of the near CSR: rowScale_i (sum over the
// panels a of star i and s of star j of block entry (la, lb) of record (a, s)
// plus the P1 mass term of the panels holding both i and j). One CTA per row, in
// two steps: first the sums over star i for every trial panel s of the near list
// (the CSR row of i's first panel holds all of them; kNearTile panels at a time),
// then each entry's sum over star j from shared memory. Reading the 36 records of
// every entry, each found by its own binary search in global memory, took 11.2 ms
// for the 8k-triangle horn; the sums over star i are shared by the star's
// neighbours and the searches of the second step stay in shared memory: 1.9 ms.
constexpr uint32_t kNearTile = 2048, kNearThreads = 256;
constexpr size_t kNearValuesSmem = kNearTile * (3 * sizeof(double2) + sizeof(uint32_t) + 1);

__global__ void __launch_bounds__(kNearThreads) nearValuesKernel(
    const double *__restrict__ records, SlotMap map, const uint32_t *__restrict__ nearRow,
    const uint32_t *__restrict__ nearCol, const uint32_t *__restrict__ incOffsets, const uint32_t *__restrict__ incPanel,
    const uint8_t *__restrict__ incLocal, const DPanel *__restrict__ panels, const double *__restrict__ rowScale,
    uint32_t T, double2 *vals, int *error) {
    extern __shared__ __align__(16) unsigned char rawSmem[];
    double2 *sums = reinterpret_cast<double2 *>(rawSmem);             // [3][kNearTile]: sum over star i, trial vertex lb
    uint32_t *trial = reinterpret_cast<uint32_t *>(sums + 3 * kNearTile);  // sorted trial panels
    uint8_t *missing = reinterpret_cast<uint8_t *>(trial + kNearTile);     // some panel of star i has no record of it
    const uint32_t i = blockIdx.x, o0 = incOffsets[i], o1 = incOffsets[i + 1];
    if (o0 == o1)
        return;
    const uint32_t list = map.row[incPanel[o0]], length = map.row[incPanel[o0] + 1] - list;
    const double sc = rowScale[i];
    bool escaped = false;
    for (uint32_t base = 0; base == 0 || base < length; base += kNearTile) {
        const uint32_t count = min(kNearTile, length - base);
        const bool last = base + count >= length;
        const uint32_t previous = base ? map.col[list + base - 1] : 0;
        for (uint32_t p = threadIdx.x; p < count; p += kNearThreads) {
            const uint32_t s = map.col[list + base + p];
            double2 acc[3] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
            bool absent = false;
            for (uint32_t oa = o0; oa < o1; ++oa) {
                const size_t slot = oa == o0 ? size_t(list + base + p) : mapSlot(map, T, incPanel[oa], s);
                if (slot == kNoSlot) {
                    absent = true;
                    continue;
                }
                const int la = incLocal[oa];
#pragma unroll
                for (int lb = 0; lb < 3; ++lb) {
                    const double2 r =
                        *reinterpret_cast<const double2 *>(records + mapOffset(map.planeSlots, slot, 3 * la + lb));
                    acc[lb].x += r.x;
                    acc[lb].y += r.y;
                }
            }
#pragma unroll
            for (int lb = 0; lb < 3; ++lb)
                sums[lb * kNearTile + p] = acc[lb];
            trial[p] = s;
            missing[p] = absent;
        }
        __syncthreads();
        for (uint32_t e = nearRow[i] + threadIdx.x; e < nearRow[i + 1]; e += kNearThreads) {
            const uint32_t j = nearCol[e];
            double2 v = base ? vals[e] : make_double2(0, 0);
            for (uint32_t os = incOffsets[j]; os < incOffsets[j + 1]; ++os) {
                const uint32_t s = incPanel[os];
                const uint32_t at = nearTilePlace(trial, count, s);
                if (at < count && trial[at] == s) {
                    escaped |= missing[at] != 0;
                    const double2 r = sums[incLocal[os] * kNearTile + at];
                    v.x += r.x;
                    v.y += r.y;
                } else  // in another tile, or in none
                    escaped |= nearTileMisses(at, count, base == 0, last, previous, s);
            }
            if (last) {
                for (uint32_t oa = o0; oa < o1; ++oa) {
                    const DPanel &p = panels[incPanel[oa]];
                    if (p.nodes[0] == j || p.nodes[1] == j || p.nodes[2] == j)
                        v.x += p.area * (i == j ? 2.0 : 1.0) / 24.0;
                }
                v.x *= sc;
                v.y *= sc;
            }
            vals[e] = v;
        }
        __syncthreads();
    }
    if (escaped)
        flagError(error, kErrEscapedPlan);
}

// Near right-hand side: rhs_i = rowScale_i sum over near j, panels s of star j
// (weight 1/3: a panel's flux is emitted through its three vertex supports)
// and panels a of star i of rhs moment la of record (a, s) times q_s.
__global__ void nearRhsKernel(const double *__restrict__ records, SlotMap map, const uint32_t *__restrict__ nearRow,
                              const uint32_t *__restrict__ nearCol, const uint32_t *__restrict__ incOffsets,
                              const uint32_t *__restrict__ incPanel, const uint8_t *__restrict__ incLocal,
                              const double2 *__restrict__ flux, const double *__restrict__ rowScale, uint32_t T,
                              uint32_t N, uint32_t E, double2 *rhs, int *error) {
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const uint32_t ex = blockIdx.y;
    if (i >= N)
        return;
    const double2 *q = flux + size_t(ex) * T;
    double re = 0, im = 0;
    for (uint32_t e = nearRow[i] + lane; e < nearRow[i + 1]; e += 32) {
        const uint32_t j = nearCol[e];
        for (uint32_t os = incOffsets[j]; os < incOffsets[j + 1]; ++os) {
            const uint32_t sp = incPanel[os];
            const double2 qs = q[sp];
            if (qs.x == 0 && qs.y == 0)
                continue;
            double mr = 0, mi = 0;
            for (uint32_t oa = incOffsets[i]; oa < incOffsets[i + 1]; ++oa) {
                const size_t slot = mapSlot(map, T, incPanel[oa], sp);
                if (slot == kNoSlot) {
                    flagError(error, kErrEscapedPlan);
                    continue;
                }
                const double *r = records + mapOffset(map.planeSlots, slot, 9 + incLocal[oa]);
                mr += r[0];
                mi += r[1];
            }
            re += (mr * qs.x - mi * qs.y) / 3.0;
            im += (mr * qs.y + mi * qs.x) / 3.0;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (lane == 0)
        rhs[size_t(ex) * N + i] = make_double2(re * rowScale[i], im * rowScale[i]);
}

}  // namespace

size_t nearFieldWorkspaceBytes(size_t pairSlots, uint64_t pairCount) {
    return pairSlots * kRecordDoubles * 8 + kBins * pairCount * sizeof(uint2) + kBins * 16;
}

void assembleNearField(const AssemblyGeometry &g, const double *k, const double *singularTuples, const double *flux,
                       uint32_t E, const NearFieldLayout &nf, void *workspace, double *vals, double *rhsNear,
                       int *error, cudaStream_t stream, KernelTimer *timer) {
    char *w = static_cast<char *>(workspace);
    AssemblyWorkspace ws{};
    ws.records = w;
    ws.bins = reinterpret_cast<uint2 *>(w + nf.pairSlots * kRecordDoubles * 8);
    ws.binCounts = reinterpret_cast<uint32_t *>(w + nf.pairSlots * kRecordDoubles * 8 + kBins * nf.pairCount * sizeof(uint2));
    ws.binCapacity = nf.pairCount;
    ws.binOffsets = nullptr;
    SlotMap map;
    map.row = nf.pairRow;
    map.col = nf.pairCol;
    map.planeSlots = nf.pairSlots;
    cudaCheck(cudaMemsetAsync(ws.records, 0, nf.pairSlots * kRecordDoubles * 8, stream), "near record reset");
    computeRecords(g, k, singularTuples, 1, ws, map, nf.pairList, nf.pairCount, error, stream, timer, false);
    {
        TimedScope scope(timer, "fmm_near_values", stream);
        static PerDeviceOnce attribute;
        attribute.run([]() {
            cudaCheck(cudaFuncSetAttribute(nearValuesKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           int(kNearValuesSmem)),
                      "near values smem attribute");
        });
        nearValuesKernel<<<g.N, kNearThreads, kNearValuesSmem, stream>>>(
            static_cast<const double *>(ws.records), map, nf.nearRow, nf.nearCol, g.incOffsets, g.incPanel, g.incLocal,
            g.panels, g.rowScale, g.T, reinterpret_cast<double2 *>(vals), error);
        cudaCheck(cudaGetLastError(), "near values launch");
    }
    {
        TimedScope scope(timer, "fmm_near_rhs", stream);
        nearRhsKernel<<<dim3((g.N * 32 + 255) / 256, E), 256, 0, stream>>>(
            static_cast<const double *>(ws.records), map, nf.nearRow, nf.nearCol, g.incOffsets, g.incPanel,
            g.incLocal, reinterpret_cast<const double2 *>(flux), g.rowScale, g.T, g.N, E,
            reinterpret_cast<double2 *>(rhsNear), error);
        cudaCheck(cudaGetLastError(), "near rhs launch");
    }
}

}  // namespace hsb
