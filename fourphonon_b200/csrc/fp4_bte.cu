// Linearised-BTE sweep and thermal conductivity on the device.
//
// iteration (Src/iterations.f90:34-92) and iteration_4ph (95-215, the same
// sweep with the ++, +- and -- lists added) are in-place Gauss-Seidel sweeps:
// modes are visited in the order (ll, i, kk) and each update reads F_n values
// already overwritten earlier in the same sweep.  The device sweep keeps that
// order exactly: one CTA walks the (ll, i, kk) steps in sequence and spreads
// each step's sum over the mode's processes across its threads (a tree
// reduction, so only the summation order inside one step differs from the
// reference's left-to-right loop).  F_n stays in the Fortran layout
// F_n(nbands,nptk,3).  The three-phonon sweep keeps the order with far less in the
// chain (k_block_sums, k_block_steps).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "../../include/fourphonon_b200.h"
#include "fp4_ctx.h"
#include "fp4_internal.h"

using namespace fp4;

namespace {

struct BteParams {
    int nb, nptk, nlist, nsr;
    const int* nequi;
    const int* allequi;   // ALLEquiList(nsr, *) column-major
    const int* typeofsym; // TypeofSymmetry(nsr, *)
    const int* id_equi;   // ID_equi(nsr, nptk)
    const double* symm;   // symmetrizers(3,3,nptk)
    const int* n_plus;
    const int* n_minus;
    const long long* off_plus;
    const long long* off_minus;
    const int* i2p;
    const int* i3p;
    const int* i2m;
    const int* i3m;
    const double* gp;
    const double* gm;
    const double* energy;    // energy(nptk,nb)
    const double* velocity;  // velocity(nptk,nb,3)
    const double* tau_zero;  // tau_zero(nb,nlist)
    double* F;               // F_n(nb,nptk,3)
    // four-phonon lists of iteration_4ph (n4[0] == nullptr: three-phonon sweep)
    const long long* n4[3];
    const long long* off4[3];
    const long long* i2_4[3];
    const long long* i3_4[3];
    const long long* i4_4[3];
    const double* g4[3];
    int* err;
};

__device__ __forceinline__ double& Fat(const BteParams& p, int b, int q, int d) {
    return p.F[((size_t)d * p.nptk + q) * p.nb + b];
}

// This thread's share (x = t0, t0 + dt, ...) of one step's sum over the mode's
// processes, with the q-points mapped by symmetry operation `sym`, reading F.
__device__ __forceinline__ void step_sum(const BteParams& p, const double* F, int mm, int sym, long long t0,
                                         long long dt, double& a0, double& a1, double& a2) {
    const int nb = p.nb;
    auto Fv = [&](int b, int q, int d) { return F[((size_t)d * p.nptk + q) * nb + b]; };
    const int np_ = p.n_plus[mm], nm_ = p.n_minus[mm];
    const long long op = p.off_plus[mm], om = p.off_minus[mm];
    long long c4[3] = {0, 0, 0};
    if (p.n4[0])
        for (int ch = 0; ch < 3; ch++) c4[ch] = p.n4[ch][mm];
    const long long n3ph = (long long)np_ + nm_, ntot = n3ph + c4[0] + c4[1] + c4[2];
    const long long lim = (long long)p.nptk * nb;
    for (long long x = t0; x < ntot; x += dt) {
        if (x >= n3ph) {
            // iteration_4ph: ++ Gamma(F_l - F_j - F_k), +- Gamma(F_l - F_j + F_k),
            // -- Gamma(F_l + F_j + F_k), q-points mapped by the same symmetry
            long long y = x - n3ph;
            int ch = 0;
            while (ch < 2 && y >= c4[ch]) {
                y -= c4[ch];
                ch++;
            }
            const long long o = p.off4[ch][mm] + y;
            const long long y2 = p.i2_4[ch][o] - 1, y3 = p.i3_4[ch][o] - 1, y4 = p.i4_4[ch][o] - 1;
            if (y2 < 0 || y2 >= lim || y3 < 0 || y3 >= lim || y4 < 0 || y4 >= lim) {
                atomicOr(p.err, kErrList);
                continue;
            }
            const int j = (int)(y2 % nb), k = (int)(y3 % nb), l = (int)(y4 % nb);
            const int qj = p.id_equi[(y2 / nb) * p.nsr + sym] - 1;
            const int qk = p.id_equi[(y3 / nb) * p.nsr + sym] - 1;
            const int ql = p.id_equi[(y4 / nb) * p.nsr + sym] - 1;
            const double g = p.g4[ch][o];
            const double sj = (ch == 2) ? 1.0 : -1.0, sk = (ch == 0) ? -1.0 : 1.0;
            // F_l -+ F_j -+ F_k with the reference's left-to-right order
            a0 += g * ((Fv(l, ql, 0) + sj * Fv(j, qj, 0)) + sk * Fv(k, qk, 0));
            a1 += g * ((Fv(l, ql, 1) + sj * Fv(j, qj, 1)) + sk * Fv(k, qk, 1));
            a2 += g * ((Fv(l, ql, 2) + sj * Fv(j, qj, 2)) + sk * Fv(k, qk, 2));
            continue;
        }
        const bool plus = x < np_;
        const long long o = plus ? op + x : om + (x - np_);
        const int x2 = (plus ? p.i2p : p.i2m)[o] - 1, x3 = (plus ? p.i3p : p.i3m)[o] - 1;
        if (x2 < 0 || x2 >= lim || x3 < 0 || x3 >= lim) {
            atomicOr(p.err, kErrList);
            continue;
        }
        const int j = x2 % nb, m2 = x2 / nb, k = x3 % nb, n3 = x3 / nb;
        const int qa = p.id_equi[(size_t)n3 * p.nsr + sym] - 1;
        const int qb = p.id_equi[(size_t)m2 * p.nsr + sym] - 1;
        const double g = (plus ? p.gp : p.gm)[o];
        double t0_, t1_, t2_;
        if (plus) {
            t0_ = g * (Fv(k, qa, 0) - Fv(j, qb, 0));
            t1_ = g * (Fv(k, qa, 1) - Fv(j, qb, 1));
            t2_ = g * (Fv(k, qa, 2) - Fv(j, qb, 2));
        } else {
            t0_ = g * (Fv(k, qa, 0) + Fv(j, qb, 0)) * 5.e-1;
            t1_ = g * (Fv(k, qa, 1) + Fv(j, qb, 1)) * 5.e-1;
            t2_ = g * (Fv(k, qa, 2) + Fv(j, qb, 2)) * 5.e-1;
        }
        a0 += t0_;
        a1 += t1_;
        a2 += t2_;
    }
}

// Block sum of (a0, a1, a2) into thread 0 (red: 3 x 32 doubles of shared memory).
__device__ __forceinline__ void block_sum3(double& a0, double& a1, double& a2, double (*red)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_down_sync(0xffffffffu, a0, o);
        a1 += __shfl_down_sync(0xffffffffu, a1, o);
        a2 += __shfl_down_sync(0xffffffffu, a2, o);
    }
    if (lane == 0) {
        red[0][warp] = a0;
        red[1][warp] = a1;
        red[2][warp] = a2;
    }
    __syncthreads();
    if (warp == 0) {
        a0 = lane < nwarp ? red[0][lane] : 0.0;
        a1 = lane < nwarp ? red[1][lane] : 0.0;
        a2 = lane < nwarp ? red[2][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a0 += __shfl_down_sync(0xffffffffu, a0, o);
            a1 += __shfl_down_sync(0xffffffffu, a1, o);
            a2 += __shfl_down_sync(0xffffffffu, a2, o);
        }
    }
}

// iteration / iteration_4ph (iterations.f90:34-215): one Gauss-Seidel sweep in the
// reference's order (ll, i, kk), updating F in place; one CTA.
__global__ void __launch_bounds__(1024) k_sweep(BteParams p) {
    __shared__ double red[3][32];
    const int nb = p.nb;
    for (int ll = 0; ll < p.nlist; ll++) {
        for (int i = 0; i < nb; i++) {
            const int mm = ll * nb + i;
            for (int kk = 0; kk < p.nequi[ll]; kk++) {
                const int qq = p.allequi[ll * p.nsr + kk] - 1;
                const int sym = p.typeofsym[ll * p.nsr + kk] - 1;
                double a0 = 0.0, a1 = 0.0, a2 = 0.0;
                step_sum(p, p.F, mm, sym, threadIdx.x, blockDim.x, a0, a1, a2);
                block_sum3(a0, a1, a2, red);
                if (threadIdx.x == 0) {
                    const double tz = p.tau_zero[ll * nb + i];
                    const size_t e = (size_t)i * p.nptk + qq, pl = (size_t)p.nptk * nb;
                    const double w = p.energy[e];
                    Fat(p, i, qq, 0) = tz * p.velocity[e] * w + tz * a0;
                    Fat(p, i, qq, 1) = tz * p.velocity[e + pl] * w + tz * a1;
                    Fat(p, i, qq, 2) = tz * p.velocity[e + 2 * pl] * w + tz * a2;
                }
                __syncthreads();
                // F_n(:,qq,:) = transpose(matmul(symmetrizers(:,:,qq), transpose(F_n(:,qq,:))))
                if (threadIdx.x < nb) {
                    const int b = threadIdx.x;
                    const double* Sq = p.symm + 9 * (size_t)qq;
                    double x0 = Fat(p, b, qq, 0), x1 = Fat(p, b, qq, 1), x2 = Fat(p, b, qq, 2);
                    double y[3];
#pragma unroll
                    for (int a = 0; a < 3; a++) y[a] = Sq[a] * x0 + Sq[a + 3] * x1 + Sq[a + 6] * x2;
                    Fat(p, b, qq, 0) = y[0];
                    Fat(p, b, qq, 1) = y[1];
                    Fat(p, b, qq, 2) = y[2];
                }
                __syncthreads();
            }
        }
    }
}

// The three-phonon sweep in blocks of consecutive irreducible points.  While the steps
// of a block run, F changes only at the block's own points (the stars of its
// irreducible points), so each step's sum splits into the terms at all other points,
// which k_block_sums forms for every step of the block at once on the whole GPU, and
// the few at the block's points (about 2 n B / nptk of a mode's 2 n terms for B points),
// which it lists and k_block_steps adds in the reference's step order from shared
// memory.  k_sweep puts every term of a step into the chain: 12.5 us a step on the 12^3
// diamond grid (130 ms a sweep).  Here a step of the chain is two barriers and a few
// hundred terms, and the sweep's kernels take 13.0 ms.
constexpr int kBlockPoints = 64;   // most points of a block (one star may have more)
constexpr int kStepThreads = 128;  // threads of k_block_steps

struct StepInfo {
    double base[3];  // tau v omega
    double sum[3];   // the terms outside the block
    double tau;
    long long term;       // its first listed term
    int cnt, slot, band;  // listed terms inside the block, the step's point and branch
};
struct BlockParams {
    const int* step0;           // first step of each irreducible point, over the whole sweep
    const long long* term0;     // first listed term of each mode's steps, within its block
    int* slot_of;               // point -> its slot in the block, -1 outside
    StepInfo* info;             // [step of the block]
    int* idx;                   // listed terms: slot * nb + branch
    double* coef;               //               and signed amplitude
};

// Slots of the points of the stars [l0, l1); a point met twice keeps its first slot.
__device__ void mark_block(const BteParams& p, const BlockParams& q, int l0, int l1) {
    int s = 0;
    for (int ll = l0; ll < l1; ll++) {
        for (int kk = threadIdx.x; kk < p.nequi[ll]; kk += blockDim.x)  // -1 is the largest unsigned value
            atomicMin(reinterpret_cast<unsigned*>(q.slot_of + p.allequi[ll * p.nsr + kk] - 1), (unsigned)(s + kk));
        s += p.nequi[ll];
    }
}

__global__ void k_block_begin(BteParams p, BlockParams q, int l1) {
    for (int x = threadIdx.x; x < p.nptk; x += blockDim.x) q.slot_of[x] = -1;
    __syncthreads();
    mark_block(p, q, 0, l1);
}

// One CTA per step of the block [l0, l1).  The listed terms keep a fixed order (by passes
// of kSumRows rows of kSumThreads processes, row and warp; a warp's first terms before its
// second ones), so that a sweep gives the same bits every time.  Several rows to a barrier,
// since a row is four dependent loads: sweep of diamond 16^3, 1, 2 and 4 rows 35.9, 35.0,
// 34.7 ms (34.9 with places from an atomic counter, which leave the order open), 20^3 78.2,
// 75.2, 74.5 (75.3).
constexpr int kSumThreads = 256, kSumWarps = kSumThreads / 32;
constexpr int kSumRows = 4;  // rows between two barriers
__global__ void __launch_bounds__(kSumThreads) k_block_sums(BteParams p, BlockParams q, int l0, int l1) {
    __shared__ double red[3][32];
    __shared__ int s_cnt[2][kSumRows * kSumWarps];  // listed terms of each (row, warp), alternately
    const int nb = p.nb;
    const int step = q.step0[l0] + blockIdx.x;
    int ll = l0;
    while (q.step0[ll + 1] <= step) ll++;
    const int neq = p.nequi[ll], rest = step - q.step0[ll], i = rest / neq, kk = rest - i * neq;
    const int mm = ll * nb + i;
    const int qq = p.allequi[ll * p.nsr + kk] - 1, sym = p.typeofsym[ll * p.nsr + kk] - 1;
    const int np_ = p.n_plus[mm], nt = np_ + p.n_minus[mm];
    const long long op = p.off_plus[mm], om = p.off_minus[mm];
    const long long out = q.term0[mm] + (long long)kk * 2 * nt;
    const int lim = p.nptk * nb;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    double a[3] = {0.0, 0.0, 0.0};
    const size_t pl = (size_t)lim;
    int listed = 0;
    for (int x0 = 0, buf = 0; x0 < nt; x0 += kSumRows * kSumThreads, buf ^= 1) {
        int ia[kSumRows], ib[kSumRows];  // the processes' listed terms: slot * nb + branch
        double g[kSumRows];
        unsigned ma[kSumRows], mb[kSumRows];
        bool plus[kSumRows];
#pragma unroll
        for (int y = 0; y < kSumRows; y++) {
            const int x = x0 + y * kSumThreads + threadIdx.x;
            ia[y] = ib[y] = -1;
            g[y] = 0.0;
            plus[y] = x < np_;
            if (x < nt) {
                const long long o = plus[y] ? op + x : om + (x - np_);
                const int x2 = (plus[y] ? p.i2p : p.i2m)[o] - 1, x3 = (plus[y] ? p.i3p : p.i3m)[o] - 1;
                if (x2 < 0 || x2 >= lim || x3 < 0 || x3 >= lim) {
                    atomicOr(p.err, kErrList);
                } else {
                    const int m2 = x2 / nb, j = x2 - m2 * nb, n3 = x3 / nb, k = x3 - n3 * nb;
                    const int qa = p.id_equi[(size_t)n3 * p.nsr + sym] - 1, qb = p.id_equi[(size_t)m2 * p.nsr + sym] - 1;
                    const int sa = q.slot_of[qa], sb = q.slot_of[qb];
                    const double* fa = p.F + (size_t)qa * nb + k;
                    const double* fb = p.F + (size_t)qb * nb + j;
                    const double sg = plus[y] ? -1.0 : 1.0;
                    g[y] = plus[y] ? p.gp[o] : p.gm[o] * 5.e-1;
                    // as step_sum: the amplitude times F_a -+ F_b, without what is listed
                    double f[3] = {0.0, 0.0, 0.0};
                    if (sa >= 0) {
                        ia[y] = sa * nb + k;
                    } else {
#pragma unroll
                        for (int d = 0; d < 3; d++) f[d] = fa[d * pl];
                    }
                    if (sb >= 0) {
                        ib[y] = sb * nb + j;
                    } else {
#pragma unroll
                        for (int d = 0; d < 3; d++) f[d] = fma(sg, fb[d * pl], f[d]);
                    }
                    if (sa < 0 || sb < 0) {
#pragma unroll
                        for (int d = 0; d < 3; d++) a[d] = fma(g[y], f[d], a[d]);
                    }
                }
            }
        }
#pragma unroll
        for (int y = 0; y < kSumRows; y++) {
            ma[y] = __ballot_sync(0xffffffffu, ia[y] >= 0);
            mb[y] = __ballot_sync(0xffffffffu, ib[y] >= 0);
            if (lane == 0) s_cnt[buf][y * kSumWarps + warp] = __popc(ma[y]) + __popc(mb[y]);
        }
        __syncthreads();  // (the next rows write the other counts)
#pragma unroll
        for (int y = 0; y < kSumRows; y++) {
            long long pos = out + listed;
#pragma unroll
            for (int w = 0; w < kSumWarps; w++) {
                const int n = s_cnt[buf][y * kSumWarps + w];
                pos += w < warp ? n : 0;
                listed += n;
            }
            if (ia[y] >= 0) {
                q.idx[pos + __popc(ma[y] & below)] = ia[y];
                q.coef[pos + __popc(ma[y] & below)] = g[y];
            }
            pos += __popc(ma[y]);
            if (ib[y] >= 0) {
                q.idx[pos + __popc(mb[y] & below)] = ib[y];
                q.coef[pos + __popc(mb[y] & below)] = plus[y] ? -g[y] : g[y];
            }
        }
    }
    block_sum3(a[0], a[1], a[2], red);
    if (threadIdx.x == 0) {
        const double tz = p.tau_zero[mm];
        const size_t e = (size_t)i * p.nptk + qq;
        const double w = p.energy[e];
        StepInfo s;
        for (int d = 0; d < 3; d++) {
            s.base[d] = tz * p.velocity[e + d * pl] * w;
            s.sum[d] = a[d];
        }
        s.tau = tz;
        s.term = out;
        s.cnt = listed;
        s.slot = q.slot_of[qq];
        s.band = i;
        q.info[blockIdx.x] = s;
    }
}

// The block's steps in order, on one CTA; then the marks of the next block [l1, l2).
// Shared memory: F and the symmetrizer of each of the block's npts points.
__global__ void __launch_bounds__(kStepThreads) k_block_steps(BteParams p, BlockParams q, int l0, int l1, int l2,
                                                              int npts) {
    extern __shared__ double sm[];
    __shared__ double red[3][kStepThreads / 32];
    const int nb = p.nb, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* Fs = sm;                        // [slot][band][3]
    double* Ss = sm + (size_t)npts * nb * 3;  // [slot][9]
    int s0 = 0;
    for (int ll = l0; ll < l1; ll++) {
        const int neq = p.nequi[ll];
        for (int x = threadIdx.x; x < neq * nb; x += blockDim.x) {
            const int kk = x / nb, b = x - kk * nb, qq = p.allequi[ll * p.nsr + kk] - 1;
            for (int d = 0; d < 3; d++) Fs[((s0 + kk) * nb + b) * 3 + d] = Fat(p, b, qq, d);
        }
        for (int x = threadIdx.x; x < neq * 9; x += blockDim.x)
            Ss[s0 * 9 + x] = p.symm[9 * (size_t)(p.allequi[ll * p.nsr + x / 9] - 1) + x % 9];
        s0 += neq;
    }
    __syncthreads();
    // a step's record is read two steps ahead, each thread's first two of its terms one
    // step ahead: no load of the chain's own step is waited for
    const int nsteps = q.step0[l1] - q.step0[l0];
    auto record = [&](int st) { return q.info[min(st, nsteps - 1)]; };
    auto terms = [&](const StepInfo& s, int (&ix)[2], double (&cf)[2]) {
#pragma unroll
        for (int y = 0; y < 2; y++) {
            const int x = threadIdx.x + y * kStepThreads;
            ix[y] = x < s.cnt ? q.idx[s.term + x] : 0;
            cf[y] = x < s.cnt ? q.coef[s.term + x] : 0.0;
        }
    };
    StepInfo s_1{}, s_2{};
    int ix_1[2] = {0, 0};
    double cf_1[2] = {0.0, 0.0};
    if (nsteps > 0) {
        s_1 = record(0);
        s_2 = record(1);
        terms(s_1, ix_1, cf_1);
    }
    for (int st = 0; st < nsteps; st++) {
        const StepInfo s = s_1;
        const int ix[2] = {ix_1[0], ix_1[1]};
        const double cf[2] = {cf_1[0], cf_1[1]};
        s_1 = s_2;
        s_2 = record(st + 2);
        terms(s_1, ix_1, cf_1);
        double a[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int y = 0; y < 2; y++)
            if (threadIdx.x + y * kStepThreads < s.cnt)
                for (int d = 0; d < 3; d++) a[d] = fma(cf[y], Fs[ix[y] * 3 + d], a[d]);
        for (int x = threadIdx.x + 2 * kStepThreads; x < s.cnt; x += kStepThreads) {
            const int ii = q.idx[s.term + x];
            const double g = q.coef[s.term + x];
            for (int d = 0; d < 3; d++) a[d] = fma(g, Fs[ii * 3 + d], a[d]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int d = 0; d < 3; d++) a[d] += __shfl_down_sync(0xffffffffu, a[d], o);
        if (lane == 0)
            for (int d = 0; d < 3; d++) red[d][warp] = a[d];
        __syncthreads();
        // the step's branch takes its new value, then F_n(:,qq,:) is symmetrised
        if (threadIdx.x < nb) {
            double* f = Fs + (s.slot * nb + threadIdx.x) * 3;
            double y[3] = {f[0], f[1], f[2]};
            if (threadIdx.x == s.band) {
                for (int d = 0; d < 3; d++) {
                    double in = 0.0;
#pragma unroll
                    for (int w = 0; w < kStepThreads / 32; w++) in += red[d][w];
                    y[d] = s.base[d] + s.tau * (s.sum[d] + in);
                }
            }
            const double* Sq = Ss + s.slot * 9;
            for (int d = 0; d < 3; d++) f[d] = Sq[d] * y[0] + Sq[d + 3] * y[1] + Sq[d + 6] * y[2];
        }
        __syncthreads();
    }
    s0 = 0;
    for (int l = l0; l < l1; l++) {
        const int neq = p.nequi[l];
        for (int x = threadIdx.x; x < neq * nb; x += blockDim.x) {
            const int k = x / nb, b = x - k * nb, qq = p.allequi[l * p.nsr + k] - 1;
            if (q.slot_of[qq] != s0 + k) continue;  // a repeated point lives in its first slot
            for (int d = 0; d < 3; d++) Fat(p, b, qq, d) = Fs[((s0 + k) * nb + b) * 3 + d];
        }
        s0 += neq;
    }
    __syncthreads();
    for (int l = l0; l < l1; l++)
        for (int k = threadIdx.x; k < p.nequi[l]; k += blockDim.x) q.slot_of[p.allequi[l * p.nsr + k] - 1] = -1;
    __syncthreads();
    mark_block(p, q, l1, l2);
}

// The Jacobi form of the same update (no counterpart in the reference, whose
// sweep is Gauss-Seidel): every step reads the previous iterate F and writes
// Fout, so all steps run at once, one CTA per (mode, equivalent point).  The
// site symmetrizer is applied afterwards (k_symmetrize) to every point, which is
// what the in-place sweep's per-step projection does to the band it has just
// updated.  Converges to the same fixed point, in more sweeps.
__global__ void __launch_bounds__(256) k_jacobi_step(BteParams p, double* Fout) {
    __shared__ double red[3][32];
    const int nb = p.nb;
    const int mm = blockIdx.x, kk = blockIdx.y;
    const int ll = mm / nb, i = mm - ll * nb;
    if (kk >= p.nequi[ll]) return;
    const int qq = p.allequi[ll * p.nsr + kk] - 1;
    const int sym = p.typeofsym[ll * p.nsr + kk] - 1;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    step_sum(p, p.F, mm, sym, threadIdx.x, blockDim.x, a0, a1, a2);
    block_sum3(a0, a1, a2, red);
    if (threadIdx.x == 0) {
        const double tz = p.tau_zero[ll * nb + i];
        const size_t e = (size_t)i * p.nptk + qq, pl = (size_t)p.nptk * nb;
        const double w = p.energy[e];
        Fout[((size_t)0 * p.nptk + qq) * nb + i] = tz * p.velocity[e] * w + tz * a0;
        Fout[((size_t)1 * p.nptk + qq) * nb + i] = tz * p.velocity[e + pl] * w + tz * a1;
        Fout[((size_t)2 * p.nptk + qq) * nb + i] = tz * p.velocity[e + 2 * pl] * w + tz * a2;
    }
}

__global__ void k_iteration0(int nb, int nptk, int nlist, int nsr, const int* nequi, const int* allequi,
                             const double* energy, const double* velocity, const double* tau_zero, double* F) {
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < nlist * nb * nsr; x += gridDim.x * blockDim.x) {
        int kk = x % nsr, rest = x / nsr, i = rest % nb, ll = rest / nb;
        if (kk >= nequi[ll]) continue;
        int qq = allequi[ll * nsr + kk] - 1;
        size_t e = (size_t)i * nptk + qq, pl = (size_t)nptk * nb;
        double tz = tau_zero[ll * nb + i], w = energy[e];
        for (int d = 0; d < 3; d++) F[((size_t)d * nptk + qq) * nb + i] = tz * velocity[e + d * pl] * w;
    }
}

__global__ void k_symmetrize(int nb, int nptk, const double* symm, double* F) {
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < nb * nptk; x += gridDim.x * blockDim.x) {
        int b = x % nb, q = x / nb;
        const double* Sq = symm + 9 * (size_t)q;
        double v[3];
        for (int d = 0; d < 3; d++) v[d] = F[((size_t)d * nptk + q) * nb + b];
        for (int a = 0; a < 3; a++) F[((size_t)a * nptk + q) * nb + b] = Sq[a] * v[0] + Sq[a + 3] * v[1] + Sq[a + 6] * v[2];
    }
}

// TConduct (conductivity.f90:11-37): one CTA per branch, q >= 2, fixed-order tree sum.
__global__ void k_tconduct(int nb, int nptk, double T, double scale, const double* energy, const double* velocity,
                           const double* F, double* kappa, double* kmode) {
    __shared__ double red[9][32];
    const int jj = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const double hbar = 1.05457172647e-22, kb = 1.380648813e-23;
    double acc[9];
    for (int x = 0; x < 9; x++) acc[x] = 0.0;
    const size_t pl = (size_t)nptk * nb;
    for (int ii = 1 + threadIdx.x; ii < nptk; ii += blockDim.x) {
        size_t e = (size_t)jj * nptk + ii;
        double w = energy[e];
        double f = 1.0 / (exp(hbar * w / kb / T) - 1.0);
        double c = f * (f + 1) * w;
        for (int d2 = 0; d2 < 3; d2++) {
            double Fd = F[((size_t)d2 * nptk + ii) * nb + jj];
            for (int d1 = 0; d1 < 3; d1++) {
                double m = c * (velocity[e + d1 * pl] * Fd);
                acc[d2 * 3 + d1] += m;
                if (kmode) kmode[(((size_t)(d2 * 3 + d1)) * nb + jj) * nptk + ii] = scale * m;
            }
        }
    }
    for (int x = 0; x < 9; x++) {
        double v = acc[x];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[x][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < 9) {
        double t = 0.0;
        for (int w = 0; w < nwarp; w++) t += red[threadIdx.x][w];
        kappa[threadIdx.x * nb + jj] = scale * t;  // ThConductivity(jj,d1,d2): [(d2*3+d1)*nb + jj]
    }
}

// Euclidean norm of a 3-vector by the scaled sum of squares of reference BLAS
// dnrm2, unfused so that it rounds as the host evaluation does.
__device__ double nrm2_3(double x0, double x1, double x2) {
    double scale = 0.0, ssq = 1.0;
    const double x[3] = {x0, x1, x2};
    for (int i = 0; i < 3; i++) {
        if (x[i] != 0.0) {
            const double a = fabs(x[i]);
            if (scale < a) {
                const double q = scale / a;
                ssq = __dadd_rn(1.0, __dmul_rn(__dmul_rn(ssq, q), q));
                scale = a;
            } else {
                const double q = a / scale;
                ssq = __dadd_rn(ssq, __dmul_rn(q, q));
            }
        }
    }
    return __dmul_rn(scale, sqrt(ssq));
}

// CumulativeTConduct / CumulativeTConductOmega (conductivity.f90:64-148): one CTA
// per (tick, branch) sums the modes whose mean free path (or omega) is below
// the tick.  results(nb,3,3,nticks) as [((k*3 + d2)*3 + d1)*nb + b].
__global__ void k_cumulative(int nb, int nptk, int nticks, int omega_mode, double T, double scale,
                             const double* energy, const double* velocity, const double* F, const double* ticks,
                             double* results) {
    __shared__ double red[9][32];
    const int k = blockIdx.x, jj = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const double hbar = 1.05457172647e-22, kb = 1.380648813e-23;
    const double tick = ticks[k];
    double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const size_t pl = (size_t)nptk * nb;
    for (int ii = 1 + threadIdx.x; ii < nptk; ii += blockDim.x) {  // reference q index 2..nptk
        const size_t e = (size_t)jj * nptk + ii;
        const double w = energy[e];
        const double v[3] = {velocity[e], velocity[e + pl], velocity[e + 2 * pl]};
        const double f[3] = {F[(size_t)ii * nb + jj], F[((size_t)nptk + ii) * nb + jj], F[((size_t)2 * nptk + ii) * nb + jj]};
        double lambda;
        if (omega_mode) {
            lambda = w;
        } else {
            const double dot = __dadd_rn(__dadd_rn(__dmul_rn(f[0], v[0]), __dmul_rn(f[1], v[1])), __dmul_rn(f[2], v[2]));
            lambda = dot / __dmul_rn(__dadd_rn(w, 1e-12), nrm2_3(v[0], v[1], v[2]));
        }
        if (!(tick > lambda)) continue;
        const double fbe = 1.0 / (exp(hbar * w / kb / T) - 1.0);
        const double pre = fbe * (fbe + 1) * w;
        for (int d1 = 0; d1 < 3; d1++)
            for (int d2 = 0; d2 < 3; d2++) acc[d2 * 3 + d1] += pre * (v[d1] * f[d2]);
    }
    for (int x = 0; x < 9; x++) {
        double t = acc[x];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) red[x][warp] = t;
    }
    __syncthreads();
    if (threadIdx.x < 9) {
        double t = 0.0;
        for (int w = 0; w < nwarp; w++) t += red[threadIdx.x][w];
        results[((size_t)k * 9 + threadIdx.x) * nb + jj] = scale * t;
    }
}

}  // namespace

namespace fp4 {
cudaError_t launch_iteration0(int nb, int nptk, int nlist, int nsr, const int* nequi, const int* allequi,
                              const double* energy, const double* velocity, const double* tau_zero, double* F,
                              cudaStream_t st) {
    k_iteration0<<<256, 256, 0, st>>>(nb, nptk, nlist, nsr, nequi, allequi, energy, velocity, tau_zero, F);
    return cudaGetLastError();
}

cudaError_t launch_tconduct(int nb, int nptk, double T, double V, const double* energy, const double* velocity,
                            const double* F, double* kappa, cudaStream_t st) {
    const double hbar = 1.05457172647e-22, kb = 1.380648813e-23;
    const double scale = (double)1e21f * (hbar * hbar) / (kb * T * T * V * nptk);
    k_tconduct<<<nb, 256, 0, st>>>(nb, nptk, T, scale, energy, velocity, F, kappa, nullptr);
    return cudaGetLastError();
}
}  // namespace fp4

#define CK(call)                                                                                      \
    do {                                                                                              \
        cudaError_t e_ = (call);                                                                      \
        if (e_ != cudaSuccess) return fp4_fail(c, FP4_E_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

static int check_g(fp4_ctx* c, const fp4_globals* g) {
    if (!g) return fp4_fail(c, FP4_E_ARG, "null globals");
    for (int d = 0; d < 3; d++)
        if (g->ngrid[d] < 1) return fp4_fail(c, FP4_E_ARG, "ngrid must be >0");
    if (g->nbands < 3) return fp4_fail(c, FP4_E_ARG, "nbands must be >=3");
    return FP4_OK;
}

extern "C" int fp4_iteration0(fp4_ctx* c, const fp4_globals* g, int32_t nlist, const int32_t* nequi,
                              const int32_t* allequi, int32_t nsr, const double* omega, const double* velocity,
                              const double* tau_zero, double* f_n) {
    FP4_TRACE();
    if (!c) return FP4_E_ARG;
    int r;
    if ((r = check_g(c, g))) return r;
    if (!nequi || !allequi || !omega || !velocity || !tau_zero || !f_n || nlist < 1 || nsr < 1)
        return fp4_fail(c, FP4_E_ARG, "bad argument");
    if ((r = fp4_begin(c))) return r;
    const int nb = g->nbands, nptk = g->ngrid[0] * g->ngrid[1] * g->ngrid[2];
    DevBuffer* B = c->b_bte;
    if ((r = B[0].upload(c, nequi, nlist * sizeof(int))) || (r = B[1].upload(c, allequi, (size_t)nlist * nsr * sizeof(int))) ||
        (r = B[2].upload(c, omega, (size_t)nptk * nb * sizeof(double))) ||
        (r = B[3].upload(c, velocity, (size_t)nptk * nb * 3 * sizeof(double))) ||
        (r = B[4].upload(c, tau_zero, (size_t)nlist * nb * sizeof(double))) ||
        (r = B[5].reserve(c, (size_t)nptk * nb * 3 * sizeof(double))))
        return r;
    CK(cudaMemsetAsync(B[5].ptr, 0, (size_t)nptk * nb * 3 * sizeof(double), c->stream));
    k_iteration0<<<256, 256, 0, c->stream>>>(nb, nptk, nlist, nsr, B[0].as<int>(), B[1].as<int>(), B[2].as<double>(),
                                            B[3].as<double>(), B[4].as<double>(), B[5].as<double>());
    CK(cudaGetLastError());
    c->launches++;
    CK(cudaMemcpyAsync(f_n, B[5].ptr, (size_t)nptk * nb * 3 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    return fp4_end(c);
}

namespace {
// The four-phonon arguments of iteration_4ph (all null for the three-phonon sweep).
struct Lists4 {
    const int64_t* n[3];
    int64_t ntotal[3];
    const int64_t* i2[3];
    const int64_t* i3[3];
    const int64_t* i4[3];
    const double* g[3];
};
}  // namespace

static size_t block_smem(int nb, int pts) { return (size_t)pts * (nb * 3 + 9) * sizeof(double); }

// Cuts the irreducible points into blocks of at most B points (or one star), and lays out
// their steps and, for the worst case that every term falls inside the block, their listed
// terms; terms, steps and pts are the largest block's.
//   B: of a mode's m terms a block of B points lists m B / nptk for the chain, whose threads
// read two of them ahead each; more are waited for.  So B is the most points whose steps
// keep to 2 kStepThreads terms, and kBlockPoints where that is more: a block costs two
// launches and the serial rows of k_block_sums, about 10 us and 9 ns for each of m / 2
// processes.  3-atom cell on 8^3, B = 13 (2, 8, 16, 64 points: 17.4, 8.3, 8.8, 19.4 ms; k_sweep
// 40.2); 8-atom cell on 4^3, B = 1, two points to a star (2, 8, 64 points: 3.3, 7.0, 76 ms;
// k_sweep 14.2); diamond 16^3, B = 63 (32, 64 points: 38.2, 34.4 ms; k_sweep 583).
//   False, and the sweep runs on k_sweep, where that is the cheaper one (a few points with
// many processes, half of whose terms lie inside a star), when a block's terms or points
// would take too much memory, or when there are more branches than k_block_steps has
// threads.  (The worst case is far from the listed share of about B / nptk: the 12^3 diamond
// grid gets 16 MB and lists 3 % of it.  One star of 48 points passes the limit when its
// modes have 350,000 processes in all.)
static bool plan_blocks(int nb, int nptk, int nlist, const int32_t* nequi, const int32_t* n_plus,
                        const int32_t* n_minus, long long nproc, std::vector<int>& cut, std::vector<int>& step0,
                        std::vector<long long>& term0, size_t& terms, size_t& steps, int& pts) {
    const size_t kMaxTerms = (size_t)32 << 20;  // 384 MB of indices and amplitudes
    const size_t kMaxSmem = 200 * 1024;
    const double m = 2.0 * nproc / ((double)nb * nlist);      // a mode's terms
    const double kBlockNs = 10000.0 + 4.5 * m;
    const double kStepNs = 650.0, kTermNs = 3.0;              // a step of the chain, and each of its listed terms
    const double kSweepStepNs = 1900.0, kSweepTermNs = 0.65;  // a step of k_sweep, and each of its terms
    const int B = (int)std::max(1.0, std::min((double)kBlockPoints, 2.0 * kStepThreads * nptk / (m + 1.0)));
    double blocks_ns = 0.0, sweep_ns = 0.0;
    auto add_cost = [&](double points, double all) {  // of a block whose steps have `all` terms together
        blocks_ns += kBlockNs + points * nb * kStepNs + kTermNs * all * points / nptk;
        sweep_ns += points * nb * kSweepStepNs + kSweepTermNs * all;
    };
    cut.assign(1, 0);
    step0.assign(nlist + 1, 0);
    term0.assign((size_t)nb * nlist, 0);
    terms = steps = 0;
    pts = 0;
    size_t bt = 0;
    int bp = 0;
    for (int ll = 0; ll < nlist; ll++) {
        size_t lt = 0;
        for (int i = 0; i < nb; i++) lt += (size_t)2 * ((size_t)n_plus[ll * nb + i] + n_minus[ll * nb + i]) * nequi[ll];
        if (ll > cut.back() && (bp + nequi[ll] > B || bt + lt > kMaxTerms)) {
            add_cost(bp, (double)bt);
            cut.push_back(ll);
            bt = 0;
            bp = 0;
        }
        for (int i = 0; i < nb; i++) {
            term0[(size_t)ll * nb + i] = (long long)bt;
            bt += (size_t)2 * ((size_t)n_plus[ll * nb + i] + n_minus[ll * nb + i]) * nequi[ll];
        }
        bp += nequi[ll];
        step0[ll + 1] = step0[ll] + nb * nequi[ll];
        terms = std::max(terms, bt);
        steps = std::max(steps, (size_t)(step0[ll + 1] - step0[cut.back()]));
        pts = std::max(pts, bp);
    }
    add_cost(bp, (double)bt);
    cut.push_back(nlist);
    return blocks_ns < sweep_ns && nb <= kStepThreads && terms <= kMaxTerms && block_smem(nb, pts) <= kMaxSmem;
}

static int run_sweep(fp4_ctx* c, const fp4_globals* g, int32_t nlist, const int32_t* nequi, const int32_t* allequi,
                     const int32_t* typeofsym, int32_t nsr, const int32_t* id_equi, const double* symmetrizers,
                     const int32_t* n_plus, const int32_t* n_minus, int32_t ntotal_plus, int32_t ntotal_minus,
                     const int32_t* i2p, const int32_t* i3p, const int32_t* i2m, const int32_t* i3m,
                     const double* omega, const double* velocity, const double* gp, const double* gm,
                     const double* tau_zero, double* f_n, const Lists4* l4, bool jacobi = false) {
    if (!c) return FP4_E_ARG;
    int r;
    if ((r = check_g(c, g))) return r;
    if (!nequi || !allequi || !typeofsym || !id_equi || !symmetrizers || !n_plus || !n_minus || !omega || !velocity ||
        !tau_zero || !f_n || nlist < 1 || nsr < 1 || ntotal_plus < 0 || ntotal_minus < 0)
        return fp4_fail(c, FP4_E_ARG, "bad argument");
    if ((ntotal_plus && (!i2p || !i3p || !gp)) || (ntotal_minus && (!i2m || !i3m || !gm)))
        return fp4_fail(c, FP4_E_ARG, "null process list");
    const int nb = g->nbands, nptk = g->ngrid[0] * g->ngrid[1] * g->ngrid[2], nm = nb * nlist;
    std::vector<long long> op(nm + 1, 0), om(nm + 1, 0);
    for (int m = 0; m < nm; m++) {
        if (n_plus[m] < 0 || n_minus[m] < 0) return fp4_fail(c, FP4_E_ARG, "negative count");
        op[m + 1] = op[m] + n_plus[m];
        om[m + 1] = om[m] + n_minus[m];
    }
    if (op[nm] != ntotal_plus || om[nm] != ntotal_minus)
        return fp4_fail(c, FP4_E_ARG, "sum(N_plus)/sum(N_minus) differ from Ntotal_plus/Ntotal_minus");
    for (int q = 0; q < nptk * nsr; q++)
        if (id_equi[q] < 1 || id_equi[q] > nptk) return fp4_fail(c, FP4_E_ARG, "ID_equi entry outside [1,nptk]");
    for (int ll = 0; ll < nlist; ll++) {
        if (nequi[ll] < 0 || nequi[ll] > nsr) return fp4_fail(c, FP4_E_ARG, "Nequi entry outside [0,nsymm_rot]");
        for (int kk = 0; kk < nequi[ll]; kk++) {
            const int q = ll * nsr + kk;
            if (typeofsym[q] < 1 || typeofsym[q] > nsr || allequi[q] < 1 || allequi[q] > nptk)
                return fp4_fail(c, FP4_E_ARG, "TypeofSymmetry/ALLEquiList entry out of range");
        }
    }
    std::vector<long long> off4;
    if (l4) {
        off4.assign((size_t)3 * (nm + 1), 0);
        for (int ch = 0; ch < 3; ch++) {
            if (!l4->n[ch]) return fp4_fail(c, FP4_E_ARG, "null 4-phonon counts");
            long long* o = off4.data() + (size_t)ch * (nm + 1);
            for (int m = 0; m < nm; m++) {
                if (l4->n[ch][m] < 0) return fp4_fail(c, FP4_E_ARG, "negative count");
                o[m + 1] = o[m] + l4->n[ch][m];
            }
            if (o[nm] != l4->ntotal[ch])
                return fp4_fail(c, FP4_E_ARG, "sum(N_plusplus/plusminus/minusminus) differs from its Ntotal");
            if (o[nm] && (!l4->i2[ch] || !l4->i3[ch] || !l4->i4[ch] || !l4->g[ch]))
                return fp4_fail(c, FP4_E_ARG, "null 4-phonon process list");
        }
    }
    if ((r = fp4_begin(c))) return r;
    DevBuffer* B = c->b_bte;
    if ((r = B[0].upload(c, nequi, nlist * sizeof(int))) || (r = B[1].upload(c, allequi, (size_t)nlist * nsr * sizeof(int))) ||
        (r = B[2].upload(c, omega, (size_t)nptk * nb * sizeof(double))) ||
        (r = B[3].upload(c, velocity, (size_t)nptk * nb * 3 * sizeof(double))) ||
        (r = B[4].upload(c, tau_zero, (size_t)nlist * nb * sizeof(double))) ||
        (r = B[5].upload(c, f_n, (size_t)nptk * nb * 3 * sizeof(double))) ||
        (r = B[6].upload(c, typeofsym, (size_t)nlist * nsr * sizeof(int))) ||
        (r = B[7].upload(c, id_equi, (size_t)nptk * nsr * sizeof(int))) ||
        (r = B[8].upload(c, symmetrizers, (size_t)nptk * 9 * sizeof(double))))
        return r;
    // process lists: [n_plus|n_minus|off_plus|off_minus] and [i2p|i3p|i2m|i3m] and [gp|gm]
    std::vector<unsigned char> meta((size_t)nm * 2 * sizeof(int) + (size_t)(nm + 1) * 2 * sizeof(long long));
    memcpy(meta.data(), n_plus, nm * sizeof(int));
    memcpy(meta.data() + nm * sizeof(int), n_minus, nm * sizeof(int));
    memcpy(meta.data() + 2 * nm * sizeof(int), op.data(), (nm + 1) * sizeof(long long));
    memcpy(meta.data() + 2 * nm * sizeof(int) + (nm + 1) * sizeof(long long), om.data(), (nm + 1) * sizeof(long long));
    if ((r = B[9].upload(c, meta.data(), meta.size()))) return r;
    const size_t tp = ntotal_plus, tm = ntotal_minus;
    if ((r = B[10].reserve(c, (2 * tp + 2 * tm) * sizeof(int) + 64)) || (r = B[11].reserve(c, (tp + tm) * sizeof(double) + 64)))
        return r;
    int* L = B[10].as<int>();
    double* G = B[11].as<double>();
    auto host = [](const void* x) { return const_cast<void*>(x); };
    const HostCopy in[6] = {{host(i2p), L, tp * sizeof(int)},
                            {host(i3p), L + tp, tp * sizeof(int)},
                            {host(gp), G, tp * sizeof(double)},
                            {host(i2m), L + 2 * tp, tm * sizeof(int)},
                            {host(i3m), L + 2 * tp + tm, tm * sizeof(int)},
                            {host(gm), G + tp, tm * sizeof(double)}};
    if ((r = fp4_copy_lists(c, in, 6, false))) return r;
    BteParams p{};
    p.nb = nb;
    p.nptk = nptk;
    p.nlist = nlist;
    p.nsr = nsr;
    p.nequi = B[0].as<int>();
    p.allequi = B[1].as<int>();
    p.energy = B[2].as<double>();
    p.velocity = B[3].as<double>();
    p.tau_zero = B[4].as<double>();
    p.F = B[5].as<double>();
    p.typeofsym = B[6].as<int>();
    p.id_equi = B[7].as<int>();
    p.symm = B[8].as<double>();
    const unsigned char* mb = static_cast<const unsigned char*>(B[9].ptr);
    p.n_plus = reinterpret_cast<const int*>(mb);
    p.n_minus = p.n_plus + nm;
    p.off_plus = reinterpret_cast<const long long*>(mb + 2 * nm * sizeof(int));
    p.off_minus = p.off_plus + nm + 1;
    p.i2p = L;
    p.i3p = L + tp;
    p.i2m = L + 2 * tp;
    p.i3m = L + 2 * tp + tm;
    p.gp = G;
    p.gm = G + tp;
    p.err = c->b_err.as<int>();
    if (l4) {
        // [n4 (3 x nm) | off4 (3 x (nm+1))] and [i2|i3|i4 per channel] and [gamma per channel]
        const size_t t4 = (size_t)(l4->ntotal[0] + l4->ntotal[1] + l4->ntotal[2]);
        if ((r = c->b_counts.reserve(c, ((size_t)3 * nm + off4.size()) * sizeof(long long))) ||
            (r = c->b_lists.reserve(c, t4 * 3 * sizeof(long long) + 64)) ||
            (r = c->b_gamma.reserve(c, t4 * sizeof(double) + 64)))
            return r;
        long long* dn = c->b_counts.as<long long>();
        long long* doff = dn + 3 * nm;
        long long* L4 = c->b_lists.as<long long>();
        double* G4 = c->b_gamma.as<double>();
        CK(cudaMemcpyAsync(doff, off4.data(), off4.size() * sizeof(long long), cudaMemcpyHostToDevice, c->stream));
        size_t base = 0;
        for (int ch = 0; ch < 3; ch++) {
            const size_t t = (size_t)l4->ntotal[ch];
            CK(cudaMemcpyAsync(dn + (size_t)ch * nm, l4->n[ch], nm * sizeof(long long), cudaMemcpyHostToDevice, c->stream));
            long long* l = L4 + 3 * base;
            if (t) {
                CK(cudaMemcpyAsync(l, l4->i2[ch], t * sizeof(long long), cudaMemcpyHostToDevice, c->stream));
                CK(cudaMemcpyAsync(l + t, l4->i3[ch], t * sizeof(long long), cudaMemcpyHostToDevice, c->stream));
                CK(cudaMemcpyAsync(l + 2 * t, l4->i4[ch], t * sizeof(long long), cudaMemcpyHostToDevice, c->stream));
                CK(cudaMemcpyAsync(G4 + base, l4->g[ch], t * sizeof(double), cudaMemcpyHostToDevice, c->stream));
            }
            p.n4[ch] = dn + (size_t)ch * nm;
            p.off4[ch] = doff + (size_t)ch * (nm + 1);
            p.i2_4[ch] = l;
            p.i3_4[ch] = l + t;
            p.i4_4[ch] = l + 2 * t;
            p.g4[ch] = G4 + base;
            base += t;
        }
    }
    if (jacobi) {
        if ((r = B[12].reserve(c, (size_t)nptk * nb * 3 * sizeof(double)))) return r;
        double* Fout = B[12].as<double>();
        CK(cudaEventRecord(c->evk0, c->stream));
        k_jacobi_step<<<dim3((unsigned)nm, (unsigned)nsr), 256, 0, c->stream>>>(p, Fout);
        CK(cudaGetLastError());
        k_symmetrize<<<256, 256, 0, c->stream>>>(nb, nptk, B[8].as<double>(), Fout);
        CK(cudaGetLastError());
        CK(cudaEventRecord(c->evk1, c->stream));
        c->kernel_timed = true;
        c->launches += 2;
        CK(cudaMemcpyAsync(f_n, Fout, (size_t)nptk * nb * 3 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
        return fp4_end(c);
    }
    std::vector<int> cut;  // blocks [cut[x], cut[x+1]) of irreducible points
    std::vector<int> step0;
    std::vector<long long> term0;
    size_t terms = 0, steps = 0;
    int pts = 0;
    bool blocks = !l4 && plan_blocks(nb, nptk, nlist, nequi, n_plus, n_minus, op[nm] + om[nm], cut, step0, term0, terms, steps, pts);
    // [slot_of | step0] and [term0], [records], [coef], [idx] in one buffer
    auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t o1 = up((size_t)nptk * sizeof(int)), o2 = o1 + up((nlist + 1) * sizeof(int)),
                 o3 = o2 + up(nm * sizeof(long long)), o4 = o3 + up(steps * sizeof(StepInfo)),
                 o5 = o4 + up(terms * sizeof(double)), o6 = o5 + up(terms * sizeof(int));
    if (blocks && B[12].reserve(c, o6) != FP4_OK) {  // no room: k_sweep needs none
        cudaGetLastError();
        c->err.clear();
        blocks = false;
    }
    if (blocks) {
        unsigned char* d = B[12].as<unsigned char>();
        BlockParams q{};
        q.slot_of = reinterpret_cast<int*>(d);
        q.step0 = reinterpret_cast<const int*>(d + o1);
        q.term0 = reinterpret_cast<const long long*>(d + o2);
        q.info = reinterpret_cast<StepInfo*>(d + o3);
        q.coef = reinterpret_cast<double*>(d + o4);
        q.idx = reinterpret_cast<int*>(d + o5);
        CK(cudaMemcpyAsync(d + o1, step0.data(), (nlist + 1) * sizeof(int), cudaMemcpyHostToDevice, c->stream));
        CK(cudaMemcpyAsync(d + o2, term0.data(), nm * sizeof(long long), cudaMemcpyHostToDevice, c->stream));
        const size_t smem = block_smem(nb, pts);
        CK(cudaFuncSetAttribute(k_block_steps, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        CK(cudaEventRecord(c->evk0, c->stream));
        k_block_begin<<<1, 1024, 0, c->stream>>>(p, q, cut[1]);
        CK(cudaGetLastError());
        c->launches++;
        for (size_t x = 0; x + 1 < cut.size(); x++) {
            const int l0 = cut[x], l1 = cut[x + 1], l2 = x + 2 < cut.size() ? cut[x + 2] : l1;
            const int ns = step0[l1] - step0[l0];
            if (ns) {
                k_block_sums<<<ns, kSumThreads, 0, c->stream>>>(p, q, l0, l1);
                CK(cudaGetLastError());
                c->launches++;
            }
            int np = 0;
            for (int ll = l0; ll < l1; ll++) np += nequi[ll];
            k_block_steps<<<1, kStepThreads, smem, c->stream>>>(p, q, l0, l1, l2, np);
            CK(cudaGetLastError());
            c->launches++;
        }
        CK(cudaEventRecord(c->evk1, c->stream));
    } else {
        CK(cudaEventRecord(c->evk0, c->stream));
        k_sweep<<<1, 1024, 0, c->stream>>>(p);
        CK(cudaGetLastError());
        CK(cudaEventRecord(c->evk1, c->stream));
        c->launches++;
    }
    c->kernel_timed = true;
    CK(cudaMemcpyAsync(f_n, B[5].ptr, (size_t)nptk * nb * 3 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    B[5].key = 0;  // device copy now differs from the caller's previous F_n
    return fp4_end(c);
}

extern "C" int fp4_iteration(fp4_ctx* c, const fp4_globals* g, int32_t nlist, const int32_t* nequi,
                             const int32_t* allequi, const int32_t* typeofsym, int32_t nsr, const int32_t* id_equi,
                             const double* symmetrizers, const int32_t* n_plus, const int32_t* n_minus,
                             int32_t ntotal_plus, int32_t ntotal_minus, const int32_t* i2p, const int32_t* i3p,
                             const int32_t* i2m, const int32_t* i3m, const double* omega, const double* velocity,
                             const double* gp, const double* gm, const double* tau_zero, double* f_n) {
    FP4_TRACE();
    return run_sweep(c, g, nlist, nequi, allequi, typeofsym, nsr, id_equi, symmetrizers, n_plus, n_minus, ntotal_plus,
                     ntotal_minus, i2p, i3p, i2m, i3m, omega, velocity, gp, gm, tau_zero, f_n, nullptr);
}

extern "C" int fp4_iteration_jacobi(fp4_ctx* c, const fp4_globals* g, int32_t nlist, const int32_t* nequi,
                                    const int32_t* allequi, const int32_t* typeofsym, int32_t nsr,
                                    const int32_t* id_equi, const double* symmetrizers, const int32_t* n_plus,
                                    const int32_t* n_minus, int32_t ntotal_plus, int32_t ntotal_minus,
                                    const int32_t* i2p, const int32_t* i3p, const int32_t* i2m, const int32_t* i3m,
                                    const double* omega, const double* velocity, const double* gp, const double* gm,
                                    const double* tau_zero, double* f_n) {
    FP4_TRACE();
    return run_sweep(c, g, nlist, nequi, allequi, typeofsym, nsr, id_equi, symmetrizers, n_plus, n_minus, ntotal_plus,
                     ntotal_minus, i2p, i3p, i2m, i3m, omega, velocity, gp, gm, tau_zero, f_n, nullptr, true);
}

extern "C" int fp4_iteration_4ph(fp4_ctx* c, const fp4_globals* g, int32_t nlist, const int32_t* nequi,
                                 const int32_t* allequi, const int32_t* typeofsym, int32_t nsr,
                                 const int32_t* id_equi, const double* symmetrizers, const int32_t* n_plus,
                                 const int32_t* n_minus, int32_t ntotal_plus, int32_t ntotal_minus,
                                 const int64_t* n_pp, const int64_t* n_pm, const int64_t* n_mm, int64_t ntotal_pp,
                                 int64_t ntotal_pm, int64_t ntotal_mm, const int32_t* i2p, const int32_t* i3p,
                                 const int32_t* i2m, const int32_t* i3m, const int64_t* i2pp, const int64_t* i3pp,
                                 const int64_t* i4pp, const int64_t* i2pm, const int64_t* i3pm, const int64_t* i4pm,
                                 const int64_t* i2mm, const int64_t* i3mm, const int64_t* i4mm, const double* omega,
                                 const double* velocity, const double* gp, const double* gm, const double* gpp,
                                 const double* gpm, const double* gmm, const double* tau_zero, double* f_n) {
    FP4_TRACE();
    Lists4 l4{{n_pp, n_pm, n_mm}, {ntotal_pp, ntotal_pm, ntotal_mm}, {i2pp, i2pm, i2mm}, {i3pp, i3pm, i3mm},
              {i4pp, i4pm, i4mm}, {gpp, gpm, gmm}};
    return run_sweep(c, g, nlist, nequi, allequi, typeofsym, nsr, id_equi, symmetrizers, n_plus, n_minus, ntotal_plus,
                     ntotal_minus, i2p, i3p, i2m, i3m, omega, velocity, gp, gm, tau_zero, f_n, &l4);
}

extern "C" int fp4_symmetrize_fn(fp4_ctx* c, const fp4_globals* g, const double* symmetrizers, double* f_n) {
    FP4_TRACE();
    if (!c) return FP4_E_ARG;
    int r;
    if ((r = check_g(c, g))) return r;
    if (!symmetrizers || !f_n) return fp4_fail(c, FP4_E_ARG, "null argument");
    const int nb = g->nbands, nptk = g->ngrid[0] * g->ngrid[1] * g->ngrid[2];
    if ((r = fp4_begin(c))) return r;
    DevBuffer* B = c->b_bte;
    if ((r = B[8].upload(c, symmetrizers, (size_t)nptk * 9 * sizeof(double))) ||
        (r = B[5].upload(c, f_n, (size_t)nptk * nb * 3 * sizeof(double))))
        return r;
    k_symmetrize<<<256, 256, 0, c->stream>>>(nb, nptk, B[8].as<double>(), B[5].as<double>());
    CK(cudaGetLastError());
    c->launches++;
    CK(cudaMemcpyAsync(f_n, B[5].ptr, (size_t)nptk * nb * 3 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    B[5].key = 0;
    return fp4_end(c);
}

extern "C" int fp4_tconduct(fp4_ctx* c, const fp4_globals* g, double V, const double* omega, const double* velocity,
                            const double* f_n, double* kappa, double* kmode) {
    FP4_TRACE();
    if (!c) return FP4_E_ARG;
    int r;
    if ((r = check_g(c, g))) return r;
    if (!omega || !velocity || !f_n || !kappa || !(V > 0.0) || !(g->T > 0.0)) return fp4_fail(c, FP4_E_ARG, "bad argument");
    const int nb = g->nbands, nptk = g->ngrid[0] * g->ngrid[1] * g->ngrid[2];
    if ((r = fp4_begin(c))) return r;
    DevBuffer* B = c->b_bte;
    if ((r = B[2].upload(c, omega, (size_t)nptk * nb * sizeof(double))) ||
        (r = B[3].upload(c, velocity, (size_t)nptk * nb * 3 * sizeof(double))) ||
        (r = B[5].upload(c, f_n, (size_t)nptk * nb * 3 * sizeof(double))) || (r = c->b_out.reserve(c, nb * 9 * sizeof(double))))
        return r;
    double* km = nullptr;
    if (kmode) {
        if ((r = B[10].reserve(c, (size_t)nptk * nb * 9 * sizeof(double)))) return r;
        km = B[10].as<double>();
        CK(cudaMemsetAsync(km, 0, (size_t)nptk * nb * 9 * sizeof(double), c->stream));
        B[10].key = 0;
    }
    const double hbar = 1.05457172647e-22, kb = 1.380648813e-23;
    // 1e21*hbar**2*ThConductivity/(kB*T*T*V*nptk), 1e21 a default-REAL literal
    const double scale = (double)1e21f * (hbar * hbar) / (kb * g->T * g->T * V * nptk);
    k_tconduct<<<nb, 256, 0, c->stream>>>(nb, nptk, g->T, scale, B[2].as<double>(), B[3].as<double>(),
                                          B[5].as<double>(), c->b_out.as<double>(), km);
    CK(cudaGetLastError());
    c->launches++;
    CK(cudaMemcpyAsync(kappa, c->b_out.ptr, nb * 9 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    if (kmode) CK(cudaMemcpyAsync(kmode, km, (size_t)nptk * nb * 9 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    return fp4_end(c);
}

// CumulativeTConduct (omega_mode 0) and CumulativeTConductOmega (1).
static int run_cumulative(fp4_ctx* c, const fp4_globals* g, double V, const double* omega, const double* velocity,
                          const double* f_n, int32_t nticks, double* ticks, double* results, int omega_mode) {
    if (!c) return FP4_E_ARG;
    int r;
    if ((r = check_g(c, g))) return r;
    if (!omega || !velocity || !f_n || !ticks || !results || !(V > 0.0) || !(g->T > 0.0) || nticks < 2)
        return fp4_fail(c, FP4_E_ARG, "bad argument");
    const int nb = g->nbands, nptk = g->ngrid[0] * g->ngrid[1] * g->ngrid[2];
    // the thresholds, computed on the host as the reference computes them
    if (omega_mode == 0) {
        for (int ii = 1; ii <= nticks; ii++)  // 10.**(8.*(ii-1.)/(nticks-1.)-2.) in default REAL
            ticks[ii - 1] = (double)powf(10.0f, 8.0f * ((float)ii - 1.0f) / ((float)nticks - 1.0f) - 2.0f);
    } else {
        double emin = 1.e10, emax = -1.e10;
        for (size_t x = 0; x < (size_t)nptk * nb; x++) {
            emin = std::min(emin, omega[x]);
            emax = std::max(emax, omega[x]);
        }
        emax = emax * 1.1;
        for (int ii = 1; ii <= nticks; ii++) ticks[ii - 1] = emin + (emax - emin) * ii / nticks;
    }
    if ((r = fp4_begin(c))) return r;
    DevBuffer* B = c->b_bte;
    if ((r = B[2].upload(c, omega, (size_t)nptk * nb * sizeof(double))) ||
        (r = B[3].upload(c, velocity, (size_t)nptk * nb * 3 * sizeof(double))) ||
        (r = B[5].upload(c, f_n, (size_t)nptk * nb * 3 * sizeof(double))) ||
        (r = B[9].upload(c, ticks, (size_t)nticks * sizeof(double))) ||
        (r = c->b_out.reserve(c, (size_t)nb * 9 * nticks * sizeof(double))))
        return r;
    const double hbar = 1.05457172647e-22, kb = 1.380648813e-23;
    const double scale = (double)1e21f * (hbar * hbar) / (kb * g->T * g->T * V * nptk);
    k_cumulative<<<dim3(nticks, nb), 128, 0, c->stream>>>(nb, nptk, nticks, omega_mode, g->T, scale,
                                                          B[2].as<double>(), B[3].as<double>(), B[5].as<double>(),
                                                          B[9].as<double>(), c->b_out.as<double>());
    CK(cudaGetLastError());
    c->launches++;
    CK(cudaMemcpyAsync(results, c->b_out.ptr, (size_t)nb * 9 * nticks * sizeof(double), cudaMemcpyDeviceToHost,
                       c->stream));
    B[9].key = 0;
    return fp4_end(c);
}

extern "C" int fp4_cumulative_tconduct(fp4_ctx* c, const fp4_globals* g, double V, const double* omega,
                                       const double* velocity, const double* f_n, int32_t nticks, double* ticks,
                                       double* results) {
    FP4_TRACE();
    return run_cumulative(c, g, V, omega, velocity, f_n, nticks, ticks, results, 0);
}

extern "C" int fp4_cumulative_tconduct_omega(fp4_ctx* c, const fp4_globals* g, double V, const double* omega,
                                             const double* velocity, const double* f_n, int32_t nticks,
                                             double* ticks, double* results) {
    FP4_TRACE();
    return run_cumulative(c, g, V, omega, velocity, f_n, nticks, ticks, results, 1);
}
