// FP64 kernels of the drop-in path.
//
// This translation unit is compiled with -fmad=false: every multiply and add
// is rounded on its own, in the order the reference's C++ evaluates it, and
// double division and square root are IEEE round-to-nearest (by the compiler's
// operators, or by pd_rn.cuh inside its range).  A node's lanes take its bonds
// or contributors side by side; every sum adds its terms one after another in
// family order, which is the order of the reference's loops, so the force,
// gather and state vectors are bit-for-bit those of the reference CPU path
// (pdDataManager.cpp:1767-2134).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <type_traits>
#include <vector>

#include "pd_gather.cuh"
#include "pd_internal.cuh"
#include "pd_rn.cuh"
#include "pd_stage.cuh"

namespace pd {

namespace {

constexpr double kMega = DBL_MAX;  // pdIntgManager.h:26
constexpr double kTiny = DBL_MIN;  // pdIntgManager.h:27

__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }  // std::min

// pdBdryCondition*::GetTimeFactor (pdBdryConditionDispl.cpp:15, ...Veloc.cpp:15,
// ...DisplGrad.cpp:16, ...Tract.cpp:15)
__device__ __forceinline__ double time_factor(const BcDev& b, double t) {
    if (b.type == PD_BC_VELOC) return (t <= b.end_time) ? 1.0 : 0.0;
    if (b.load_type == 1.0) return (t <= b.end_time) ? t / b.end_time : 1.0;
    return 1.0;
}

// pdDataManager::CalcBetaFactor, pdDataManager3.cpp:1801-1829
__device__ __forceinline__ double beta_factor(double dist, double delta, double dx, bool cci_original) {
    double inner = delta - 0.5 * dx;
    double outer = delta + 0.5 * dx;
    if (cci_original) outer = delta;
    if (dist <= inner) return 1.0;
    if (dist > inner && dist <= outer) return (delta + 0.5 * dx - dist) / dx;
    return 0.0;
}

// ------------------------------------------------------------------ force


// p - r = (p^2 - r^2) / (p + r) with p^2 - r^2 = eta.(2 xi + eta): no
// cancellation when the strain is small (PD_PREC_FP64A)
__device__ __forceinline__ double extension(double x0, double x1, double x2, double e0, double e1, double e2,
                                            double r, double p) {
    const double q = e0 * (2.0 * x0 + e0) + e1 * (2.0 * x1 + e1) + e2 * (2.0 * x2 + e2);
    return q / (p + r);
}

// The force of one Gauss point on node i (CalcBondForceCCI, pdDataManager2.cpp:
// 1293-1351) with the compiler's IEEE square roots and divisions: any operands.
struct PointIn {
    double bE, c, ecrit, delta, dxe, pw3;
    bool cci_orig;
};
template <bool CCI, bool ENERGY, bool ACC>
__device__ __noinline__ void point_any(const PointIn& P, double vol, double x0, double x1, double x2, double e0,
                                       double e1, double e2, double* f) {
    const double r = sqrt(x0 * x0 + x1 * x1 + x2 * x2);
    const double y0 = x0 + e0, y1 = x1 + e1, y2 = x2 + e2;
    const double pl = sqrt(y0 * y0 + y1 * y1 + y2 * y2);
    const double beta = beta_factor(r, P.delta, P.dxe, P.cci_orig);
    const double u = ACC ? extension(x0, x1, x2, e0, e1, e2, r, pl) : pl - r;
    const double s = u / r;
    f[0] = f[1] = f[2] = f[3] = 0.0;
    if (u <= 0.0 || (u > 0.0 && s <= P.ecrit)) {
        const double t = CCI ? P.bE * vol * beta * P.c * s : P.bE * beta * P.c * s;
        f[0] = t * y0 / pl;
        f[1] = t * y1 / pl;
        f[2] = t * y2 / pl;
        if (ENERGY) f[3] = P.bE * 0.5 * (0.5 * beta * (P.c / r) * u * u) * P.pw3;
    }
}

// The limits of beta_factor and the reciprocal of its divisor.
struct BetaIn {
    double inner, outer, top, dxe, ydxe;  // ydxe = 1 / dxe rounded to nearest
};
__device__ __forceinline__ BetaIn beta_in(double delta, double dxe, bool cci_orig) {
    BetaIn B;
    B.inner = delta - 0.5 * dxe;
    B.outer = cci_orig ? delta : delta + 0.5 * dxe;
    B.top = delta + 0.5 * dxe;
    B.dxe = dxe;
    B.ydxe = 1.0 / dxe;
    return B;
}

// v <= w for v, w >= 0 (finite): their bit patterns compare as integers, off
// the FP64 pipe
__device__ __forceinline__ bool le_pos(double v, double w) {
    return __double_as_longlong(v) <= __double_as_longlong(w);
}

// point_any's arithmetic in the same order, straight-line: the square roots,
// the two reciprocals and the six quotients of pd_rn.cuh.  ecp: the critical
// stretch, +0 where it is negative or NaN.  False when an operand is outside
// the range those are exact in (the caller then takes point_any).
template <bool CCI, bool ENERGY, bool ACC>
__device__ __forceinline__ bool point_rn(const BetaIn& B, double bE, double c, double ecp, double vol, double pw3,
                                         double x0, double x1, double x2, double r2, double e0, double e1, double e2,
                                         double& f0, double& f1, double& f2, double& el) {
    const double y0 = x0 + e0, y1 = x1 + e1, y2 = x2 + e2;
    const double p2 = y0 * y0 + y1 * y1 + y2 * y2;
    double r, yr, pl, yp;
    rn_sqrt_rcp(r2, r, yr);
    rn_sqrt_rcp(p2, pl, yp);
    const double u = ACC ? extension(x0, x1, x2, e0, e1, e2, r, pl) : pl - r;
    const double s = rn_div(u, r, yr);
    double beta = rn_div(B.top - r, B.dxe, B.ydxe);
    beta = le_pos(r, B.outer) ? beta : 0.0;
    beta = le_pos(r, B.inner) ? 1.0 : beta;
    const double t = CCI ? bE * vol * beta * c * s : bE * beta * c * s;
    const double n0 = t * y0, n1 = t * y1, n2 = t * y2;
    // s <= ecrit as signed integers: true for every negative s
    const bool on = __double_as_longlong(s) <= __double_as_longlong(ecp);
    f0 = on ? (CCI ? rn_div_signed(n0, pl, yp) : rn_div(n0, pl, yp)) : 0.0;
    f1 = on ? (CCI ? rn_div_signed(n1, pl, yp) : rn_div(n1, pl, yp)) : 0.0;
    f2 = on ? (CCI ? rn_div_signed(n2, pl, yp) : rn_div(n2, pl, yp)) : 0.0;
    if (ENERGY) el = on ? bE * 0.5 * (0.5 * beta * rn_div(c, r, yr) * u * u) * pw3 : 0.0;
    const unsigned far = max(max(rn_dividend(n0), rn_dividend(n1)), max(rn_dividend(n2), ACC ? rn_dividend(u) : 0u));
    return rn_range(r2) && rn_range(p2) && far < rn_span;
}

// L lanes per node.  FGI: the Gauss-point summation branch of
// CalcBondBasedMotionRK4 (pdDataManager.cpp:1917-1962) with the per-point
// CalcBondForceCCI (pdDataManager2.cpp:1293-1351).  CCI: the one-point
// branch (pdDataManager.cpp:1818-1866).
//
// Each lane evaluates one bond of its node (all its points, in point order)
// and leaves the velocity increment (F + b) dt / rho, and the points' energy
// terms, in shared memory; three lanes of the group (a fourth for the energy)
// then add the round's L bonds in family order, so every sum has the
// reference's terms in the reference's order, bit for bit.  Lanes past the
// family's end store -0.0, which changes no sum.  UNI: the 2x2x2 rule with
// equal weights, its points in four pairs (their offsets are two per axis, so
// they share squares); else any rule, point by point.  stage 1..4: the stage's
// epilogue follows on the same lanes (stage_axis), which saves a launch and a
// round trip of vbuf per stage; the one-point scheme, whose bonds read their
// far nodes' displacements, then reads ue and leaves the next stage's in
// ue_next.
//
// Bound by the FP64 pipe and the latency of its chains: 154 instructions per
// evaluation, about 71 of them FP64 (pipe 57 % busy), and no faster with more
// warps (five blocks per SM 1.51 ms, six 1.48, against 1.45 with four; four
// points side by side at three blocks 1.50, all eight 1.67-1.91).  200x200x4
// cracked plate, per launch: 3.86 -> 1.45 ms against one thread per node with
// the compiler's square roots and divisions (474 instructions); 20x10x10 bar
// with energies 560 -> 62 us, 10x10x10 CCI cube 568 -> 17 us, where one thread
// (or eight lanes) per node left a serial chain of 250 bonds on a few SMs.
template <bool CCI, bool ENERGY, bool SFAC, bool ACC, bool UNI, int L>
__global__ void __launch_bounds__(128, 4) k_force_f64(Dev d, double dts, int stage, double dt) {
    constexpr int GS = 3 * L + 4;  // shared doubles per group: 4 more than its bonds, so that groups differ in bank
    constexpr int G = 32 / L;
    extern __shared__ double sh64[];
    const int64_t N = d.n;
    const int npt = CCI ? 1 : (UNI ? 8 : d.npt);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ql = lane % L, grp = lane / L;
    const int ES = ENERGY ? L * npt + 2 : 0;  // shared doubles of a group's energy terms
    double* sw = sh64 + warp * (G * (GS + ES)) + grp * GS;
    double* se = sh64 + warp * (G * (GS + ES)) + G * GS + grp * ES;
    const int64_t slot = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / L;
    const bool live = slot < N;
    const int64_t i = live ? d.order[slot] : 0;
    const MatDev Mi = d.mats[d.mat[i]];
    const double rho = Mi.density, yrho = 1.0 / rho;
    const bool rho_ok = rn_range(rho);
    const double b0 = Mi.grav[0] * rho, b1 = Mi.grav[1] * rho, b2 = Mi.grav[2] * rho;
    const double* src = CCI && d.ue ? d.ue : ((d.bc[i] >= 0) ? d.U : d.us);
    const double ui0 = src[i], ui1 = src[N + i], ui2 = src[2 * N + i];
    const double xi0 = d.x[i], xi1 = d.x[N + i], xi2 = d.x[2 * N + i];
    const double bEi = d.bdry[i];
    const double sfi = SFAC ? d.sfac[i] : 0.0;
    // lane ql < 3 sums component ql of the velocity, lane 3 the energy
    double acc = -0.0;
    if (live && ql < 3) acc = d.vbuf[(int64_t)ql * N + i];
    if (ENERGY && live && ql == 3) acc = d.eed[i];
    const int64_t row = d.arow[i];
    const int cnt = live ? (int)(d.arow[i + 1] - row) : 0;
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    BetaIn B = beta_in(d.delta, CCI ? 2.0 * d.dx / 2.0 : d.gc[0].dxe, CCI && !d.cci_mdf);
    double hlo = 0.0, hhi = 0.0, W = 0.0, pw3 = 1.0;
    if (UNI) {
        hlo = d.gc[0].hg[2];
        hhi = d.gc[1].hg[2];
        W = d.gc[0].W;
        pw3 = d.gc[0].pw3;
    }
    for (int base = 0; base < most; base += L) {
        const bool valid = base + ql < cnt;
        double w0 = -0.0, w1 = -0.0, w2 = -0.0;
        if (valid) {
            const int64_t j = d.acol[row + base + ql];
            double ecrit = Mi.ecrit, c = Mi.spring;
            if (d.nmat > 1) {
                const MatDev& Mj = d.mats[d.mat[j]];
                ecrit = dmin(Mi.ecrit, Mj.ecrit);
                c = dmin(Mi.spring, Mj.spring);
            }
            if (SFAC) c = c * (0.5 * (sfi + d.sfac[j]));
            const double bE = 0.5 * (bEi + d.bdry[j]);
            const double xj0 = d.x[j], xj1 = d.x[N + j], xj2 = d.x[2 * N + j];
            const double ecp = ecrit > 0.0 ? ecrit : 0.0;
            const bool c_ok = !ENERGY || rn_quotient_ok(c);
            double F0 = 0.0, F1 = 0.0, F2 = 0.0;
            if (CCI) {
                const double* sj = d.ue ? d.ue : ((d.bc[j] >= 0) ? d.U : d.us);
                const double x0 = xj0 - xi0, x1 = xj1 - xi1, x2 = xj2 - xi2;
                const double e0 = sj[j] - ui0, e1 = sj[N + j] - ui1, e2 = sj[2 * N + j] - ui2;
                double el = 0.0;
                if (!point_rn<true, ENERGY, ACC>(B, bE, c, ecp, d.vol_cci, 1.0, x0, x1, x2, x0 * x0 + x1 * x1 + x2 * x2,
                                                 e0, e1, e2, F0, F1, F2, el) || !c_ok) {
                    double f[4];
                    const PointIn P{bE, c, ecrit, d.delta, B.dxe, 1.0, !d.cci_mdf};
                    point_any<true, ENERGY, ACC>(P, d.vol_cci, x0, x1, x2, e0, e1, e2, f);
                    F0 = f[0];
                    F1 = f[1];
                    F2 = f[2];
                    el = f[3];
                }
                if (ENERGY) se[ql] = el;
            } else if (UNI) {
                const double xa[2] = {(hlo + xj0) - xi0, (hhi + xj0) - xi0};
                const double xb[2] = {(hlo + xj1) - xi1, (hhi + xj1) - xi1};
                const double xc[2] = {(hlo + xj2) - xi2, (hhi + xj2) - xi2};
                bool ok = c_ok;
#pragma unroll 1
                for (int a = 0; a < 4; ++a) {
                    const double x0 = a & 2 ? xa[1] : xa[0], x1 = a & 1 ? xb[1] : xb[0];
                    const double x01 = x0 * x0 + x1 * x1;
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int g = 2 * a + q;
                        const double x2 = xc[q];
                        const double* ugp = d.ug + (int64_t)(3 * g) * N + j;
                        double f0, f1, f2, el;
                        ok &= point_rn<false, ENERGY, ACC>(B, bE, c, ecp, 0.0, pw3, x0, x1, x2, x01 + x2 * x2,
                                                           ugp[0] - ui0, ugp[N] - ui1, ugp[2 * N] - ui2, f0, f1, f2,
                                                           el);
                        F0 += W * f0;
                        F1 += W * f1;
                        F2 += W * f2;
                        if (ENERGY) se[ql * 8 + g] = el;
                    }
                }
                if (!ok) {
                    const PointIn P{bE, c, ecrit, d.delta, B.dxe, pw3, false};
                    F0 = F1 = F2 = 0.0;
                    for (int g = 0; g < 8; ++g) {
                        const double* ugp = d.ug + (int64_t)(3 * g) * N + j;
                        double f[4];
                        point_any<false, ENERGY, ACC>(P, 0.0, (d.gc[g].hg[0] + xj0) - xi0, (d.gc[g].hg[1] + xj1) - xi1,
                                                      (d.gc[g].hg[2] + xj2) - xi2, ugp[0] - ui0, ugp[N] - ui1,
                                                      ugp[2 * N] - ui2, f);
                        F0 += W * f[0];
                        F1 += W * f[1];
                        F2 += W * f[2];
                        if (ENERGY) se[ql * 8 + g] = f[3];
                    }
                }
            } else {
                for (int g = 0; g < npt; ++g) {
                    const GaussConst& Gc = d.gc[g];
                    const double x0 = (Gc.hg[0] + xj0) - xi0, x1 = (Gc.hg[1] + xj1) - xi1, x2 = (Gc.hg[2] + xj2) - xi2;
                    const double* ugp = d.ug + (int64_t)(3 * g) * N + j;
                    const double e0 = ugp[0] - ui0, e1 = ugp[N] - ui1, e2 = ugp[2 * N] - ui2;
                    if (Gc.dxe != B.dxe) B = beta_in(d.delta, Gc.dxe, false);
                    double f[4];
                    f[3] = 0.0;
                    if (!point_rn<false, ENERGY, ACC>(B, bE, c, ecp, 0.0, Gc.pw3, x0, x1, x2,
                                                      x0 * x0 + x1 * x1 + x2 * x2, e0, e1, e2, f[0], f[1], f[2], f[3]) ||
                        !c_ok) {
                        const PointIn P{bE, c, ecrit, d.delta, Gc.dxe, Gc.pw3, false};
                        point_any<false, ENERGY, ACC>(P, 0.0, x0, x1, x2, e0, e1, e2, f);
                    }
                    F0 += Gc.W * f[0];
                    F1 += Gc.W * f[1];
                    F2 += Gc.W * f[2];
                    if (ENERGY) se[ql * npt + g] = f[3];
                }
            }
            const double n0 = (F0 + b0) * dts, n1 = (F1 + b1) * dts, n2 = (F2 + b2) * dts;
            if (rho_ok && max(max(rn_dividend(n0), rn_dividend(n1)), rn_dividend(n2)) < rn_span) {
                w0 = rn_div_signed(n0, rho, yrho);
                w1 = rn_div_signed(n1, rho, yrho);
                w2 = rn_div_signed(n2, rho, yrho);
            } else {
                w0 = n0 / rho;
                w1 = n1 / rho;
                w2 = n2 / rho;
            }
        } else if (ENERGY) {
            for (int g = 0; g < npt; ++g) se[ql * npt + g] = -0.0;
        }
        sw[3 * ql] = w0;
        sw[3 * ql + 1] = w1;
        sw[3 * ql + 2] = w2;
        __syncwarp();
        if (ql < 3) {
#pragma unroll 8
            for (int q = 0; q < L; ++q) acc += sw[3 * q + ql];
        } else if (ENERGY && ql == 3) {
#pragma unroll 8
            for (int q = 0; q < L * npt; ++q) acc += se[q];
        }
        __syncwarp();
    }
    if (ENERGY && live && ql == 3) d.eed[i] = acc;
    if (stage < 0) {
        if (live && ql < 3) d.vbuf[(int64_t)ql * N + i] = acc;
        return;
    }
    double v = acc;
    if (live && ql < 3) {
        double eff;
        v = stage_axis<false>(d, i, ql, stage, dts, dt, *d.tdev, rho, acc, eff);
        if (CCI) d.ue_next[(int64_t)ql * N + i] = eff;
    }
    if (ENERGY && stage == 4) {  // the lanes of a group hold v0, v1, v2 and the energy density
        const int first = lane - ql;
        const double v0 = __shfl_sync(0xffffffffu, v, first), v1 = __shfl_sync(0xffffffffu, v, first + 1),
                     v2 = __shfl_sync(0xffffffffu, v, first + 2), e = __shfl_sync(0xffffffffu, v, first + 3);
        if (live && ql == 0) stage_energy(d, i, rho, v0, v1, v2, e);
    }
}

// ----------------------------------------------------------------- gather

// The Gauss-point displacement of a node with a boundary condition
// (UpdateIntgPointStatusWithBC, pdDataManager.cpp:2604-2703): its flagged
// directions.
__device__ __forceinline__ void gather_bc(const Dev& d, int64_t i, int g, double t, double* ug) {
    const int64_t N = d.n;
    const BcDev& B = d.bcs[d.bc[i]];
    const double fac = time_factor(B, t);
    const GaussConst& G = d.gc[g];
    const double q0 = G.hg[0] + d.x[i], q1 = G.hg[1] + d.x[N + i], q2 = G.hg[2] + d.x[2 * N + i];
    for (int a = 0; a < 3; ++a) {
        if (B.dir[a] != 1) continue;
        if (B.type == PD_BC_DISPL) ug[a * N] = B.val[a] * fac;
        else if (B.type == PD_BC_DISPLGRAD)
            ug[a * N] = (B.val[3 * a] * q0 + B.val[3 * a + 1] * q1 + B.val[3 * a + 2] * q2) * fac;
    }
}

// One thread per (node, Gauss point): CalcIntgPointDisplRK4 (pdDataManager.cpp:
// 2402-2495) with UpdateIntgPointStatusWithBC (:2604-2703).  Nodes with a
// boundary condition keep the displacement of their unflagged directions
// (VELOC and TRACTION nodes keep all three), exactly as the reference's
// Gaussian points do.
__global__ void k_gather_f64(Dev d, const double* __restrict__ us) {
    const int64_t N = d.n;
    const double t = *d.tdev;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (tid >= N * d.npt) return;
    const int64_t i = d.order[tid / d.npt];
    const int g = (int)(tid % d.npt);
    double* ug = d.ug + (int64_t)(3 * g) * N + i;
    if (d.bc[i] >= 0) {
        gather_bc(d, i, g, t, ug);
        return;
    }
    if (d.mls) {
        const int64_t c0 = d.cbptr[i], nc = d.cbptr[i + 1] - c0;
        const double* cf = d.coeff + c0 * d.npt + g;
        const int32_t* cb = d.cbidx + c0;
        double a0 = 0.0, a1 = 0.0, a2 = 0.0;
        int64_t k = 0;
        // loads of four contributors are issued together; the sums still run
        // in contributor order
        for (; k + 4 <= nc; k += 4) {
            int64_t m[4];
            double c[4], v[4][3];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                m[u] = cb[k + u];
                c[u] = cf[(k + u) * d.npt];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                v[u][0] = us[m[u]];
                v[u][1] = us[N + m[u]];
                v[u][2] = us[2 * N + m[u]];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                a0 += v[u][0] * c[u];
                a1 += v[u][1] * c[u];
                a2 += v[u][2] * c[u];
            }
        }
        for (; k < nc; ++k) {
            const int64_t m = cb[k];
            const double c = cf[k * d.npt];
            a0 += us[m] * c;
            a1 += us[N + m] * c;
            a2 += us[2 * N + m] * c;
        }
        ug[0] = a0;
        ug[N] = a1;
        ug[2 * N] = a2;
    } else {
        ug[0] = us[i];
        ug[N] = us[N + i];
        ug[2 * N] = us[2 * N + i];
    }
}

// The same for the 2x2x2 rule (gather_chunks): 20x10x10 bar 21 -> 13 us, plate
// 200x200x4 272 -> 171 us per launch (844 MB: 4.9 TB/s, 0.75 of the copy rate).
constexpr int kGatherStages = 4;
__global__ void __launch_bounds__(128) k_gather_f64_lanes(Dev d, const double* __restrict__ us) {
    extern __shared__ __align__(16) char gather_sm[];
    const int64_t N = d.n;
    const int64_t slot = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3;
    const int g = threadIdx.x & 7;
    const bool live = slot < N;
    const int64_t i = d.order[live ? slot : 0];
    const bool free = live && d.bc[i] < 0;
    const int64_t c0 = d.cbptr[i];
    const int nc = free ? (int)(d.cbptr[i + 1] - c0) : 0;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    gather_chunks<double, kGatherStages>(
        gather_sm + (threadIdx.x >> 5) * gather_warp_bytes<double>(kGatherStages), d.coeff + c0 * 8, d.cbidx + c0, nc,
        [&](int m, double* v) {
            v[0] = us[m];
            v[1] = us[N + m];
            v[2] = us[2 * N + m];
        },
        [&](double c, const double* v) {
            a0 += v[0] * c;
            a1 += v[1] * c;
            a2 += v[2] * c;
        });
    if (!live) return;
    double* ug = d.ug + (int64_t)(3 * g) * N + i;
    if (!free) {
        gather_bc(d, i, g, *d.tdev, ug);
        return;
    }
    ug[0] = a0;
    ug[N] = a1;
    ug[2 * N] = a2;
}

// --------------------------------------------------------------- epilogue

// Per node, after the force kernel of stage `stage` (1..4): the traction load
// (project rule), UpdateNodeStatusWithBC (pdDataManager.cpp:2497-2602),
// k = vbuf*dt_s (:1977-1990) and the RK4 bookkeeping of pdDataManager::RK4
// (:2027-2092): next trial displacement, k3 += k2, and at stage 4 the
// combination, the damping and the new velocity.
// Bound by memory: a thread per component (per node where the energies need
// all three).  640,000 nodes: 27 us with a thread per node and U and vbuf
// always rewritten, 20 us now.
template <int STAGE>
__global__ void k_epilogue(Dev d, double dts, double dt) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= 3 * d.n) return;
    const int a = k >= 2 * d.n ? 2 : (k >= d.n ? 1 : 0);
    const int64_t i = k - a * d.n;
    double eff;
    stage_axis<true>(d, i, a, STAGE, dts, dt, *d.tdev, d.mats[d.mat[i]].density, __ldcg(d.vbuf + k), eff);
}
__global__ void k_epilogue_energy(Dev d, int stage, double dts, double dt) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < d.n) stage_epilogue<true>(d, i, stage, dts, dt, *d.tdev);
}

// Deterministic two-level sum of red[0..N) and red[N..2N) into red[2N], red[2N+1].
__global__ void k_energy_partial(const double* __restrict__ red, int64_t N, double* __restrict__ part) {
    __shared__ double s0[256], s1[256];
    double a = 0.0, c = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
        a += red[i];
        c += red[N + i];
    }
    s0[threadIdx.x] = a;
    s1[threadIdx.x] = c;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            s0[threadIdx.x] += s0[threadIdx.x + w];
            s1[threadIdx.x] += s1[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = s0[0];
        part[2 * blockIdx.x + 1] = s1[0];
    }
}

// The sums of the blocks' partial sums in block order: all loads first, then
// one thread per sum.
__global__ void __launch_bounds__(256) k_energy_final(const double* __restrict__ part, int nb, double* __restrict__ out) {
    __shared__ double sp[2 * 256];
    for (int k = threadIdx.x; k < 2 * nb; k += blockDim.x) sp[k] = part[k];
    __syncthreads();
    if (threadIdx.x >= 2) return;
    double a = 0.0;
#pragma unroll 8
    for (int k = 0; k < nb; ++k) a += sp[2 * k + threadIdx.x];
    out[threadIdx.x] = a;
}

__global__ void k_to_soa(const double* __restrict__ aos, double* __restrict__ soa, int64_t n, int comps) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n * comps) return;
    const int64_t i = t / comps;
    const int c = (int)(t - i * comps);
    soa[c * n + i] = aos[t];
}

// k_to_soa that also records whether any value changed (bit pattern), so a
// caller can tell a round trip of the device state from a new state
__global__ void k_to_soa_changed(const double* __restrict__ aos, double* __restrict__ soa, int64_t n, int comps,
                                 int* __restrict__ changed) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n * comps) return;
    const int64_t i = t / comps;
    const int c = (int)(t - i * comps);
    const double v = aos[t];
    if (__double_as_longlong(soa[c * n + i]) != __double_as_longlong(v)) *changed = 1;
    soa[c * n + i] = v;
}

__global__ void k_to_aos(const double* __restrict__ soa, double* __restrict__ aos, int64_t n, int comps) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n * comps) return;
    const int64_t i = t / comps;
    const int c = (int)(t - i * comps);
    aos[t] = soa[c * n + i];
}

__global__ void k_fill(double* p, double v, int64_t n) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < n) p[t] = v;
}

inline unsigned blocks_for(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

}  // namespace

bool launch_force_f64(const Dev& d, double dts, cudaStream_t s, int stage, double dt) {
    if (d.n == 0) return true;
    if (d.ai) {
        launch_ai_force(d, dts, s);
        return false;
    }
    if (d.cci && !d.ue) stage = -1;
    // The 2x2x2 rule with equal weights takes the unrolled form.  A small
    // problem gives a node a whole warp, so that the SMs fill; a larger one
    // eight lanes, which waste fewer on a family's last round and add its bonds
    // in fewer steps.  Measured, 8 against 32 lanes: 2,000 nodes 80 / 39 us,
    // 8,192 145 / 119, 16,384 234 / 234, 32,768 424 / 458, 160,000 1501 / 1791;
    // with energies 113 / 62 us at 2,000 and 563 / 743 at 32,768; the lighter
    // CCI points 33 / 17 us at 1,000 and 78 / 94 at 19,800.
    constexpr int64_t kWarpPerNodeBelow = 12288;
    const bool uni = !d.cci && d.npt == 8 && d.gc_uniform;
    const int lanes = d.n < std::min(d.f64_lanes_below, kWarpPerNodeBelow) ? 32 : 8;
    const size_t warp_bytes =
        sizeof(double) * (32 / lanes) * (3 * lanes + 4 + (d.energy ? lanes * (d.cci ? 1 : d.npt) + 2 : 0));
    const int warps = std::max(1, std::min(4, (int)(200 * 1024 / warp_bytes)));
    const unsigned nb = blocks_for(lanes * d.n, 32 * warps);
    const size_t sh = warps * warp_bytes;
    const bool sf = d.sfac != nullptr;
    auto go = [&](auto kernel) {
        if (sh > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh);
        kernel<<<nb, 32 * warps, sh, s>>>(d, dts, stage, dt);
    };
    auto lanes_of = [&](auto C, auto E, auto S, auto A, auto Un) {
        constexpr bool c = decltype(C)::value, e = decltype(E)::value, f = decltype(S)::value;
        constexpr bool a = decltype(A)::value, u = decltype(Un)::value;
        if (lanes == 32) go(k_force_f64<c, e, f, a, u, 32>);
        else go(k_force_f64<c, e, f, a, u, 8>);
    };
    auto rule = [&](auto E, auto S, auto A) {
        if (d.cci) lanes_of(std::true_type{}, E, S, A, std::false_type{});
        else if (uni) lanes_of(std::false_type{}, E, S, A, std::true_type{});
        else lanes_of(std::false_type{}, E, S, A, std::false_type{});
    };
    auto form = [&](auto E, auto S) {
        if (d.acc_stretch) rule(E, S, std::true_type{});
        else rule(E, S, std::false_type{});
    };
    if (d.energy) { if (sf) form(std::true_type{}, std::true_type{}); else form(std::true_type{}, std::false_type{}); }
    else { if (sf) form(std::false_type{}, std::true_type{}); else form(std::false_type{}, std::false_type{}); }
    return stage > 0;
}

void launch_gather_f64(const Dev& d, const double* us, cudaStream_t s) {
    if (d.ai) {
        launch_ai_gather(d, us, s);
        return;
    }
    if (d.cci || d.n == 0) return;
    if (d.npt == 8 && d.mls) {
        k_gather_f64_lanes<<<blocks_for(8 * d.n, 128), 128, 4 * gather_warp_bytes<double>(kGatherStages), s>>>(d, us);
        return;
    }
    const int bs = 256;
    k_gather_f64<<<blocks_for(d.n * d.npt, bs), bs, 0, s>>>(d, us);
}

void launch_epilogue(const Dev& d, int stage, double dts, double dt, cudaStream_t s) {
    if (d.n == 0) return;
    const int bs = 256;
    const unsigned nb = blocks_for(3 * d.n, bs);
    if (d.energy) k_epilogue_energy<<<blocks_for(d.n, bs), bs, 0, s>>>(d, stage, dts, dt);
    else if (stage == 0) k_epilogue<0><<<nb, bs, 0, s>>>(d, dts, dt);
    else if (stage == 1) k_epilogue<1><<<nb, bs, 0, s>>>(d, dts, dt);
    else if (stage == 2) k_epilogue<2><<<nb, bs, 0, s>>>(d, dts, dt);
    else if (stage == 3) k_epilogue<3><<<nb, bs, 0, s>>>(d, dts, dt);
    else k_epilogue<4><<<nb, bs, 0, s>>>(d, dts, dt);
}

// t += dt on the device, as pdSolve.cpp:61 advances currentTime
__global__ void k_advance_time(double* t, double dt) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *t = *t + dt;
}

void launch_advance_time(double* t, double dt, cudaStream_t s) { k_advance_time<<<1, 32, 0, s>>>(t, dt); }

__global__ void k_set_time(double* t, double v) { *t = v; }
void launch_set_time(double* t, double v, cudaStream_t s) { k_set_time<<<1, 1, 0, s>>>(t, v); }

// One launch for what were three copies, one or two fills and the time's
// advance: at a few thousand nodes each cost a launch of about 2 us.
__global__ void k_step_begin(Dev d, double dt, int advance, double* ue) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k == 0 && advance) *d.tdev = *d.tdev + dt;
    if (k >= 3 * d.n) return;
    const double U = d.U[k];
    d.vbuf[k] = d.V[k];
    d.u1[k] = U;
    d.us[k] = U;
    if (ue) ue[k] = U;
    if (k >= d.n) return;
    if (d.energy) d.eed[k] = 0.0;
    if (d.ai) d.ai_dmg[k] = 0;
}
void launch_step_begin(const Dev& d, double dt, bool advance, double* ue, cudaStream_t s) {
    k_step_begin<<<std::max(1u, blocks_for(3 * d.n, 256)), 256, 0, s>>>(d, dt, advance, ue);
}

void launch_energy_reduce(const Dev& d, cudaStream_t s) {
    const int nb = 148;
    double* part = d.red + 2 * d.n + 2;
    k_energy_partial<<<nb, 256, 0, s>>>(d.red, d.n, part);
    k_energy_final<<<1, 256, 0, s>>>(part, nb, d.red + 2 * d.n);
}

// ============================================================ MLS setup
//
// InitIntegrationPoint (pdDataManager2.cpp:118-256) on the device: the
// contributor lists and the coefficients of every Gauss point, in the
// reference's operation order (this unit is compiled with -fmad=false).  The
// one difference: the spline weight's d^3 and d^4, which the reference takes
// from glibc's pow, are rounded once here (Dekker's exact product, formed with
// FMA), and glibc's pow is off the correctly rounded value for about 4 in
// 10,000 arguments; through the ill-conditioned moment matrix (global
// coordinates) such a weight moves the coefficients by round-off amplified
// like the reference's own (1e-10..1e-5 of the largest coefficient).

__device__ __forceinline__ double cube_rn(double d) {
    const double p = d * d, ep = fma(d, d, -p);  // d^2 = p + ep exactly
    const double h = p * d, eh = fma(p, d, -h);  // p d = h + eh exactly
    return h + (eh + ep * d);
}

__device__ __forceinline__ double quart_rn(double d) {
    const double p = d * d, ep = fma(d, d, -p);
    const double q = p * p, eq = fma(p, p, -q);  // d^4 = q + eq + 2 p ep + ep^2
    return q + (eq + 2.0 * p * ep);
}

// quadratic basis in global coordinates, pdDataManager2.cpp:1547-1563
__device__ __forceinline__ void mls_basis(double q0, double q1, double q2, double* p) {
    p[0] = 1.0;
    p[1] = q0;
    p[2] = q1;
    p[3] = q2;
    p[4] = q0 * q1;
    p[5] = q0 * q2;
    p[6] = q1 * q2;
    p[7] = q0 * q0;
    p[8] = q1 * q1;
    p[9] = q2 * q2;
}

// quartic spline of |q - node| / rw, pdDataManager2.cpp:1565-1578
// (yrw = 1 / rw rounded to nearest; rw_ok: rw in rn_range)
__device__ __forceinline__ double mls_weight(double n0, double n1, double n2, double q0, double q1, double q2,
                                             double rw, double yrw, bool rw_ok) {
    const double e1 = q0 - n0, e2 = q1 - n1, e3 = q2 - n2;
    const double r2 = e1 * e1 + e2 * e2 + e3 * e3;
    double r, y, d;
    rn_sqrt_rcp(r2, r, y);
    d = rn_div(r, rw, yrw);
    if (!(rn_range(r2) && rw_ok)) {
        r = sqrt(r2);
        d = r / rw;
    }
    if (d > 1.0) return 0.0;
    return (1 - 6.0 * d * d + 8.0 * cube_rn(d) - 3.0 * quart_rn(d));
}

// contributors: the node, then its family members (ascending id) within rw,
// or within 1.5 rw when fewer than 10 qualify (pdDataManager2.cpp:118-171).
// A warp per node, its family read side by side and compacted in order by
// ballots.  cut: the largest squared distance whose root is <= the radius (the
// root is monotone, so the comparison is the reference's without it).
template <bool FILL>
__global__ void __launch_bounds__(256) k_mls_contrib(Dev d, const double* __restrict__ xm, double cut, double cut15,
                                                     int64_t* __restrict__ cnt, const int64_t* __restrict__ cbptr,
                                                     int32_t* __restrict__ cbidx) {
    const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= d.n) return;
    const int64_t N = d.n, row = d.frow[i], end = d.frow[i + 1];
    const double x0 = xm[i], x1 = xm[N + i], x2 = xm[2 * N + i];
    double lim = cut;
    int64_t c = 1;
    if (FILL) {
        const int64_t o = cbptr[i];
        // the count tells which radius was taken: 10 or more within rw, else 1.5 rw
        for (int pass = 0; pass < 2; ++pass) {
            lim = pass == 0 ? cut : cut15;
            c = 1;
            for (int64_t p = row; p < end; p += 32) {
                bool in = false;
                int32_t j = 0;
                if (p + lane < end) {
                    j = d.fcol[p + lane];
                    const double d1 = xm[j] - x0, d2 = xm[N + j] - x1, d3 = xm[2 * N + j] - x2;
                    in = d1 * d1 + d2 * d2 + d3 * d3 <= lim;
                }
                const unsigned m = __ballot_sync(0xffffffffu, in);
                const int64_t at = c + __popc(m & ((1u << lane) - 1u));
                if (in && o + at < cbptr[i + 1]) cbidx[o + at] = j;
                c += __popc(m);
            }
            if (c >= 10) break;
            __syncwarp();  // the wider pass stores over these entries, from other lanes
        }
        if (lane == 0) cbidx[o] = (int32_t)i;
        return;
    }
    for (int pass = 0; pass < 2; ++pass) {
        lim = pass == 0 ? cut : cut15;
        c = 1;
        for (int64_t p = row; p < end; p += 32) {
            bool in = false;
            if (p + lane < end) {
                const int32_t j = d.fcol[p + lane];
                const double d1 = xm[j] - x0, d2 = xm[N + j] - x1, d3 = xm[2 * N + j] - x2;
                in = d1 * d1 + d2 * d2 + d3 * d3 <= lim;
            }
            c += __popc(__ballot_sync(0xffffffffu, in));
        }
        if (c >= 10) break;
    }
    if (lane == 0) cnt[i] = c;
}

// One thread per (node, Gauss point): the 10x10 moment matrix sum_k w_k p_k
// p_k^T, the full-pivot Gauss-Jordan solve of pdMatrix::Gauss
// (pdMatrix.cpp:251-391) for A s = p(x_g), and coeff_k = w_k p_k^T s, laid
// out [node][contributor][point], with its FP32 copy and the partition-of-unity
// defect sum_k c_k - 1.  A singular matrix records its node in *bad.
//
// The sums run over the contributors in registers, each entry in the
// reference's order; (w p_r) p_c and (w p_c) p_r round differently, so all 100
// entries are kept except the first column, which equals the first row bit for
// bit.  Only the solve, whose pivots index the matrix, has it in shared memory
// (entry-major, so that a warp's accesses hit distinct banks).  With the sums
// in shared memory too, two loads or stores per product bounded the kernel:
// 2.88 ms for 40,000 nodes with 2x2x2 points (plate 100x100x4), 1.19 ms now, the
// coordinates loaded one contributor ahead and the pivot searched row by row in
// parallel.  Eight warps per SM: bound by the latency of the FP64 chains.
__global__ void __launch_bounds__(128, 2) k_mls_coeff(Dev d, const double* __restrict__ xm, double rw,
                                                   const double* __restrict__ absc, int n1,
                                                   const int64_t* __restrict__ cbptr,
                                                   const int32_t* __restrict__ cbidx, double* __restrict__ coeff,
                                                   float* __restrict__ coeff32, float* __restrict__ csum,
                                                   unsigned long long* __restrict__ bad) {
    extern __shared__ double smA[];
    const int bs = blockDim.x, tl = threadIdx.x;
    const int npt = n1 * n1 * n1;
    const int64_t t = blockIdx.x * (int64_t)bs + tl;
    if (t >= d.n * npt) return;
    const int64_t N = d.n;
    const int64_t i = t / npt;
    const int g = (int)(t - i * npt);
    const int gi = g / (n1 * n1), gj = (g / n1) % n1, gk = g % n1;
    const double q0 = 0.5 * d.dx * absc[gi] + xm[i];
    const double q1 = 0.5 * d.dx * absc[gj] + xm[N + i];
    const double q2 = 0.5 * d.dx * absc[gk] + xm[2 * N + i];
    const double yrw = 1.0 / rw;
    const bool rw_ok = rn_range(rw);
#define PD_A(r, c) smA[((r) * 10 + (c)) * bs + tl]
    const int64_t b = cbptr[i], nc = cbptr[i + 1] - b;
    {
        double A[10][10];
#pragma unroll
        for (int r = 0; r < 10; ++r)
#pragma unroll
            for (int c = 0; c < 10; ++c) A[r][c] = 0.0;
        // the next contributor's coordinates are loaded behind the products
        int64_t next = cbidx[b];
        double n0 = xm[next], n1v = xm[N + next], n2 = xm[2 * N + next];
#pragma unroll 1
        for (int64_t k = 0; k < nc; ++k) {
            const double m0 = n0, m1 = n1v, m2 = n2;
            next = cbidx[b + (k + 1 < nc ? k + 1 : k)];
            n0 = xm[next], n1v = xm[N + next], n2 = xm[2 * N + next];
            double e[10];
            mls_basis(m0, m1, m2, e);
            const double w = mls_weight(m0, m1, m2, q0, q1, q2, rw, yrw, rw_ok);
#pragma unroll
            for (int r = 0; r < 10; ++r) {
                const double wr = w * e[r];
#pragma unroll
                for (int c = r ? 1 : 0; c < 10; ++c) A[r][c] = A[r][c] + wr * e[c];
            }
        }
#pragma unroll
        for (int r = 0; r < 10; ++r)
#pragma unroll
            for (int c = 0; c < 10; ++c) PD_A(r, c) = c ? A[r][c] : A[0][r];
    }
    double s[10];
    mls_basis(q0, q1, q2, s);
    // The pivot: the largest entry outside the rows and columns taken, the last
    // in row order among equals; every row is searched on its own (ten chains
    // side by side) and the rows are then compared in order.  A step that finds
    // none (NaN) takes column 0 again, which the next step reports, as the
    // reference's counts do.
    unsigned used = 0;
    bool ok = true, twice = false;
    for (int step = 0; step < 10 && ok; ++step) {
        if (twice) {
            ok = false;
            break;
        }
        double big = 0.0;
        int prow = 0, pcol = 0;
        double rbig[10];
        int rcol[10];
#pragma unroll
        for (int r = 0; r < 10; ++r) rbig[r] = -1.0, rcol[r] = 0;
#pragma unroll
        for (int c = 0; c < 10; ++c) {
            if (used >> c & 1) continue;
#pragma unroll
            for (int r = 0; r < 10; ++r) {
                const double v = fabs(PD_A(r, c));
                if (v >= rbig[r]) rbig[r] = v, rcol[r] = c;
            }
        }
#pragma unroll
        for (int r = 0; r < 10; ++r)
            if (!(used >> r & 1) && rbig[r] >= big) big = rbig[r], prow = r, pcol = rcol[r];
        twice = used >> pcol & 1;
        used |= 1u << pcol;
        if (prow != pcol) {
            for (int c = 0; c < 10; ++c) {
                const double tmp = PD_A(prow, c);
                PD_A(prow, c) = PD_A(pcol, c);
                PD_A(pcol, c) = tmp;
            }
            const double tmp = s[prow];
            s[prow] = s[pcol];
            s[pcol] = tmp;
        }
        if (PD_A(pcol, pcol) == 0.0) {
            ok = false;
            break;
        }
        const double inv = 1.0 / PD_A(pcol, pcol);
        PD_A(pcol, pcol) = 1.0;
        double pr[10];
#pragma unroll
        for (int c = 0; c < 10; ++c) PD_A(pcol, c) = pr[c] = PD_A(pcol, c) * inv;
        const double sp = s[pcol] * inv;
        s[pcol] = sp;
#pragma unroll
        for (int r = 0; r < 10; ++r) {
            if (r == pcol) continue;
            const double mm = PD_A(r, pcol);
            PD_A(r, pcol) = 0.0;
#pragma unroll
            for (int c = 0; c < 10; ++c) PD_A(r, c) = PD_A(r, c) - pr[c] * mm;
            s[r] = s[r] + -mm * sp;
        }
    }
#undef PD_A
    if (!ok) {
        atomicMin(bad, (unsigned long long)i);
        for (int64_t k = 0; k < nc; ++k) {
            coeff[(b + k) * npt + g] = 0.0;
            coeff32[(b + k) * npt + g] = 0.0f;
        }
        csum[t] = -1.0f;
        return;
    }
    double unity = 0.0;
#pragma unroll 2
    for (int64_t k = 0; k < nc; ++k) {
        const int64_t m = cbidx[b + k];
        const double m0 = xm[m], m1 = xm[N + m], m2 = xm[2 * N + m];
        double e[10];
        mls_basis(m0, m1, m2, e);
        const double w = mls_weight(m0, m1, m2, q0, q1, q2, rw, yrw, rw_ok);
        double sum = 0.0;
        for (int r = 0; r < 10; ++r) sum += (e[r] * w) * s[r];
        coeff[(b + k) * npt + g] = sum;
        coeff32[(b + k) * npt + g] = (float)sum;
        unity += sum;
    }
    csum[t] = (float)(unity - 1.0);
}

int mls_setup(const Dev& d, const double* xm, double rw, const double* absc, int n1, int64_t* cnt, int64_t* cbptr,
              int32_t** cbidx, double** coeff, float** coeff32, float** csum, int64_t* total, int64_t* bad_node,
              void* (*alloc)(void*, size_t), void* actx, cudaStream_t s) {
    const int64_t N = d.n;
    const int npt = n1 * n1 * n1;
    *bad_node = -1;
    if (N == 0) return PD_OK;
    // the largest squared distance with a root <= radius
    auto cut_of = [](double radius) {
        double v = radius * radius;
        while (std::sqrt(v) <= radius && v < DBL_MAX) v = std::nextafter(v, DBL_MAX);
        while (v > 0.0 && std::sqrt(v) > radius) v = std::nextafter(v, 0.0);
        return v;
    };
    const double cut = cut_of(rw), cut15 = cut_of(rw * 1.5);
    k_mls_contrib<false><<<blocks_for(32 * N, 256), 256, 0, s>>>(d, xm, cut, cut15, cnt, nullptr, nullptr);
    if (exclusive_scan_i64(cnt, cbptr, N, s) != PD_OK) return PD_ERR_CUDA;
    if (cudaMemcpyAsync(total, cbptr + N, sizeof(int64_t), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return PD_ERR_CUDA;
    const int64_t T = *total;
    *cbidx = (int32_t*)alloc(actx, sizeof(int32_t) * (size_t)std::max<int64_t>(T, 1));
    *coeff = (double*)alloc(actx, sizeof(double) * (size_t)std::max<int64_t>(T * npt, 1));
    *coeff32 = (float*)alloc(actx, sizeof(float) * (size_t)std::max<int64_t>(T * npt, 1));
    *csum = (float*)alloc(actx, sizeof(float) * (size_t)(N * npt));
    if (!*cbidx || !*coeff || !*coeff32 || !*csum) return PD_ERR_OOM;
    k_mls_contrib<true><<<blocks_for(32 * N, 256), 256, 0, s>>>(d, xm, cut, cut15, nullptr, cbptr, *cbidx);
    unsigned long long* dbad = reinterpret_cast<unsigned long long*>(cnt);  // the counts are no longer needed
    const unsigned long long none = ~0ull;
    if (cudaMemcpyAsync(dbad, &none, sizeof none, cudaMemcpyHostToDevice, s) != cudaSuccess) return PD_ERR_CUDA;
    const int bs = 128;
    const size_t smem = sizeof(double) * 100 * bs;
    if (cudaFuncSetAttribute(k_mls_coeff, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return PD_ERR_CUDA;
    k_mls_coeff<<<(unsigned)((N * npt + bs - 1) / bs), bs, smem, s>>>(d, xm, rw, absc, n1, cbptr, *cbidx, *coeff,
                                                                      *coeff32, *csum, dbad);
    unsigned long long hb = none;
    if (cudaMemcpyAsync(&hb, dbad, sizeof hb, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return PD_ERR_CUDA;
    if (hb != none) {
        *bad_node = (int64_t)hb;
        return PD_ERR_SINGULAR;
    }
    return cudaGetLastError() == cudaSuccess ? PD_OK : PD_ERR_CUDA;
}

void launch_to_soa(const double* aos, double* soa, int64_t n, int comps, cudaStream_t s) {
    if (n == 0) return;
    k_to_soa<<<blocks_for(n * comps, 256), 256, 0, s>>>(aos, soa, n, comps);
}

void launch_to_soa_changed(const double* aos, double* soa, int64_t n, int comps, int* changed, cudaStream_t s) {
    if (n == 0) return;
    k_to_soa_changed<<<blocks_for(n * comps, 256), 256, 0, s>>>(aos, soa, n, comps, changed);
}

void launch_to_aos(const double* soa, double* aos, int64_t n, int comps, cudaStream_t s) {
    if (n == 0) return;
    k_to_aos<<<blocks_for(n * comps, 256), 256, 0, s>>>(soa, aos, n, comps);
}

void launch_fill(double* p, double v, int64_t n, cudaStream_t s) {
    if (n == 0) return;
    k_fill<<<blocks_for(n, 256), 256, 0, s>>>(p, v, n);
}

// ============================================================ bond search

namespace {

__device__ __forceinline__ double shortest_between(double v, double lo, double hi, double tol) {
    if (v < lo - tol) return fabs(v - lo);
    if (v > hi + tol) return fabs(v - hi);
    return 0.0;
}

__device__ __forceinline__ double longest_between(double v, double lo, double hi, double tol) {
    if (v < lo - tol) return fabs(v - hi);
    if (v > hi + tol) return fabs(v - lo);
    if (v > 0.5 * (hi + lo)) return fabs(v - lo);
    return fabs(v - hi);
}

// pdDataManager::CalcDistanceToFace, pdDataManager3.cpp:1573-1661
__device__ void dist_to_face(int nrm, double xf, const double* pi, const double* pj, double dx, double* dmn,
                             double* dmx) {
    const double tol = 1e-4 * dx;
    const int n1 = nrm == 1, n2 = nrm == 2, n3 = nrm == 3;
    const double xi1 = pi[0], xi2 = pi[1], xi3 = pi[2];
    const double xj1 = pj[0], xj2 = pj[1], xj3 = pj[2];
    if (fabs((xi1 - xj1) * n1 + (xi2 - xj2) * n2 + (xi3 - xj3) * n3) < tol) {
        *dmn = kMega;
        *dmx = kTiny;
        return;
    }
    const double x1lo = xj1 - 0.5 * dx, x1hi = xj1 + 0.5 * dx;
    const double x2lo = xj2 - 0.5 * dx, x2hi = xj2 + 0.5 * dx;
    const double x3lo = xj3 - 0.5 * dx, x3hi = xj3 + 0.5 * dx;
    const double x_i = xi1 * n1 + xi2 * n2 + xi3 * n3;
    const double x_j = xj1 * n1 + xj2 * n2 + xj3 * n3;
    const double fac = (xf - x_i) / (x_j - x_i);
    const double x1int = xi1 + fac * (xj1 - xi1);
    const double x2int = xi2 + fac * (xj2 - xi2);
    const double x3int = xi3 + fac * (xj3 - xi3);
    if (x1int > x1lo - tol && x1int < x1hi + tol && x2int > x2lo - tol && x2int < x2hi + tol && x3int > x3lo - tol &&
        x3int < x3hi + tol) {
        const double f1 = (1 - n1) * xi1 + n1 * xf;
        const double f2 = (1 - n2) * xi2 + n2 * xf;
        const double f3 = (1 - n3) * xi3 + n3 * xf;
        const double s1 = (1 - n1) * shortest_between(f1, x1lo, x1hi, tol);
        const double s2 = (1 - n2) * shortest_between(f2, x2lo, x2hi, tol);
        const double s3 = (1 - n3) * shortest_between(f3, x3lo, x3hi, tol);
        const double l1 = (1 - n1) * longest_between(f1, x1lo, x1hi, tol);
        const double l2 = (1 - n2) * longest_between(f2, x2lo, x2hi, tol);
        const double l3 = (1 - n3) * longest_between(f3, x3lo, x3hi, tol);
        const double ffs = sqrt(s1 * s1 + s2 * s2 + s3 * s3);
        const double ffl = sqrt(l1 * l1 + l2 * l2 + l3 * l3);
        const double itf = sqrt((f1 - xi1) * (f1 - xi1) + (f2 - xi2) * (f2 - xi2) + (f3 - xi3) * (f3 - xi3));
        *dmn = sqrt(ffs * ffs + itf * itf);
        *dmx = sqrt(ffl * ffl + itf * itf);
        return;
    }
    *dmn = kMega;
    *dmx = kTiny;
}

// InitBond's membership test for the pair (a < b): the rough distance
// reject of pdDataManager2.cpp:34-38, then CalcDistanceToCube's minimum
// (pdDataManager3.cpp:637-685) against horizon + tolerance.
__device__ bool pair_bonded(const double* pa, const double* pb, double dx, double delta, double tol, double* dist) {
    const double d1 = pb[0] - pa[0], d2 = pb[1] - pa[1], d3 = pb[2] - pa[2];
    *dist = sqrt(d1 * d1 + d2 * d2 + d3 * d3);
    if (delta < *dist - 1.5 * dx) return false;
    double mn = kMega, a, b;
    for (int ax = 0; ax < 3; ++ax) {
        dist_to_face(ax + 1, pb[ax] - 0.5 * dx, pa, pb, dx, &a, &b);
        mn = dmin(mn, a);
        dist_to_face(ax + 1, pb[ax] + 0.5 * dx, pa, pb, dx, &a, &b);
        mn = dmin(mn, a);
    }
    return mn < delta + tol;
}

// The same out of line with its operands by value, so that the search's common
// path keeps neither its registers nor its arrays.
__device__ __noinline__ bool pair_bonded_any(double a0, double a1, double a2, double b0, double b1, double b2, double dx,
                                             double delta, double tol) {
    const double pa[3] = {a0, a1, a2}, pb[3] = {b0, b1, b2};
    double dist;
    return pair_bonded(pa, pb, dx, delta, tol, &dist);
}

// Project rule for pdSlit (pdSlit.h:6-10 fixes only the keyword): the segment
// from the lower-id to the higher-id node crosses the rectangle.
__device__ __forceinline__ int slit_plane(const double* s, double* c) {
    int nrm = 0;
    double ext = s[1] - s[0];
    for (int k = 1; k < 3; ++k)
        if (s[2 * k + 1] - s[2 * k] < ext) {
            ext = s[2 * k + 1] - s[2 * k];
            nrm = k;
        }
    *c = 0.5 * (s[2 * nrm] + s[2 * nrm + 1]);
    return nrm;
}
__device__ bool slit_crosses(const double* s, const double* a, const double* b) {
    double c;
    const int nrm = slit_plane(s, &c);
    const double da = a[nrm] - c, db = b[nrm] - c;
    if (!((da < 0.0 && db > 0.0) || (da > 0.0 && db < 0.0))) return false;
    const double t = (c - a[nrm]) / (b[nrm] - a[nrm]);
    for (int k = 0; k < 3; ++k) {
        if (k == nrm) continue;
        const double p = a[k] + t * (b[k] - a[k]);
        if (p < s[2 * k] || p > s[2 * k + 1]) return false;
    }
    return true;
}

// pair_bonded decided from the separation alone wherever that cannot differ
// from it.  The line from a node through the centre of the other's cell enters
// the cell by the face across the longest component of the separation, and the
// nearest point of that face is |d_k| - dx/2 away along every component longer
// than dx/2.  pair_bonded reaches the same distance through intersections that
// allow 1e-4 dx of tolerance; a pair whose distance lies more than a hundred
// times that from the limit, with the node well outside the cell and the rough
// reject not in doubt, is decided here, and the rest (none on the decks'
// lattices) by pair_bonded itself.
struct PairLimits {
    double far2, near2;  // squared: beyond far2 the rough reject holds, within near2 it does not
    double lo2, hi2;     // squared distance to the cell: member below lo2, none above hi2
    double half, out;    // dx / 2, and the least longest component of a pair decided here
};
__host__ inline PairLimits pair_limits(double dx, double delta, double tol, double reach) {
    PairLimits P;
    const double rough = delta + 1.5 * dx, lim = delta + tol, margin = 0.01 * dx;
    // coordinates so large that their rounding nears the margin: nothing is decided here
    const bool fine = reach * 1e-14 < 1e-4 * dx;
    P.far2 = fine ? rough * rough * (1.0 + 1e-9) : HUGE_VAL;
    P.near2 = rough * rough * (1.0 - 1e-9);
    P.lo2 = lim > margin ? (lim - margin) * (lim - margin) : 0.0;
    P.hi2 = (lim + margin) * (lim + margin);
    P.half = 0.5 * dx;
    P.out = fine ? 0.51 * dx : HUGE_VAL;
    return P;
}
// d: separation, d2 = |d|^2 (d1^2 + d2^2 + d3^2 as pair_bonded sums it)
__device__ __forceinline__ int pair_quick(const PairLimits& P, double d1, double d2, double d3, double dd) {
    if (dd > P.far2) return 0;
    const double a1 = fabs(d1), a2 = fabs(d2), a3 = fabs(d3);
    const double g1 = fmax(a1 - P.half, 0.0), g2 = fmax(a2 - P.half, 0.0), g3 = fmax(a3 - P.half, 0.0);
    const double m2 = g1 * g1 + g2 * g2 + g3 * g3;
    if (dd < P.near2 && fmax(fmax(a1, a2), a3) > P.out) {
        if (m2 < P.lo2) return 1;
        if (m2 > P.hi2) return 0;
    }
    return -1;  // pair_bonded decides
}

struct SearchArgs {
    const double* x;  // [3][N]
    int64_t n;
    double dx, delta, tol;
    SearchGrid g;
    PairLimits lim;
    const int64_t* cstart;     // [ncell+1] by cell, x fastest
    const int32_t* sorted;     // nodes ordered by cell
    const double* xs;          // [3][N] their coordinates in that order
    int nslit;
    const double* slits;
};

__device__ __forceinline__ void load_x(const SearchArgs& A, int64_t i, double* p) {
    p[0] = A.x[i];
    p[1] = A.x[A.n + i];
    p[2] = A.x[2 * A.n + i];
}

__device__ __forceinline__ int64_t cell_coord(const SearchArgs& A, double v, int a) {
    int64_t c = (int64_t)floor((v - A.g.lo[a]) / A.g.h);
    if (c < 0) c = 0;
    if (c >= A.g.nc[a]) c = A.g.nc[a] - 1;
    return c;
}

__global__ void k_cell_count(SearchArgs A, int32_t* node_cell, int64_t* cnt) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    double p[3];
    load_x(A, i, p);
    const int64_t cx = cell_coord(A, p[0], 0), cy = cell_coord(A, p[1], 1), cz = cell_coord(A, p[2], 2);
    const int32_t r = (int32_t)((cz * A.g.nc[1] + cy) * A.g.nc[0] + cx);
    node_cell[i] = r;
    atomicAdd((unsigned long long*)&cnt[r], 1ull);
}

__global__ void k_cell_scatter(SearchArgs A, const int32_t* node_cell, const int64_t* cstart, int64_t* fillc,
                               int32_t* sorted, double* xs) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    const int32_t r = node_cell[i];
    const int64_t at = cstart[r] + (int64_t)atomicAdd((unsigned long long*)&fillc[r], 1ull);
    sorted[at] = (int32_t)i;
    for (int a = 0; a < 3; ++a) xs[a * A.n + at] = A.x[a * A.n + i];
}

// Sorts the n <= 32 R keys of buf in the lanes' registers (bitonic; element
// 32 r + lane in v[r]); places past n come last.
template <int R>
__device__ __forceinline__ void warp_sort(const uint32_t* buf, int n, int lane, uint32_t (&v)[R]) {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = 32 * r + lane < n ? buf[32 * r + lane] : 0xffffffffu;
#pragma unroll
    for (int k = 2; k <= 32 * R; k *= 2) {
#pragma unroll
        for (int j = k / 2; j > 0; j /= 2) {
            if (j >= 32) {
                const int q = j / 32;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (r & q) continue;
                    const bool up = ((32 * r) & k) == 0;
                    const uint32_t lo = min(v[r], v[r | q]), hi = max(v[r], v[r | q]);
                    v[r] = up ? lo : hi;
                    v[r | q] = up ? hi : lo;
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const uint32_t o = __shfl_xor_sync(0xffffffffu, v[r], j);
                    const bool up = ((32 * r + lane) & k) == 0, low = (lane & j) == 0;
                    v[r] = (up == low) ? min(v[r], o) : max(v[r], o);
                }
            }
        }
    }
}

// The sorted keys (2 id + broken) of one node as its rows of both CSRs.
template <int R>
__device__ __forceinline__ void write_rows(const uint32_t* buf, int n, int lane, int64_t fo, int64_t ao, int32_t* fcol,
                                           uint8_t* fbroken, int32_t* acol) {
    uint32_t v[R];
    warp_sort<R>(buf, n, lane, v);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int e = 32 * r + lane;
        const bool in = e < n, whole = in && !(v[r] & 1u);
        const unsigned m = __ballot_sync(0xffffffffu, whole);
        if (in) {
            fcol[fo + e] = (int32_t)(v[r] >> 1);
            fbroken[fo + e] = (uint8_t)(v[r] & 1u);
        }
        if (whole) acol[ao + __popc(m & ((1u << lane) - 1u))] = (int32_t)(v[r] >> 1);
        ao += __popc(m);
    }
}

// What pair_quick leaves open for the pair of i and j, out of line: bit 0 the
// membership (known where quick > 0), bit 1 whether a slit breaks the bond.
__device__ __noinline__ int pair_rest(const SearchArgs& A, int64_t i, int64_t j, int quick) {
    double pa[3], pb[3], dist;
    load_x(A, i < j ? i : j, pa);
    load_x(A, i < j ? j : i, pb);
    if (quick < 0 && !pair_bonded(pa, pb, A.dx, A.delta, A.tol, &dist)) return 0;
    for (int k = 0; k < A.nslit; ++k)
        if (slit_crosses(A.slits + 6 * k, pa, pb)) return 3;
    return 1;
}

// One warp per node (taken in cell order so that neighbouring warps scan
// overlapping cells); the three cells of a row along x are one run of the
// sorted nodes.  PASS 0 counts family and unbroken entries and the minimum
// bond length; PASS 1 collects the family into shared memory as keys 2 id +
// broken, orders it by id and writes both CSRs.
//
// Bound by instruction issue.  Deciding a pair from its separation (pair_quick)
// instead of six face intersections with their roots and divisions, and
// sorting in registers instead of ranking every entry against all others, took
// the two passes over 40,000 nodes (100x100x4 with a slit) from 0.59 and 0.78 ms
// to 0.17 and 0.21 ms; over 160,000 nodes 0.67 and 0.82 ms
// (issue 76 % active, 170 instructions per 32 candidates).
template <int PASS>
__global__ void __launch_bounds__(128, 6) k_search(const __grid_constant__ SearchArgs A, int64_t* cnt_full, int64_t* cnt_act,
                                                unsigned long long* min_bits, unsigned long long* max_cnt,
                                                const int64_t* frow, int32_t* fcol, uint8_t* fbroken,
                                                const int64_t* arow, int32_t* acol, int cap) {
    extern __shared__ uint32_t sbuf[];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (w >= A.n) return;
    const int64_t N = A.n;
    uint32_t* buf = sbuf + (size_t)wib * cap;
    const int64_t i = A.sorted[w];
    const double pi0 = A.xs[w], pi1 = A.xs[N + w], pi2 = A.xs[2 * N + w];
    const int64_t cx = cell_coord(A, pi0, 0), cy = cell_coord(A, pi1, 1), cz = cell_coord(A, pi2, 2);
    const int64_t x0 = cx > 0 ? cx - 1 : 0, x1 = cx + 1 < A.g.nc[0] ? cx + 1 : cx;
    int nfull = 0, nact = 0;
    double mb2 = HUGE_VAL;  // least squared bond length
    for (int64_t qz = cz > 0 ? cz - 1 : 0; qz <= cz + 1 && qz < A.g.nc[2]; ++qz) {
        for (int64_t qy = cy > 0 ? cy - 1 : 0; qy <= cy + 1 && qy < A.g.nc[1]; ++qy) {
            const int64_t rowc = (qz * A.g.nc[1] + qy) * A.g.nc[0];
            const int64_t s0 = A.cstart[rowc + x0], s1 = A.cstart[rowc + x1 + 1];
            for (int64_t s = s0; s < s1; s += 32) {
                bool hit = false, br = false;
                int32_t j = -1;
                if (s + lane < s1 && s + lane != w) {
                    const double d1 = A.xs[s + lane] - pi0, d2 = A.xs[N + s + lane] - pi1,
                                 d3 = A.xs[2 * N + s + lane] - pi2;
                    const double dd = d1 * d1 + d2 * d2 + d3 * d3;
                    const int q = pair_quick(A.lim, d1, d2, d3, dd);
                    if (q != 0) {
                        j = A.sorted[s + lane];
                        bool open = q < 0;
                        for (int k = 0; k < A.nslit && !open; ++k) {  // only ends on both sides can cross
                            double c;
                            const int nrm = slit_plane(A.slits + 6 * k, &c);
                            const double da = (nrm == 0 ? pi0 : (nrm == 1 ? pi1 : pi2)) - c;
                            const double db = A.xs[nrm * N + s + lane] - c;
                            open = (da < 0.0 && db > 0.0) || (da > 0.0 && db < 0.0);
                        }
                        const int rest = open ? pair_rest(A, i, j, q) : 1;
                        hit = rest & 1;
                        br = rest & 2;
                        if (hit) mb2 = fmin(mb2, dd);
                    }
                }
                const unsigned hm = __ballot_sync(0xffffffffu, hit);
                if (PASS == 1 && hit) {
                    const int slot = nfull + __popc(hm & ((1u << lane) - 1u));
                    if (slot < cap) buf[slot] = (uint32_t)j << 1 | (br ? 1u : 0u);
                }
                nfull += __popc(hm);
                if (PASS == 0) nact += __popc(__ballot_sync(0xffffffffu, hit && !br));
            }
        }
    }
    if (PASS == 0) {
        for (int o = 16; o > 0; o >>= 1) mb2 = fmin(mb2, __shfl_xor_sync(0xffffffffu, mb2, o));
        if (lane == 0) {
            cnt_full[i] = nfull;
            cnt_act[i] = nact;
            // the root is monotone: the least length is the root of the least square
            const double mb = dmin(A.delta, sqrt(mb2));
            atomicMin(min_bits, (unsigned long long)__double_as_longlong(mb));
            atomicMax(max_cnt, (unsigned long long)nfull);
        }
        return;
    }
    __syncwarp();
    const int nf = nfull < cap ? nfull : cap;
    const int64_t fo = frow[i], ao = arow[i];
    if (nf <= 128) {
        write_rows<4>(buf, nf, lane, fo, ao, fcol, fbroken, acol);
    } else if (nf <= 256) {
        write_rows<8>(buf, nf, lane, fo, ao, fcol, fbroken, acol);
    } else {  // families beyond 256: every entry's rank among the others
        for (int e = lane; e < nf; e += 32) {
            const uint32_t v = buf[e];
            int rk = 0, ra = 0;
            for (int k = 0; k < nf; ++k) {
                if (buf[k] < v) {
                    ++rk;
                    ra += buf[k] & 1u ? 0 : 1;
                }
            }
            fcol[fo + rk] = (int32_t)(v >> 1);
            fbroken[fo + rk] = (uint8_t)(v & 1u);
            if (!(v & 1u)) acol[ao + ra] = (int32_t)(v >> 1);
        }
    }
}

}  // namespace

int bond_search(const Dev& d, const SearchGrid& g, int64_t ncell, double reach, int nslit, const double* slits_dev,
                int64_t** frow_o, int32_t** fcol_o, uint8_t** fbroken_o, int64_t** arow_o, int32_t** acol_o,
                int64_t* nh, int64_t* nb, double* min_bond, cudaStream_t s) {
    const int64_t N = d.n;
    SearchArgs A;
    A.x = d.x;
    A.n = N;
    A.dx = d.dx;
    A.delta = d.delta;
    A.tol = 1.0e-4 * d.dx;
    A.g = g;
    A.lim = pair_limits(A.dx, A.delta, A.tol, reach);
    A.nslit = nslit;
    A.slits = slits_dev;
    // one allocation for the call's working memory
    char* work = nullptr;
    int64_t *frow = nullptr, *arow = nullptr;
    int32_t *fcol = nullptr, *acol = nullptr;
    uint8_t* fbr = nullptr;
    int rc = PD_OK;
    auto release = [&](int code) {
        cudaFree(work); cudaFree(frow); cudaFree(arow); cudaFree(fcol); cudaFree(acol); cudaFree(fbr);
        return code;
    };
#define PD_S_TRY(expr)                                                        \
    do {                                                                      \
        cudaError_t _e = (expr);                                              \
        if (_e != cudaSuccess) {                                              \
            rc = fail_cuda(_e, #expr, __FILE__, __LINE__);                    \
            return release(rc);                                               \
        }                                                                     \
    } while (0)
    const int64_t Nw = (N + 2) / 2 * 2;  // keeps the 8-byte arrays aligned
    const int64_t nscan = scan_words(std::max(N, ncell));
    const size_t words = 2 + 3 * (size_t)(ncell + 1) + 2 * (size_t)(N + 1) + 3 * (size_t)N + (size_t)nscan;
    PD_S_TRY(cudaMalloc(&work, sizeof(int64_t) * words + sizeof(int32_t) * 2 * (size_t)Nw));
    unsigned long long* scal = reinterpret_cast<unsigned long long*>(work);
    int64_t* ccnt = reinterpret_cast<int64_t*>(scal + 2);
    int64_t* fillc = ccnt + (ncell + 1);
    int64_t* cstart = fillc + (ncell + 1);
    int64_t *cf = cstart + (ncell + 1), *ca = cf + (N + 1);
    double* xs = reinterpret_cast<double*>(ca + (N + 1));
    int64_t* scan = reinterpret_cast<int64_t*>(xs + 3 * N);
    int32_t *node_cell = reinterpret_cast<int32_t*>(scan + nscan), *sorted = node_cell + Nw;
    PD_S_TRY(cudaMalloc(&frow, sizeof(int64_t) * (N + 1)));
    PD_S_TRY(cudaMalloc(&arow, sizeof(int64_t) * (N + 1)));
    PD_S_TRY(cudaMemsetAsync(ccnt, 0, sizeof(int64_t) * 2 * (ncell + 1), s));
    unsigned long long init[2] = {(unsigned long long)__builtin_bit_cast(unsigned long long, d.delta), 0ull};
    PD_S_TRY(cudaMemcpyAsync(scal, init, sizeof(init), cudaMemcpyHostToDevice, s));
    const int bs = 256;
    if (N > 0) {
        k_cell_count<<<blocks_for(N, bs), bs, 0, s>>>(A, node_cell, ccnt);
        PD_S_TRY(cudaGetLastError());
    }
    if (exclusive_scan_i64(ccnt, cstart, ncell, s, scan) != PD_OK) return release(fail(PD_ERR_CUDA, "scan failed"));
    if (N > 0) {
        k_cell_scatter<<<blocks_for(N, bs), bs, 0, s>>>(A, node_cell, cstart, fillc, sorted, xs);
        PD_S_TRY(cudaGetLastError());
    }
    A.cstart = cstart;
    A.sorted = sorted;
    A.xs = xs;
    const int wpb = 4;  // warps per block
    if (N > 0) {
        k_search<0><<<blocks_for(N * 32, 32 * wpb), 32 * wpb, 0, s>>>(A, cf, ca, scal, scal + 1, nullptr, nullptr,
                                                                      nullptr, nullptr, nullptr, 0);
        PD_S_TRY(cudaGetLastError());
    }
    if (exclusive_scan_i64(cf, frow, N, s, scan) != PD_OK || exclusive_scan_i64(ca, arow, N, s, scan) != PD_OK)
        return release(fail(PD_ERR_CUDA, "scan failed"));
    unsigned long long hs[2];
    int64_t tot[2] = {0, 0};
    PD_S_TRY(cudaMemcpyAsync(hs, scal, sizeof(hs), cudaMemcpyDeviceToHost, s));
    PD_S_TRY(cudaMemcpyAsync(&tot[0], frow + N, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    PD_S_TRY(cudaMemcpyAsync(&tot[1], arow + N, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    PD_S_TRY(cudaStreamSynchronize(s));
    PD_S_TRY(cudaMalloc(&fcol, sizeof(int32_t) * (tot[0] + 1)));
    PD_S_TRY(cudaMalloc(&fbr, sizeof(uint8_t) * (tot[0] + 1)));
    PD_S_TRY(cudaMalloc(&acol, sizeof(int32_t) * (tot[1] + 1)));
    const int cap = (int)hs[1] + 1;
    const size_t sh = (size_t)wpb * cap * sizeof(uint32_t);
    // Largest family taken: 10,239 members.  The keys themselves (four bytes)
    // would allow a quarter more; what is refused does not follow their size.
    if ((size_t)wpb * cap * 5 > 200 * 1024)
        return release(fail(PD_ERR_CAPACITY, "family larger than the search kernel's shared buffer"));
    if (sh > 48 * 1024)
        PD_S_TRY(cudaFuncSetAttribute(k_search<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh));
    if (N > 0) {
        k_search<1><<<blocks_for(N * 32, 32 * wpb), 32 * wpb, sh, s>>>(A, nullptr, nullptr, nullptr, nullptr, frow,
                                                                       fcol, fbr, arow, acol, cap);
        PD_S_TRY(cudaGetLastError());
    }
    PD_S_TRY(cudaStreamSynchronize(s));
#undef PD_S_TRY
    cudaFree(work);
    *frow_o = frow;
    *fcol_o = fcol;
    *fbroken_o = fbr;
    *arow_o = arow;
    *acol_o = acol;
    *nh = tot[0];
    *nb = tot[0] - tot[1];
    *min_bond = __builtin_bit_cast(double, hs[0]);
    return PD_OK;
}

// ======================================= bond search without allocation

// pd_bond_search_noalloc works entirely in this fixed device array, carved
// into the regions below.  Every GPU that loads the library holds it until
// the process exits; all calls share it.
namespace na {
constexpr int64_t kNodes = PD_NOALLOC_MAX_NODES;
constexpr int64_t kCells = PD_NOALLOC_MAX_CELLS;
constexpr int kSlits = PD_NOALLOC_MAX_SLITS;
constexpr size_t kOffSorted = sizeof(int32_t) * kNodes;                 // node_cell [kNodes] at 0
constexpr size_t kOffCnt = kOffSorted + sizeof(int32_t) * kNodes;       // sorted [kNodes]
constexpr size_t kOffCellCnt = kOffCnt + sizeof(int64_t) * kNodes;      // cnt [kNodes]
constexpr size_t kOffCstart = kOffCellCnt + sizeof(int64_t) * (kCells + 1);
constexpr size_t kOffFill = kOffCstart + sizeof(int64_t) * (kCells + 1);
constexpr size_t kOffSlits = kOffFill + sizeof(int64_t) * (kCells + 1);
constexpr size_t kOffScal = kOffSlits + sizeof(double) * 6 * kSlits;   // bbox[6], min bits, max count
constexpr size_t kBytes = kOffScal + 16 * sizeof(double);
static_assert(kBytes == PD_NOALLOC_SCRATCH_BYTES, "scratch size stated in pdmtel_b200.h");
}  // namespace na

static __device__ __align__(256) unsigned char g_noalloc_scratch[na::kBytes];

namespace {

struct NaArgs {
    const double* x;  // [n][3], caller's device buffer
    int64_t n;
    double dx, delta, tol;
    SearchGrid g;
    unsigned char* s;  // device address of g_noalloc_scratch
    int nslit;
    PairLimits lim;
};

__device__ __forceinline__ int32_t* na_node_cell(unsigned char* s) { return (int32_t*)s; }
__device__ __forceinline__ int32_t* na_sorted(unsigned char* s) { return (int32_t*)(s + na::kOffSorted); }
__device__ __forceinline__ int64_t* na_cnt(unsigned char* s) { return (int64_t*)(s + na::kOffCnt); }
__device__ __forceinline__ int64_t* na_cell_cnt(unsigned char* s) { return (int64_t*)(s + na::kOffCellCnt); }
__device__ __forceinline__ int64_t* na_cstart(unsigned char* s) { return (int64_t*)(s + na::kOffCstart); }
__device__ __forceinline__ int64_t* na_fill(unsigned char* s) { return (int64_t*)(s + na::kOffFill); }
__device__ __forceinline__ double* na_slits(unsigned char* s) { return (double*)(s + na::kOffSlits); }
__device__ __forceinline__ double* na_scal(unsigned char* s) { return (double*)(s + na::kOffScal); }

// bounding box of the nodes into scal[0..5]; one block
__global__ void k_na_bbox(const double* __restrict__ x, int64_t n, unsigned char* s) {
    __shared__ double red[6][32];
    __shared__ int nonfinite;
    if (threadIdx.x == 0) nonfinite = 0;
    __syncthreads();
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    bool bad = false;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
        for (int a = 0; a < 3; ++a) {
            bad = bad || !isfinite(x[3 * i + a]);
            lo[a] = dmin(lo[a], x[3 * i + a]);
            hi[a] = -dmin(-hi[a], -x[3 * i + a]);
        }
    if (bad) nonfinite = 1;
    for (int o = 16; o > 0; o >>= 1)
        for (int a = 0; a < 3; ++a) {
            lo[a] = dmin(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = -dmin(-hi[a], -__shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int a = 0; a < 3; ++a) {
            red[a][w] = lo[a];
            red[3 + a][w] = hi[a];
        }
    __syncthreads();
    if (threadIdx.x == 0) {
        double* sc = na_scal(s);
        for (int a = 0; a < 3; ++a) {
            double l = red[a][0], h = red[3 + a][0];
            for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
                l = dmin(l, red[a][k]);
                h = -dmin(-h, -red[3 + a][k]);
            }
            sc[a] = nonfinite ? __longlong_as_double(0x7ff8000000000000LL) : l;  // a non-finite coordinate is reported as a NaN box
            sc[3 + a] = h;
        }
        ((unsigned long long*)sc)[6] = (unsigned long long)__double_as_longlong(0.0);
        ((unsigned long long*)sc)[7] = 0ull;
    }
}

__device__ __forceinline__ int64_t na_cell_of(const NaArgs& A, const double* p, int64_t* c) {
    for (int a = 0; a < 3; ++a) {
        int64_t v = (int64_t)floor((p[a] - A.g.lo[a]) / A.g.h);
        c[a] = v < 0 ? 0 : (v >= A.g.nc[a] ? A.g.nc[a] - 1 : v);
    }
    return (c[2] * A.g.nc[1] + c[1]) * A.g.nc[0] + c[0];
}

__global__ void k_na_cell_count(NaArgs A) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    int64_t c[3];
    const int64_t cell = na_cell_of(A, A.x + 3 * i, c);
    na_node_cell(A.s)[i] = (int32_t)cell;
    atomicAdd((unsigned long long*)&na_cell_cnt(A.s)[cell], 1ull);
}

// exclusive scan of in[0..n) into out[0..n], out[n] = total; one block of
// 1024 threads, each thread owning a contiguous run
__global__ void k_na_scan(const int64_t* __restrict__ in, int64_t* __restrict__ out, int64_t n) {
    __shared__ int64_t part[1024];
    const int64_t per = (n + 1023) / 1024;
    const int64_t b = threadIdx.x * per, e = b + per < n ? b + per : n;
    int64_t sum = 0;
    for (int64_t k = b; k < e; ++k) sum += in[k];
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int64_t v = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    int64_t run = part[threadIdx.x] - sum;
    for (int64_t k = b; k < e; ++k) {
        const int64_t v = in[k];
        out[k] = run;
        run += v;
    }
    if (threadIdx.x == 1023) out[n] = part[1023];
}

__global__ void k_na_scatter(NaArgs A) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    const int32_t cell = na_node_cell(A.s)[i];
    const int64_t pos = (int64_t)atomicAdd((unsigned long long*)&na_fill(A.s)[cell], 1ull);
    na_sorted(A.s)[na_cstart(A.s)[cell] + pos] = (int32_t)i;
}

// One warp per node, the membership test of InitBond (pdDataManager2.cpp:
// 12-70).  PASS 0 counts; PASS 1 sorts the family by id in shared memory and
// writes it with the slit marks.
template <int PASS>
__global__ void k_na_search(NaArgs A, int64_t* row_ptr, int32_t* col, uint8_t* broken, int cap) {
    extern __shared__ int32_t sb[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (i >= A.n) return;
    int32_t* buf = sb + (size_t)wib * cap;
    uint8_t* brk = (uint8_t*)(sb + (size_t)(blockDim.x >> 5) * cap) + (size_t)wib * cap;
    const double* sl = na_slits(A.s);
    double pi[3] = {A.x[3 * i], A.x[3 * i + 1], A.x[3 * i + 2]};
    int64_t c[3];
    na_cell_of(A, pi, c);
    int64_t nf = 0;
    double mb = A.delta;
    for (int64_t dz = -1; dz <= 1; ++dz)
        for (int64_t dy = -1; dy <= 1; ++dy)
            for (int64_t dxc = -1; dxc <= 1; ++dxc) {
                const int64_t qx = c[0] + dxc, qy = c[1] + dy, qz = c[2] + dz;
                if (qx < 0 || qy < 0 || qz < 0 || qx >= A.g.nc[0] || qy >= A.g.nc[1] || qz >= A.g.nc[2]) continue;
                const int64_t q = (qz * A.g.nc[1] + qy) * A.g.nc[0] + qx;
                const int64_t s0 = na_cstart(A.s)[q], s1 = na_cstart(A.s)[q + 1];
                for (int64_t s = s0; s < s1; s += 32) {
                    bool hit = false, br = false;
                    int64_t j = -1;
                    if (s + lane < s1) {
                        j = na_sorted(A.s)[s + lane];
                        if (j != i) {
                            const double pj[3] = {A.x[3 * j], A.x[3 * j + 1], A.x[3 * j + 2]};
                            const double* pa = (i < j) ? pi : pj;
                            const double* pb = (i < j) ? pj : pi;
                            const double d1 = pj[0] - pi[0], d2 = pj[1] - pi[1], d3 = pj[2] - pi[2];
                            const double dd = d1 * d1 + d2 * d2 + d3 * d3;
                            const int quick = pair_quick(A.lim, d1, d2, d3, dd);
                            hit = quick > 0 || (quick < 0 && pair_bonded_any(pa[0], pa[1], pa[2], pb[0], pb[1], pb[2],
                                                                             A.dx, A.delta, A.tol));
                            if (hit) {
                                if (i < j) mb = dmin(mb, sqrt(dd));
                                for (int k = 0; k < A.nslit; ++k) br = br || slit_crosses(sl + 6 * k, pa, pb);
                            }
                        }
                    }
                    const unsigned hm = __ballot_sync(0xffffffffu, hit);
                    if (PASS == 1 && hit) {
                        const int slot = (int)nf + __popc(hm & ((1u << lane) - 1u));
                        if (slot < cap) {
                            buf[slot] = (int32_t)j;
                            brk[slot] = br ? 1 : 0;
                        }
                    }
                    nf += __popc(hm);
                }
            }
    if (PASS == 0) {
        for (int o = 16; o > 0; o >>= 1) mb = dmin(mb, __shfl_xor_sync(0xffffffffu, mb, o));
        if (lane == 0) {
            na_cnt(A.s)[i] = nf;
            unsigned long long* sc = (unsigned long long*)na_scal(A.s);
            atomicMin(&sc[6], (unsigned long long)__double_as_longlong(mb));
            atomicMax(&sc[7], (unsigned long long)nf);
        }
        return;
    }
    __syncwarp();
    const int n = (int)(nf < cap ? nf : cap);
    const int64_t o = row_ptr[i];
    for (int e = lane; e < n; e += 32) {
        const int32_t v = buf[e];
        int rk = 0;
        for (int k = 0; k < n; ++k) rk += buf[k] < v ? 1 : 0;
        col[o + rk] = v;
        if (broken) broken[o + rk] = brk[e];
    }
}

std::mutex g_na_mu;
void* g_na_addr[64] = {};

}  // namespace

}  // namespace pd

extern "C" int pd_bond_search_noalloc(const double* coords, int64_t n, double grid_spacing, double horizon,
                                      int32_t num_slits, const double* slits, int64_t* row_ptr, int32_t* col,
                                      uint8_t* broken, int64_t capacity, void* stream, int64_t* num_halves,
                                      double* min_bond_length) {
    using namespace pd;
    if (n < 0 || n > na::kNodes) return fail(PD_ERR_CAPACITY, "pd_bond_search_noalloc: more nodes than PD_NOALLOC_MAX_NODES");
    if (num_slits < 0 || num_slits > na::kSlits || (num_slits > 0 && !slits))
        return fail(PD_ERR_ARG, "pd_bond_search_noalloc: bad slit list");
    if (!row_ptr || (n > 0 && !coords) || capacity < 0 || (capacity > 0 && !col) || !(grid_spacing > 0.0) ||
        !(horizon > 0.0))
        return fail(PD_ERR_ARG, "pd_bond_search_noalloc: bad argument");
    int dev = 0;
    PD_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(PD_ERR_ARG, "pd_bond_search_noalloc: device index above 63");
    unsigned char* s = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_na_mu);
        if (!g_na_addr[dev]) {
            void* p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess) return fail_cuda(e, "cudaGetSymbolAddress(g_noalloc_scratch)", __FILE__, __LINE__);
            g_na_addr[dev] = p;
        }
        s = (unsigned char*)g_na_addr[dev];
    }
    cudaStream_t st = (cudaStream_t)stream;
    double bb[6] = {0, 0, 0, 0, 0, 0};
    if (n > 0) {
        k_na_bbox<<<1, 1024, 0, st>>>(coords, n, s);
        PD_CUDA_TRY(cudaGetLastError());
        PD_CUDA_TRY(cudaMemcpyAsync(bb, s + na::kOffScal, sizeof bb, cudaMemcpyDeviceToHost, st));
        PD_CUDA_TRY(cudaStreamSynchronize(st));
    }
    NaArgs A;
    A.x = coords;
    A.n = n;
    A.dx = grid_spacing;
    A.delta = horizon;
    A.tol = 1.0e-4 * grid_spacing;
    A.s = s;
    A.nslit = num_slits;
    A.g.h = horizon + grid_spacing;
    // Cells per axis are counted in double and checked against the array's
    // limit before any conversion to an integer: a non-finite coordinate or a
    // horizon tiny next to the extent must not reach an undefined cast or an
    // overflowing product.
    int64_t ncell = 1;
    for (int a = 0; a < 3; ++a) {
        if (!std::isfinite(bb[a]) || !std::isfinite(bb[3 + a]))
            return fail(PD_ERR_ARG, "pd_bond_search_noalloc: non-finite coordinate");
        const double cells = std::floor((bb[3 + a] - bb[a]) / A.g.h) + 1.0;
        if (!(cells >= 1.0) || cells > (double)na::kCells)
            return fail(PD_ERR_CAPACITY, "pd_bond_search_noalloc: more cells than PD_NOALLOC_MAX_CELLS");
        A.g.lo[a] = bb[a];
        A.g.nc[a] = (int64_t)cells;
        ncell *= A.g.nc[a];  // each factor <= kCells and the partial product too: no overflow
        if (ncell > na::kCells)
            return fail(PD_ERR_CAPACITY, "pd_bond_search_noalloc: more cells than PD_NOALLOC_MAX_CELLS");
    }
    double reach = 0.0;
    for (double v : bb) reach = std::max(reach, std::fabs(v));
    A.lim = pair_limits(A.dx, A.delta, A.tol, reach);
    // the regions read before they are written start at zero
    PD_CUDA_TRY(cudaMemsetAsync(s + na::kOffCellCnt, 0, sizeof(int64_t) * (ncell + 1), st));
    PD_CUDA_TRY(cudaMemsetAsync(s + na::kOffFill, 0, sizeof(int64_t) * (ncell + 1), st));
    if (num_slits > 0)
        PD_CUDA_TRY(cudaMemcpyAsync(s + na::kOffSlits, slits, sizeof(double) * 6 * num_slits, cudaMemcpyHostToDevice, st));
    unsigned long long sc[2] = {(unsigned long long)__builtin_bit_cast(unsigned long long, horizon), 0ull};
    PD_CUDA_TRY(cudaMemcpyAsync(s + na::kOffScal + 6 * sizeof(double), sc, sizeof sc, cudaMemcpyHostToDevice, st));
    const int bs = 256, wpb = 4;
    const unsigned nb = (unsigned)((n + bs - 1) / bs), nw = (unsigned)((n * 32 + 32 * wpb - 1) / (32 * wpb));
    if (n > 0) k_na_cell_count<<<nb, bs, 0, st>>>(A);
    k_na_scan<<<1, 1024, 0, st>>>((const int64_t*)(s + na::kOffCellCnt), (int64_t*)(s + na::kOffCstart), ncell);
    if (n > 0) {
        k_na_scatter<<<nb, bs, 0, st>>>(A);
        k_na_search<0><<<nw, 32 * wpb, 0, st>>>(A, nullptr, nullptr, nullptr, 0);
    }
    k_na_scan<<<1, 1024, 0, st>>>((const int64_t*)(s + na::kOffCnt), row_ptr, n);
    PD_CUDA_TRY(cudaGetLastError());
    int64_t total = 0;
    unsigned long long back[2] = {0, 0};
    PD_CUDA_TRY(cudaMemcpyAsync(&total, row_ptr + n, sizeof total, cudaMemcpyDeviceToHost, st));
    PD_CUDA_TRY(cudaMemcpyAsync(back, s + na::kOffScal + 6 * sizeof(double), sizeof back, cudaMemcpyDeviceToHost, st));
    PD_CUDA_TRY(cudaStreamSynchronize(st));
    if (num_halves) *num_halves = total;
    if (min_bond_length) *min_bond_length = n > 0 ? __builtin_bit_cast(double, back[0]) : horizon;
    if (total > capacity) return fail(PD_ERR_CAPACITY, "pd_bond_search_noalloc: col capacity below the family size");
    const int cap = (int)back[1] + 1;
    const size_t sh = (size_t)wpb * cap * (sizeof(int32_t) + sizeof(uint8_t));
    if (sh > 48 * 1024) return fail(PD_ERR_CAPACITY, "pd_bond_search_noalloc: family larger than the shared buffer");
    if (n > 0) k_na_search<1><<<nw, 32 * wpb, sh, st>>>(A, row_ptr, col, broken, cap);
    PD_CUDA_TRY(cudaGetLastError());
    PD_CUDA_TRY(cudaStreamSynchronize(st));
    return PD_OK;
}

namespace pd {

// ================================================== areal force density
//
// pdSolve::PostAFD (pdSolve.cpp:810-834, pdDataManager3.cpp:442-635,
// 1101-1223): the stress tensor at a source node s from the areal force
// density.  For each direction d and each node i at s - (1 + is) dx e_d
// (is < int(horizon / dx)), the bond forces of i with every node j of its
// family that lies in the source's half space x_j,d >= x_s,d are summed.
// Here one thread takes one (i, s, d) item; the host builds the items and
// adds them up in the reference's order.

// Gauss-point displacements as PostAFD derives them from a Tecplot dump
// (pdDataManager.cpp:2704-2752, CalcApproxDispl, or the copy of the one-point
// rule): the MLS sum of the nodal displacements u_k c_k on every node, except
// that a direction a boundary condition flags keeps its Gauss points at zero
// (they are never set in a post-processing run).
__global__ void k_afd_gauss(Dev d, const double* __restrict__ U, double* __restrict__ ug) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    const int64_t N = d.n;
    const int npt = d.npt;
    bool flagged[3] = {false, false, false};
    if (d.bc[i] >= 0)
        for (int a = 0; a < 3; ++a) flagged[a] = d.bcs[d.bc[i]].dir[a] == 1;
    for (int g = 0; g < npt; ++g) {
        double v[3] = {0.0, 0.0, 0.0};
        if (d.mls) {
            const int64_t b = d.cbptr[i], nc = d.cbptr[i + 1] - b;
            for (int64_t k = 0; k < nc; ++k) {
                const int64_t m = d.cbidx[b + k];
                const double c = d.coeff[(b + k) * npt + g];
                v[0] += U[m] * c;
                v[1] += U[N + m] * c;
                v[2] += U[2 * N + m] * c;
            }
            for (int a = 0; a < 3; ++a)
                if (flagged[a]) v[a] = 0.0;
        } else {
            for (int a = 0; a < 3; ++a) v[a] = U[a * N + i];
        }
        for (int a = 0; a < 3; ++a) ug[(int64_t)(3 * g + a) * N + i] = v[a];
    }
}

// pdIntgManager::CalcBondBasedForce (pdIntgManager2.cpp:92-310), fixed
// Gauss points: the point at local position (X, Y, Z) from node i, with the
// displacement of cell j's point g
__device__ __forceinline__ void afd_point(const Dev& d, double X, double Y, double Z, const double* ugj, double ui0,
                                          double ui1, double ui2, double bE, double spring, double ecrit,
                                          double dxe, double* f) {
    const double xi1 = X - 0.0, xi2 = Y - 0.0, xi3 = Z - 0.0;
    const double eta1 = ugj[0] - ui0, eta2 = ugj[1] - ui1, eta3 = ugj[2] - ui2;
    const double r = sqrt(xi1 * xi1 + xi2 * xi2 + xi3 * xi3);
    const double y1 = xi1 + eta1, y2 = xi2 + eta2, y3 = xi3 + eta3;
    const double p = sqrt(y1 * y1 + y2 * y2 + y3 * y3);
    const double beta = beta_factor(r, d.delta, dxe, false);
    const double u = p - r;
    const double stretch = u / r;
    if (u <= 0.0 || (u > 0.0 && stretch <= ecrit)) {
        f[0] = bE * beta * spring * stretch * y1 / p;
        f[1] = bE * beta * spring * stretch * y2 / p;
        f[2] = bE * beta * spring * stretch * y3 / p;
    } else {
        f[0] = f[1] = f[2] = 0.0;
    }
}

__global__ void k_afd_items(Dev d, const double* __restrict__ U, const double* __restrict__ bE,
                            const double* __restrict__ ug, const double* __restrict__ absc,
                            const double* __restrict__ wts, int n1, int64_t n_items,
                            const int64_t* __restrict__ item_i, const int64_t* __restrict__ item_s,
                            const int32_t* __restrict__ item_d, double* __restrict__ out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n_items) return;
    const int64_t N = d.n;
    const int64_t i = item_i[t], s = item_s[t];
    const int dir = item_d[t] - 1;
    const double pi[3] = {d.x[i], d.x[N + i], d.x[2 * N + i]};
    const double xs_d = d.x[dir * N + s];
    const double ui0 = U[i], ui1 = U[N + i], ui2 = U[2 * N + i];
    const MatDev& Mi = d.mats[d.mat[i]];
    const double dx = d.dx, tol = 1.0e-4 * dx;
    double sum0 = 0.0, sum1 = 0.0, sum2 = 0.0;
    for (int64_t p = d.frow[i]; p < d.frow[i + 1]; ++p) {
        const int64_t j = d.fcol[p];
        const double pj[3] = {d.x[j], d.x[N + j], d.x[2 * N + j]};
        if (!(pj[dir] - xs_d >= 0.0)) continue;  // the source's R+ space
        const MatDev& Mj = d.mats[d.mat[j]];
        const double ecrit = dmin(Mi.ecrit, Mj.ecrit);
        const double spring = dmin(Mi.spring, Mj.spring);
        const double bEij = 0.5 * (bE[i] + bE[j]);
        double f[3] = {0.0, 0.0, 0.0};
        if (d.cci) {
            // pdDataManager::CalcBondForceCCI(bond, i, j), pdDataManager2.cpp:1087-1154
            const double xi1 = pj[0] - pi[0], xi2 = pj[1] - pi[1], xi3 = pj[2] - pi[2];
            const double eta1 = U[j] - ui0, eta2 = U[N + j] - ui1, eta3 = U[2 * N + j] - ui2;
            const double r = sqrt(xi1 * xi1 + xi2 * xi2 + xi3 * xi3);
            const double y1 = xi1 + eta1, y2 = xi2 + eta2, y3 = xi3 + eta3;
            const double pl = sqrt(y1 * y1 + y2 * y2 + y3 * y3);
            const double u = pl - r;
            const double stretch = u / r;
            if (u <= 0.0 || (u > 0.0 && stretch <= ecrit)) {
                const double beta = beta_factor(r, d.delta, dx, !d.cci_mdf);
                const double vol = d.vol;
                f[0] = bEij * vol * beta * spring * stretch * y1 / pl;
                f[1] = bEij * vol * beta * spring * stretch * y2 / pl;
                f[2] = bEij * vol * beta * spring * stretch * y3 / pl;
            }
        } else {
            // CalcBondForceIntg (pdDataManager2.cpp:1156-1215): nothing when
            // the cell lies beyond the horizon, else the cell's fixed Gauss
            // rule as pdIntgManager::CalcConfigurationType3 / CalcIntg3D /
            // CalcGaussianQuad nest it (pdIntgManager.cpp:49-128,453-509,
            // 3471-3482), in local coordinates x_j - x_i
            double mn = kMega, a, b;
            for (int ax = 0; ax < 3; ++ax) {
                dist_to_face(ax + 1, pj[ax] - 0.5 * dx, pi, pj, dx, &a, &b);
                mn = dmin(mn, a);
                dist_to_face(ax + 1, pj[ax] + 0.5 * dx, pi, pj, dx, &a, &b);
                mn = dmin(mn, a);
            }
            if (!(d.delta <= mn)) {
                const double x1j = pj[0] - pi[0], x2j = pj[1] - pi[1], x3j = pj[2] - pi[2];
                const double lo1 = x1j - 0.5 * dx, hi1 = x1j + 0.5 * dx;
                const double lo2 = x2j - 0.5 * dx, hi2 = x2j + 0.5 * dx;
                const double lo3 = x3j - 0.5 * dx, hi3 = x3j + 0.5 * dx;
                int counter = 0;  // _intgPointCounter: the Gauss point of cell j
                if (fabs(lo1 - hi1) > 1.0e-10) {
                    double S1[3] = {0.0, 0.0, 0.0};
                    for (int q1 = 0; q1 < n1; ++q1) {
                        const double X = 0.5 * dx * absc[q1] + x1j;
                        double F2[3] = {0.0, 0.0, 0.0};
                        if (fabs(lo2 - hi2) > 1.0e-10) {
                            double S2[3] = {0.0, 0.0, 0.0};
                            for (int q2 = 0; q2 < n1; ++q2) {
                                const double Y = 0.5 * dx * absc[q2] + x2j;
                                double F3[3] = {0.0, 0.0, 0.0};
                                if (fabs(lo3 - hi3) > 1.0e-10) {
                                    double S3[3] = {0.0, 0.0, 0.0};
                                    for (int q3 = 0; q3 < n1; ++q3) {
                                        const double Z = 0.5 * dx * absc[q3] + x3j;
                                        const double ugj[3] = {ug[(int64_t)(3 * counter) * N + j],
                                                               ug[(int64_t)(3 * counter + 1) * N + j],
                                                               ug[(int64_t)(3 * counter + 2) * N + j]};
                                        double fp[3];
                                        afd_point(d, X, Y, Z, ugj, ui0, ui1, ui2, bEij, spring, ecrit,
                                                  d.gc[counter].dxe, fp);
                                        ++counter;
                                        for (int c = 0; c < 3; ++c) S3[c] += wts[q3] * fp[c];
                                    }
                                    for (int c = 0; c < 3; ++c) F3[c] = S3[c] * (0.5 * (hi3 - lo3));
                                }
                                for (int c = 0; c < 3; ++c) S2[c] += wts[q2] * F3[c];
                            }
                            for (int c = 0; c < 3; ++c) F2[c] = S2[c] * (0.5 * (hi2 - lo2));
                        }
                        for (int c = 0; c < 3; ++c) S1[c] += wts[q1] * F2[c];
                    }
                    for (int c = 0; c < 3; ++c) f[c] = S1[c] * (0.5 * (hi1 - lo1));
                }
            }
        }
        sum0 += f[0];
        sum1 += f[1];
        sum2 += f[2];
    }
    (void)tol;
    out[3 * t] = sum0;
    out[3 * t + 1] = sum1;
    out[3 * t + 2] = sum2;
}

int afd_forces(const Dev& d, const double* U, const double* bE, double* ug, const double* absc, const double* wts,
               int n1, int64_t n_items, const int64_t* item_i, const int64_t* item_s, const int32_t* item_d,
               double* out, cudaStream_t s) {
    if (d.n == 0 || n_items == 0) return PD_OK;
    k_afd_gauss<<<(unsigned)((d.n + 127) / 128), 128, 0, s>>>(d, U, ug);
    k_afd_items<<<(unsigned)((n_items + 63) / 64), 64, 0, s>>>(d, U, bE, ug, absc, wts, n1, n_items, item_i, item_s,
                                                               item_d, out);
    return cudaGetLastError() == cudaSuccess ? PD_OK : PD_ERR_CUDA;
}

}  // namespace pd
