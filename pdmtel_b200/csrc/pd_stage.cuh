// The per-node end of an RK4 stage, shared by the stage kernel of every form
// and by the persistent kernel.
//
// Every operation is an explicit round-to-nearest intrinsic, in the order the
// reference writes it, so the result is the same bit for bit whatever the
// contraction flags of the translation unit that includes this file.  Loads
// of the state go through L2 (ld.global.cg): inside one persistent launch
// another SM may have rewritten a line this SM still holds in L1.
#pragma once

#include "pd_internal.cuh"

namespace pd {

// GetTimeFactor: VELOC is on until its end time; DISPL/DISPLGRAD ramp as
// t/t_end when load_type == 1, else full (pdDataManager.cpp:2507-2522)
__device__ __forceinline__ double bc_time_factor(const BcDev& b, double t) {
    if (b.type == PD_BC_VELOC) return (t <= b.end_time) ? 1.0 : 0.0;
    if (b.load_type == 1.0) return (t <= b.end_time) ? __ddiv_rn(t, b.end_time) : 1.0;
    return 1.0;
}

// After the bond forces of stage `stage` (1..4; 0 for a lone stage whose k
// goes to k1) have been added to vbuf at time t, component a of node i: the
// traction load (project rule: value*factor/dx added to vbuf once per stage),
// UpdateNodeStatusWithBC (pdDataManager.cpp:2497-2602), k = vbuf*dt_s
// (:1977-1990) and the RK4 bookkeeping of pdDataManager::RK4 (:2027-2092).  v:
// the component of vbuf with the stage's forces (HELD: vbuf itself holds it);
// returns its final value.  eff: the displacement a one-point force of the next
// stage uses for the node.  U and a held vbuf are touched only where a
// condition or the last stage may change them: two passes over each less in
// three stages of four.
template <bool HELD>
__device__ __forceinline__ double stage_axis(const Dev& d, int64_t i, int a, int stage, double dts, double dt, double t,
                                             double rho, double v, double& eff) {
    const int64_t N = d.n, r = a * N + i;
    const int b = d.bc[i];
    const bool changes = b >= 0 || stage == 4;
    double U = changes ? __ldcg(d.U + r) : 0.0;
    if (b >= 0) {
        const BcDev& B = d.bcs[b];
        if (B.dir[a] == 1) {
            const double fac = bc_time_factor(B, t);
            if (B.type == PD_BC_TRACTION) {
                const double tb = __ddiv_rn(__dmul_rn(B.val[a], fac), d.dx);
                v = __dadd_rn(v, __ddiv_rn(__dmul_rn(tb, dts), rho));
            } else if (B.type == PD_BC_DISPL) {
                U = __dmul_rn(B.val[a], fac);
                v = 0.0;
            } else if (B.type == PD_BC_VELOC) {
                v = __dmul_rn(B.val[a], fac);
            } else if (B.type == PD_BC_DISPLGRAD) {
                const double e = __dadd_rn(__dadd_rn(__dmul_rn(B.val[3 * a], d.x[i]),
                                                     __dmul_rn(B.val[3 * a + 1], d.x[N + i])),
                                           __dmul_rn(B.val[3 * a + 2], d.x[2 * N + i]));
                U = __dmul_rn(e, fac);
                v = 0.0;
            }
        }
    }
    const double dt6 = 1.0 / 6.0;
    const double k = __dmul_rn(v, dts);
    double us = 0.0;
    if (stage == 0) {
        d.k1[r] = k;
    } else if (stage == 1) {
        d.k1[r] = k;
        d.us[r] = us = __dadd_rn(__ldcg(d.u1 + r), __dmul_rn(0.5, k));
    } else if (stage == 2) {
        d.k2[r] = k;
        d.us[r] = us = __dadd_rn(__ldcg(d.u1 + r), __dmul_rn(0.5, k));
    } else if (stage == 3) {
        d.us[r] = us = __dadd_rn(__ldcg(d.u1 + r), k);
        d.k32[r] = __dadd_rn(k, __ldcg(d.k2 + r));
    } else {
        const double Vold = __ldcg(d.V + r);
        const double inc = __dmul_rn(dt6, __dadd_rn(__dadd_rn(__ldcg(d.k1 + r), k), __dmul_rn(2.0, __ldcg(d.k32 + r))));
        if (b >= 0) {
            U = __dadd_rn(U, inc);
        } else {
            const double damp = __ddiv_rn(__dmul_rn(__dmul_rn(__dmul_rn(dt, d.damping), Vold), dt), rho);
            U = __dsub_rn(__dadd_rn(U, inc), damp);
        }
        v = __dadd_rn(v, __ddiv_rn(__dmul_rn(__dmul_rn(-d.damping, Vold), dt), rho));
        d.V[r] = v;
        d.u1[r] = U;
        d.us[r] = us = U;
    }
    if (!HELD || changes) d.vbuf[r] = v;
    if (changes) d.U[r] = U;
    eff = b >= 0 ? U : us;
    return v;
}

// The node's kinetic and elastic energy of a step, from its final velocity and
// energy density, into red[i], red[N+i].
__device__ __forceinline__ void stage_energy(const Dev& d, int64_t i, double rho, double v0, double v1, double v2,
                                             double eed) {
    const double velsq = __dadd_rn(__dadd_rn(__dmul_rn(v0, v0), __dmul_rn(v1, v1)), __dmul_rn(v2, v2));
    d.red[i] = __dmul_rn(__dmul_rn(__dmul_rn(0.5, rho), velsq), d.vol);
    d.red[d.n + i] = __dmul_rn(d.vol, eed);
}

// All of node i at the end of a stage; with ENERGY, stage 4 leaves its energies.
template <bool ENERGY>
__device__ __forceinline__ void stage_epilogue(const Dev& d, int64_t i, int stage, double dts, double dt, double t) {
    const int64_t N = d.n;
    const double rho = d.mats[d.mat[i]].density;
    double v[3], eff;
    for (int a = 0; a < 3; ++a)
        v[a] = stage_axis<true>(d, i, a, stage, dts, dt, t, rho, __ldcg(d.vbuf + a * N + i), eff);
    if (ENERGY && stage == 4) stage_energy(d, i, rho, v[0], v[1], v[2], __ldcg(d.eed + i));
}

}  // namespace pd
