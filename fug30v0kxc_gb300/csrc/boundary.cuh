// boundary.cuh -- the boundary conditions of one column (src/dbydz.F90:3686-4197
// and :4205-4791), shared by the kernels that apply them.
#pragma once
#include "common.cuh"
#include "engine.h"
#include "fpconv.cuh"

// In the split form (m != nullptr) the FP32 mirrors of the two boundary
// planes are written here too: m = {u32, v32, w32, t32}, t0 = T0(z).
__device__ __forceinline__ void boundary_column(double *u, double *v, double *w, double *t, size_t np, int nz,
                                                double theta, double dz, int radbc, int constflux,
                                                const BoundaryMirrors &mb, size_t q)
{
    const double elf = 1.0 / 11.0;
#define P(f, kk) f[(size_t)(kk) * np + q]
    P(w, 0) = 0.0;
    P(u, 0) = elf * (18.0 * P(u, 1) - 9.0 * P(u, 2) + 2.0 * P(u, 3));
    P(v, 0) = elf * (18.0 * P(v, 1) - 9.0 * P(v, 2) + 2.0 * P(v, 3));
    P(w, nz - 1) = 0.0;
    P(u, nz - 1) = elf * (18.0 * P(u, nz - 2) - 9.0 * P(u, nz - 3) + 2.0 * P(u, nz - 4));
    P(v, nz - 1) = elf * (18.0 * P(v, nz - 2) - 9.0 * P(v, nz - 3) + 2.0 * P(v, nz - 4));
    if (radbc) {   // :4036-4055, Newton iterations on the radiative condition
        double t1old = P(t, 0);
        for (int it = 0; it < 10; it++) {
            double ft1 = 6.0 * theta * dz * t1old * t1old * t1old * t1old + 11.0 * t1old - 18.0 * P(t, 1)
                         + 9.0 * P(t, 2) - 2.0 * P(t, 3);
            double dft1 = 24.0 * theta * dz * t1old * t1old * t1old + 11.0;
            t1old = t1old - (ft1 / dft1);
        }
        P(t, 0) = t1old;
    } else {
        P(t, 0) = 1.0;
    }
    if (constflux)
        P(t, nz - 1) = elf * (18.0 * P(t, nz - 2) - 9.0 * P(t, nz - 3) + 2.0 * P(t, nz - 4) + 6.0 * theta * dz);
    else
        P(t, nz - 1) = 1.0 + theta;
    if (mb.u32) {
        const int ks[2] = { 0, nz - 1 };
        for (int e = 0; e < 2; e++) {
            const int kk = ks[e];
            mb.u32[(size_t)kk * np + q] = d2f_rn(P(u, kk));
            mb.v32[(size_t)kk * np + q] = d2f_rn(P(v, kk));
            mb.w32[(size_t)kk * np + q] = d2f_rn(P(w, kk));
            mb.t32[(size_t)kk * np + q] = d2f_rn(P(t, kk) - mb.t0[kk]);
        }
    }
#undef P
}

// arguments of k_boundary / k_boundaries
struct BndArgs {
    double *u, *v, *w, *t, *pol, *tor, *bxb, *byb;
    size_t np;
    int nz;
    double theta, dz;
    int radbc, constflux, perfect;
    BoundaryMirrors mb;
};

static inline BndArgs bnd_args(Engine *E)
{
    BndArgs a;
    BoundaryMirrors mb = {};
    if (E->split) {
        mb.u32 = E->u32; mb.v32 = E->v32; mb.w32 = E->w32; mb.t32 = E->t32; mb.t0 = split_bg_t0(E);
        mb.pol32 = E->pol32; mb.tor32 = E->tor32;
    }
    a.u = E->u; a.v = E->v; a.w = E->w; a.t = E->t; a.pol = E->pol; a.tor = E->tor; a.bxb = E->bxbar; a.byb = E->bybar;
    a.np = E->np; a.nz = E->nz; a.theta = E->p.theta; a.dz = E->k.dz;
    a.radbc = E->p.radbc; a.constflux = E->p.constflux; a.perfect = E->p.perfect; a.mb = mb;
    return a;
}

__device__ __forceinline__ void mag_boundary_column(double *pol, double *tor, double *bxb, double *byb, size_t np,
                                                    int nz, int perfect, const BoundaryMirrors &mb, size_t q)
{
    const double elf = 1.0 / 11.0;
    if (q == 0) {
        if (perfect) {
            bxb[0] = elf * (18.0 * bxb[1] - 9.0 * bxb[2] + 2.0 * bxb[3]);
            byb[0] = elf * (18.0 * byb[1] - 9.0 * byb[2] + 2.0 * byb[3]);
            bxb[nz - 1] = elf * (18.0 * bxb[nz - 2] - 9.0 * bxb[nz - 3] + 2.0 * bxb[nz - 4]);
            byb[nz - 1] = elf * (18.0 * byb[nz - 2] - 9.0 * byb[nz - 3] + 2.0 * byb[nz - 4]);
        } else {
            bxb[0] = 0.0; byb[0] = 0.0; bxb[nz - 1] = 0.0; byb[nz - 1] = 0.0;
        }
    }
    if (q >= np) return;
#define P(f, kk) f[(size_t)(kk) * np + q]
    if (perfect) {   // :4407-4560
        P(pol, 0) = 0.0;
        P(tor, 0) = elf * (18.0 * P(tor, 1) - 9.0 * P(tor, 2) + 2.0 * P(tor, 3));
        P(pol, nz - 1) = 0.0;
        P(tor, nz - 1) = elf * (18.0 * P(tor, nz - 2) - 9.0 * P(tor, nz - 3) + 2.0 * P(tor, nz - 4));
    } else {         // :4663-4780
        P(tor, 0) = 0.0;
        P(pol, 0) = elf * (18.0 * P(pol, 1) - 9.0 * P(pol, 2) + 2.0 * P(pol, 3));
        P(tor, nz - 1) = 0.0;
        P(pol, nz - 1) = elf * (18.0 * P(pol, nz - 2) - 9.0 * P(pol, nz - 3) + 2.0 * P(pol, nz - 4));
    }
    if (mb.pol32) {
        mb.pol32[q] = d2f_rn(P(pol, 0));
        mb.tor32[q] = d2f_rn(P(tor, 0));
        mb.pol32[(size_t)(nz - 1) * np + q] = d2f_rn(P(pol, nz - 1));
        mb.tor32[(size_t)(nz - 1) * np + q] = d2f_rn(P(tor, nz - 1));
    }
#undef P
}
