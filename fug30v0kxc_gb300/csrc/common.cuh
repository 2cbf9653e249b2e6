// common.cuh -- shared types of the GB300 VarElecCond library (internal).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include "../../include/vec.h"

// complex type per real precision
template <typename R> struct CT;
template <> struct CT<double> { using T = double2; };
template <> struct CT<float> { using T = float2; };

// operations of one line job
enum LineOp {
    OP_NONE = 0,
    OP_D1 = 1,       // first derivative (+ik), DC and Nyquist dropped: src/fft.F90:292-302
    OP_D2 = 2,       // second derivative (-k^2), Nyquist kept: src/fft.F90:442-454
    OP_DEALIAS = 3,  // 2/3-rule truncation: src/fft.F90:618-626
    OP_FWD = 4,      // real -> halfcomplex, unnormalised (rfftw forward)
    OP_INV = 5,      // halfcomplex -> real, divided by n (rfftw backward / n); op2
                     // OP_D1 adds the derivative of that inverse as a second output
};

template <typename R>
struct LineJob {
    const R *in;
    R *out1, *out2;
    R alpha1, alpha2;   // outputs are alpha * result (+ old value when acc)
    int op1, op2;
    int acc1, acc2;
    const double *addk; // OP_INV only: out1 += addk[plane] + addc
    double addc;
};

// line jobs per launch: a batch of 16 members carries up to 96 (five hydro
// jobs, and the Lorentz fluxes' and E's transforms, per member); the job
// and tensor-map packs then take 24 KB of the 32 KB kernel parameter space
#define MAX_JOBS 128
// Parameters cost a launch time by their size: with room for MAX_JOBS jobs and TMA
// descriptors, 24 KB, a derivative pair at 64^2 x 65 took 12.0 (x) and 10.4 us (y),
// with room for eight jobs 8.9 and 8.5.  So launches of a few jobs (one solver's; a
// batch of members has more) have kernels of their own.
#define NJ_SMALL 8

// spectral tables of one direction (device pointers)
template <typename R>
struct LineTables {
    typename CT<R>::T *tw;  // exp(-2 pi i e / n), e = 0..n-1
    R *m1;                  // d1 multiplier (imaginary part, sign and 1/n folded in)
    R *m2;                  // d2 multiplier (k2 / n, DC zeroed)
    R *mda;                 // dealias mask (1/n or 0)
};

// the FP64 line kernel's passes for a length n (lines_fx.cu): radix, block and
// stride of each, ceil(2^31 / stride), and where its twiddles start
struct FxPlan {
    int n, nb;              // length; elements of a buffer (n rounded up to 8)
    int np;                 // passes
    int R[6], L[6], M[6], tw[6], kind[6];
    unsigned mg[6];
    int ntw;                // twiddles in all
    int hf, hi;             // halvings of a forward, an inverse transform
    unsigned fup, iup;      // passes (bits) that leave their halving out: lines_fx_long.cu
    int gb;                 // its values stay below 2^gb times the norm
    int Q;                  // sequences per warp
    int cut;                // wavenumbers below it survive the dealiasing
    float rn;               // 1 / n
    float floor1, floor2;   // least sums of squares of a first, second derivative's spectrum
};
// its tables: twiddles by pass; position of wavenumber k in the spectrum and
// back; the constants of dealias and inverse, d1 and d2
struct TwX;
struct FxTables {
    TwX *tw;                // (one allocation with pos and kof)
    unsigned short *pos, *kof;
    double c0, c1, c2;
};

// the FP32 general line kernel's passes (lines.cu): radices, the strides of the forward and
// the inverse pass of each, ceil(2^31 / stride), and where their twiddles start
struct FsPlan {
    int n, np, R[8];
    int fM[8], iM[8], ftw[8], itw[8];
    unsigned fmg[8], img[8];
    int ntw;                // twiddles in all
    int Q;                  // sequences per warp
    int nb, sha, shb;       // words of a buffer; padding of the first and the second one
};
// its tables: twiddles by pass; multipliers, wavenumber and place in the spectrum by the
// element of the first inverse pass
struct FsTables {
    float2 *tw;             // (one allocation with the others)
    float *m1, *m2, *mda;
    unsigned short *pos, *gat;
};

// horizontal wavenumber tables in one precision: akx1, aky1 and the
// plane table akx2[i] + aky2[j] (summed in FP64, then rounded once)
template <typename R>
struct HTab {
    const R *kx1, *ky1, *kh2;
    const R *kh2inv;        // 1 / kh2 (0 at the mean, kh2 = 0), rounded once from FP64
};

// ---- per-context derived constants: src/constants.f90:56-109 -----------
struct Consts {
    double dx, dy, dz, dd, xn, xzn, taylt, cpsi, spsi, cor;
    double gck, sck, zck, scko3, sckg, fzckg, thmplus1, fo2, g1, gm1, nusstmp;
    double dtvisc0x, dtvisc0z, dtdiff0x, dtdiff0z;
    double ho12, sc1;
    double f, gamma, theta, sf;
    double eta_max;
    int var_eta;            // eta_contrast != 1
    int icutoffx, icutoffy;
};

// order-preserving keys (see okey in physics.cu) of -DBL_MAX and +DBL_MAX
#define OKEY_NEG_HUGE 0x0010000000000000ull
#define OKEY_POS_HUGE 0xffefffffffffffffull

// time-loop scalars living on the device (src/main.F90:84-103)
struct DevScalars {
    double dt, dt1, dt2, ttime;
    double c0, c1, c2;
    int first, second;
    // reductions
    unsigned long long velmxx, velmxz, denmn;  // order-preserving keys of the reductions
    double res[64];                            // diagnostics results
    // the last calcdt met a non-finite value (NaN or infinity) in the state
    // or in the CFL expression; the time loop reports it as VEC_ERR_NAN
    int nonfinite, pad_nf;
};

// AB3 coefficients of src/main.F90:381-403 from the step sizes (read-only)
__device__ __forceinline__ void ab3_coefs(const DevScalars *ds, double *c)
{
    const double dt = ds->dt;
    if (ds->first) {
        c[0] = dt; c[1] = 0.0; c[2] = 0.0;
    } else if (ds->second) {
        c[0] = dt * (1.0 + 0.5 * (dt / ds->dt1));
        c[1] = -0.5 * dt * (dt / ds->dt1);
        c[2] = 0.0;
    } else {
        const double dt1 = ds->dt1, dt2 = ds->dt2;
        c[0] = dt + (((dt * dt) / (dt1 * dt2)) * ((dt / 3.0) + 0.5 * (dt1 + dt2)));
        c[1] = ((dt * dt) / (dt1 * (dt1 - dt2))) * ((dt / 3.0) + 0.5 * dt2);
        c[2] = -((dt * dt) / (dt2 * (dt1 - dt2))) * ((dt / 3.0) + 0.5 * dt1);
    }
}
// the scalar updates of one step: ttime (:345), the Euler / AB2 start flags
// and dt1, dt2 (:488-489); c are this step's coefficients
__device__ __forceinline__ void ab3_advance(DevScalars *ds, const double *c)
{
    const double dt = ds->dt;
    ds->ttime = ds->ttime + dt;
    if (ds->first) {
        ds->first = 0; ds->second = 1;
        ds->dt1 = 0.0; ds->dt2 = 0.0;
    } else if (ds->second) {
        ds->first = 0; ds->second = 0;
        ds->dt2 = 0.0;
    }
    ds->c0 = c[0]; ds->c1 = c[1]; ds->c2 = c[2];
    ds->dt2 = dt + ds->dt1;
    ds->dt1 = dt;
}

// RHS histories in logical slot order (0 oldest .. 2 newest), kept in device
// memory so that kernels read their slot pointers at run time and a one-
// thread kernel performs the shift of src/main.F90:448-461 by rotating it;
// kernel arguments are then the same on every step (graph capture).
struct HistTable {
    void *p[7][3];          // r, t, u, v, w, pol, tor
    double *bx[3], *by[3];  // bxbardot, bybardot
};

// The arguments of one kernel for each member of a batch: equally sized
// contexts (one grid size of an ensemble) whose step runs as one launch per
// kernel, blockIdx.z picking the member.  A single context is a batch of
// one (NB = 1, member index 0).
#define BATCH_MAX 16
template <typename A, int NB> struct Batch { A a[NB]; };
#define BATCH_MEMBER(bt, NB) ((bt).a[(NB) > 1 ? blockIdx.z : 0])

// First statement of the step's kernels: with programmatic dependent launch
// a kernel may be started while its predecessor in the stream still runs,
// and this waits until every predecessor grid has completed and its memory
// is visible (a no-op for an ordinary launch).
#define PDL_WAIT() asm volatile("griddepcontrol.wait;" ::: "memory")

// ---- error helper --------------------------------------------------------
void vec_set_error(const char *fmt, ...);

#define CUDA_TRY(x)                                                                   \
    do {                                                                              \
        cudaError_t e_ = (x);                                                         \
        if (e_ != cudaSuccess) {                                                      \
            vec_set_error("%s:%d %s: %s", __FILE__, __LINE__, #x, cudaGetErrorString(e_)); \
            return VEC_ERR_CUDA;                                                      \
        }                                                                             \
    } while (0)
