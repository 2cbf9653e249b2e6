// lines_fx.cu -- the FP64 horizontal spectral operators (src/fft.F90): every
// line length 2^a 3^b 5^c, in 64-bit fixed point (fx.cuh).
//
// A group of G = 32 / Q lanes owns a sequence z = a + i b of two real lines in
// shared memory (Q sequences per warp, so that short lines fill it).  The
// forward transform is a chain of radix-8/6/5/4/3/2 passes by decimation in
// frequency, in place, which leaves the spectrum in digit-reversed order; the
// Hermitian multipliers of the operators (+ik, -k^2, 2/3 truncation) are
// stored in that order, and the inverse runs the same passes backwards, so
// that nothing is reordered (only the halfcomplex transforms read or write
// through the permutation).  Passes are synchronised per warp.  x lines:
// warps are independent.  y lines: a CTA's sequences are adjacent columns,
// loaded and stored by all its threads row by row.
//
// Why passes through shared memory rather than 16-point DFTs in registers:
// the work is bound by integer instructions, and with 8 elements a thread
// three times as many warps fit and the code stays in the instruction cache.
// The register form (the FP32 kernel's) issued in 20 % of the cycles, this one
// in 57 % (three CTAs per SM at 80 registers).
//
// Measured at 256^2 x 129, mean of d2bydx and d1bydx: 618 us in FP64 (the FP64
// pipe 83 % busy) -> 168 us, y the same; the 12 passes of an FP64 time step:
// 14.6 -> 7.3 ms; error against long double 2 to 3 times smaller for white
// noise, 10^3 times for a constant plus little.
#include <math.h>
#include <string.h>

#include <vector>

#include "common.cuh"
#include "engine.h"
#include "fx.cuh"

struct FxPack { LineJob<double> j[MAX_JOBS]; };

#define FX_TPB 256

// element i of a sequence's buffer: the eight 16-byte words of a 128-byte row
// are permuted by the row (and, y lines, by the sequence), so that strides of
// 2, 4 and 8 elements, and the same element of eight sequences, fall on
// different banks
__device__ __forceinline__ int fx_at(int i, int s7) { return i ^ ((i >> 3) & 7) ^ s7; }

struct FxPassArgs { int n, L, M, G, l, s7; unsigned mg; const TwX *tw; };

// one decimation-in-frequency pass: DFT_R over the elements j + m M of every
// block of L, then W_L^(j r) / 2.  FIRST: the elements are (a - mean) 2^sh.
template <int R, bool FIRST>
__device__ __forceinline__ void fx_fwd(X2 *buf, const FxPassArgs &a, long long mx, long long my, int sh)
{
    for (int b = a.l; b < a.n / R; b += a.G) {
        const int q = (int)(((unsigned long long)(unsigned)b * a.mg) >> 31), j = b - q * a.M;
        int at[R];
        X2 v[R];
#pragma unroll
        for (int m = 0; m < R; m++) {
            at[m] = fx_at(q * a.L + j + m * a.M, a.s7);
            v[m] = buf[at[m]];
            if (FIRST) { v[m].x = fx_shift(v[m].x - mx, sh); v[m].y = fx_shift(v[m].y - my, sh); }
        }
        XDft<R, false>::run(v);
        buf[at[0]] = a.M > 1 ? fx_half(v[0]) : v[0];
#pragma unroll
        for (int r = 1; r < R; r++) buf[at[r]] = a.M > 1 ? fx_mulc(v[r], a.tw[(r - 1) * a.M + j]) : v[r];
    }
    __syncwarp();
}
// the reverse: conj(W_L^(j r)) / 2, then the inverse DFT_R.  MUL: the elements
// are those of src times 2^(d - 1) and the multiplier (i times it for D1).
template <int R, bool MUL>
__device__ __forceinline__ void fx_inv(X2 *buf, const X2 *src, const FxPassArgs &a, const int2 *mul, bool d1, int d)
{
    for (int b = a.l; b < a.n / R; b += a.G) {
        const int q = (int)(((unsigned long long)(unsigned)b * a.mg) >> 31), j = b - q * a.M;
        int at[R];
        X2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int i = q * a.L + j + r * a.M;
            at[r] = fx_at(i, a.s7);
            if (MUL) {
                const X2 z = src[at[r]];
                const int2 m = __ldg(mul + i);
                const long long p = fx_muls(z.x, m.x, m.y, d), w = fx_muls(z.y, m.x, m.y, d);
                v[r].x = d1 ? -w : p;
                v[r].y = d1 ? p : w;
            } else {
                v[r] = buf[at[r]];
                if (r == 0) v[r] = a.M > 1 ? fx_half(v[r]) : v[r];
                else if (a.M > 1) v[r] = fx_mulcj(v[r], a.tw[(r - 1) * a.M + j]);
            }
        }
        XDft<R, true>::run(v);
#pragma unroll
        for (int r = 0; r < R; r++) buf[at[r]] = v[r];
    }
    __syncwarp();
}

#define FX_RADIX(R, CALL)                                                                  \
    switch (R) {                                                                           \
    case 8: { constexpr int RR = 8; CALL; break; }                                         \
    case 6: { constexpr int RR = 6; CALL; break; }                                         \
    case 5: { constexpr int RR = 5; CALL; break; }                                         \
    case 4: { constexpr int RR = 4; CALL; break; }                                         \
    case 3: { constexpr int RR = 3; CALL; break; }                                         \
    default: { constexpr int RR = 2; CALL; break; }                                        \
    }

// what the store of a sequence needs (y lines: through shared memory)
struct FxOut { double cx, cy; int xe, nonfin; };

// DIR 0: x lines (sequence = two rows), DIR 1: y lines (two columns).  tpp
// tiles per plane: of Q sequences (one warp's, x) or S = warps Q (a CTA's, y).
template <int DIR>
__global__ void __launch_bounds__(FX_TPB, 3)
line_fx(const __grid_constant__ FxPack jobs, const __grid_constant__ FxPlan pl, FxTables tb, int nx, int ny, int nz,
        int tpp, int total, int two)
{
    PDL_WAIT();
    extern __shared__ __align__(128) unsigned char smem[];
    const int n = pl.n, Q = pl.Q, G = 32 / Q, W = (int)blockDim.x / 32, S = W * Q;
    TwX *tw = reinterpret_cast<TwX *>(smem);
    X2 *bufA = reinterpret_cast<X2 *>(tw + pl.ntw);
    X2 *bufB = bufA + (size_t)S * pl.nb;               // (two)
    FxOut *so = reinterpret_cast<FxOut *>(bufB + (two ? (size_t)S * pl.nb : 0));
    const int tid = threadIdx.x, wid = tid >> 5, g = (tid & 31) / G, l = (tid & 31) % G;
    const int s = wid * Q + g;
    const int s7 = DIR == 1 ? s & 7 : 0;
    X2 *A = bufA + (size_t)s * pl.nb, *B = two ? bufB + (size_t)s * pl.nb : A;
    const size_t np = (size_t)nx * ny;
    const int pairs = (DIR == 0 ? ny : nx) / 2;

    for (int e = tid; e < pl.ntw; e += blockDim.x) tw[e] = tb.tw[e];
    __syncthreads();
    auto args = [&](int p) {
        FxPassArgs a;
        a.n = n; a.L = pl.L[p]; a.M = pl.M[p]; a.G = G; a.l = l; a.s7 = s7; a.mg = pl.mg[p]; a.tw = tw + pl.tw[p];
        return a;
    };
    const int t0 = DIR == 0 ? blockIdx.x * W + wid : blockIdx.x, dt = DIR == 0 ? gridDim.x * W : gridDim.x;
    for (int t = t0; t < total; t += dt) {
        const int job = t / (nz * tpp), rem = t - job * (nz * tpp);
        const int plane = rem / tpp, tile = rem - plane * tpp;
        const LineJob<double> &jb = jobs.j[job];
        const int op1 = jb.op1, op2 = jb.op2;
        const size_t pb = (size_t)plane * np;
        const int pair = tile * (DIR == 0 ? Q : S) + (DIR == 0 ? g : s);     // this group's lines 2 pair, 2 pair + 1
        const bool valid = pair < pairs;

        // ---- load the bits
        unsigned mxh = 0u;
        if (DIR == 0) {
            const double *r0 = jb.in + pb + (size_t)(valid ? 2 * pair : 0) * nx, *r1 = r0 + nx;
            for (int e0 = l; e0 < n; e0 += 8 * G) {
                X2 v[8];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int e = e0 + c * G;
                    const bool in = valid && e < n;
                    v[c].x = in ? __double_as_longlong(r0[e]) : 0;
                    v[c].y = in ? __double_as_longlong(r1[e]) : 0;
                }
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int e = e0 + c * G;
                    if (e >= n) break;
                    mxh = max(mxh, (unsigned)fx_hi(v[c].x) & 0x7fffffffu);
                    mxh = max(mxh, (unsigned)fx_hi(v[c].y) & 0x7fffffffu);
                    A[fx_at(e, s7)] = v[c];
                }
            }
        } else {
            const int ls = 31 - __clz(S);
            const double *in = jb.in + pb + 2 * (size_t)tile * S;
            for (int i0 = tid; i0 < n * S; i0 += 8 * (int)blockDim.x) {
                double2 v[8];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int i = i0 + c * (int)blockDim.x, e = i >> ls, q = i & (S - 1);
                    v[c] = i < n * S && tile * S + q < pairs ? *reinterpret_cast<const double2 *>(in + (size_t)e * nx + 2 * q)
                                                             : make_double2(0.0, 0.0);
                }
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int i = i0 + c * (int)blockDim.x, e = i >> ls, q = i & (S - 1);
                    if (i < n * S) *reinterpret_cast<double2 *>(bufA + (size_t)q * pl.nb + fx_at(e, q & 7)) = v[c];
                }
            }
            __syncthreads();
            for (int e = l; e < n; e += G) {
                const X2 v = A[fx_at(e, s7)];
                mxh = max(mxh, (unsigned)fx_hi(v.x) & 0x7fffffffu);
                mxh = max(mxh, (unsigned)fx_hi(v.y) & 0x7fffffffu);
            }
        }
        for (int o = G >> 1; o > 0; o >>= 1) mxh = max(mxh, __shfl_xor_sync(0xffffffffu, mxh, o));
        const int E = (int)max(mxh >> 20, 1u);
        FxOut out;
        out.nonfin = E == 0x7ff;
        out.cx = out.cy = 0.0;

        // ---- to integers; the mean of a real line, or a spectrum's constant, off
        int sx = 0, sy = 0;
        const bool low = E < 64;
        const bool inv = op1 == OP_INV;
        double dcx = 0.0, dcy = 0.0;
        for (int e = l; e < n; e += G) {
            X2 v = A[fx_at(e, s7)];
            if (inv && e == 0) {
                dcx = __longlong_as_double(v.x);
                dcy = __longlong_as_double(v.y);
                v.x = v.y = 0;
            }
            if (low) {
                v.x = fx_from_low((unsigned)fx_hi(v.x), (unsigned)v.x, E);
                v.y = fx_from_low((unsigned)fx_hi(v.y), (unsigned)v.y, E);
            } else {
                v.x = fx_from((unsigned)fx_hi(v.x), (unsigned)v.x, E);
                v.y = fx_from((unsigned)fx_hi(v.y), (unsigned)v.y, E);
            }
            sx += fx_hi(v.x) >> 9;
            sy += fx_hi(v.y) >> 9;
            A[fx_at(e, s7)] = v;
        }
        long long mx = 0, my = 0;
        if (inv) {
            const int src = (tid & 31) - l;
            out.cx = __shfl_sync(0xffffffffu, dcx, src) / (double)n;
            out.cy = __shfl_sync(0xffffffffu, dcy, src) / (double)n;
        } else {
            for (int o = G >> 1; o > 0; o >>= 1) {
                sx += __shfl_xor_sync(0xffffffffu, sx, o);
                sy += __shfl_xor_sync(0xffffffffu, sy, o);
            }
            // (to 21 bits, a multiple of 2^41 units)
            mx = (long long)(int)((float)sx * pl.rn) << 41;
            my = (long long)(int)((float)sy * pl.rn) << 41;
            const int ex = E - 1084;
            out.cx = fx_to(mx, ex, fx_safe(ex));
            out.cy = fx_to(my, ex, fx_safe(ex));
        }
        // ---- the norm and with it the exponent
        long long ss = 0;
        for (int e = l; e < n; e += G) {
            const X2 v = A[fx_at(e, s7)];
            const int qx = fx_hi(v.x - mx) >> 4, qy = fx_hi(v.y - my) >> 4;
            ss += fx_wide(qx, qx) + fx_wide(qy, qy);
        }
        auto log2sum = [&](long long v) {
            float f = (float)v;
            for (int o = G >> 1; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
            return fx_log2(f);
        };
        // (a halfcomplex element stands for two of the spectrum)
        const int K = log2sum(ss) + (inv ? 1 : 0);
        const int sh = min(25 - pl.gb - ((K + 1) >> 1), 15);
        const int F = E - 1084 - sh;
        __syncwarp();

        if (!inv) {
            { const FxPassArgs a = args(0); FX_RADIX(pl.R[0], (fx_fwd<RR, true>(A, a, mx, my, sh))) }
            for (int p = 1; p < pl.np; p++) { const FxPassArgs a = args(p); FX_RADIX(pl.R[p], (fx_fwd<RR, false>(A, a, 0, 0, 0))) }
        }

        if (op1 == OP_FWD) {
            // separate Z into the halfcomplex spectra of the two real lines
            out.xe = F + pl.halvings - 1;
            const bool scale = jb.alpha1 != 1.0;
            auto sep = [&](const X2 *Z, int z7, int p, const FxOut &o, bool safe, double *va, double *vb) {
                const X2 zp = Z[fx_at(__ldg(tb.pos + p), z7)], zq = Z[fx_at(__ldg(tb.pos + (p == 0 ? 0 : n - p)), z7)];
                const bool re = 2 * p <= n;
                *va = fx_to(re ? zp.x + zq.x : zq.y - zp.y, o.xe, safe);
                *vb = fx_to(re ? zp.y + zq.y : zp.x - zq.x, o.xe, safe);
                if (p == 0) { *va += (double)n * o.cx; *vb += (double)n * o.cy; }
                if (o.nonfin) *va = *vb = FX_NAN;
                if (scale) { *va *= jb.alpha1; *vb *= jb.alpha1; }
            };
            if (DIR == 0) {
                if (valid) {
                    double *oa = jb.out1 + pb + 2 * (size_t)pair * nx, *ob = oa + nx;
                    const bool safe = fx_safe(out.xe);
                    for (int p = l; p < n; p += G) {
                        double va, vb;
                        sep(A, s7, p, out, safe, &va, &vb);
                        oa[p] = jb.acc1 ? oa[p] + va : va;
                        ob[p] = jb.acc1 ? ob[p] + vb : vb;
                    }
                }
                __syncwarp();
            } else {
                if (l == 0) so[s] = out;
                __syncthreads();
                const int ls = 31 - __clz(S);
                double *op = jb.out1 + pb + 2 * (size_t)tile * S;
                for (int i = tid; i < n * S; i += (int)blockDim.x) {
                    const int p = i >> ls, q = i & (S - 1);
                    if (tile * S + q >= pairs) continue;
                    const FxOut o = so[q];
                    double2 v;
                    sep(bufA + (size_t)q * pl.nb, q & 7, p, o, fx_safe(o.xe), &v.x, &v.y);
                    double2 *d = reinterpret_cast<double2 *>(op + (size_t)p * nx + 2 * q);
                    if (jb.acc1) { const double2 w = *d; v.x = w.x + v.x; v.y = w.y + v.y; }
                    *d = v;
                }
                __syncthreads();
            }
            continue;
        }

        const int nout = op2 != OP_NONE && (!inv || op2 == OP_D1) ? 2 : 1;
        for (int o = 0; o < nout; o++) {
            const int op = o == 0 ? op1 : op2;
            const X2 *src = A;
            X2 *dst = o + 1 < nout ? B : A;
            int sh1 = 0;               // exponent of the multiplier step
            if (inv) {
                // Z_k = A_k + i B_k from the halfcomplex lines a (re), b (im),
                // into the digit-reversed order of the passes
                for (int i = l; i < n; i += G) {
                    const int k = __ldg(tb.kof + i), kk = 2 * k <= n ? k : n - k;
                    const bool edge = kk == 0 || 2 * kk == n;
                    X2 pa = A[fx_at(kk, s7)], pbb = A[fx_at(edge ? 0 : n - kk, s7)];
                    if (edge) pbb.x = pbb.y = 0;
                    pa.x = fx_shift(pa.x, sh); pa.y = fx_shift(pa.y, sh);
                    pbb.x = fx_shift(pbb.x, sh); pbb.y = fx_shift(pbb.y, sh);
                    if (2 * k > n) { pbb.x = -pbb.x; pbb.y = -pbb.y; }
                    X2 z;
                    z.x = pa.x - pbb.y;
                    z.y = pbb.x + pa.y;
                    B[fx_at(i, s7)] = z;
                }
                __syncwarp();
                src = dst = B;
            }
            const int2 *mul = op == OP_D1 ? tb.m1 : op == OP_D2 ? tb.m2 : tb.mda;
            int d = 1 - pl.gb;
            if (op == OP_D1 || op == OP_D2) {
                // the spectrum's norm from a quarter of the products to 27 bits
                long long sy2 = 0;
                for (int i = l; i < n; i += G) {
                    const X2 z = src[fx_at(i, s7)];
                    const int m = __ldg(&mul[i].x);
                    const int qx = fx_hi(fx_wide(fx_hi(z.x), m)), qy = fx_hi(fx_wide(fx_hi(z.y), m));
                    sy2 += fx_wide(qx, qx) + fx_wide(qy, qy);
                }
                d = min(max(28 - pl.gb - ((log2sum(sy2) + 1) >> 1), -1), 20);
                __syncwarp();
            }
            int p = pl.np - 1;
            if (op != OP_INV || !pl.pow2) {
                sh1 = 1 - d + (op == OP_D1 ? tb.p1 : op == OP_D2 ? tb.p2 : op == OP_INV ? tb.pinv : tb.pda);
                const int2 *mm = op == OP_INV ? tb.minv : mul;
                const FxPassArgs a = args(p);
                FX_RADIX(pl.R[p], (fx_inv<RR, true>(dst, src, a, mm, op == OP_D1, d)))
                p--;
            } else {
                sh1 = tb.pinv;
            }
            for (; p >= 0; p--) { const FxPassArgs a = args(p); FX_RADIX(pl.R[p], (fx_inv<RR, false>(dst, dst, a, nullptr, false, 0))) }

            out.xe = F + sh1 + (inv ? 1 : 2) * pl.halvings;
            const double alpha = o == 0 ? jb.alpha1 : jb.alpha2;
            const int acc = o == 0 ? jb.acc1 : jb.acc2;
            double *ot = o == 0 ? jb.out1 : jb.out2;
            // what is added back: the mean of a dealiased line, the constant of an
            // inverse and its addk, addc
            const bool con = op == OP_DEALIAS || op == OP_INV;
            double addv = 0.0;
            if (op == OP_INV) addv = (jb.addk ? jb.addk[plane] : 0.0) + jb.addc;
            // (what is only stored takes loops of its own: FP64 operations,
            // predicated off or not, would keep the FP64 pipe busier than the
            // conversions do)
            const bool store = !acc && alpha == 1.0;
            if (store && op == OP_INV) { out.cx += addv; out.cy += addv; }
            auto fin = [&](const X2 v, const FxOut &q, const double *old, double *va, double *vb, size_t step) {
                const bool safe = fx_safe(q.xe);
                *va = fx_to(v.x, q.xe, safe);
                *vb = fx_to(v.y, q.xe, safe);
                if (con) { *va += q.cx; *vb += q.cy; }
                if (q.nonfin) *va = *vb = FX_NAN;
                *va *= alpha;
                *vb *= alpha;
                if (acc) { *va = old[0] + *va; *vb = old[step] + *vb; }
                if (op == OP_INV && !store) { *va += addv; *vb += addv; }
            };
            if (DIR == 0) {
                double *oa = ot + pb + 2 * (size_t)pair * nx, *ob = oa + nx;
                if (valid && store && !out.nonfin && fx_safe(out.xe)) {
                    if (con)
                        for (int e = l; e < n; e += G) {
                            const X2 v = dst[fx_at(e, s7)];
                            oa[e] = fx_to(v.x, out.xe, true) + out.cx;
                            ob[e] = fx_to(v.y, out.xe, true) + out.cy;
                        }
                    else
                        for (int e = l; e < n; e += G) {
                            const X2 v = dst[fx_at(e, s7)];
                            oa[e] = fx_to(v.x, out.xe, true);
                            ob[e] = fx_to(v.y, out.xe, true);
                        }
                } else if (valid) {
                    for (int e = l; e < n; e += G) {
                        double va, vb;
                        fin(dst[fx_at(e, s7)], out, oa + e, &va, &vb, nx);
                        oa[e] = va;
                        ob[e] = vb;
                    }
                }
                __syncwarp();
            } else {
                if (l == 0) so[s] = out;
                const bool fast = __syncthreads_and(store && !out.nonfin && fx_safe(out.xe));
                const int ls = 31 - __clz(S), q = tid & (S - 1);     // (S divides the CTA: one sequence per thread)
                const X2 *bs = (dst == A ? bufA : bufB) + (size_t)q * pl.nb;
                double *od = ot + pb + 2 * ((size_t)tile * S + q);
                if (tile * S + q < pairs) {
                    const FxOut f = so[q];
                    if (fast && con) {
                        for (int e = tid >> ls; e < n; e += (int)blockDim.x >> ls) {
                            const X2 v = bs[fx_at(e, q & 7)];
                            *reinterpret_cast<double2 *>(od + (size_t)e * nx) =
                                make_double2(fx_to(v.x, f.xe, true) + f.cx, fx_to(v.y, f.xe, true) + f.cy);
                        }
                    } else if (fast) {
                        for (int e = tid >> ls; e < n; e += (int)blockDim.x >> ls) {
                            const X2 v = bs[fx_at(e, q & 7)];
                            *reinterpret_cast<double2 *>(od + (size_t)e * nx) = make_double2(fx_to(v.x, f.xe, true), fx_to(v.y, f.xe, true));
                        }
                    } else {
                        for (int e = tid >> ls; e < n; e += (int)blockDim.x >> ls) {
                            double *dd = od + (size_t)e * nx;
                            double2 v;
                            fin(bs[fx_at(e, q & 7)], f, dd, &v.x, &v.y, 1);
                            *reinterpret_cast<double2 *>(dd) = v;
                        }
                    }
                }
                __syncthreads();
            }
        }
    }
}

// ---- host side ------------------------------------------------------------------
// v with 62 fractional bits as a high word and a signed low word (that is not
// INT32_MIN: the kernels negate it)
static FxConst fx_const(long double v)
{
    long long q = llroundl(v * 0x1p62L);
    if ((int)q == INT32_MIN) q++;
    FxConst c;
    c.l = (int)q;
    c.h = (int)((q - (int)q) >> 32);
    return c;
}
// exp(-2 pi i e/n) in long double, exact at the quadrants
static TwX tw_unit(long e, long n)
{
    e %= n;
    const long q = (4 * e) / n, r = 4 * e - q * n;     // quadrant, and the angle (pi/2) r/n in it
    const long double h = 1.57079632679489661923132169163975144L;
    long double c, s;
    if (2 * r <= n) { c = cosl(h * (long double)r / n); s = sinl(h * (long double)r / n); }
    else { c = sinl(h * (long double)(n - r) / n); s = cosl(h * (long double)(n - r) / n); }
    const long double cc[4] = { c, -s, -c, s }, ss[4] = { s, c, -s, -c };
    const FxConst x = fx_const(cc[q]), y = fx_const(-ss[q]);
    return TwX{ x.h, x.l, y.h, y.l };
}

int line_fx_configure()
{
    const long double h = 3.14159265358979323846264338327950288L;
    const FxConst r8 = fx_const(cosl(h / 4)), r3 = fx_const(sinl(h / 3));
    const FxConst c5 = fx_const((cosl(2 * h / 5) - cosl(4 * h / 5)) / 2), sa = fx_const(sinl(2 * h / 5)), sb = fx_const(sinl(4 * h / 5));
    CUDA_TRY(cudaMemcpyToSymbol(c_fx_r8, &r8, sizeof(r8)));
    CUDA_TRY(cudaMemcpyToSymbol(c_fx_r3, &r3, sizeof(r3)));
    CUDA_TRY(cudaMemcpyToSymbol(c_fx_c5, &c5, sizeof(c5)));
    CUDA_TRY(cudaMemcpyToSymbol(c_fx_s5a, &sa, sizeof(sa)));
    CUDA_TRY(cudaMemcpyToSymbol(c_fx_s5b, &sb, sizeof(sb)));
    return VEC_OK;
}

// the radices of n with the fewest passes, larger ones first
static bool radices(int n, std::vector<int> &r)
{
    static const int all[] = { 8, 6, 5, 4, 3, 2 };
    std::vector<int> best;
    std::vector<int> cur;
    auto go = [&](auto &self, int m, int from) -> void {
        if (!best.empty() && cur.size() >= best.size()) return;
        if (m == 1) { best = cur; return; }
        for (int q = from; q < 6; q++)
            if (m % all[q] == 0) {
                cur.push_back(all[q]);
                self(self, m / all[q], q);
                cur.pop_back();
            }
    };
    go(go, n, 0);
    r = best;
    return !r.empty();
}

int fx_plan_make(int n, FxPlan *pl)
{
    *pl = FxPlan{};
    std::vector<int> r;
    if (n > 2048 || !radices(n, r) || r.size() > 6) return VEC_ERR_SIZE;
    pl->n = n;
    pl->nb = (n + 7) & ~7;
    pl->np = (int)r.size();
    pl->rn = 1.0f / (float)n;
    pl->pow2 = (n & (n - 1)) == 0;
    int L = n;
    double P = 1.0, top = 0.0;     // growth sqrt(P) 2^-halvings
    for (int p = 0; p < pl->np; p++) {
        const int R = r[p], M = L / R;
        pl->R[p] = R; pl->L[p] = L; pl->M[p] = M;
        pl->mg[p] = (unsigned)(((1ull << 31) + M - 1) / M);
        pl->tw[p] = pl->ntw;
        if (M > 1) pl->ntw += (R - 1) * M;
        // sums inside the radix: 2 x 4 and 3 x 2 with a halving between
        const int in[2] = { R == 8 ? 2 : R == 6 ? 3 : R, R == 8 ? 4 : R == 6 ? 2 : 1 };
        for (int q = 0; q < 2; q++) {
            P *= in[q];
            top = fmax(top, sqrt(P) * exp2(-(double)pl->halvings));
            if (q == 0 && in[1] > 1) pl->halvings++;
        }
        if (p + 1 < pl->np) pl->halvings++;
        L = M;
    }
    // (the inverse takes the radices backwards: the same bound on its growth
    // from the other end)
    P = 1.0;
    int h = 0;
    for (int p = pl->np - 1; p >= 0; p--) {
        const int R = r[p], in[2] = { R == 8 ? 2 : R == 6 ? 3 : R, R == 8 ? 4 : R == 6 ? 2 : 1 };
        for (int q = 0; q < 2; q++) {
            P *= in[q];
            top = fmax(top, sqrt(P) * exp2(-(double)h));
            if (q == 0 && in[1] > 1) h++;
        }
        h++;
    }
    pl->gb = top <= 2.0 ? 1 : 2;
    if (top > 4.0) return VEC_ERR_SIZE;
    // sequences per warp: about 256 elements, at least four lanes each
    pl->Q = n <= 32 ? 8 : n <= 64 ? 4 : n <= 128 ? 2 : 1;
    return VEC_OK;
}

// the tables of one direction: the twiddles of each pass, the order of the
// spectrum, and the multipliers of line_tables_make in that order, scaled by a
// power of two per table to at most one in magnitude
int fx_tables_make(int n, const FxPlan &pl, const double *k1, const double *k2, int icut, FxTables *tb)
{
    std::vector<TwX> tw;
    for (int p = 0; p < pl.np; p++)
        if (pl.M[p] > 1)
            for (int r = 1; r < pl.R[p]; r++)
                for (int j = 0; j < pl.M[p]; j++) tw.push_back(tw_unit((long)j * r, pl.L[p]));
    std::vector<unsigned short> pos(n), kof(n);
    for (int k = 0; k < n; k++) {
        int rest = k, at = 0;
        for (int p = 0; p < pl.np; p++) {
            at += (rest % pl.R[p]) * pl.M[p];
            rest /= pl.R[p];
        }
        pos[k] = (unsigned short)at;
        kof[at] = (unsigned short)k;
    }
    std::vector<long double> m[4];
    for (auto &v : m) v.assign(n, 0.0L);
    for (int e = 0; e < n; e++) {
        if (e > 0 && 2 * e < n) m[0][e] = (long double)k1[e] / n;
        else if (2 * e > n) m[0][e] = -(long double)k1[e] / n;
        if (e) m[1][e] = (long double)k2[e] / n;
        const int kk = e <= n / 2 ? e : n - e;
        m[2][e] = kk >= n / 2 - icut ? 0.0L : 1.0L / n;
        m[3][e] = 1.0L / n;
    }
    int2 **dst[4] = { &tb->m1, &tb->m2, &tb->mda, &tb->minv };
    int *px[4] = { &tb->p1, &tb->p2, &tb->pda, &tb->pinv };
    auto up = [](void **d, const void *s, size_t bytes) {
        if (cudaMalloc(d, bytes ? bytes : 16) != cudaSuccess) { cudaGetLastError(); return (int)VEC_ERR_ALLOC; }
        return cudaMemcpy(*d, s, bytes, cudaMemcpyHostToDevice) == cudaSuccess ? (int)VEC_OK : (int)VEC_ERR_CUDA;
    };
    int st;
    if ((st = up((void **)&tb->tw, tw.data(), tw.size() * sizeof(TwX))) ||
        (st = up((void **)&tb->pos, pos.data(), n * sizeof(short))) || (st = up((void **)&tb->kof, kof.data(), n * sizeof(short))))
        return st;
    for (int t = 0; t < 4; t++) {
        long double mx = 0.0L;
        for (auto v : m[t]) mx = fmaxl(mx, fabsl(v));
        int p = 0;
        if (mx > 0.0L && frexpl(mx, &p) == 0.5L) p--;     // mx = f 2^p, f in (1/2, 1]
        *px[t] = p;
        std::vector<int2> q(n);
        for (int i = 0; i < n; i++) {
            const FxConst c = fx_const(ldexpl(m[t][kof[i]], -p));
            q[i] = make_int2(c.h, c.l);
        }
        if ((st = up((void **)dst[t], q.data(), n * sizeof(int2)))) return st;
    }
    return VEC_OK;
}
void fx_tables_free(FxTables *tb)
{
    cudaFree(tb->tw); cudaFree(tb->m1); cudaFree(tb->m2); cudaFree(tb->mda); cudaFree(tb->minv);
    cudaFree(tb->pos); cudaFree(tb->kof);
    *tb = FxTables{};
}

template <int DIR>
static int run_fx(Engine *E, const LineJob<double> *jobs, int nj)
{
    const FxPlan &pl = DIR == 0 ? E->fpx : E->fpy;
    FxPack pk;
    memset(&pk, 0, sizeof(pk));
    double fields = 0.0;
    int two = 0;                   // a second buffer per sequence
    for (int j = 0; j < nj; j++) {
        pk.j[j] = jobs[j];
        fields += 2.0 + (jobs[j].acc1 ? 1.0 : 0.0);
        if (jobs[j].op2 != OP_NONE) fields += 1.0 + (jobs[j].acc2 ? 1.0 : 0.0);
        if (jobs[j].op2 != OP_NONE || jobs[j].op1 == OP_INV) two = 1;
    }
    const int pairs = (DIR == 0 ? E->ny : E->nx) / 2;
    // warps per CTA: 8, fewer where the buffers do not fit half an SM or where
    // there would be less than a CTA per SM
    int W = FX_TPB / 32;
    auto smem_of = [&](int w) {
        const size_t S = (size_t)w * pl.Q;
        return sizeof(TwX) * pl.ntw + S * pl.nb * sizeof(X2) * (two ? 2 : 1) + S * sizeof(FxOut) + 16;
    };
    auto tiles_of = [&](int w) {
        const int S = DIR == 0 ? pl.Q : w * pl.Q;
        return (long long)nj * E->nz * ((pairs + S - 1) / S);
    };
    while (W > 1 && (smem_of(W) > 75 * 1024 || (DIR == 0 ? tiles_of(W) / W : tiles_of(W)) < E->num_sms)) W >>= 1;
    const size_t smem = smem_of(W);
    static bool attr = false;
    if (!attr) {
        CUDA_TRY(cudaFuncSetAttribute(line_fx<DIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        attr = true;
    }
    if (smem > 226 * 1024) return VEC_ERR_SIZE;
    int per_sm = 1;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, line_fx<DIR>, W * 32, smem));
    if (per_sm < 1) per_sm = 1;
    const int S = DIR == 0 ? pl.Q : W * pl.Q, tpp = (pairs + S - 1) / S;
    const long long total = tiles_of(W);
    long long grid = DIR == 0 ? (total + W - 1) / W : total;
    if (grid > (long long)E->num_sms * per_sm) grid = (long long)E->num_sms * per_sm;
    E->prof_begin(DIR == 0 ? "line_x_f64" : "line_y_f64", fields * (double)E->n * 8.0);
    CUDA_TRY(launch_k(*E, line_fx<DIR>, dim3((unsigned)grid), dim3(W * 32), smem, pk, pl, DIR == 0 ? E->fxx : E->fxy, E->nx,
                      E->ny, E->nz, tpp, (int)total, two));
    E->prof_end();
    CUDA_TRY(cudaGetLastError());
    return VEC_OK;
}

template <>
int launch_lines<double>(Engine *E, int dir, const LineJob<double> *jobs, int njobs)
{
    for (int j0 = 0; j0 < njobs; j0 += MAX_JOBS) {
        const int nj = njobs - j0 < MAX_JOBS ? njobs - j0 : MAX_JOBS;
        const int st = dir == 0 ? run_fx<0>(E, jobs + j0, nj) : run_fx<1>(E, jobs + j0, nj);
        if (st) return st;
    }
    return VEC_OK;
}
