// lines_fx.cu -- the FP64 horizontal spectral operators (src/fft.F90): every
// line length 2^a 3^b 5^c, in 64-bit fixed point (fx.cuh).
//
// A group of G = 32 / Q lanes owns a sequence z = a + i b of two real lines in
// shared memory (Q sequences per warp, so that short lines fill it).  The
// forward transform is a chain of radix-8/6/5/4/3/2 passes by decimation in
// frequency, in place, which leaves the spectrum in digit-reversed order; the
// Hermitian multipliers of the operators (+ik, -k^2, 2/3 truncation) are
// applied in that order, and the inverse runs the same passes backwards, so
// that nothing is reordered (only the halfcomplex transforms read or write
// through the permutation).  Passes are synchronised per warp.  x lines:
// warps are independent.  y lines: a CTA's sequences are adjacent columns,
// loaded and stored by all its threads row by row.
//
// Why passes through shared memory rather than 16-point DFTs in registers:
// the work is bound by integer instructions, and with 8 elements a thread three
// times as many warps fit (three CTAs per SM at 80 registers).  The register form
// (lines_ct.cu's, on integers) issued in 20 % of the cycles.
//
// Measured at 256^2 x 129, mean of d2bydx and d1bydx: 618 us in FP64 (the FP64
// pipe 83 % busy) -> 150 us, y the same.  (168 us with every element's place
// computed, a table of multipliers, and x results stored by a loop of their
// own.)  It issues in 45 % of the cycles, the rest being instruction fetches and
// the latency of shared memory and conversions; synchronising the passes of a
// CTA's warps, so that they fetch the same code, changed nothing, nor did rolled
// loops of twiddle products (13 % less code).  Error (rms) of
// derivatives against long double, in parts of that of the register FFT in FP64: 0.3 to
// 0.5 for white noise, 0.1 to 0.5 for lines of few waves, 10^-3 to 4 10^-3 for a constant plus
// 1 % of waves.
#include <math.h>
#include <string.h>

#include <type_traits>
#include <vector>

#include "common.cuh"
#include "engine.h"
#include "fx.cuh"

template <int NJ> struct FxPack { LineJob<double> j[NJ]; };

#define FX_TPB 256
// lines above that many points: lines_fx_long.cu, which compiles this file once more
#define FX_SHORT 512

// element i of a sequence's buffer: the eight 16-byte words of a 128-byte row
// are permuted by the row (and, y lines, by the sequence), so that strides of
// 2, 4 and 8 elements, and the same element of eight sequences, fall on
// different banks
__device__ __forceinline__ int fx_at(int i, int s7) { return i ^ ((i >> 3) & 7) ^ s7; }

// One pass of a sequence: radix R over the elements j + m M of every block of
// L = R M.  KIND: how the elements' places in the buffer follow from the first's
// (the permutation of fx_at costs three instructions per element in general):
// K64: M a multiple of 64, K8: R = M = 8, K1: R = 8, M = 1.
enum { KG, K64, K8, K1 };
struct FxPassArgs { int n, L, M, G, l, s7, up; unsigned mg; const TwX *tw; };
// the value that a pass takes its twiddle product of (which halves it), and the one it
// halves itself; long lines leave some halvings out
__device__ __forceinline__ X2 fx_up(X2 v, const FxPassArgs &a)
{
#if FX_LONG
    v.x <<= a.up;
    v.y <<= a.up;
#endif
    return v;
}
__device__ __forceinline__ X2 fx_half(X2 v, const FxPassArgs &a) { return FX_LONG && a.up ? v : fx_half(v); }

template <int R, int KIND>
__device__ __forceinline__ void fx_places(const FxPassArgs &a, int b, int &j, int *at)
{
    if (KIND == K1) {
        j = 0;
        const int base = 8 * b + ((b & 7) ^ a.s7);
#pragma unroll
        for (int m = 0; m < R; m++) at[m] = base ^ m;
    } else if (KIND == K8) {
        j = b & 7;
        const int base = 8 * (b - j) + (j ^ a.s7);
#pragma unroll
        for (int m = 0; m < R; m++) at[m] = (base ^ m) + 8 * m;
    } else {
        const int q = (int)(((unsigned long long)(unsigned)b * a.mg) >> 31);
        j = b - q * a.M;
        const int i = q * a.L + j;
        at[0] = fx_at(i, a.s7);
#pragma unroll
        for (int m = 1; m < R; m++) at[m] = KIND == K64 ? at[0] + m * a.M : fx_at(i + m * a.M, a.s7);
    }
}
template <int KIND> __device__ __forceinline__ int fx_stride(const FxPassArgs &a) { return KIND == K8 ? 8 : a.M; }

// decimation in frequency: DFT_R, then W_L^(j r) / 2
template <int R, int KIND>
__device__ __forceinline__ void fx_fwd(X2 *buf, const FxPassArgs &a)
{
    const int M = fx_stride<KIND>(a);
    for (int b = a.l; b < a.n / R; b += a.G) {
        int j, at[R];
        X2 v[R];
        fx_places<R, KIND>(a, b, j, at);
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = buf[at[m]];
        XDft<R, false>::run(v);
        buf[at[0]] = fx_half(v[0], a);
        const TwX *w = a.tw + j;
#pragma unroll
        for (int r = 1; r < R; r++) buf[at[r]] = fx_mulc(fx_up(v[r], a), w[(r - 1) * M]);
    }
    __syncwarp();
}
// The last pass (M = 1) has no twiddles.  Its results are the spectrum: with
// key, the sums of |k X|^2 (s1) and |k^2 X|^2 (s2) over it, in units of 2^39
// for X.  (Its element m of butterfly b is wavenumber kof[b R] + m n / R.)
template <int R, int KIND>
__device__ __forceinline__ void fx_last(X2 *buf, const FxPassArgs &a, const unsigned short *kof, bool key, float &s1, float &s2)
{
    for (int b = a.l; b < a.n / R; b += a.G) {
        int j, at[R];
        X2 v[R];
        fx_places<R, KIND>(a, b, j, at);
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = buf[at[m]];
        XDft<R, false>::run(v);
#pragma unroll
        for (int m = 0; m < R; m++) buf[at[m]] = v[m];
        if (key) {
            const int k0 = __ldg(kof + b * R), dk = a.n / R;
#pragma unroll
            for (int m = 0; m < R; m++) {
                const int k = k0 + m * dk;
                const float kf = (float)min(k, a.n - k), x = fx_float((fx_hi(v[m].x) + 64) >> 7), y = fx_float((fx_hi(v[m].y) + 64) >> 7);
                const float p = x * x + y * y, k2 = kf * kf;
                s1 = fmaf(p, k2, s1);
                s2 = fmaf(p * k2, k2, s2);
            }
        }
    }
    __syncwarp();
}
// what the first inverse pass does to the spectrum: the operators' multipliers
// are i k, -k^2 and a mask, up to the constant in the results' scale
__device__ __forceinline__ X2 fx_op(X2 z, int op, int k, int n, int t, int cut)
{
    if (op == OP_INV) return z;
    const int kk = min(k, n - k);
    X2 y;
    if (op == OP_DEALIAS) {
        y.x = kk < cut ? z.x >> t : 0;
        y.y = kk < cut ? z.y >> t : 0;
        return y;
    }
    const bool d1 = op == OP_D1;
    const int m = !d1 ? kk * kk : 2 * k < n ? k : 2 * k == n ? 0 : k - n;
    y.x = fx_mulk(d1 ? z.y : z.x, d1 ? -m : m, t);
    y.y = fx_mulk(d1 ? z.x : z.y, m, t);
    return y;
}
// the reverse of fx_last, from src into buf
template <int R, int KIND>
__device__ __forceinline__ void fx_inv_first(X2 *buf, const X2 *src, const FxPassArgs &a, const unsigned short *kof, int op, int t,
                                             int cut)
{
    for (int b = a.l; b < a.n / R; b += a.G) {
        int j, at[R];
        X2 v[R];
        fx_places<R, KIND>(a, b, j, at);
        const int k0 = op == OP_INV ? 0 : (int)__ldg(kof + b * R), dk = a.n / R;
#pragma unroll
        for (int m = 0; m < R; m++) v[m] = fx_op(src[at[m]], op, k0 + m * dk, a.n, t, cut);
        XDft<R, true>::run(v);
#pragma unroll
        for (int m = 0; m < R; m++) buf[at[m]] = v[m];
    }
    __syncwarp();
}
// conj(W_L^(j r)) / 2, then the inverse DFT_R.  OUT (the last pass of an x line):
// the results times sc to the two rows; plus ca, cb or what the rows hold.
enum { FX_SET, FX_CONST, FX_ACC };
template <int R, int KIND, bool OUT>
__device__ __forceinline__ void fx_inv(X2 *buf, const FxPassArgs &a, double *oa, double *ob, double sc, double ca, double cb, int mode)
{
    const int M = fx_stride<KIND>(a);
    for (int b = a.l; b < a.n / R; b += a.G) {
        int j, at[R];
        X2 v[R];
        fx_places<R, KIND>(a, b, j, at);
        const TwX *w = a.tw + j;
        v[0] = fx_half(buf[at[0]], a);
#pragma unroll
        for (int r = 1; r < R; r++) v[r] = fx_mulcj(fx_up(buf[at[r]], a), w[(r - 1) * M]);
        XDft<R, true>::run(v);
        if (OUT) {
            // (one block: elements j + r M)
            if (mode == FX_ACC) {
                double xa[R], xb[R];
#pragma unroll
                for (int r = 0; r < R; r++) { xa[r] = oa[j + r * M]; xb[r] = ob[j + r * M]; }
#pragma unroll
                for (int r = 0; r < R; r++) {
                    oa[j + r * M] = fma(__ll2double_rn(v[r].x), sc, xa[r]);
                    ob[j + r * M] = fma(__ll2double_rn(v[r].y), sc, xb[r]);
                }
            } else if (mode == FX_CONST) {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    oa[j + r * M] = fma(__ll2double_rn(v[r].x), sc, ca);
                    ob[j + r * M] = fma(__ll2double_rn(v[r].y), sc, cb);
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    oa[j + r * M] = __ll2double_rn(v[r].x) * sc;
                    ob[j + r * M] = __ll2double_rn(v[r].y) * sc;
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; r++) buf[at[r]] = v[r];
        }
    }
    __syncwarp();
}

// a pass's template by its radix and kind
#define FX_SWITCH(pl, p, CALL)                                                             \
    if (pl.kind[p] == K64) {                                                               \
        switch (pl.R[p]) {                                                                 \
        case 8: CALL(8, K64); break;                                                       \
        case 6: CALL(6, K64); break;                                                       \
        case 5: CALL(5, K64); break;                                                       \
        case 4: CALL(4, K64); break;                                                       \
        case 3: CALL(3, K64); break;                                                       \
        default: CALL(2, K64); break;                                                      \
        }                                                                                  \
    } else if (pl.kind[p] == K8) {                                                         \
        CALL(8, K8);                                                                       \
    } else {                                                                               \
        switch (pl.R[p]) {                                                                 \
        case 8: CALL(8, KG); break;                                                        \
        case 6: CALL(6, KG); break;                                                        \
        case 5: CALL(5, KG); break;                                                        \
        case 4: CALL(4, KG); break;                                                        \
        case 3: CALL(3, KG); break;                                                        \
        default: CALL(2, KG); break;                                                       \
        }                                                                                  \
    }
// the last pass: K1 or general
#define FX_SWITCH_LAST(pl, CALL)                                                           \
    if (pl.kind[pl.np - 1] == K1) {                                                        \
        CALL(8, K1);                                                                       \
    } else {                                                                               \
        switch (pl.R[pl.np - 1]) {                                                         \
        case 8: CALL(8, KG); break;                                                        \
        case 6: CALL(6, KG); break;                                                        \
        case 5: CALL(5, KG); break;                                                        \
        case 4: CALL(4, KG); break;                                                        \
        case 3: CALL(3, KG); break;                                                        \
        default: CALL(2, KG); break;                                                       \
        }                                                                                  \
    }

// what the store of a sequence needs (y lines: through shared memory): results
// are integers times sc, plus c; or, where sc would leave the normal range or
// the line is not finite, times con 2^xe
struct FxOut { double cx, cy, sc; int xe, bad; };

// DIR 0: x lines (sequence = two rows), DIR 1: y lines (two columns).  tpp
// tiles per plane: of Q sequences (one warp's, x) or S = warps Q (a CTA's, y).
template <int DIR, int NJ, int LONG>
__global__ void __launch_bounds__(FX_TPB, 3)
line_fx(const __grid_constant__ FxPack<NJ> jobs, const __grid_constant__ FxPlan pl, FxTables tb, int nx, int ny, int nz,
        int tpp, int total, int two)
{
    PDL_WAIT();
    extern __shared__ __align__(128) unsigned char smem[];
    const int n = pl.n, Q = pl.Q, G = 32 / Q, W = (int)blockDim.x / 32, S = W * Q;
    X2 *bufA = reinterpret_cast<X2 *>(smem);
    X2 *bufB = bufA + (size_t)S * pl.nb;               // (two)
    TwX *tw = reinterpret_cast<TwX *>(bufB + (two ? (size_t)S * pl.nb : 0));
    FxOut *so = reinterpret_cast<FxOut *>(tw + pl.ntw);
    const int tid = threadIdx.x, wid = tid >> 5, g = (tid & 31) / G, l = (tid & 31) % G;
    const int s = wid * Q + g;
    const int s7 = DIR == 1 ? s & 7 : 0;
    X2 *A = bufA + (size_t)s * pl.nb, *B = two ? bufB + (size_t)s * pl.nb : A;
    const size_t np = (size_t)nx * ny;
    const int pairs = (DIR == 0 ? ny : nx) / 2;

    for (int e = tid; e < pl.ntw; e += blockDim.x) tw[e] = tb.tw[e];
    __syncthreads();
    auto args = [&](int p, unsigned up) {
        FxPassArgs a;
        a.up = (up >> p) & 1;
        a.n = n; a.L = pl.L[p]; a.M = pl.M[p]; a.G = G; a.l = l; a.s7 = s7; a.mg = pl.mg[p]; a.tw = tw + pl.tw[p];
        return a;
    };
    const int t0 = DIR == 0 ? blockIdx.x * W + wid : blockIdx.x, dt = DIR == 0 ? gridDim.x * W : gridDim.x;
    for (int t = t0; t < total; t += dt) {
        const int job = t / (nz * tpp), rem = t - job * (nz * tpp);
        const int plane = rem / tpp, tile = rem - plane * tpp;
        const LineJob<double> &jb = jobs.j[job];
        const int op1 = jb.op1, op2 = jb.op2;
        const bool inv = op1 == OP_INV;
        const size_t pb = (size_t)plane * np;
        const int pair = tile * (DIR == 0 ? Q : S) + (DIR == 0 ? g : s);     // this group's lines 2 pair, 2 pair + 1
        const bool valid = pair < pairs;

        // ---- y lines: the bits into shared memory, row by row
        const double *r0 = jb.in + pb + (size_t)(valid ? 2 * pair : 0) * nx;
        if (DIR == 1) {
            const int ls = 31 - __clz(S), q = tid & (S - 1), de = (int)blockDim.x >> ls;     // (S divides the CTA)
            const double *in = jb.in + pb + 2 * ((size_t)tile * S + q);
            const bool have = tile * S + q < pairs;
            double2 *to = reinterpret_cast<double2 *>(bufA + (size_t)q * pl.nb);
            for (int e0 = tid >> ls; e0 < n; e0 += 8 * de) {
                double2 v[8];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int e = e0 + c * de;
                    v[c] = have && e < n ? *reinterpret_cast<const double2 *>(in + (size_t)e * nx) : make_double2(0.0, 0.0);
                }
#pragma unroll
                for (int c = 0; c < 8; c++)
                    if (e0 + c * de < n) to[fx_at(e0 + c * de, q & 7)] = v[c];
            }
            __syncthreads();
        }
        auto raw = [&](int e) -> X2 {
            X2 v;
            if (DIR == 0) {
                v.x = valid ? __double_as_longlong(r0[e]) : 0;
                v.y = valid ? __double_as_longlong(r0[e + nx]) : 0;
            } else {
                v = A[fx_at(e, s7)];
            }
            return v;
        };
        // (a spectrum's constant, lane 0's first element, is kept apart; where a derivative
        // is asked for, which does not contain it, it must not set the exponent either)
        double dcx = 0.0, dcy = 0.0;
        auto constant = [&](X2 &v) {
            if (inv && l == 0) {
                dcx = __longlong_as_double(v.x);
                dcy = __longlong_as_double(v.y);
                if (op2 == OP_D1) v.x = v.y = 0;
            }
        };
        // the largest high word; 0 only for a line of zeros (at rest, truncated, or a
        // partial tile's), which takes the exponent of 1 and no slow path
        unsigned low = 0u;
        auto top = [&](unsigned m, const X2 &v) {
            low |= (unsigned)v.x | (unsigned)v.y;
            return max(max(m, (unsigned)fx_hi(v.x) & 0x7fffffffu), (unsigned)fx_hi(v.y) & 0x7fffffffu);
        };
        auto group_max = [&](unsigned m) {
            m = max(m, min(low, 1u));
            for (int o = G >> 1; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            return m == 0 ? 1023 : (int)max(m >> 20, 1u);
        };
        auto group_sum = [&](float f) {
            for (int o = G >> 1; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
            return f;
        };

        // ---- to integers; the mean of a real line, or a spectrum's constant, off;
        // then the norm and with it the exponent F
        FxOut out;
        out.cx = out.cy = 0.0;
        int E = 1, F = 0, sx = 0, sy = 0;
        long long mx = 0, my = 0;
        auto conv = [&](int e, X2 v) {
            if (inv && e == 0) v.x = v.y = 0;
            v.x = fx_from((unsigned)fx_hi(v.x), (unsigned)v.x, E);
            v.y = fx_from((unsigned)fx_hi(v.y), (unsigned)v.y, E);
            sx += fx_hi(v.x) >> 9;
            sy += fx_hi(v.y) >> 9;
            return v;
        };
        auto means = [&]() {
            if (inv) {
                const int src = (tid & 31) - l;
                out.cx = __shfl_sync(0xffffffffu, dcx, src);
                out.cy = __shfl_sync(0xffffffffu, dcy, src);
                // (the division takes zeros on a slow path)
                if (out.cx != 0.0) out.cx /= (double)n;
                if (out.cy != 0.0) out.cy /= (double)n;
                return;
            }
            // (an element is 2^21 at most, a lane's sum 2^27: the line's fits 32 bits up
            // to 1024 elements, and without its last two bits above that)
            const int cut = n > 1024 ? 2 : 0;
            sx >>= cut;
            sy >>= cut;
            for (int o = G >> 1; o > 0; o >>= 1) {
                sx += __shfl_xor_sync(0xffffffffu, sx, o);
                sy += __shfl_xor_sync(0xffffffffu, sy, o);
            }
            // (to 21 bits, a multiple of 2^41 units)
            const float rn = cut ? 4.0f * pl.rn : pl.rn;
            mx = (long long)(int)((float)sx * rn) << 41;
            my = (long long)(int)((float)sy * rn) << 41;
        };
        auto square = [&](const X2 &v) {     // in units of 2^41
            const float x = fx_float(fx_hi(v.x) >> 9), y = fx_float(fx_hi(v.y) >> 9);
            return x * x + y * y;
        };
        auto shift = [&](float sq) {
            // (the squares are of truncated values: 8 n for what they leave out; a
            // halfcomplex element stands for two of the spectrum)
            const int K = fx_log2((sq + 8.0f * (float)n) * (inv ? 2.0f : 1.0f));
            const int sh = 20 - pl.gb - ((K + 1) >> 1);
            F = E - 1084 - sh;
            return sh;
        };
        // (rare: near the bottom of the exponent range, where subnormals count,
        // the elements become integers one by one, in shared memory)
        auto conv_low = [&](int e) {
            X2 v = A[fx_at(e, s7)];
            if (inv && e == 0) v.x = v.y = 0;
            v.x = fx_from_low((unsigned)fx_hi(v.x), (unsigned)v.x, E);
            v.y = fx_from_low((unsigned)fx_hi(v.y), (unsigned)v.y, E);
            sx += fx_hi(v.x) >> 9;
            sy += fx_hi(v.y) >> 9;
            A[fx_at(e, s7)] = v;
        };
        // CH elements per lane in registers
        auto in_registers = [&](auto chunk) {
            constexpr int CH = decltype(chunk)::value;
            X2 v[CH];
            unsigned m = 0u;
#pragma unroll
            for (int c = 0; c < CH; c++) {
                const int e = l + c * G;
                if (e < n) v[c] = raw(e);
                else v[c].x = v[c].y = 0;
            }
            constant(v[0]);
#pragma unroll
            for (int c = 0; c < CH; c++) m = top(m, v[c]);
            E = group_max(m);
            if (E >= 64) {
#pragma unroll
                for (int c = 0; c < CH; c++) v[c] = conv(l + c * G, v[c]);
            } else {
#pragma unroll
                for (int c = 0; c < CH; c++)
                    if (l + c * G < n) A[fx_at(l + c * G, s7)] = v[c];
                for (int e = l; e < n; e += G) conv_low(e);
#pragma unroll
                for (int c = 0; c < CH; c++)
                    if (l + c * G < n) v[c] = A[fx_at(l + c * G, s7)];
            }
            means();
            float sq = 0.0f;
#pragma unroll
            for (int c = 0; c < CH; c++) {
                if (l + c * G < n) {
                    v[c].x -= mx;
                    v[c].y -= my;
                }
                sq += square(v[c]);
            }
            const int sh = shift(group_sum(sq));
#pragma unroll
            for (int c = 0; c < CH; c++) {
                const int e = l + c * G;
                v[c].x = fx_shift(v[c].x, sh);
                v[c].y = fx_shift(v[c].y, sh);
                if (e < n) A[fx_at(e, s7)] = v[c];
            }
        };
        if (n <= 2 * G) {
            in_registers(std::integral_constant<int, 2>());
        } else if (n <= 8 * G) {
            in_registers(std::integral_constant<int, 8>());
        } else {
            unsigned m = 0u;
            for (int e0 = l; e0 < n; e0 += 8 * G) {
                X2 v[8];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int e = e0 + c * G;
                    if (e < n) v[c] = raw(e);
                    else v[c].x = v[c].y = 0;
                }
                if (e0 == l) constant(v[0]);
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    m = top(m, v[c]);
                    if (DIR == 0 && e0 + c * G < n) A[fx_at(e0 + c * G, s7)] = v[c];
                }
            }
            E = group_max(m);
            if (E >= 64)
                for (int e = l; e < n; e += G) A[fx_at(e, s7)] = conv(e, A[fx_at(e, s7)]);
            else
                for (int e = l; e < n; e += G) conv_low(e);
            means();
            float sq = 0.0f;
            for (int e = l; e < n; e += G) {
                X2 v = A[fx_at(e, s7)];
                v.x -= mx;
                v.y -= my;
                sq += square(v);
            }
            const int sh = shift(group_sum(sq));
            for (int e = l; e < n; e += G) {
                X2 v = A[fx_at(e, s7)];
                v.x = fx_shift(v.x - mx, sh);
                v.y = fx_shift(v.y - my, sh);
                A[fx_at(e, s7)] = v;
            }
        }
        out.bad = E == 0x7ff;
        if (inv) out.bad = out.bad || !(isfinite(out.cx) && isfinite(out.cy));
        if (op1 == OP_FWD || op1 == OP_DEALIAS || op2 == OP_DEALIAS) {
            const int ex = E - 1084;
            out.cx = fx_to(mx, ex, fx_safe(ex));
            out.cy = fx_to(my, ex, fx_safe(ex));
        }
        __syncwarp();

        // ---- forward
        float s1 = 0.0f, s2 = 0.0f;
        if (!inv) {
            for (int p = 0; p < pl.np - 1; p++) {
                const FxPassArgs a = args(p, pl.fup);
#define CALL(R, K) fx_fwd<R, K>(A, a)
                FX_SWITCH(pl, p, CALL)
#undef CALL
            }
            const bool key = op1 == OP_D1 || op1 == OP_D2 || op2 == OP_D1 || op2 == OP_D2;
            const FxPassArgs a = args(pl.np - 1, 0);
#define CALL(R, K) fx_last<R, K>(A, a, tb.kof, key, s1, s2)
            FX_SWITCH_LAST(pl, CALL)
#undef CALL
            if (key) {
                s1 = group_sum(s1);
                s2 = group_sum(s2);
            }
        }

        if (op1 == OP_FWD) {
            // separate Z into the halfcomplex spectra of the two real lines
            out.xe = F + pl.hf - 1;
            const bool scale = jb.alpha1 != 1.0;
            auto sep = [&](const X2 *Z, int z7, int p, const FxOut &o, double *va, double *vb) {
                const X2 zp = Z[fx_at(__ldg(tb.pos + p), z7)], zq = Z[fx_at(__ldg(tb.pos + (p == 0 ? 0 : n - p)), z7)];
                const bool re = 2 * p <= n, safe = fx_safe(o.xe);
                *va = fx_to(re ? zp.x + zq.x : zq.y - zp.y, o.xe, safe);
                *vb = fx_to(re ? zp.y + zq.y : zp.x - zq.x, o.xe, safe);
                if (p == 0) { *va += (double)n * o.cx; *vb += (double)n * o.cy; }
                if (o.bad) *va = *vb = FX_NAN;
                if (scale) { *va *= jb.alpha1; *vb *= jb.alpha1; }
            };
            if (DIR == 0) {
                if (valid) {
                    double *oa = jb.out1 + pb + 2 * (size_t)pair * nx, *ob = oa + nx;
                    for (int p = l; p < n; p += G) {
                        double va, vb;
                        sep(A, s7, p, out, &va, &vb);
                        oa[p] = jb.acc1 ? oa[p] + va : va;
                        ob[p] = jb.acc1 ? ob[p] + vb : vb;
                    }
                }
                __syncwarp();
            } else {
                if (l == 0) so[s] = out;
                __syncthreads();
                const int ls = 31 - __clz(S), q = tid & (S - 1);
                if (tile * S + q < pairs) {
                    const FxOut o = so[q];
                    double *op = jb.out1 + pb + 2 * ((size_t)tile * S + q);
                    for (int p = tid >> ls; p < n; p += (int)blockDim.x >> ls) {
                        double2 v;
                        sep(bufA + (size_t)q * pl.nb, q & 7, p, o, &v.x, &v.y);
                        double2 *d = reinterpret_cast<double2 *>(op + (size_t)p * nx);
                        if (jb.acc1) { const double2 w = *d; v.x = w.x + v.x; v.y = w.y + v.y; }
                        *d = v;
                    }
                }
                __syncthreads();
            }
            continue;
        }

        // ---- one or two inverse transforms
        const int nout = op2 != OP_NONE && (!inv || op2 == OP_D1) ? 2 : 1;
        for (int o = 0; o < nout; o++) {
            const int op = o == 0 ? op1 : op2;
            const X2 *src = A;
            X2 *dst = o + 1 < nout ? B : A;
            if (inv) {
                // Z_k = A_k + i B_k from the halfcomplex lines a (re), b (im),
                // into the digit-reversed order of the passes
                float q1 = 0.0f;
                for (int i = l; i < n; i += G) {
                    const int k = __ldg(tb.kof + i), kk = min(k, n - k);
                    const bool edge = kk == 0 || 2 * kk == n;
                    const X2 pa = A[fx_at(kk, s7)];
                    X2 pc = A[fx_at(edge ? 0 : n - kk, s7)];
                    if (edge) pc.x = pc.y = 0;
                    if (2 * k > n) { pc.x = -pc.x; pc.y = -pc.y; }
                    X2 z;
                    z.x = pa.x - pc.y;
                    z.y = pc.x + pa.y;
                    B[fx_at(i, s7)] = z;
                    const float x = fx_float((fx_hi(z.x) + 64) >> 7), y = fx_float((fx_hi(z.y) + 64) >> 7), kf = (float)kk;
                    q1 = fmaf((x * x + y * y) * kf, kf, q1);
                }
                if (op == OP_D1) s1 = group_sum(q1);
                __syncwarp();
                src = dst = B;
            }
            // the multiplier's shift: a derivative's from its norm (what the
            // squares cannot resolve counted in), a mask's for the growth
            int sh = 0;
            if (op == OP_D1) sh = max(((fx_log2(s1 + pl.floor1) + 1) >> 1) + pl.gb - 22, -20);
            else if (op == OP_D2) sh = max(((fx_log2(s2 + pl.floor2) + 1) >> 1) + pl.gb - 22, -20);
            else if (op == OP_DEALIAS) sh = pl.gb;
            {
                const FxPassArgs a = args(pl.np - 1, 0);
                if (op == OP_INV && pl.kind[pl.np - 1] == K1) {
                    fx_inv_first<8, K1>(dst, src, a, tb.kof, OP_INV, 0, 0);
                } else {
#define CALL(R, K) fx_inv_first<R, K>(dst, src, a, tb.kof, op, sh, pl.cut)
                    FX_SWITCH_LAST(pl, CALL)
#undef CALL
                }
            }
            out.xe = F + sh + pl.hi + (inv ? 0 : pl.hf);
            const double con = op == OP_D1 ? tb.c1 : op == OP_D2 ? tb.c2 : tb.c0;
            // (con 2^xe, and with it every result, in the normal range)
            const bool safe = out.xe >= -700 && out.xe <= 700;
            out.sc = safe ? con * fx_pow2(out.xe) : 0.0;
            const double alpha = o == 0 ? jb.alpha1 : jb.alpha2;
            const int acc = o == 0 ? jb.acc1 : jb.acc2;
            double *ot = o == 0 ? jb.out1 : jb.out2;
            // what is added back: the mean of a dealiased line, the constant of an
            // inverse, and its addk, addc.  (What is stored or accumulated as it is takes
            // paths of its own: FP64 operations, predicated off or not, would keep the FP64 pipe
            // busier than the conversions do.)
            const bool add = op == OP_DEALIAS || op == OP_INV;
            double addv = 0.0;
            if (op == OP_INV) addv = (jb.addk ? jb.addk[plane] : 0.0) + jb.addc;
            const bool store = !acc && alpha == 1.0;
            double ca = out.cx, cb = out.cy;
            if (store && op == OP_INV) { ca += addv; cb += addv; }
            double *oa = ot + pb + 2 * (size_t)pair * nx, *ob = oa + nx;
            const bool plain = alpha == 1.0 && !(acc && add) && safe && !out.bad;
            const int mode = acc ? FX_ACC : add ? FX_CONST : FX_SET;
            // x lines: the last pass stores its results
            const bool fused = DIR == 0 && pl.np > 1 && __all_sync(0xffffffffu, plain && valid);
            for (int p = pl.np - 2; p >= (fused ? 1 : 0); p--) {
                const FxPassArgs a = args(p, pl.iup);
#define CALL(R, K) fx_inv<R, K, false>(dst, a, nullptr, nullptr, 0.0, 0.0, 0.0, FX_SET)
                FX_SWITCH(pl, p, CALL)
#undef CALL
            }
            if (fused) {
                const FxPassArgs a = args(0, pl.iup);
#define CALL(R, K) fx_inv<R, K, true>(dst, a, oa, ob, out.sc, ca, cb, mode)
                FX_SWITCH(pl, 0, CALL)
#undef CALL
                continue;
            }
            auto fin = [&](const X2 v, const FxOut &q, double *va, double *vb, const double *old, size_t step) {
                const bool ok = q.xe >= -700 && q.xe <= 700;
                *va = ok ? __ll2double_rn(v.x) * q.sc : fx_to_far(v.x, q.xe, con);
                *vb = ok ? __ll2double_rn(v.y) * q.sc : fx_to_far(v.y, q.xe, con);
                if (add) { *va += q.cx; *vb += q.cy; }
                if (q.bad) *va = *vb = FX_NAN;
                *va *= alpha;
                *vb *= alpha;
                if (acc) { *va = old[0] + *va; *vb = old[step] + *vb; }
                if (op == OP_INV && !store) { *va += addv; *vb += addv; }
            };
            const FxOut mine = { ca, cb, out.sc, out.xe, out.bad };
            if (DIR == 0) {
                if (valid)
                    for (int e = l; e < n; e += G) {
                        double va, vb;
                        fin(dst[fx_at(e, s7)], mine, &va, &vb, oa + e, nx);
                        oa[e] = va;
                        ob[e] = vb;
                    }
                __syncwarp();
            } else {
                if (l == 0) so[s] = mine;
                const bool fast = __syncthreads_and(plain);
                const int ls = 31 - __clz(S), q = tid & (S - 1), de = (int)blockDim.x >> ls;
                const X2 *bs = (dst == A ? bufA : bufB) + (size_t)q * pl.nb;
                double *od = ot + pb + 2 * ((size_t)tile * S + q);
                if (tile * S + q < pairs) {
                    const FxOut f = so[q];
                    if (fast && acc) {
                        for (int e = tid >> ls; e < n; e += de) {
                            const X2 v = bs[fx_at(e, q & 7)];
                            double2 *o2 = reinterpret_cast<double2 *>(od + (size_t)e * nx);
                            const double2 x = *o2;
                            *o2 = make_double2(fma(__ll2double_rn(v.x), f.sc, x.x), fma(__ll2double_rn(v.y), f.sc, x.y));
                        }
                    } else if (fast && add) {
                        for (int e = tid >> ls; e < n; e += de) {
                            const X2 v = bs[fx_at(e, q & 7)];
                            *reinterpret_cast<double2 *>(od + (size_t)e * nx) =
                                make_double2(fma(__ll2double_rn(v.x), f.sc, f.cx), fma(__ll2double_rn(v.y), f.sc, f.cy));
                        }
                    } else if (fast) {
                        for (int e = tid >> ls; e < n; e += de) {
                            const X2 v = bs[fx_at(e, q & 7)];
                            *reinterpret_cast<double2 *>(od + (size_t)e * nx) =
                                make_double2(__ll2double_rn(v.x) * f.sc, __ll2double_rn(v.y) * f.sc);
                        }
                    } else {
                        for (int e = tid >> ls; e < n; e += de) {
                            double *dd = od + (size_t)e * nx;
                            double2 v;
                            fin(bs[fx_at(e, q & 7)], f, &v.x, &v.y, dd, 1);
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
#if !FX_LONG
// exp(-2 pi i e/n), computed in long double, exact at the quadrants; the angles
// of an octant are computed once
struct UnitCircle {
    long n;
    std::vector<FxConst> c, s;      // cos, sin of (pi/2) r/n, r = 0 .. n/2; c.h = 0: not yet
    explicit UnitCircle(int n_) : n(n_), c(n_ / 2 + 1, FxConst{ 0, 0 }), s(n_ / 2 + 1) {}
    TwX operator()(long e)
    {
        e %= n;
        const long q = (4 * e) / n, r = 4 * e - q * n, a = 2 * r <= n ? r : n - r;
        if (!c[a].h) {
            const long double t = 1.57079632679489661923132169163975144L * (long double)a / n;
            c[a] = fx_const(cosl(t));
            s[a] = fx_const(sinl(t));
        }
        const FxConst cr = a == r ? c[a] : s[a], sr = a == r ? s[a] : c[a];
        const FxConst cn = { -cr.h, -cr.l }, sn = { -sr.h, -sr.l };
        const FxConst re[4] = { cr, sn, cn, sr }, im[4] = { sn, cn, sr, cr };     // exp(-i t): (c, -s) turned by -q
        return TwX{ re[q].h, re[q].l, im[q].h, im[q].l };
    }
};
#endif

#if FX_LONG
int line_fx_long_configure()
#else
int line_fx_configure()
#endif
{
    const long double h = 3.14159265358979323846264338327950288L;
    const FxConst r8 = fx_const(cosl(h / 4)), r3 = fx_const(sinl(h / 3));
    const FxConst c5 = fx_const((cosl(2 * h / 5) - cosl(4 * h / 5)) / 2), sa = fx_const(sinl(2 * h / 5)), sb = fx_const(sinl(4 * h / 5));
    CUDA_TRY(cudaMemcpyToSymbol(c_fx_r8, &r8, sizeof(r8)));
    CUDA_TRY(cudaMemcpyToSymbol(c_fx_r3, &r3, sizeof(r3)));
    CUDA_TRY(cudaMemcpyToSymbol(c_fx_c5, &c5, sizeof(c5)));
    CUDA_TRY(cudaMemcpyToSymbol(c_fx_s5a, &sa, sizeof(sa)));
    CUDA_TRY(cudaMemcpyToSymbol(c_fx_s5b, &sb, sizeof(sb)));
#if FX_LONG
    return VEC_OK;
#else
    return line_fx_long_configure();
#endif
}

#if !FX_LONG
// the radices of n with the fewest passes; 8 where it divides, and last: the
// strides of the other passes are then multiples of 8 or 64
static bool radices(int n, std::vector<int> &r)
{
    static const int all[] = { 2, 3, 4, 5, 6, 8 };
    std::vector<int> best;
    std::vector<int> cur;
    auto go = [&](auto &self, int m, int from) -> void {
        if (!best.empty() && cur.size() >= best.size()) return;
        if (m == 1) { best = cur; return; }
        for (int q = from; q >= 0; q--)
            if (m % all[q] == 0) {
                cur.push_back(all[q]);
                self(self, m / all[q], q);
                cur.pop_back();
            }
    };
    go(go, n, 5);
    r.assign(best.rbegin(), best.rend());
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
    // (what the squares' unit leaves out, half of it at every wavenumber: with
    // (x + y)^2 <= 1.25 x^2 + 5 y^2, and the mean of k^2 and k^4)
    const double kmax = n / 2;
    pl->floor1 = (float)(n * kmax * kmax);
    pl->floor2 = (float)(n * kmax * kmax * kmax * kmax);
    // the sums of a pass: 2 x 4 and 3 x 2 with a halving between
    auto sums = [&](int p, int q) {
        const int R = r[p];
        return q == 0 ? (R == 8 ? 2 : R == 6 ? 3 : R) : R == 8 ? 4 : R == 6 ? 2 : 1;
    };
    int L = n;
    for (int p = 0; p < pl->np; p++) {
        const int R = r[p], M = L / R;
        pl->R[p] = R; pl->L[p] = L; pl->M[p] = M;
        pl->mg[p] = (unsigned)(((1ull << 31) + M - 1) / M);
        pl->kind[p] = M % 64 == 0 ? K64 : R == 8 && M == 8 ? K8 : R == 8 && M == 1 ? K1 : KG;
        pl->tw[p] = pl->ntw;
        if (M > 1) pl->ntw += (R - 1) * M;
        L = M;
    }
    // growth sqrt(P) 2^-halvings along the forward passes, and along the inverse ones, which
    // take the radices backwards; a halving between two passes.  Long lines leave out those
    // that the bound does not need: each costs a bit
    double top = 0.0;
    for (int d = 0; d < 2; d++)
        for (int o = 0; o < pl->np; o++)
            for (int q = 0; q < 2; q++) {
                double P = 1.0;
                int h = 0;
                for (int t = 0; t <= o; t++) {
                    const int p = d ? pl->np - 1 - t : t;
                    P *= sums(p, 0);
                    if (t == o && q == 0) break;
                    h += sums(p, 1) > 1;
                    P *= sums(p, 1);
                    if (t < o) h++;
                }
                top = fmax(top, sqrt(P) * exp2(-(double)h));
            }
    pl->gb = top <= 2.0 ? 1 : 2;
    if (top > 4.0) return VEC_ERR_SIZE;
    for (int d = 0; d < 2; d++) {
        double P = 1.0;
        int h = 0;
        for (int t = 0; t < pl->np; t++) {
            const int p = d ? pl->np - 1 - t : t, next = d ? p - 1 : p + 1;
            P *= r[p];
            h += sums(p, 1) > 1;
            if (t + 1 == pl->np) break;
            if (n > FX_SHORT && sqrt(P * sums(next, 0)) * exp2(-(double)h) <= exp2((double)pl->gb))
                (d ? pl->iup : pl->fup) |= 1u << (d ? next : p);
            else
                h++;
        }
        (d ? pl->hi : pl->hf) = h;
    }
    // sequences per warp: about 256 elements, at least four lanes each
    pl->Q = n <= 32 ? 8 : n <= 64 ? 4 : n <= 128 ? 2 : 1;
    return VEC_OK;
}

// the tables of one direction: the twiddles of each pass, the order of the
// spectrum, and the operators' constants (k1, k2: the multipliers' tables)
int fx_tables_make(int n, FxPlan *pl, const double *k1, const double *k2, int icut, FxTables *tb)
{
    pl->cut = n / 2 - icut;
    tb->c0 = 1.0 / n;
    tb->c1 = k1[1] / n;
    tb->c2 = k2[1] / n;
    UnitCircle unit(n);
    std::vector<TwX> tw;
    for (int p = 0; p < pl->np; p++)
        if (pl->M[p] > 1)
            for (int r = 1; r < pl->R[p]; r++)
                for (int j = 0; j < pl->M[p]; j++) tw.push_back(unit((long)j * r * (n / pl->L[p])));
    std::vector<unsigned short> pos(2 * n);       // and kof
    for (int k = 0; k < n; k++) {
        int rest = k, at = 0;
        for (int p = 0; p < pl->np; p++) {
            at += (rest % pl->R[p]) * pl->M[p];
            rest /= pl->R[p];
        }
        pos[k] = (unsigned short)at;
        pos[n + at] = (unsigned short)k;
    }
    const size_t bt = tw.size() * sizeof(TwX), bp = pos.size() * sizeof(short);
    std::vector<char> all(bt + bp);
    if (bt) memcpy(all.data(), tw.data(), bt);
    memcpy(all.data() + bt, pos.data(), bp);
    if (cudaMalloc(&tb->tw, all.size()) != cudaSuccess) {
        cudaGetLastError();
        return VEC_ERR_ALLOC;
    }
    tb->pos = reinterpret_cast<unsigned short *>(reinterpret_cast<char *>(tb->tw) + bt);
    tb->kof = tb->pos + n;
    CUDA_TRY(cudaMemcpy(tb->tw, all.data(), all.size(), cudaMemcpyHostToDevice));
    return VEC_OK;
}
void fx_tables_free(FxTables *tb)
{
    cudaFree(tb->tw);
    *tb = FxTables{};
}
#endif

template <int DIR, int NJ>
static int run_fx(Engine *E, const LineJob<double> *jobs, int nj)
{
    FxPlan pl = DIR == 0 ? E->fpx : E->fpy;
    FxPack<NJ> pk;
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
    // fewer sequences per warp where the device would not be full (8 warps per
    // SM): the time is then that of one warp's tile, which more lanes per
    // sequence shorten if its passes take fewer rounds (30 x 30 x 60: 36 -> 26 us;
    // 64 points take as many with 8 lanes as with 32, and lose: 23 -> 28 us)
    while (pl.Q > 1 && (long long)nj * E->nz * pairs < (long long)E->num_sms * 8 * pl.Q && fx_rounds(pl, pl.Q / 2) < fx_rounds(pl, pl.Q))
        pl.Q >>= 1;
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
    static SmemLimit limit;
    CUDA_TRY(limit.raise((const void *)line_fx<DIR, NJ, FX_LONG>, 226 * 1024));
    if (smem > 226 * 1024) return VEC_ERR_SIZE;
    int per_sm = 1;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, line_fx<DIR, NJ, FX_LONG>, W * 32, smem));
    if (per_sm < 1) per_sm = 1;
    const int S = DIR == 0 ? pl.Q : W * pl.Q, tpp = (pairs + S - 1) / S;
    const long long total = tiles_of(W);
    long long grid = DIR == 0 ? (total + W - 1) / W : total;
    if (grid > (long long)E->num_sms * per_sm) grid = (long long)E->num_sms * per_sm;
    E->prof_begin(DIR == 0 ? "line_x_f64" : "line_y_f64", fields * (double)E->n * 8.0);
    CUDA_TRY(launch_k(*E, line_fx<DIR, NJ, FX_LONG>, dim3((unsigned)grid), dim3(W * 32), smem, pk, pl, DIR == 0 ? E->fxx : E->fxy, E->nx,
                      E->ny, E->nz, tpp, (int)total, two));
    E->prof_end();
    CUDA_TRY(cudaGetLastError());
    return VEC_OK;
}

#if FX_LONG
int launch_lines_fx_long(Engine *E, int dir, const LineJob<double> *jobs, int njobs)
{
#else
template <>
int launch_lines<double>(Engine *E, int dir, const LineJob<double> *jobs, int njobs)
{
    if ((dir == 0 ? E->nx : E->ny) > FX_SHORT) return launch_lines_fx_long(E, dir, jobs, njobs);
#endif
    for (int j0 = 0; j0 < njobs; j0 += MAX_JOBS) {
        const int nj = njobs - j0 < MAX_JOBS ? njobs - j0 : MAX_JOBS;
        const LineJob<double> *j = jobs + j0;
        const int st = nj <= NJ_SMALL ? (dir == 0 ? run_fx<0, NJ_SMALL>(E, j, nj) : run_fx<1, NJ_SMALL>(E, j, nj))
                                      : (dir == 0 ? run_fx<0, MAX_JOBS>(E, j, nj) : run_fx<1, MAX_JOBS>(E, j, nj));
        if (st) return st;
    }
    return VEC_OK;
}
