// fx.cuh -- 64-bit fixed-point complex arithmetic of the FP64 line transforms.
//
// GB300 executes about two FP64 operations per clock and SM, 28 widening 32-bit
// multiply-adds (32 x 32 + 64) on operands that change, and 64 to 128 other 32-bit
// integer ones (measured: 1.7 DFMA, 28 mad.wide, 128 IADD, 64 logic operations and
// shifts per clock and SM).
// An FFT is linear, and the rounding of a floating-point one is relative to
// the norm of the whole line, not to the single element.  So the FP64 lines
// are transformed in block floating point: one exponent per sequence (a pair
// of real lines, which a floating-point transform packed as a + i b mixes in
// the same way) and 64-bit integers.  A complex addition is 4 integer
// instructions instead of 2 FP64 ones, a twiddle product as much as 46 instructions
// of 64 a clock instead of 4: 0.04 clocks instead of 1.2, and 0.7 instead of 2.3.
//
// Scaling.  The values of a sequence are integers times 2^F with
// 2^gb ||z||_2 2^-F <= 2^61.  A transform is a chain of small DFTs; between
// any two of them its values are multiplied by a twiddle and 1/2.  By
// Cauchy-Schwarz a sum of P elements is at most sqrt(P) ||z||_2; gb bounds
// sqrt(P) 2^-halvings over the chain (1 for 2^a 3^b, 2 for some 5^c).  Above 512
// points (FX_LONG) the halvings that this bound can do without are left out: passes of six
// points halve twice for a growth of 2.4, and four of them gave two bits away.  A
// product is rounded to the nearest integer with an error below one unit,
// about 2^-55 of the rms value against FP64's 2^-52.
// A floating-point transform is better than that where the line is a large
// constant plus little, or where a derivative is small: the differences it
// forms are exact there.  So the line's mean (any number near it) is taken
// off before the exponent is chosen, and a derivative's spectrum gets an
// exponent of its own before it is transformed back.
#pragma once
#include <stdint.h>

struct __align__(16) X2 { long long x, y; };
// w = (xh 2^32 + xl, yh 2^32 + yl) 2^-62 with signed low words
struct __align__(16) TwX { int xh, xl, yh, yl; };

__device__ __forceinline__ long long fx_wide(int a, int b) { return (long long)a * (long long)b; }
__device__ __forceinline__ int fx_hi(long long a) { return (int)(a >> 32); }
// the high word for a signed low word: a = fx_h(a) 2^32 + (int)a
__device__ __forceinline__ int fx_h(long long a) { return fx_hi(a) + (int)((unsigned)a >> 31); }

// a m / 2 for |a| < 2^62, m = (mh 2^32 + ml) 2^-62, |m| <= 1
__device__ __forceinline__ long long fx_mulr(long long a, int mh, int ml)
{
    const int h = fx_h(a), l = (int)a;
    const long long mid = fx_wide(h, ml) + fx_wide(l, mh) + (1LL << 30);
    return fx_wide(h << 1, mh) + (mid >> 31);
}
// a w / 2 for |a| < 2^62, |w| <= 1 (CONJ: a conj(w) / 2)
template <bool CONJ> __device__ __forceinline__ X2 fx_mulw(X2 a, TwX w)
{
    const int xh = fx_h(a.x), xl = (int)a.x, yh = fx_h(a.y), yl = (int)a.y;
    const int nh = -w.yh, nl = -w.yl;
    const int ph = CONJ ? w.yh : nh, pl = CONJ ? w.yl : nl;    // times a.y in the real part
    const int qh = CONJ ? nh : w.yh, ql = CONJ ? nl : w.yl;    // times a.x in the imaginary part
    const long long mr = fx_wide(xh, w.xl) + fx_wide(xl, w.xh) + fx_wide(yh, pl) + fx_wide(yl, ph) + (1LL << 30);
    const long long mi = fx_wide(xh, ql) + fx_wide(xl, qh) + fx_wide(yh, w.xl) + fx_wide(yl, w.xh) + (1LL << 30);
    const int x2 = xh << 1, y2 = yh << 1;
    X2 r;
    r.x = fx_wide(x2, w.xh) + fx_wide(y2, ph) + (mr >> 31);
    r.y = fx_wide(x2, qh) + fx_wide(y2, w.xh) + (mi >> 31);
    return r;
}
__device__ __forceinline__ X2 fx_mulc(X2 a, TwX w) { return fx_mulw<false>(a, w); }
__device__ __forceinline__ X2 fx_mulcj(X2 a, TwX w) { return fx_mulw<true>(a, w); }
// a / 2, a / 4.  Rounded down they leave out a quarter and three eighths of a unit on
// average, the same for all elements of a pass: in long lines these add up, at the lowest
// wavenumbers and, on the way back, at the first elements (three times the other
// elements' error).  There (FX_LONG) they are rounded by the other part's last bit.  Both
// together: the rms error of 1080 to 1944 points 0.8 to 1.5 times that of the FP64 register
// transforms -> 0.4 to 0.6, the largest up to 3.7 (1.3 at 648 to 972) -> 0.4 to 0.8, for 3 to
// 6 % of the time.
#ifndef FX_LONG
#define FX_LONG 0
#endif
__device__ __forceinline__ X2 fx_half(X2 a)
{
    X2 r;
    r.x = (a.x + (FX_LONG ? (long long)((int)a.y & 1) : 0)) >> 1;
    r.y = (a.y + (FX_LONG ? (long long)((int)a.x & 1) : 0)) >> 1;
    return r;
}
__device__ __forceinline__ X2 fx_quarter(X2 a)
{
    X2 r;
    r.x = (a.x + (FX_LONG ? 1 + (long long)((int)a.y & 1) : 0)) >> 2;
    r.y = (a.y + (FX_LONG ? 1 + (long long)((int)a.x & 1) : 0)) >> 2;
    return r;
}

// a k 2^-t for -20 <= t <= 31 where the result is below 2^62, |k| < 2^21
__device__ __forceinline__ long long fx_mulk(long long a, int k, int t)
{
    if (t <= 0) {
        a <<= -t;
        const long long p = fx_wide((int)a, k);
        return (long long)(((unsigned long long)(unsigned)(fx_hi(p) + fx_h(a) * k) << 32) | (unsigned)p);
    }
    const long long p = fx_wide((int)a, k) + (1LL << (t - 1));
    const long long q = fx_wide(fx_h(a), k) + (p >> 32);
    return (q << (32 - t)) + (long long)((unsigned)p >> t);
}
// a signed 23-bit integer as a float, without the conversion unit
__device__ __forceinline__ float fx_float(int v) { return __int_as_float(0x4b400000 + v) - 12582912.0f; }

// ---- double <-> fixed ---------------------------------------------------------
// The FP64 pipe converts 1.9 values per clock and SM, beside the integer pipe.

// the double with bits (h, l) as an integer multiple of 2^(E - 1084)
// (truncated), E its sequence's largest exponent field: below 2^62
__device__ __forceinline__ long long fx_from(unsigned h, unsigned l, int E)
{
    // the exponent moved by 1084 - E; what falls out of the normal range is
    // below 2^-960 of the largest value
    const int s = (1084 - E) << 20;
    const bool in = (int)(h & 0x7ff00000u) > -s && (h & 0x7ff00000u);
    const double d = __hiloint2double((int)(in ? h + (unsigned)s : 0u), (int)(in ? l : 0u));
    return __double2ll_rz(d);
}
// the same for sequences near the bottom of the exponent range, where
// subnormals count
static __device__ __noinline__ long long fx_from_low(unsigned h, unsigned l, int E)
{
    const unsigned e = (h >> 20) & 0x7ffu;
    const unsigned long long m = ((unsigned long long)((h & 0xfffffu) | (e ? 0x100000u : 0u)) << 32) | l;
    const long long p = (long long)((m << 9) >> min(E - (int)max(e, 1u), 63));
    return (int)h < 0 ? -p : p;
}
// 2^e in the normal range
__device__ __forceinline__ double fx_pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }
static __device__ __noinline__ double fx_to_slow(long long a, int ex) { return scalbn((double)a, ex); }
// a con 2^ex for -1100 < ex < 1100 and 2^-400 < con < 2^400, rounded once where it leaves the normal range
static __device__ __noinline__ double fx_to_far(long long a, int ex, double con)
{
    return (double)a * (con * fx_pow2(ex >> 1)) * fx_pow2(ex - (ex >> 1));
}
// a 2^ex rounded to double; safe: ex lies in [-1022, 960], where no result
// with |a| < 2^62 leaves the normal range
__device__ __forceinline__ bool fx_safe(int ex) { return ex >= -1022 && ex <= 960; }
__device__ __forceinline__ double fx_to(long long a, int ex, bool safe)
{
    if (!safe) return fx_to_slow(a, ex);
    const double d = __ll2double_rn(a);
    const int h = __double2hiint(d);
    return __hiloint2double(h == 0 ? 0 : h + (ex << 20), __double2loint(d));
}
// a 2^r (truncated)
__device__ __forceinline__ long long fx_shift(long long a, int r) { return r >= 0 ? a << r : a >> -r; }
// ceil(log2 s) for s > 0 (0 stands for the smallest normal number)
__device__ __forceinline__ int fx_log2(float s) { return (int)(__float_as_uint(s) >> 23) - 126; }

// ---- in-register DFTs -----------------------------------------------------------
// W_8^1, W_12^1 (real part sqrt(3)/2), and of W_5: (cos 72 - cos 144) / 2,
// sin 72, sin 144 (degrees), with 62 fractional bits as high word and signed
// low word; set by line_fx_configure
#define FX_NAN __longlong_as_double(0x7ff8000000000000ll)
struct FxConst { int h, l; };
static __constant__ FxConst c_fx_r8, c_fx_r3, c_fx_c5, c_fx_s5a, c_fx_s5b;

__device__ __forceinline__ X2 operator+(X2 a, X2 b) { X2 r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
__device__ __forceinline__ X2 operator-(X2 a, X2 b) { X2 r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
// times -i (forward), i (INV)
template <bool INV> __device__ __forceinline__ X2 fx_rot(X2 a)
{
    X2 r;
    if (INV) { r.x = -a.y; r.y = a.x; }
    else { r.x = a.y; r.y = -a.x; }
    return r;
}
// times a real constant (|a| < 2^61: doubled, for the product's 1/2)
__device__ __forceinline__ X2 fx_scale(X2 a, FxConst c)
{
    X2 r;
    r.x = fx_mulr(a.x << 1, c.h, c.l);
    r.y = fx_mulr(a.y << 1, c.h, c.l);
    return r;
}
// times W_8 / 2 (conjugate for INV)
template <bool INV> __device__ __forceinline__ X2 fx_w8(X2 a)
{
    const FxConst c = c_fx_r8;
    X2 r;
    r.x = fx_mulr(INV ? a.x - a.y : a.x + a.y, c.h, c.l);
    r.y = fx_mulr(INV ? a.x + a.y : a.y - a.x, c.h, c.l);
    return r;
}

template <int N, bool INV> struct XDft;
template <bool INV> struct XDft<2, INV> {
    static __device__ __forceinline__ void run(X2 *v) { const X2 a = v[0], b = v[1]; v[0] = a + b; v[1] = a - b; }
};
template <bool INV> struct XDft<3, INV> {
    static __device__ __forceinline__ void run(X2 *v)
    {
        const X2 t = v[1] + v[2], r = fx_scale(fx_rot<INV>(v[1] - v[2]), c_fx_r3), m = v[0] - fx_half(t);
        v[0] = v[0] + t;
        v[1] = m + r;
        v[2] = m - r;
    }
};
template <bool INV> struct XDft<4, INV> {
    static __device__ __forceinline__ void run(X2 *v)
    {
        const X2 a0 = v[0] + v[2], a1 = v[0] - v[2], b0 = v[1] + v[3], b1 = fx_rot<INV>(v[1] - v[3]);
        v[0] = a0 + b0; v[1] = a1 + b1; v[2] = a0 - b0; v[3] = a1 - b1;
    }
};
// cos 72 + cos 144 = -1/2: the cosine sums take one product
template <bool INV> struct XDft<5, INV> {
    static __device__ __forceinline__ void run(X2 *v)
    {
        const X2 t1 = v[1] + v[4], t2 = v[2] + v[3], d1 = fx_rot<INV>(v[1] - v[4]), d2 = fx_rot<INV>(v[2] - v[3]);
        const X2 t = t1 + t2, m = v[0] - fx_half(fx_half(t)), c = fx_scale(t1 - t2, c_fx_c5);
        const X2 a1 = m + c, a2 = m - c;
        const X2 b1 = fx_scale(d1, c_fx_s5a) + fx_scale(d2, c_fx_s5b);
        const X2 b2 = fx_scale(d1, c_fx_s5b) - fx_scale(d2, c_fx_s5a);
        v[0] = v[0] + t;
        v[1] = a1 + b1; v[4] = a1 - b1; v[2] = a2 + b2; v[3] = a2 - b2;
    }
};
// 3 x 2 and 2 x 4 with one halving between
template <bool INV> struct XDft<6, INV> {
    static __device__ __forceinline__ void run(X2 *v)
    {
        X2 a[3] = { v[0], v[2], v[4] }, b[3] = { v[1], v[3], v[5] };
        XDft<3, INV>::run(a);
        XDft<3, INV>::run(b);
        // b_k W_6^k / 2: W_6 = (1 - i sqrt 3) / 2, W_6^2 = -(1 + i sqrt 3) / 2 (forward)
        const X2 r1 = fx_rot<INV>(b[1]), r2 = fx_rot<INV>(b[2]);
        X2 w1, w2;
        const FxConst c = c_fx_r3;
        const X2 q1 = fx_quarter(b[1]), q2 = fx_quarter(b[2]);
        w1.x = q1.x + fx_mulr(r1.x, c.h, c.l); w1.y = q1.y + fx_mulr(r1.y, c.h, c.l);
        w2.x = fx_mulr(r2.x, c.h, c.l) - q2.x; w2.y = fx_mulr(r2.y, c.h, c.l) - q2.y;
        const X2 h0 = fx_half(a[0]), h1 = fx_half(a[1]), h2 = fx_half(a[2]), g0 = fx_half(b[0]);
        v[0] = h0 + g0; v[3] = h0 - g0;
        v[1] = h1 + w1; v[4] = h1 - w1;
        v[2] = h2 + w2; v[5] = h2 - w2;
    }
};
template <bool INV> struct XDft<8, INV> {
    static __device__ __forceinline__ void run(X2 *v)
    {
        X2 a[4], b[4];
#pragma unroll
        for (int j = 0; j < 4; j++) { a[j] = fx_half(v[j] + v[j + 4]); b[j] = v[j] - v[j + 4]; }
        b[0] = fx_half(b[0]);
        b[1] = fx_w8<INV>(b[1]);
        b[2] = fx_half(fx_rot<INV>(b[2]));
        b[3] = fx_w8<INV>(fx_rot<INV>(b[3]));
        XDft<4, INV>::run(a);
        XDft<4, INV>::run(b);
#pragma unroll
        for (int m = 0; m < 4; m++) { v[2 * m] = a[m]; v[2 * m + 1] = b[m]; }
    }
};
