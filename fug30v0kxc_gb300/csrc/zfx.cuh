// zfx.cuh -- z stencils of FP64 fields summed in integers.
//
// A stencil is a sum of up to seven neighbours with small integer weights, four
// or five FP64 operations of 37 issue slots each on GB300 (2 per clock and SM).
// Here the neighbours are aligned to their largest exponent (14 integer
// instructions each, shared by all the stencils of a field at a point), summed
// in integers, and the sum rounded once (20 instructions).  Three bits below the
// largest value's last one are kept, so that neighbours of up to an eighth of it
// enter whole; what smaller ones lose, less than a unit of 2^-3 each, enters with
// the weights (their absolute sum is at most 64, and the sum below 2^62): at most 8
// units in the last place of the largest neighbour, and the one rounding, where the
// FP64 sum has a rounding per operation.
#pragma once
#include <stdint.h>

#include "zstencil.cuh"

// The values f as integers times 2^(E - 1078), E the largest exponent field (64
// for zeros: the truncated modes of a spectrum); false (and FP64 is to be used)
// if one is not finite or all are tiny.
template <int N> __device__ __forceinline__ bool zi_align(const double (&f)[N], long long (&v)[N], int &E)
{
    unsigned m = 0u, any = 0u;
#pragma unroll
    for (int i = 0; i < N; i++) {
        m = max(m, (unsigned)__double2hiint(f[i]) & 0x7fffffffu);
        any |= (unsigned)__double2loint(f[i]);
    }
    E = (m | any) ? (int)(m >> 20) : 64;
#pragma unroll
    for (int i = 0; i < N; i++) {
        const unsigned h = (unsigned)__double2hiint(f[i]), e = (h >> 20) & 0x7ffu;
        // (an exponent field of 0 is at least 64 below E: shifted out)
        const unsigned long long p = ((unsigned long long)((h & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(f[i]);
        const long long q = (long long)((p << 3) >> min((unsigned)E - e, 63u)), s = (long long)(int)h >> 63;
        v[i] = (q ^ s) - s;
    }
    return E >= 64 && E <= 2030;
}
// s 2^(E - 1078) rounded to the nearest double
__device__ __forceinline__ double zi_to(long long s, int E)
{
    const unsigned long long a = (unsigned long long)(s < 0 ? -s : s);
    const int lz = __clzll((long long)a);
    const unsigned long long m = a << lz;
    // (a carry out of the fraction moves into the exponent)
    const unsigned long long r = (m >> 11) + ((m >> 10) & 1u) + ((unsigned long long)(unsigned)(E + 7 - lz) << 52);
    return s == 0 ? 0.0 : __longlong_as_double((long long)(r | ((unsigned long long)s & 0x8000000000000000ull)));
}

// the same with the conversion on the FP64 pipe (one operation; 4 integer
// instructions instead of 24), for kernels that leave it idle
__device__ __forceinline__ double zi_to_pipe(long long s, int E)
{
    const double d = __ll2double_rn(s);
    const int h = __double2hiint(d);
    return __hiloint2double(h == 0 ? 0 : h + (E - 1078) * (1 << 20), __double2loint(d));
}

// The interior rows of zstencil.cuh without their factors h and s, on
// v[d] = f(k - 3 + d)
__device__ __forceinline__ long long zi_sum1(const long long (&v)[7]) { return (v[1] - v[5]) + ((v[4] - v[2]) << 3); }
__device__ __forceinline__ long long zi_sum2(const long long (&v)[7])
{
    return ((v[2] + v[4]) << 4) - (v[3] << 5) + (v[3] << 1) - (v[1] + v[5]);
}
// (against the flow the mirror image with the other sign)
__device__ __forceinline__ long long zi_sumup(const long long (&v)[7], bool pos)
{
    const long long a = pos ? v[0] : v[6], b = pos ? v[1] : v[5], c = pos ? v[2] : v[4], e = pos ? v[4] : v[2];
    const long long t = b - c - (c << 1);
    const long long s = (t << 2) + (t << 1) - a + (v[3] << 3) + (v[3] << 1) + e + (e << 1);
    return pos ? s : -s;
}

// which stencils of a field a kernel wants
// (ZPIPE: the sums' conversion on the FP64 pipe)
enum { ZD1 = 1, ZD2 = 2, ZUP = 4, ZPIPE = 8 };
struct ZSum { double d1, d2, up; };

// the stencils W of one column at plane k without their factors (F(k): plane k
// of the column; the wall rows' flags f1, f2 for d1 and up, d2)
//
// The stencils share one alignment, to the largest of all planes that any of them
// reads.  One whose own planes are more than four times smaller would lose bits to a
// plane it does not read, more than its FP64 sum rounds off (at four times as large
// the truncation is at most 4 / 8 of the weights' sum in the last bits of its own
// largest plane, 9, 32 and 19, and the FP64 sums' intermediate results round off 17,
// 57 and 35): there all are summed in FP64.
template <int W, typename A>
__device__ __forceinline__ ZSum zsum(const A &F, int k, int nz, int f1, int f2, double w0)
{
    ZSum z = { 0.0, 0.0, 0.0 };
    if (k >= 3 && k <= nz - 4) {
        const bool pos = w0 >= 0.0;
        int E;
        if constexpr ((W & (ZD1 | ZD2 | ZUP)) == ZUP) {
            // (the five planes it reads, against the flow in mirror image)
            double f[5];
            long long v[5];
#pragma unroll
            for (int d = 0; d < 5; d++) f[d] = F(pos ? k - 3 + d : k + 3 - d);
            if (zi_align<5>(f, v, E)) {
                const long long t = v[1] - v[2] - (v[2] << 1);
                const long long s = (t << 2) + (t << 1) - v[0] + (v[3] << 3) + (v[3] << 1) + v[4] + (v[4] << 1);
                z.up = W & ZPIPE ? zi_to_pipe(pos ? s : -s, E) : zi_to(pos ? s : -s, E);
                return z;
            }
            z.up = zd1upa(F, k, nz, f1, 1.0, w0);
            return z;
        }
        double f[7];
        long long v[7];
        // (the planes the wanted stencils do not read count as zero)
#pragma unroll
        for (int d = 0; d < 7; d++) f[d] = (d == 0 || d == 6) && !(W & ZUP) ? 0.0 : d == 3 && !(W & (ZD2 | ZUP)) ? 0.0 : F(k - 3 + d);
        // the smallest of the stencils' own largest planes
        auto top = [&](int d) { return (unsigned)__double2hiint(f[d]) & 0x7fffffffu; };
        unsigned m = 0xffffffffu;
        if (W & ZUP) m = max(max(max(top(2), top(4)), top(3)), pos ? max(top(0), top(1)) : max(top(5), top(6)));
        if ((W & ZD1) && (W & (ZD2 | ZUP))) m = min(m, max(max(top(1), top(5)), max(top(2), top(4))));
        else if ((W & ZD2) && (W & ZUP)) m = min(m, max(max(max(top(1), top(5)), max(top(2), top(4))), top(3)));
        if (zi_align<7>(f, v, E) && (m >= (unsigned)(E - 2) << 20 || E <= 66)) {     // (E = 64: all zeros)
            auto to = [&](long long s) { return W & ZPIPE ? zi_to_pipe(s, E) : zi_to(s, E); };
            if (W & ZD1) z.d1 = to(zi_sum1(v));
            if (W & ZD2) z.d2 = to(zi_sum2(v));
            if (W & ZUP) z.up = to(zi_sumup(v, pos));
            return z;
        }
    }
    if (W & ZD1) z.d1 = zd1a(F, k, nz, f1, 1.0);
    if (W & ZD2) z.d2 = zd2a(F, k, nz, f2, 1.0);
    if (W & ZUP) z.up = zd1upa(F, k, nz, f1, 1.0, w0);
    return z;
}
template <int W>
__device__ __forceinline__ ZSum zsum(const double *f, size_t np, int k, int nz, int f1, int f2, double w0 = 0.0)
{
    return zsum<W>(ZCol<double>{ f, np }, k, nz, f1, f2, w0);
}
