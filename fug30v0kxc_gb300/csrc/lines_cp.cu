// lines_cp.cu -- horizontal spectral operators (src/fft.F90) in FP32 for line
// lengths n = 384, 512, 768 and 1024, the hot path of the split step.
//
// Per tile a CTA owns 2S real lines of one z-plane.  The tile is brought into
// shared memory by TMA bulk copies (cp.async.bulk + mbarrier): one copy per four
// contiguous x rows, or a 2S-wide box of y columns.  CTAs are persistent over
// tiles and the next tile is prefetched into the second buffer while the current
// one is transformed.
//
// Each length-n FFT is held in registers, in three levels n = A B C: with
// m = BC m1 + C b + c and k = k1 + A k2 + AB k3, thread m' = C b + c does an A-point
// DFT over m1 and applies W_n^(m' k1); thread (k1, c) a B-point DFT over b and
// W_BC^(c k2); thread (k1, k2) a C-point DFT over c.  The spectral operator (k, -k^2,
// 2/3 truncation, all Hermitian-symmetric multipliers) is a product in registers, and
// the inverse runs the same levels backwards, so that every thread writes to an
// exchange what it read from it and one barrier per exchange is enough.
//
// A group of threads transforms two complex sequences together, of four adjacent
// lines l + i (l+2) and (l+1) + i (l+3): a point is a pair of real parts and a pair
// of imaginary parts (Z), every butterfly is an FP32x2 instruction on a pair (a sign
// is an operand modifier and free), an exchange moves 16 bytes per point and a y
// line's store as many.  Instructions bound the kernel, not memory: one sequence per
// group in scalar FP32 and two levels (lines_ct.cu) took 65 % of the issue slots, with
// half of a 512-point line's threads idle on the first of 32 x 16 levels.  Pairs halve
// the arithmetic, the exchanges and the stores at once, and three levels of 8 keep
// all 64 threads busy with 32 registers per spectrum.  (A factor of 3 is in the last level,
// C = 6 or 12, and an 8 ends on fours: what a last stage rounds off repeats at n / its
// radix, and a second derivative weighs it by the fourth power.  With the 3 in the middle
// the second derivative of a smooth 384- or 768-point line erred 6 % more than with two
// levels, of a constant plus little 9 to 38 %.)  One sequence per group with
// sums on (re, im) pairs, twice the threads: 512^2 y lines 17 % slower; groups of
// eight y columns with barriers of their own: 32-byte rows, 8-30 % slower.  Nothing
// may spill: what shared memory leaves of L1 does not hold it (28 bytes a thread:
// 512^2 y lines 12-20 % slower).  A derivative pair, x and y, before -> now (us, two
// runs of one side differ by 3 %):
//    384^2 x 65    53.1  48.9 ->  43.5  41.6      768^2 x 33   104.1 100.0 ->  73.0  82.5
//    512^2 x 65    92.6  67.4 ->  60.1  62.0     1024^2 x 33   153.3 140.2 -> 122.4 133.7
// The error against FP64 (rms of d1, d2 and dealias) falls by 6 to 13 % for white noise, by
// 1 to 13 % for lines of few waves with and without noise, and stays for a constant plus
// little.
// (Up to 256 points pairs on two levels took 3-8 % less than lines_ct.cu's scalar kernel,
// 34.4 -> 31.5 at 256^2 x 129; they are not in use.)
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"
#include "engine.h"
#include "tma.cuh"

int encode_ymap(CUtensorMap *m, const float *base, int nx, int ny, int nz, int S, int BR);   // lines_ct.cu

// the jobs of one launch, and for y lines one TMA descriptor per input (3-D view
// nx x ny x nz)
template <int NJ> struct JobPackCP { LineJob<float> j[NJ]; };
template <int DIR, int NJ> struct TmapPackCP { CUtensorMap m[NJ]; };
template <int NJ> struct TmapPackCP<0, NJ> {};

// ---- arithmetic on points ------------------------------------------------------------
// a point of two sequences: their real parts and their imaginary parts
struct __align__(16) Z { float2 r, i; };

__device__ __forceinline__ float2 bc2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
// (the sign is an operand modifier: no instruction)
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }
// q quarter turns (-i)^q, or i^q in the inverse
template <bool INV> __host__ __device__ constexpr int turns(int q) { return INV ? (4 - (q & 3)) & 3 : q & 3; }
// a + (-i)^q b
template <bool INV, int Q> __device__ __forceinline__ Z zadd(const Z &a, const Z &b)
{
    constexpr int q = turns<INV>(Q);
    if constexpr (q == 0) return Z{ add2(a.r, b.r), add2(a.i, b.i) };
    else if constexpr (q == 1) return Z{ add2(a.r, b.i), sub2(a.i, b.r) };
    else if constexpr (q == 2) return Z{ sub2(a.r, b.r), sub2(a.i, b.i) };
    else return Z{ sub2(a.r, b.i), add2(a.i, b.r) };
}
// a + h (-i)^q b, h real
template <bool INV, int Q> __device__ __forceinline__ Z zfma(const Z &a, const Z &b, float h)
{
    constexpr int q = turns<INV>(Q);
    const float2 p = bc2(h), n = neg2(p);
    if constexpr (q == 0) return Z{ __ffma2_rn(b.r, p, a.r), __ffma2_rn(b.i, p, a.i) };
    else if constexpr (q == 1) return Z{ __ffma2_rn(b.i, p, a.r), __ffma2_rn(b.r, n, a.i) };
    else if constexpr (q == 2) return Z{ __ffma2_rn(b.r, n, a.r), __ffma2_rn(b.i, n, a.i) };
    else return Z{ __ffma2_rn(b.i, n, a.r), __ffma2_rn(b.r, p, a.i) };
}
// sqrt(2) W_8 b: the factor is left to the sum that takes it
template <bool INV> __device__ __forceinline__ Z zw8(const Z &b)
{
    if constexpr (INV) return Z{ sub2(b.r, b.i), add2(b.r, b.i) };
    else return Z{ add2(b.r, b.i), sub2(b.i, b.r) };
}
// (c - i s) b, (c + i s) b in the inverse
template <bool INV> __device__ __forceinline__ Z ztw(const Z &b, float c, float s)
{
    const float2 t = INV ? neg2(bc2(s)) : bc2(s);
    return Z{ __ffma2_rn(b.i, t, __fmul2_rn(b.r, bc2(c))), __ffma2_rn(b.r, neg2(t), __fmul2_rn(b.i, bc2(c))) };
}
// the same with a factor from a table, both elements of each pair alike
struct __align__(16) Tw { float2 c, s; };
template <bool INV> __device__ __forceinline__ Z ztw(const Z &b, const Tw &w)
{
    const float2 n = neg2(w.s);
    if constexpr (INV) return Z{ __ffma2_rn(b.i, n, __fmul2_rn(b.r, w.c)), __ffma2_rn(b.r, w.s, __fmul2_rn(b.i, w.c)) };
    else return Z{ __ffma2_rn(b.i, w.s, __fmul2_rn(b.r, w.c)), __ffma2_rn(b.r, n, __fmul2_rn(b.i, w.c)) };
}
__device__ __forceinline__ Tw twmul(const Tw &a, const Tw &b)
{
    return Tw{ __ffma2_rn(neg2(a.s), b.s, __fmul2_rn(a.c, b.c)), __ffma2_rn(a.s, b.c, __fmul2_rn(a.c, b.s)) };
}

// f v, f v + o, v + c, i v
__device__ __forceinline__ Z zscale(const Z &v, float f) { return Z{ __fmul2_rn(v.r, bc2(f)), __fmul2_rn(v.i, bc2(f)) }; }
__device__ __forceinline__ Z zscale(const Z &v, float2 f) { return Z{ __fmul2_rn(v.r, f), __fmul2_rn(v.i, f) }; }
__device__ __forceinline__ Z zaxpy(float f, const Z &v, const Z &o)
{
    return Z{ __ffma2_rn(v.r, bc2(f), o.r), __ffma2_rn(v.i, bc2(f), o.i) };
}
__device__ __forceinline__ Z zaddc(const Z &v, float c) { return Z{ add2(v.r, bc2(c)), add2(v.i, bc2(c)) }; }
__device__ __forceinline__ Z zi(const Z &v) { return Z{ neg2(v.i), v.r }; }

// ---- DFTs in registers, natural order ------------------------------------------------
// DFT of four points of which v2 is (-i)^Q2 times what is given, v1 and v3 (-i)^Q1
// and (-i)^Q3; h2, h13: real factors still to be applied to v2 and to v1, v3
template <bool INV, int Q1, int Q2, int Q3, bool H2, bool H13>
__device__ __forceinline__ void dft4(const Z &v0, const Z &v1, const Z &v2, const Z &v3, float h, Z &o0, Z &o1, Z &o2, Z &o3)
{
    Z a0, a1;
    if constexpr (H2) { a0 = zfma<INV, Q2>(v0, v2, h); a1 = zfma<INV, Q2 + 2>(v0, v2, h); }
    else { a0 = zadd<INV, Q2>(v0, v2); a1 = zadd<INV, Q2 + 2>(v0, v2); }
    const Z b0 = zadd<INV, Q3 - Q1 + 4>(v1, v3), b1 = zadd<INV, Q3 - Q1 + 6>(v1, v3);
    if constexpr (H13) {
        o0 = zfma<INV, Q1>(a0, b0, h); o2 = zfma<INV, Q1 + 2>(a0, b0, h);
        o1 = zfma<INV, Q1 + 1>(a1, b1, h); o3 = zfma<INV, Q1 + 3>(a1, b1, h);
    } else {
        o0 = zadd<INV, Q1>(a0, b0); o2 = zadd<INV, Q1 + 2>(a0, b0);
        o1 = zadd<INV, Q1 + 1>(a1, b1); o3 = zadd<INV, Q1 + 3>(a1, b1);
    }
}
template <bool INV> __device__ __forceinline__ void dft4(Z &a, Z &b, Z &c, Z &d)
{
    Z o0, o1, o2, o3;
    dft4<INV, 0, 0, 0, false, false>(a, b, c, d, 1.0f, o0, o1, o2, o3);
    a = o0; b = o1; c = o2; d = o3;
}
template <bool INV> __device__ __forceinline__ void dft3(Z &a, Z &b, Z &c)
{
    const float h = 0.8660254037844386f;
    const Z t = zadd<INV, 0>(b, c), d = zadd<INV, 2>(b, c);
    const Z u = zfma<INV, 2>(a, t, 0.5f);
    a = zadd<INV, 0>(a, t);
    b = zfma<INV, 1>(u, d, h);
    c = zfma<INV, 3>(u, d, h);
}
template <int N, bool INV> struct ZDft;
// 8 = 2 x 4 and 16 = 4 x 4, the fours last: what a last stage of twos rounds off lies at
// the highest wavenumbers, where a second derivative weighs it most
template <bool INV> struct ZDft<8, INV> {
    static __device__ __forceinline__ void run(Z *v)
    {
        const float h = 0.7071067811865476f;
        Z b[4];
#pragma unroll
        for (int m = 0; m < 4; m++) {
            b[m] = zadd<INV, 2>(v[m], v[m + 4]);
            v[m] = zadd<INV, 0>(v[m], v[m + 4]);
        }
        Z o[8];
        dft4<INV, 0, 0, 0, false, false>(v[0], v[1], v[2], v[3], h, o[0], o[2], o[4], o[6]);
        dft4<INV, 0, 1, 1, false, true>(b[0], zw8<INV>(b[1]), b[2], zw8<INV>(b[3]), h, o[1], o[3], o[5], o[7]);
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = o[k];
    }
};
template <bool INV> struct ZDft<16, INV> {
    static __device__ __forceinline__ void run(Z *v)
    {
        const float h = 0.7071067811865476f, c = 0.9238795325112867f, s = 0.3826834323650898f;   // W_8, W_16
#pragma unroll
        for (int m = 0; m < 4; m++) dft4<INV>(v[m], v[4 + m], v[8 + m], v[12 + m]);
        // v[4 k1 + m2] now
        Z o[16];
        dft4<INV, 0, 0, 0, false, false>(v[0], v[1], v[2], v[3], h, o[0], o[4], o[8], o[12]);
        dft4<INV, 0, 0, 0, true, false>(v[4], ztw<INV>(v[5], c, s), zw8<INV>(v[6]), ztw<INV>(v[7], s, c), h, o[1], o[5], o[9], o[13]);
        dft4<INV, 0, 1, 1, false, true>(v[8], zw8<INV>(v[9]), v[10], zw8<INV>(v[11]), h, o[2], o[6], o[10], o[14]);
        dft4<INV, 0, 1, 2, true, false>(v[12], ztw<INV>(v[13], s, c), zw8<INV>(v[14]), ztw<INV>(v[15], c, s), h, o[3], o[7], o[11], o[15]);
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = o[k];
    }
};
// 6 = 2 x 3 and 12 = 3 x 4 by the map of coprime factors (no twiddles)
template <bool INV> struct ZDft<6, INV> {
    static __device__ __forceinline__ void run(Z *v)
    {
        Z a[3], b[3];
#pragma unroll
        for (int n2 = 0; n2 < 3; n2++) {
            const Z x = v[(2 * n2) % 6], y = v[(3 + 2 * n2) % 6];
            a[n2] = zadd<INV, 0>(x, y);
            b[n2] = zadd<INV, 2>(x, y);
        }
        dft3<INV>(a[0], a[1], a[2]);
        dft3<INV>(b[0], b[1], b[2]);
#pragma unroll
        for (int k2 = 0; k2 < 3; k2++) { v[(4 * k2) % 6] = a[k2]; v[(3 + 4 * k2) % 6] = b[k2]; }
    }
};
template <bool INV> struct ZDft<12, INV> {
    static __device__ __forceinline__ void run(Z *v)
    {
        Z a[12];
#pragma unroll
        for (int n1 = 0; n1 < 3; n1++) {
            Z *t = a + 4 * n1;
#pragma unroll
            for (int n2 = 0; n2 < 4; n2++) t[n2] = v[(4 * n1 + 3 * n2) % 12];
            dft4<INV>(t[0], t[1], t[2], t[3]);
        }
#pragma unroll
        for (int k2 = 0; k2 < 4; k2++) {
            dft3<INV>(a[k2], a[4 + k2], a[8 + k2]);
#pragma unroll
            for (int k1 = 0; k1 < 3; k1++) v[(4 * k1 + 9 * k2) % 12] = a[4 * k1 + k2];
        }
    }
};

// ---- shape ---------------------------------------------------------------------------
// DIR 0: x lines (a tile = 2S contiguous rows), DIR 1: y lines (a tile = 2S adjacent
// columns over all ny rows).
template <int DIR, int A, int B, int C, int S>
struct CpShape {
    static constexpr int N = A * B * C;
    static constexpr int NG = S / 2;                      // groups of four lines
    static constexpr int RL = C;                          // radix of the last level
    static constexpr int M = N / A, NL = N / RL;          // DFTs of the first and the last level
    // threads per group: one DFT each on the first level (384-point x lines: 64
    // rather than 48, whole warps)
    static constexpr int T = DIR == 0 ? (M + 31) / 32 * 32 : M;
    static constexpr int NT = NG * T;
    // groups side by side, lane by lane: all of a y tile (what a warp stores is then as
    // wide as the tile)
    static constexpr int ST = DIR == 0 ? 1 : NG, U = ST * T;
    static constexpr int D2 = (A * C + T - 1) / T, DL = (NL + T - 1) / T;
    static constexpr int GT = 4 * N;                      // reals of a group in the tile
    static constexpr int TILE = NG * GT;
    // rows of the first exchange, in points; the lanes of its second level run over k1
    // (unless C = 8, where they run over c first), an odd row apart
    static constexpr int XS = C == 8 ? M : M + 1, GX = A * XS;
    // twiddle rows W^(j x), all of them (products of two of them in place of some err 2-3 %
    // more per exchange)
    static constexpr int R1 = A - 1, R2 = B - 1;
    static constexpr size_t SMEM = 4 * (2 * (size_t)TILE + 4 * (size_t)NG * GX + 2 * (size_t)(R1 * M) + 4 * (size_t)(R2 * C) + 6 * (size_t)N);
    static constexpr int MINB = NT <= 256 && 2 * (SMEM + 1152) <= 233472 ? 2 : 1;
    static_assert(T >= M && (C == 8 || M % 2 == 0) && SMEM + 128 <= 232448, "shape");
    static_assert(GX >= N, "spectra fit the exchange");
};

// ---- the kernel --------------------------------------------------------------------
// wsync: x lines' groups are whole warps, so the exchanges need only named barriers
// (0: CTA-wide ones).  The groups then run through their tiles
// independently; an "empty" mbarrier per tile buffer (one arrival per warp once it
// is done with the buffer) tells the thread that issues the TMA copies when a
// buffer may be refilled.
template <int DIR, int A, int B, int C, int S, int NJ>
__global__ void __launch_bounds__(CpShape<DIR, A, B, C, S>::NT, CpShape<DIR, A, B, C, S>::MINB)
line_cp(const __grid_constant__ JobPackCP<NJ> jobs, const __grid_constant__ TmapPackCP<DIR, NJ> tmaps, LineTables<float> tb,
        int nx, int ny, int nz, int tpp, int total, int wsync, int *err)
{
    PDL_WAIT();
    using P = CpShape<DIR, A, B, C, S>;
    constexpr int N = P::N, T = P::T, NT = P::NT, M = P::M, NL = P::NL, RL = P::RL, XS = P::XS, TILE = P::TILE;
    const bool WS = DIR == 0 && wsync;

    extern __shared__ __align__(128) unsigned char smem[];
    float *tile0 = reinterpret_cast<float *>(smem);
    Z *ex = reinterpret_cast<Z *>(tile0 + 2 * TILE);
    Tw *tw2 = reinterpret_cast<Tw *>(ex + P::NG * P::GX);   // [row][c]
    float2 *tw1 = reinterpret_cast<float2 *>(tw2 + P::R2 * C);  // [row][m']: cosine and sine
    float2 *mul = tw1 + P::R1 * M;  // multipliers: d1, d2, dealias
    __shared__ __align__(8) uint64_t bar[4];                   // full[2], empty[2]

    const int tid = threadIdx.x;
    constexpr int ST = P::ST, U = P::U;
    const int unit = tid / U, side = tid % ST;
    const int g = unit * ST + side, lane = (tid % U) / ST;
    const size_t np = (size_t)nx * ny;
    auto sync = [&]() {
        if (!WS) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(unit + 1), "n"(U) : "memory");
    };

    for (int e = tid; e < P::R1 * M + P::R2 * C; e += NT) {
        const bool first = e < P::R1 * M;
        const int q = first ? e : e - P::R1 * M, w = first ? M : C;
        const int r = q / w, x = q - r * w;
        const int j = r + 1;
        const float2 v = tb.tw[(first ? j * x : A * j * x) % N];
        if (first) tw1[q] = make_float2(v.x, -v.y);
        else tw2[q] = Tw{ bc2(v.x), bc2(-v.y) };
    }
    for (int e = tid; e < N; e += NT) {
        mul[e] = bc2(tb.m1[e]);
        mul[N + e] = bc2(tb.m2[e]);
        mul[2 * N + e] = bc2(tb.mda[e]);
    }
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_init(&bar[2], NT / 32);
        mbar_init(&bar[3], NT / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async();
    }
    __syncthreads();

    // (thread 0)
    auto issue = [&](int t, int buf) {
        const int job = t / (nz * tpp);
        const int rem = t - job * (nz * tpp);
        const int plane = rem / tpp;
        const int l0 = (rem - plane * tpp) * 2 * S;
        float *dst = tile0 + buf * TILE;
        mbar_expect_tx(&bar[buf], 2 * S * N * 4);
        if constexpr (DIR == 0) {
            const float *src = jobs.j[job].in + (size_t)plane * np + (size_t)l0 * nx;
#pragma unroll
            for (int c = 0; c < P::NG; c++) tma_load(dst + c * P::GT, src + (size_t)c * 4 * N, 16 * N, &bar[buf]);
        } else {
            // boxes of 2S columns x (up to 256) rows
            constexpr int BR = ybox_rows(N);
#pragma unroll
            for (int c = 0; c < N / BR; c++)
                tma_load_3d(dst + (size_t)c * BR * 2 * S, &tmaps.m[job], l0, c * BR, plane, &bar[buf]);
        }
    };
    // A wait that runs out is reported and taken as done; this thread then issues
    // no more copies and waits for no more of them but those in flight
    bool bad = false;
    auto wait = [&](int b, int parity) {
        if (!mbar_wait(&bar[b], parity, bad ? 1 : MBAR_POLLS)) {
            atomicExch(err, 1);
            bad = true;
        }
    };

    Z *exg = ex + unit * ST * P::GX + side;
    // the second level's k1 and c; the places of the second exchange, which uses the tile's
    // buffer
    auto lev2 = [](int q, int &k1, int &c) {
        k1 = C == 8 ? q / C : q % A;
        c = C == 8 ? q % C : q / A;
    };
    auto x2 = [](int k1, int k2, int c) { return C == 8 ? (k2 * A + k1) * 8 + (c ^ (k1 & 7)) : c * NL + k2 * A + k1; };

    int issued = 0;
    if (tid == 0) {
        if (blockIdx.x < total) { issue(blockIdx.x, 0); issued = 1; }
    }
    int it = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x, it++) {
        float *cur = tile0 + (it & 1) * TILE;
        if (tid == 0 && t + (int)gridDim.x < total && !bad) {
            // every warp is done with the other buffer (its use in iteration it - 1)
            if (WS && it >= 1) wait(2 + ((it + 1) & 1), ((it - 1) >> 1) & 1);
            if (!bad) {
                fence_async();
                issue(t + gridDim.x, (it + 1) & 1);
                issued++;
            }
        }
        wait(it & 1, (it >> 1) & 1);
        const int job = t / (nz * tpp);
        const int rem = t - job * (nz * tpp);
        const int plane = rem / tpp;
        const int la = (rem - plane * tpp) * 2 * S + 4 * g;   // the group's first line
        const size_t base = (size_t)plane * np + (DIR == 0 ? (size_t)la * N : (size_t)la);
        const LineJob<float> &jb = jobs.j[job];
        const int op1 = jb.op1, op2 = jb.op2;
        Z *xg = reinterpret_cast<Z *>(cur) + unit * ST * (P::GT / 4) + side;

        // element e of the group's lines in the tile; its place in a field
        auto tile_z = [&](int e) -> Z {
            if constexpr (DIR == 0) {
                const float *r = cur + g * P::GT + e;
                return Z{ make_float2(r[0], r[N]), make_float2(r[2 * N], r[3 * N]) };
            } else {
                return xg[ST * e];
            }
        };
        auto load = [&](const float *f, int e) -> Z {
            if constexpr (DIR == 0) {
                const float *r = f + base + e;
                return Z{ make_float2(r[0], r[N]), make_float2(r[2 * N], r[3 * N]) };
            } else {
                return *reinterpret_cast<const Z *>(f + base + (unsigned)(e * nx));
            }
        };
        auto store = [&](float *f, int e, const Z &v) {
            if constexpr (DIR == 0) {
                float *r = f + base + e;
                r[0] = v.r.x; r[N] = v.r.y; r[2 * N] = v.i.x; r[3 * N] = v.i.y;
            } else {
                *reinterpret_cast<Z *>(f + base + (unsigned)(e * nx)) = v;
            }
        };

        Z X[P::DL][RL];   // X[d][k3] = spectrum at lane + T d + NL k3
        if (op1 != OP_INV) {
            if (M % T == 0 || lane < M) {
                Z a[A];
#pragma unroll
                for (int m = 0; m < A; m++) a[m] = tile_z(lane + M * m);
                ZDft<A, false>::run(a);
                exg[ST * lane] = a[0];
#pragma unroll
                for (int k = 1; k < A; k++) exg[ST * (k * XS + lane)] = ztw<false>(a[k], tw1[(k - 1) * M + lane].x, tw1[(k - 1) * M + lane].y);
            }
            sync();
#pragma unroll
            for (int d = 0; d < P::D2; d++) {
                const int q = lane + T * d;
                int k1, c;
                lev2(q, k1, c);
                if ((A * C) % T == 0 || q < A * C) {
                    Z b[B];
#pragma unroll
                    for (int m = 0; m < B; m++) b[m] = exg[ST * (k1 * XS + C * m + c)];
                    ZDft<B, false>::run(b);
                    xg[ST * x2(k1, 0, c)] = b[0];
#pragma unroll
                    for (int k = 1; k < B; k++) xg[ST * x2(k1, k, c)] = ztw<false>(b[k], tw2[(k - 1) * C + c]);
                }
            }
            sync();
#pragma unroll
            for (int d = 0; d < P::DL; d++) {
                const int q = lane + T * d;
                if (NL % T == 0 || q < NL) {
#pragma unroll
                    for (int m = 0; m < RL; m++) X[d][m] = xg[ST * x2(q % A, q / A, m)];
                    ZDft<RL, false>::run(X[d]);
                }
            }
        } else {
            // halfcomplex input lines a (re) and b (im): Z_k = A_k + i B_k
#pragma unroll
            for (int d = 0; d < P::DL; d++) {
                const int q = lane + T * d;
                if (NL % T == 0 || q < NL) {
#pragma unroll
                    for (int m = 0; m < RL; m++) {
                        const int k = q + NL * m;
                        const int kk = k <= N / 2 ? k : N - k;
                        const bool edge = kk == 0 || 2 * kk == N;
                        const Z pa = tile_z(kk), pb = tile_z(edge ? kk : N - kk);   // (ha, hb)
                        X[d][m] = edge ? pa : zaxpy(k <= N / 2 ? 1.0f : -1.0f, zi(pb), pa);
                    }
                }
            }
            // (the exchanges' last readers, and the tile's)
            sync();
        }

        if (op1 == OP_FWD) {
            // separate Z into the halfcomplex spectra of the two real lines, through
            // the first exchange's rows, which no thread reads any more
#pragma unroll
            for (int d = 0; d < P::DL; d++) {
                const int q = lane + T * d;
                if (NL % T == 0 || q < NL) {
#pragma unroll
                    for (int m = 0; m < RL; m++) exg[ST * (q + NL * m)] = X[d][m];
                }
            }
            sync();
            const float f = 0.5f * jb.alpha1;
#pragma unroll 4
            for (int p = lane; p < N; p += T) {
                const int q = p == 0 ? 0 : N - p;
                const Z zp = exg[ST * p], zq = exg[ST * q];
                Z v = 2 * p <= N ? zscale(zadd<false, 0>(zp, zq), f) : zscale(zi(zadd<false, 2>(zp, zq)), f);
                if (jb.acc1) v = zadd<false, 0>(load(jb.out1, p), v);
                store(jb.out1, p, v);
            }
            fence_async();
            sync();
            if (WS && (tid & 31) == 0) mbar_arrive(&bar[2 + (it & 1)]);
            continue;
        }

        // one or two outputs: Y = m(X), inverse transform, store (a
        // halfcomplex input takes a second output only for OP_D1: the
        // derivative of its inverse)
        const int nout = (op2 != OP_NONE && (op1 != OP_INV || op2 == OP_D1)) ? 2 : 1;
#pragma unroll 1
        for (int o = 0; o < nout; o++) {
            const int op = o == 0 ? op1 : op2;
            float *out = o == 0 ? jb.out1 : jb.out2;
            const float alpha = o == 0 ? jb.alpha1 : jb.alpha2;
            const int acc = o == 0 ? jb.acc1 : jb.acc2;
            const float2 *mt = mul + (op == OP_D1 ? 0 : op == OP_D2 ? N : 2 * N);
#pragma unroll
            for (int d = 0; d < P::DL; d++) {
                const int q = lane + T * d;
                if (NL % T == 0 || q < NL) {
                    Z y[RL];
#pragma unroll
                    for (int m = 0; m < RL; m++) y[m] = X[d][m];
                    if (op != OP_INV) {
#pragma unroll
                        for (int m = 0; m < RL; m++) {
                            y[m] = zscale(y[m], mt[q + NL * m]);
                        }
                    }
                    ZDft<RL, true>::run(y);
#pragma unroll
                    for (int m = 0; m < RL; m++) {
                        xg[ST * x2(q % A, q / A, m)] = y[m];
                    }
                }
            }
            sync();
#pragma unroll
            for (int d = 0; d < P::D2; d++) {
                const int q = lane + T * d;
                int k1, c;
                lev2(q, k1, c);
                if ((A * C) % T == 0 || q < A * C) {
                    Z b[B];
                    b[0] = xg[ST * x2(k1, 0, c)];
#pragma unroll
                    for (int k = 1; k < B; k++) b[k] = ztw<true>(xg[ST * x2(k1, k, c)], tw2[(k - 1) * C + c]);
                    ZDft<B, true>::run(b);
#pragma unroll
                    for (int m = 0; m < B; m++) exg[ST * (k1 * XS + C * m + c)] = b[m];
                }
            }
            fence_async();
            sync();
            if (WS && o == nout - 1 && (tid & 31) == 0) mbar_arrive(&bar[2 + (it & 1)]);
            if (M % T == 0 || lane < M) {
                Z a[A];
                a[0] = exg[ST * lane];
#pragma unroll
                for (int k = 1; k < A; k++) a[k] = ztw<true>(exg[ST * (k * XS + lane)], tw1[(k - 1) * M + lane].x, tw1[(k - 1) * M + lane].y);
                ZDft<A, true>::run(a);
                const float f = op == OP_INV ? alpha / (float)N : alpha;
                float addv = 0.0f;
                if (op == OP_INV && jb.addk) addv = (float)jb.addk[plane];
                if (op == OP_INV) addv = addv + (float)jb.addc;
                // (an accumulation's old values are asked for CH at a time; more cost
                // y lines of 512 points spilled registers)
                constexpr int CH = DIR == 0 ? 4 : 2;
#pragma unroll
                for (int m0 = 0; m0 < A; m0 += CH) {
                    Z old[CH];
                    if (acc) {
#pragma unroll
                        for (int m = 0; m < CH; m++) old[m] = load(out, lane + M * (m0 + m));
                    }
#pragma unroll
                    for (int m = 0; m < CH; m++) {
                        // (the derivative's factor i)
                        Z v = op == OP_D1 ? zi(a[m0 + m]) : a[m0 + m];
                        v = acc ? zaxpy(f, v, old[m]) : zscale(v, f);
                        if (op == OP_INV) v = zaddc(v, addv);
                        store(out, lane + M * (m0 + m), v);
                    }
                }
            }
        }
    }
    if (tid == 0 && bad) {
        // copies still in flight land before the CTA's shared memory is released
        for (int i = issued > 2 ? issued - 2 : 0; i < issued; i++) mbar_wait(&bar[i & 1], (i >> 1) & 1);
    }
}

template <int DIR, int A, int B, int C, int S, int NJ>
static int run_nj(Engine *E, const LineJob<float> *jobs, int nj, const char *name)
{
    using P = CpShape<DIR, A, B, C, S>;
    static SmemLimit limit;
    CUDA_TRY(limit.raise((const void *)line_cp<DIR, A, B, C, S, NJ>, (int)P::SMEM));
    const int L = DIR == 0 ? E->ny : E->nx;
    const int tpp = L / (2 * S);
    JobPackCP<NJ> pk;
    memset(&pk, 0, sizeof(pk));
    double fields = 0.0;
    for (int j = 0; j < nj; j++) {
        pk.j[j] = jobs[j];
        fields += 2.0 + (jobs[j].acc1 ? 1.0 : 0.0);
        if (jobs[j].op2 != OP_NONE) fields += 1.0 + (jobs[j].acc2 ? 1.0 : 0.0);
    }
    TmapPackCP<DIR, NJ> tp;
    memset(&tp, 0, sizeof(tp));
    if constexpr (DIR == 1) {
        int st;
        for (int j = 0; j < nj; j++)
            if ((st = encode_ymap(&tp.m[j], jobs[j].in, E->nx, E->ny, E->nz, S, ybox_rows(P::N)))) return st;
    }
    const int total = nj * E->nz * tpp;
    int per_sm = 1;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, line_cp<DIR, A, B, C, S, NJ>, P::NT, P::SMEM));
    if (per_sm < 1) per_sm = 1;
    int grid = E->num_sms * per_sm;
    if (grid > total) grid = total;
    E->prof_begin(name, fields * (double)E->n * sizeof(float));
    CUDA_TRY(launch_k(*E, line_cp<DIR, A, B, C, S, NJ>, dim3(grid), dim3(P::NT), P::SMEM, pk, tp, E->tables<float>(DIR), E->nx, E->ny,
                      E->nz, tpp, total, (int)E->ct_warp, E->dev_err));
    E->prof_end();
    CUDA_TRY(cudaGetLastError());
    return VEC_OK;
}
template <int DIR, int A, int B, int C, int S>
static int run_cp(Engine *E, const LineJob<float> *jobs, int nj, const char *name)
{
    return nj <= NJ_SMALL ? run_nj<DIR, A, B, C, S, NJ_SMALL>(E, jobs, nj, name) : run_nj<DIR, A, B, C, S, MAX_JOBS>(E, jobs, nj, name);
}

// nj <= MAX_JOBS jobs of lines of 384, 512, 768 or 1024 points with tiles of 2 S
int launch_lines_cp(Engine *E, int dir, const LineJob<float> *jobs, int nj, int S, const char *name)
{
    const int n = dir == 0 ? E->nx : E->ny;
#define CP_CASE(NN, A, B, C, SS)                                                                     \
    if (n == NN && S == SS) return dir == 0 ? run_cp<0, A, B, C, SS>(E, jobs, nj, name) : run_cp<1, A, B, C, SS>(E, jobs, nj, name);
    CP_CASE(384, 8, 8, 6, 8) CP_CASE(512, 8, 8, 8, 8) CP_CASE(768, 8, 8, 12, 8) CP_CASE(1024, 16, 8, 8, 8)
    CP_CASE(768, 8, 8, 12, 4) CP_CASE(1024, 16, 8, 8, 4)
#undef CP_CASE
    return -1;
}
