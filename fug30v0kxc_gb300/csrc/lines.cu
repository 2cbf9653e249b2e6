// lines.cu -- horizontal spectral operators of src/fft.F90 in FP32 for every
// line length 2^a 3^b 5^c (FP64: lines_fx.cu; the lengths of the split step's
// usual grids: lines_ct.cu).
//
// A group of G = 32 / Q lanes owns a sequence z = a + i b of two real lines in shared
// memory and runs radix-8/4/2/3/5 passes on it in place, decimating in time both ways:
// forward from natural to digit-reversed order, and back through a second buffer, whose
// first pass gathers the spectrum in the order it needs and applies the operators'
// Hermitian multipliers (+ik, -k^2, the 2/3 truncation; tables in that order).  Warps
// synchronise their passes alone; the CTA meets for the row-by-row loads and stores of y
// lines.
//
// The eights come first and the fives last, both ways, and twiddles before the DFTs: what
// the last stages round off lies at multiples of n / radix, and a second derivative weighs it
// by the fourth power, while the first passes of the inverse meet a smooth line's spectrum
// mostly in zeros.  The errors are those of plain Stockham stages of 8, 4, 2, 3 and 5 points,
// or up to 6 % less where a two or four takes a three along.  Passes in place both ways (no
// gathering, no second buffer for a single output) with the eights last take 5 to 30 % less
// time, but err up to 20 % more on smooth lines and up to 60 % on a constant plus little.
//
// Measured (d2bydx, d2bydy) against the Stockham kernel, which kept 2048 elements per CTA,
// synchronised it between all stages and took 8 elements per thread through a call per
// stage: 240^2 x 129 220 227 -> 58 63 us, 480^2 x 65 419 446 -> 105 130, 1000^2 x 33
// 898 968 -> 314 384.  (The register kernel of lines_ct.cu is faster at its own lengths:
// 256^2 x 129 34 us.)
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <vector>

#include "common.cuh"
#include "engine.h"

template <int NJ> struct JobPack { LineJob<float> j[NJ]; };

// ---- radix kernels (natural order outputs X_0..X_{R-1}) ----------------------
template <typename C>
__device__ __forceinline__ C cmul(C a, C b) { C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r; }
template <typename C>
__device__ __forceinline__ C cadd(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C>
__device__ __forceinline__ C csub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
// multiply by -i (forward) or +i (inverse)
template <bool INV, typename C>
__device__ __forceinline__ C rot90(C a) { C r; if (INV) { r.x = -a.y; r.y = a.x; } else { r.x = a.y; r.y = -a.x; } return r; }

template <int RAD, bool INV, typename C> struct Dft;

template <bool INV, typename C> struct Dft<2, INV, C> {
    static __device__ __forceinline__ void run(C *v) { C a = v[0], b = v[1]; v[0] = cadd(a, b); v[1] = csub(a, b); }
};
template <bool INV, typename C> struct Dft<4, INV, C> {
    static __device__ __forceinline__ void run(C *v) {
        C a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
        C b0 = cadd(v[1], v[3]), b1 = rot90<INV>(csub(v[1], v[3]));
        v[0] = cadd(a0, b0); v[1] = cadd(a1, b1); v[2] = csub(a0, b0); v[3] = csub(a1, b1);
    }
};
template <bool INV, typename C> struct Dft<8, INV, C> {
    static __device__ __forceinline__ void run(C *v) {
        using R = decltype(v[0].x);
        const R h = (R)0.70710678118654752440084436210484904;   // sqrt(2)/2
        C a[4], b[4];
#pragma unroll
        for (int j = 0; j < 4; j++) { a[j] = cadd(v[j], v[j + 4]); b[j] = csub(v[j], v[j + 4]); }
        // b_j *= W8^j, W8 = exp(-+ i pi/4)
        {
            C t = b[1];
            if (!INV) { b[1].x = h * (t.x + t.y); b[1].y = h * (t.y - t.x); }
            else      { b[1].x = h * (t.x - t.y); b[1].y = h * (t.y + t.x); }
            b[2] = rot90<INV>(b[2]);
            t = b[3];
            if (!INV) { b[3].x = h * (t.y - t.x); b[3].y = -h * (t.x + t.y); }
            else      { b[3].x = -h * (t.x + t.y); b[3].y = h * (t.x - t.y); }
        }
        Dft<4, INV, C>::run(a);
        Dft<4, INV, C>::run(b);
#pragma unroll
        for (int m = 0; m < 4; m++) { v[2 * m] = a[m]; v[2 * m + 1] = b[m]; }
    }
};
template <bool INV, typename C> struct Dft<3, INV, C> {
    static __device__ __forceinline__ void run(C *v) {
        using R = decltype(v[0].x);
        const R c1 = (R)-0.5;
        const R s1 = INV ? (R)0.86602540378443864676372317075293618 : (R)-0.86602540378443864676372317075293618;
        C t1 = cadd(v[1], v[2]), t2 = csub(v[1], v[2]);
        C x0 = cadd(v[0], t1);
        C m1; m1.x = v[0].x + c1 * t1.x; m1.y = v[0].y + c1 * t1.y;
        // i*s1*t2
        C m2; m2.x = -s1 * t2.y; m2.y = s1 * t2.x;
        v[0] = x0; v[1] = cadd(m1, m2); v[2] = csub(m1, m2);
    }
};
template <bool INV, typename C> struct Dft<5, INV, C> {
    static __device__ __forceinline__ void run(C *v) {
        using R = decltype(v[0].x);
        const R c1 = (R)0.30901699437494742410229341718281906;    // cos(2pi/5)
        const R c2 = (R)-0.80901699437494742410229341718281906;   // cos(4pi/5)
        const R sg = INV ? (R)1 : (R)-1;
        const R s1 = sg * (R)0.95105651629515357211643933337938214;  // sin(2pi/5)
        const R s2 = sg * (R)0.58778525229247312916870595463907277;  // sin(4pi/5)
        C t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
        C d1 = csub(v[1], v[4]), d2 = csub(v[2], v[3]);
        C x0 = cadd(v[0], cadd(t1, t2));
        C a1, a2, b1, b2;
        a1.x = v[0].x + c1 * t1.x + c2 * t2.x; a1.y = v[0].y + c1 * t1.y + c2 * t2.y;
        a2.x = v[0].x + c2 * t1.x + c1 * t2.x; a2.y = v[0].y + c2 * t1.y + c1 * t2.y;
        // b1 = i (s1 d1 + s2 d2), b2 = i (s2 d1 - s1 d2)
        R u1x = s1 * d1.x + s2 * d2.x, u1y = s1 * d1.y + s2 * d2.y;
        R u2x = s2 * d1.x - s1 * d2.x, u2y = s2 * d1.y - s1 * d2.y;
        b1.x = -u1y; b1.y = u1x;
        b2.x = -u2y; b2.y = u2x;
        v[0] = x0; v[1] = cadd(a1, b1); v[4] = csub(a1, b1); v[2] = cadd(a2, b2); v[3] = csub(a2, b2);
    }
};
// 6 = 2 x 3 and 12 = 4 x 3 by the map of coprime factors (no twiddles)
template <int A, bool INV, typename C>
__device__ __forceinline__ void dft_a3(C *v)
{
    constexpr int N = 3 * A, E = A == 2 ? 3 : 9;      // 1 mod A, 0 mod 3
    C a[3][A];
#pragma unroll
    for (int m = 0; m < 3; m++) {
#pragma unroll
        for (int j = 0; j < A; j++) a[m][j] = v[(3 * j + A * m) % N];
        Dft<A, INV, C>::run(a[m]);
    }
#pragma unroll
    for (int k = 0; k < A; k++) {
        C b[3] = { a[0][k], a[1][k], a[2][k] };
        Dft<3, INV, C>::run(b);
#pragma unroll
        for (int m = 0; m < 3; m++) v[(E * k + 4 * m) % N] = b[m];
    }
}
template <bool INV, typename C> struct Dft<6, INV, C> { static __device__ __forceinline__ void run(C *v) { dft_a3<2, INV>(v); } };
template <bool INV, typename C> struct Dft<12, INV, C> { static __device__ __forceinline__ void run(C *v) { dft_a3<4, INV>(v); } };

#define FS_TPB 256
// element i of a sequence's buffer: a word of padding per 2^sh, against the bank conflicts
// of even strides (FsPlan: the best for the length, of either buffer)
__device__ __forceinline__ int fs_at(int i, int sh) { return i + (i >> sh); }

// one pass: radix R over the elements j + m M of every block of R M; tw: its twiddles
struct FsPass { int n, M, G, l, sh; unsigned mg; const float2 *tw; };

template <int R>
__device__ __forceinline__ void fs_places(const FsPass &a, int b, int &q, int &j, int *at)
{
    q = (int)(((unsigned long long)(unsigned)b * a.mg) >> 31);
    j = b - q * a.M;
    const int i = q * R * a.M + j;
#pragma unroll
    for (int m = 0; m < R; m++) at[m] = fs_at(i + m * a.M, a.sh);
}
// W^(r K) for block q of wavenumber K so far (not in the FIRST pass), then DFT_R
template <int R, bool FIRST>
__device__ __forceinline__ void fs_fwd(float2 *buf, const FsPass &a)
{
    const int nb = a.n / (R * a.M);
    for (int b = a.l; b < a.n / R; b += a.G) {
        int q, j, at[R];
        float2 v[R];
        fs_places<R>(a, b, q, j, at);
#pragma unroll
        for (int r = 0; r < R; r++) {
            v[r] = buf[at[r]];
            if (!FIRST && r) v[r] = cmul(v[r], a.tw[(r - 1) * nb + q]);
        }
        Dft<R, false, float2>::run(v);
#pragma unroll
        for (int r = 0; r < R; r++) buf[at[r]] = v[r];
    }
    __syncwarp();
}
// the first inverse pass (M = 1), from the spectrum src in the forward passes' order,
// times the multipliers mul (d1: i times), or from a halfcomplex line pair (HC):
// Z_k = A_k + i B_k
template <int R, bool HC>
__device__ __forceinline__ void fs_inv_first(float2 *buf, const float2 *src, const FsPass &a, int sha, const unsigned short *tab,
                                             const float *mul, bool d1)
{
    for (int b = a.l; b < a.n / R; b += a.G) {
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int i = b * R + r, t = __ldg(tab + i);
            if (HC) {
                const int kk = min(t, a.n - t);
                const bool edge = kk == 0 || 2 * kk == a.n;
                const float2 pa = src[fs_at(kk, sha)];
                float2 pc = src[fs_at(edge ? 0 : a.n - kk, sha)];
                if (edge) pc = make_float2(0.0f, 0.0f);
                if (2 * t > a.n) { pc.x = -pc.x; pc.y = -pc.y; }
                v[r] = make_float2(pa.x - pc.y, pc.x + pa.y);
            } else {
                v[r] = src[fs_at(t, sha)];
            }
            if (mul) {
                const float m = __ldg(mul + i);
                const float2 z = v[r];
                v[r].x = d1 ? -m * z.y : m * z.x;
                v[r].y = d1 ? m * z.x : m * z.y;
            }
        }
        Dft<R, true, float2>::run(v);
#pragma unroll
        for (int r = 0; r < R; r++) buf[fs_at(b * R + r, a.sh)] = v[r];
    }
    __syncwarp();
}
// the others; OUT (the last one of x lines): the results to the two rows
struct FsOut { float *a, *b; float sc, add; };
template <int R, bool OUT>
__device__ __forceinline__ void fs_inv(float2 *buf, const FsPass &a, const FsOut &o)
{
    for (int b = a.l; b < a.n / R; b += a.G) {
        int q, j, at[R];
        float2 v[R];
        fs_places<R>(a, b, q, j, at);
#pragma unroll
        for (int r = 0; r < R; r++) {
            v[r] = buf[at[r]];
            if (r) {
                float2 w = a.tw[(r - 1) * a.M + j];
                w.y = -w.y;
                v[r] = cmul(v[r], w);
            }
        }
        Dft<R, true, float2>::run(v);
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (OUT) {
                o.a[j + r * a.M] = v[r].x * o.sc + o.add;
                o.b[j + r * a.M] = v[r].y * o.sc + o.add;
            } else {
                buf[at[r]] = v[r];
            }
        }
    }
    __syncwarp();
}
#define FS_SWITCH(R, CALL)                                                                 \
    switch (R) {                                                                           \
    case 12: CALL(12); break;                                                              \
    case 8: CALL(8); break;                                                                \
    case 6: CALL(6); break;                                                                \
    case 5: CALL(5); break;                                                                \
    case 4: CALL(4); break;                                                                \
    case 3: CALL(3); break;                                                                \
    default: CALL(2); break;                                                               \
    }

// DIR 0: x lines (sequence = two rows), DIR 1: y lines (two columns).  tpp tiles
// per plane: of Q sequences (one warp's, x) or S = warps Q (a CTA's, y).
template <int DIR, int NJ>
__global__ void __launch_bounds__(FS_TPB, 4)
line_kernel(const __grid_constant__ JobPack<NJ> jobs, const __grid_constant__ FsPlan pl, FsTables tb, int nx, int ny, int nz,
            int tpp, int total, int two)
{
    PDL_WAIT();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = pl.n, Q = pl.Q, G = 32 / Q, W = (int)blockDim.x / 32, S = W * Q, nb = pl.nb, sha = pl.sha, shb = pl.shb;
    float2 *bufA = reinterpret_cast<float2 *>(smem_raw);
    float2 *bufB = bufA + (size_t)S * nb;              // (two)
    float2 *tw = bufB + (two ? (size_t)S * nb : 0);
    const int tid = threadIdx.x, wid = tid >> 5, g = (tid & 31) / G, l = (tid & 31) % G, s = wid * Q + g;
    float2 *A = bufA + (size_t)s * nb, *B = two ? bufB + (size_t)s * nb : A;
    const size_t np = (size_t)nx * ny;
    const int pairs = (DIR == 0 ? ny : nx) / 2;
    const int ls = 31 - __clz(S), yq = tid & (S - 1), ye = tid >> ls, de = (int)blockDim.x >> ls;   // y: row by row
    for (int e = tid; e < pl.ntw; e += blockDim.x) tw[e] = tb.tw[e];
    __syncthreads();
    auto args = [&](int p, bool inverse) {
        FsPass a;
        a.n = n; a.G = G; a.l = l; a.sh = inverse ? shb : sha;
        a.M = inverse ? pl.iM[p] : pl.fM[p];
        a.mg = inverse ? pl.img[p] : pl.fmg[p];
        a.tw = tw + (inverse ? pl.itw[p] : pl.ftw[p]);
        return a;
    };
    const int t0 = DIR == 0 ? blockIdx.x * W + wid : blockIdx.x, dt = DIR == 0 ? gridDim.x * W : gridDim.x;
    for (int t = t0; t < total; t += dt) {
        const int job = t / (nz * tpp), rem = t - job * (nz * tpp);
        const int plane = rem / tpp, tile = rem - plane * tpp;
        const LineJob<float> &jb = jobs.j[job];
        const int op1 = jb.op1, op2 = jb.op2;
        const bool inv = op1 == OP_INV;
        const size_t pb = (size_t)plane * np;
        const int pair = tile * (DIR == 0 ? Q : S) + (DIR == 0 ? g : s);
        const bool valid = pair < pairs, yvalid = tile * S + yq < pairs;
        const size_t xoff = pb + 2 * (size_t)pair * nx, yoff = pb + 2 * ((size_t)tile * S + yq);

        // ---- load
        if (DIR == 0) {
            const float *r0 = jb.in + (valid ? xoff : 0);
            for (int e0 = l; e0 < n; e0 += 8 * G) {
                float2 v[8];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int e = e0 + c * G;
                    const bool in = valid && e < n;
                    v[c].x = in ? r0[e] : 0.0f;
                    v[c].y = in ? r0[e + nx] : 0.0f;
                }
#pragma unroll
                for (int c = 0; c < 8; c++)
                    if (e0 + c * G < n) A[fs_at(e0 + c * G, sha)] = v[c];
            }
            __syncwarp();
        } else {
            const float *in = jb.in + yoff;
            float2 *to = bufA + (size_t)yq * nb;
            for (int e0 = ye; e0 < n; e0 += 8 * de) {
                float2 v[8];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int e = e0 + c * de;
                    v[c] = make_float2(0.0f, 0.0f);
                    if (yvalid && e < n) v[c] = *reinterpret_cast<const float2 *>(in + (size_t)e * nx);
                }
#pragma unroll
                for (int c = 0; c < 8; c++)
                    if (e0 + c * de < n) to[fs_at(e0 + c * de, sha)] = v[c];
            }
            __syncthreads();
        }

        // ---- forward
        if (!inv) {
            const FsPass a0 = args(0, false);
#define CALL(R) fs_fwd<R, true>(A, a0)
            FS_SWITCH(pl.R[0], CALL)
#undef CALL
            for (int p = 1; p < pl.np; p++) {
                const FsPass a = args(p, false);
#define CALL(R) fs_fwd<R, false>(A, a)
                FS_SWITCH(pl.R[p], CALL)
#undef CALL
            }
        }

        if (op1 == OP_FWD) {
            // separate Z into the halfcomplex spectra of the two real lines
            auto sep = [&](const float2 *Z, int p) {
                const float2 zp = Z[fs_at(__ldg(tb.pos + p), sha)], zq = Z[fs_at(__ldg(tb.pos + (p == 0 ? 0 : n - p)), sha)];
                float2 v;
                if (2 * p <= n) { v.x = 0.5f * (zp.x + zq.x); v.y = 0.5f * (zp.y + zq.y); }
                else { v.x = 0.5f * (zq.y - zp.y); v.y = 0.5f * (zp.x - zq.x); }
                v.x *= jb.alpha1;
                v.y *= jb.alpha1;
                return v;
            };
            if (DIR == 0) {
                if (valid) {
                    float *oa = jb.out1 + xoff, *ob = oa + nx;
                    for (int p = l; p < n; p += G) {
                        const float2 v = sep(A, p);
                        oa[p] = jb.acc1 ? oa[p] + v.x : v.x;
                        ob[p] = jb.acc1 ? ob[p] + v.y : v.y;
                    }
                }
                __syncwarp();
            } else {
                __syncthreads();
                if (yvalid)
                    for (int p = ye; p < n; p += de) {
                        float2 v = sep(bufA + (size_t)yq * nb, p);
                        float2 *dd = reinterpret_cast<float2 *>(jb.out1 + yoff + (size_t)p * nx);
                        if (jb.acc1) { const float2 w = *dd; v.x = w.x + v.x; v.y = w.y + v.y; }
                        *dd = v;
                    }
                __syncthreads();
            }
            continue;
        }

        // ---- one or two inverse transforms
        const int nout = op2 != OP_NONE && (!inv || op2 == OP_D1) ? 2 : 1;
        for (int o = 0; o < nout; o++) {
            const int op = o == 0 ? op1 : op2;
            const float *mul = op == OP_D1 ? tb.m1 : op == OP_D2 ? tb.m2 : op == OP_DEALIAS ? tb.mda : nullptr;
            const float alpha = o == 0 ? jb.alpha1 : jb.alpha2;
            const int acc = o == 0 ? jb.acc1 : jb.acc2;
            float *ot = o == 0 ? jb.out1 : jb.out2;
            const float sc = op == OP_INV ? 1.0f / (float)n : 1.0f;
            float addv = 0.0f;
            if (op == OP_INV && jb.addk) addv = (float)jb.addk[plane];
            if (op == OP_INV) addv = addv + (float)jb.addc;
            // x lines: the last pass stores its results
            const bool fused = DIR == 0 && pl.np > 1 && __all_sync(0xffffffffu, valid && !acc && alpha == 1.0f);
            const FsOut to = { ot + xoff, ot + xoff + nx, sc, addv };
            {
                const FsPass a = args(0, true);
                if (inv) {
#define CALL(R) fs_inv_first<R, true>(B, A, a, sha, tb.pos, mul, op == OP_D1)
                    FS_SWITCH(pl.R[0], CALL)
#undef CALL
                } else {
#define CALL(R) fs_inv_first<R, false>(B, A, a, sha, tb.gat, mul, op == OP_D1)
                    FS_SWITCH(pl.R[0], CALL)
#undef CALL
                }
            }
            for (int p = 1; p < pl.np - (fused ? 1 : 0); p++) {
                const FsPass a = args(p, true);
#define CALL(R) fs_inv<R, false>(B, a, to)
                FS_SWITCH(pl.R[p], CALL)
#undef CALL
            }
            if (fused) {
                const FsPass a = args(pl.np - 1, true);
#define CALL(R) fs_inv<R, true>(B, a, to)
                FS_SWITCH(pl.R[pl.np - 1], CALL)
#undef CALL
                continue;
            }
            if (DIR == 0) {
                if (valid)
                    for (int e = l; e < n; e += G) {
                        const float2 z = B[fs_at(e, shb)];
                        float va = alpha * (z.x * sc), vb = alpha * (z.y * sc);
                        if (acc) { va = to.a[e] + va; vb = to.b[e] + vb; }
                        to.a[e] = va + addv;
                        to.b[e] = vb + addv;
                    }
                __syncwarp();
            } else {
                __syncthreads();
                const float2 *bs = bufB + (size_t)yq * nb;
                if (yvalid)
                    for (int e = ye; e < n; e += de) {
                        const float2 z = bs[fs_at(e, shb)];
                        float2 *dd = reinterpret_cast<float2 *>(ot + yoff + (size_t)e * nx);
                        float va = alpha * (z.x * sc), vb = alpha * (z.y * sc);
                        if (acc) { const float2 w = *dd; va = w.x + va; vb = w.y + vb; }
                        *dd = make_float2(va + addv, vb + addv);
                    }
                __syncthreads();
            }
        }
    }
}

// ---- host side ------------------------------------------------------------------
// Twiddles exp(-2 pi i e/n) computed on the host in double, exact at
// multiples of n/4 (quadrant reduction of the angle).
void sincos2pi_host(long e, long n, double *c, double *s)
{
    e %= n;
    if (e < 0) e += n;
    long q = (4 * e) / n, r = 4 * e - q * n;
    double cf, sf;
    if (2 * r <= n) { double a = (M_PI / 2.0) * ((double)r / (double)n); cf = cos(a); sf = sin(a); }
    else { double a = (M_PI / 2.0) * ((double)(n - r) / (double)n); cf = sin(a); sf = cos(a); }
    switch (q) {
    case 0: *c = cf; *s = sf; break;
    case 1: *c = -sf; *s = cf; break;
    case 2: *c = -cf; *s = -sf; break;
    default: *c = sf; *s = -cf; break;
    }
}

// multipliers for a direction: k1 = akx1-like table, k2 = akx2-like table
template <typename R>
int line_tables_make(int n, const double *k1, const double *k2, int icut, LineTables<R> *tb)
{
    using C = typename CT<R>::T;
    C *tw = (C *)malloc(sizeof(C) * n);
    R *m1 = (R *)malloc(sizeof(R) * n), *m2 = (R *)malloc(sizeof(R) * n), *mda = (R *)malloc(sizeof(R) * n);
    const double dn = (double)n;
    for (int e = 0; e < n; e++) {
        double c, s;
        sincos2pi_host(e, n, &c, &s);
        tw[e].x = (R)c;
        tw[e].y = (R)(-s);
        // first derivative: +i k for 0<k<n/2, -i k for k>n/2, 0 at DC / Nyquist
        double d1 = 0.0;
        if (e > 0 && 2 * e < n) d1 = k1[e] / dn;
        else if (2 * e > n) d1 = -k1[e] / dn;
        m1[e] = (R)d1;
        m2[e] = (R)(e == 0 ? 0.0 : k2[e] / dn);
        int kk = e <= n / 2 ? e : n - e;
        mda[e] = (R)(kk >= n / 2 - icut ? 0.0 : 1.0 / dn);
    }
    int st = VEC_OK;
    if (cudaMalloc(&tb->tw, sizeof(C) * n) != cudaSuccess || cudaMalloc(&tb->m1, sizeof(R) * n) != cudaSuccess ||
        cudaMalloc(&tb->m2, sizeof(R) * n) != cudaSuccess || cudaMalloc(&tb->mda, sizeof(R) * n) != cudaSuccess)
        st = VEC_ERR_ALLOC;
    if (!st) {
        cudaMemcpy(tb->tw, tw, sizeof(C) * n, cudaMemcpyHostToDevice);
        cudaMemcpy(tb->m1, m1, sizeof(R) * n, cudaMemcpyHostToDevice);
        cudaMemcpy(tb->m2, m2, sizeof(R) * n, cudaMemcpyHostToDevice);
        cudaMemcpy(tb->mda, mda, sizeof(R) * n, cudaMemcpyHostToDevice);
    }
    free(tw); free(m1); free(m2); free(mda);
    return st;
}

// k with its digits in the radices reversed: the place of wavenumber k after the forward
// passes, and the wavenumber at place k before the inverse ones
static int fs_reverse(const FsPlan &pl, int k)
{
    int M = pl.n, at = 0;
    for (int p = 0; p < pl.np; p++) {
        M /= pl.R[p];
        at += (k % pl.R[p]) * M;
        k /= pl.R[p];
    }
    return at;
}
// the general kernel's passes: the eights first, the fives last; a two or four takes one of
// the threes along (above 64 points: below them a pass more does not show, and 60 = 12 x 5
// errs 1 % more than 4 x 3 x 5)
int fs_plan_make(int n, FsPlan *pl)
{
    *pl = FsPlan{};
    int m = n;
    auto add = [&](int r) {
        if (pl->np < 8) pl->R[pl->np++] = r;
        m /= r;
    };
    while (m % 8 == 0) add(8);
    if (m % 2 == 0) add((m % 4 == 0 ? 4 : 2) * (m % 3 == 0 && n > 64 ? 3 : 1));
    for (int r : { 3, 5 })
        while (m % r == 0) add(r);
    if (m != 1 || n > 2048 || pl->np == 0) return VEC_ERR_SIZE;
    pl->n = n;
    int nb = 1;      // blocks before a forward pass, elements of an inverse one's block
    for (int p = 0; p < pl->np; p++) {
        const int R = pl->R[p];
        pl->fM[p] = n / (nb * R);
        pl->iM[p] = nb;
        pl->fmg[p] = (unsigned)(((1ull << 31) + pl->fM[p] - 1) / pl->fM[p]);
        pl->img[p] = (unsigned)(((1ull << 31) + nb - 1) / nb);
        pl->ftw[p] = pl->ntw;
        if (p) pl->ntw += (R - 1) * nb;
        pl->itw[p] = pl->ntw;
        if (p) pl->ntw += (R - 1) * nb;
        nb *= R;
    }
    pl->Q = n <= 32 ? 8 : n <= 64 ? 4 : n <= 128 ? 2 : 1;
    // the paddings with the fewest wavefronts: half a warp's words of 8 bytes, in 16 banks,
    // of the accesses of 128 butterflies or all (first: a forward pass's, or the gathering one's and the
    // separation's; second: an inverse pass's, and the gathering one's writes)
    int best[2] = { 0, 0 };
    std::vector<int> rev(n);
    for (int k = 0; k < n; k++) rev[k] = fs_reverse(*pl, k);
    for (int sh : { 31, 6, 5, 4, 3, 2 }) {
        const int G = 32 / pl->Q, ld = (n + ((n - 1) >> sh)) | 1;
        int cost[2] = { 0, 0 };
        auto count = [&](int which, int R, auto place) {
            for (int b0 = 0; b0 < n / R && b0 < 128; b0 += G)
                for (int r = 0; r < R; r++)
                    for (int h = 0; h < 32; h += 16) {
                        int used[16] = {}, top = 0;
                        for (int t = h; t < h + 16; t++) {
                            const int b = b0 + t % G;
                            if (b >= n / R) continue;
                            const int i = place(b, r), w = t / G * ld + i + (i >> sh);
                            if (++used[w & 15] > top) top = used[w & 15];
                        }
                        cost[which] += top;
                    }
        };
        for (int p = 0; p < pl->np; p++) {
            const int R = pl->R[p];
            for (int which = 0; which < 2; which++) {
                const int M = which ? pl->iM[p] : pl->fM[p];
                count(which, R, [&](int b, int r) { return b / M * R * M + b % M + r * M; });
            }
        }
        count(0, pl->R[0], [&](int b, int r) { return rev[rev[b * pl->R[0] + r]]; });
        count(0, 1, [&](int b, int) { return rev[b]; });
        if (best[0] == 0 || cost[0] < best[0]) { best[0] = cost[0]; pl->sha = sh; }
        if (best[1] == 0 || cost[1] < best[1]) { best[1] = cost[1]; pl->shb = sh; }
    }
    // (odd: the same element of a CTA's sequences on different banks)
    pl->nb = (n + ((n - 1) >> (pl->sha < pl->shb ? pl->sha : pl->shb))) | 1;
    return VEC_OK;
}
// its tables: the passes' twiddles, and the multipliers of line_tables_make in the order of
// the first inverse pass
int fs_tables_make(const FsPlan &pl, const double *k1, const double *k2, int icut, FsTables *tb)
{
    const int n = pl.n;
    std::vector<float2> tw, unit(n);
    for (int e = 0; e < n; e++) {
        double c, s;
        sincos2pi_host(e, n, &c, &s);
        unit[e] = make_float2((float)c, (float)-s);
    }
    auto add = [&](long e) { tw.push_back(unit[e % n]); };
    for (int p = 1; p < pl.np; p++) {
        const int R = pl.R[p], nb = pl.iM[p], ts = n / (nb * R);
        for (int r = 1; r < R; r++)
            for (int q = 0; q < nb; q++) {
                int K = 0, M = nb, rest = q;     // the block's wavenumber so far
                for (int s = 0, w = 1; s < p; w *= pl.R[s++]) {
                    M /= pl.R[s];
                    K += rest / M * w;
                    rest %= M;
                }
                add((long)r * K * ts);
            }
        for (int r = 1; r < R; r++)
            for (int j = 0; j < nb; j++) add((long)r * j * ts);
    }
    std::vector<float> m(3 * n);
    std::vector<unsigned short> pos(2 * n);       // and gat
    const double dn = (double)n;
    for (int i = 0; i < n; i++) {
        const int k = fs_reverse(pl, i);
        pos[i] = (unsigned short)k;
        pos[n + i] = (unsigned short)fs_reverse(pl, k);
        m[i] = (float)(k > 0 && 2 * k < n ? k1[k] / dn : 2 * k > n ? -k1[k] / dn : 0.0);
        m[n + i] = (float)(k == 0 ? 0.0 : k2[k] / dn);
        const int kk = k <= n / 2 ? k : n - k;
        m[2 * n + i] = (float)(kk >= n / 2 - icut ? 0.0 : 1.0 / dn);
    }
    const size_t bt = tw.size() * sizeof(float2), bm = m.size() * sizeof(float), bp = pos.size() * sizeof(short);
    std::vector<char> all(bt + bm + bp);
    if (bt) memcpy(all.data(), tw.data(), bt);
    memcpy(all.data() + bt, m.data(), bm);
    memcpy(all.data() + bt + bm, pos.data(), bp);
    if (cudaMalloc(&tb->tw, all.size()) != cudaSuccess) {
        cudaGetLastError();
        return VEC_ERR_ALLOC;
    }
    tb->m1 = reinterpret_cast<float *>(reinterpret_cast<char *>(tb->tw) + bt);
    tb->m2 = tb->m1 + n;
    tb->mda = tb->m2 + n;
    tb->pos = reinterpret_cast<unsigned short *>(tb->mda + n);
    tb->gat = tb->pos + n;
    CUDA_TRY(cudaMemcpy(tb->tw, all.data(), all.size(), cudaMemcpyHostToDevice));
    return VEC_OK;
}
void fs_tables_free(FsTables *tb)
{
    cudaFree(tb->tw);
    *tb = FsTables{};
}

template <typename R>
void line_tables_free(LineTables<R> *tb)
{
    cudaFree(tb->tw); cudaFree(tb->m1); cudaFree(tb->m2); cudaFree(tb->mda);
    memset(tb, 0, sizeof(*tb));
}

template <int DIR, int NJ>
static int run_fs(Engine *E, const LineJob<float> *jobs, int nj)
{
    FsPlan pl = DIR == 0 ? E->fspx : E->fspy;
    JobPack<NJ> pk;
    memset(&pk, 0, sizeof(pk));
    double fields = 0.0;
    int two = 0;
    for (int j = 0; j < nj; j++) {
        pk.j[j] = jobs[j];
        fields += 2.0 + (jobs[j].acc1 ? 1.0 : 0.0);
        if (jobs[j].op2 != OP_NONE) fields += 1.0 + (jobs[j].acc2 ? 1.0 : 0.0);
        if (jobs[j].op1 != OP_FWD) two = 1;
    }
    const int pairs = (DIR == 0 ? E->ny : E->nx) / 2;
    // (sequences per warp and warps per CTA as in the FP64 kernel)
    while (pl.Q > 1 && (long long)nj * E->nz * pairs < (long long)E->num_sms * 8 * pl.Q && fx_rounds(pl, pl.Q / 2) < fx_rounds(pl, pl.Q))
        pl.Q >>= 1;
    auto smem_of = [&](int w) {
        return sizeof(float2) * (pl.ntw + (size_t)w * pl.Q * pl.nb * (two ? 2 : 1));
    };
    auto tiles_of = [&](int w) {
        const int S = DIR == 0 ? pl.Q : w * pl.Q;
        return (long long)nj * E->nz * ((pairs + S - 1) / S);
    };
    // warps per CTA: the most warps per SM (32 by their registers), the largest CTA of equals,
    // for wider rows of y tiles and fewer copies of the twiddles; fewer where there would be
    // less than a CTA per SM
    auto warps_of = [&](int w) {
        const size_t fit = 227 * 1024 / (smem_of(w) + 1024);
        return w * (int)(fit < (size_t)(32 / w) ? fit : (size_t)(32 / w));
    };
    int W = FS_TPB / 32;
    for (int w = W / 2; w >= 1; w >>= 1)
        if (warps_of(w) > warps_of(W)) W = w;
    while (W > 1 && (DIR == 0 ? tiles_of(W) / W : tiles_of(W)) < E->num_sms) W >>= 1;
    const size_t smem = smem_of(W);
    static SmemLimit limit;
    CUDA_TRY(limit.raise((const void *)line_kernel<DIR, NJ>, 226 * 1024));
    int per_sm = 1;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, line_kernel<DIR, NJ>, W * 32, smem));
    if (per_sm < 1) per_sm = 1;
    const int S = DIR == 0 ? pl.Q : W * pl.Q, tpp = (pairs + S - 1) / S;
    const long long total = tiles_of(W);
    long long grid = DIR == 0 ? (total + W - 1) / W : total;
    if (grid > (long long)E->num_sms * per_sm) grid = (long long)E->num_sms * per_sm;
    E->prof_begin(DIR == 0 ? "line_x_f32" : "line_y_f32", fields * (double)E->n * sizeof(float));
    CUDA_TRY(launch_k(*E, line_kernel<DIR, NJ>, dim3((unsigned)grid), dim3(W * 32), smem, pk, pl, DIR == 0 ? E->fsx : E->fsy, E->nx,
                      E->ny, E->nz, tpp, (int)total, two));
    E->prof_end();
    CUDA_TRY(cudaGetLastError());
    return VEC_OK;
}

template <>
int launch_lines<float>(Engine *E, int dir, const LineJob<float> *jobs, int njobs)
{
    if (njobs <= 0) return VEC_OK;
    if (!E->generic_lines) {
        const int h = launch_lines_ct(E, dir, jobs, njobs);
        if (h == 1) return VEC_OK;
        if (h < 0) return h;
    }
    for (int j0 = 0; j0 < njobs; j0 += MAX_JOBS) {
        const int nj = njobs - j0 < MAX_JOBS ? njobs - j0 : MAX_JOBS;
        const LineJob<float> *j = jobs + j0;
        const int st = nj <= NJ_SMALL ? (dir == 0 ? run_fs<0, NJ_SMALL>(E, j, nj) : run_fs<1, NJ_SMALL>(E, j, nj))
                                      : (dir == 0 ? run_fs<0, MAX_JOBS>(E, j, nj) : run_fs<1, MAX_JOBS>(E, j, nj));
        if (st) return st;
    }
    return VEC_OK;
}

int line_kernels_configure()
{
    int st = line_ct_configure();
    if (st || (st = line_ct64_configure()) || (st = line_fx_configure())) return st;
    return VEC_OK;
}

template int line_tables_make<double>(int, const double *, const double *, int, LineTables<double> *);
template void line_tables_free<double>(LineTables<double> *);
template int line_tables_make<float>(int, const double *, const double *, int, LineTables<float> *);
template void line_tables_free<float>(LineTables<float> *);
