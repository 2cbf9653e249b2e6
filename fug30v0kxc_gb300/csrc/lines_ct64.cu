// lines_ct64.cu -- 2-D transforms in FP64 for the start of a split run (mag_init), for
// line lengths n = N1*N2 = 2^a or 3*2^a (64..256): the scheme of lines_ct.cu in double.
//
// The FP64 form's lines run on integers (lines_fx.cu), 2.5 times as fast and more
// exact.  Where both lengths are among these, a split context's start keeps this kernel's
// bits instead: its FP32 mirrors round what mag_init makes, and 1e-16 moves some of them by
// an FP32 unit (2e-7 of a state after ten steps), from which a convecting layer takes
// another course.  (At other lengths starts are lines_fx.cu's.)  It runs once per start;
// FP64 arithmetic bounds it.
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"
#include "engine.h"
#include "tma.cuh"

#define CT64_JOBS 3
template <typename R> struct JobPackCT { LineJob<R> j[CT64_JOBS]; };
// one TMA descriptor per job input (y lines: 3-D view nx x ny x nz)
struct TmapPack { CUtensorMap m[CT64_JOBS]; };

// W_32^q = exp(-2 pi i q/32), q = 0..31, and W_96^q (the in-register radix
// kernels; radix-3 factors take their twiddles from the second table)
__constant__ double2 c_tw32d[32];
__constant__ double2 c_tw96d[96];

template <typename C> __device__ __forceinline__ C tw32(int q);
template <> __device__ __forceinline__ double2 tw32<double2>(int q) { return c_tw32d[q]; }
template <typename C> __device__ __forceinline__ C tw96(int q);
template <> __device__ __forceinline__ double2 tw96<double2>(int q) { return c_tw96d[q]; }

// x mod N for x >= 0 (N a compile-time constant)
template <int N> __device__ __forceinline__ int modn(int x) { return (N & (N - 1)) == 0 ? (x & (N - 1)) : x % N; }

template <typename C>
__device__ __forceinline__ C cmul_(C a, C b) { C r; r.x = a.x * b.x - a.y * b.y; r.y = a.x * b.y + a.y * b.x; return r; }
template <typename C>
__device__ __forceinline__ C cadd_(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C>
__device__ __forceinline__ C csub_(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
template <bool INV, typename C>
__device__ __forceinline__ C rot_(C a) { C r; if (INV) { r.x = -a.y; r.y = a.x; } else { r.x = a.y; r.y = -a.x; } return r; }

// multiply by W_N^e (e compile-time after unrolling); conjugate for INV
template <int N, bool INV, typename C>
__device__ __forceinline__ C twc(C a, int e)
{
    if constexpr (32 % N == 0) {
        const int q = (e * (32 / N)) & 31;
        if (q == 0) return a;
        if (q == 8) return rot_<INV>(a);                           // -i (fwd)
        if (q == 16) { C r; r.x = -a.x; r.y = -a.y; return r; }
        if (q == 24) return rot_<!INV>(a);                         // +i (fwd)
        C w = tw32<C>(q);
        if (INV) w.y = -w.y;
        return cmul_(a, w);
    } else {
        static_assert(96 % N == 0, "radix kernels cover divisors of 32 and 96");
        const int q = (e * (96 / N)) % 96;
        if (q == 0) return a;
        if (q == 24) return rot_<INV>(a);
        if (q == 48) { C r; r.x = -a.x; r.y = -a.y; return r; }
        if (q == 72) return rot_<!INV>(a);
        C w = tw96<C>(q);
        if (INV) w.y = -w.y;
        return cmul_(a, w);
    }
}

// in-register natural-order DFT of N points
template <int N, bool INV> struct RDft;
template <bool INV> struct RDft<1, INV> { template <typename C> static __device__ __forceinline__ void run(C *) {} };
template <bool INV> struct RDft<2, INV> {
    template <typename C> static __device__ __forceinline__ void run(C *v) { C a = v[0], b = v[1]; v[0] = cadd_(a, b); v[1] = csub_(a, b); }
};
// X1,2 = a - (b+c)/2 -+ i (sqrt(3)/2)(b-c) (forward; conjugate for INV)
template <bool INV> struct RDft<3, INV> {
    template <typename C> static __device__ __forceinline__ void run(C *v) {
        using R = decltype(v[0].x);
        const R h = (R)0.8660254037844386;
        C t1 = cadd_(v[1], v[2]), d = csub_(v[1], v[2]);
        C t2; t2.x = v[0].x - (R)0.5 * t1.x; t2.y = v[0].y - (R)0.5 * t1.y;
        C r = rot_<INV>(d);
        r.x *= h; r.y *= h;
        v[0] = cadd_(v[0], t1);
        v[1] = cadd_(t2, r);
        v[2] = csub_(t2, r);
    }
};
template <bool INV> struct RDft<4, INV> {
    template <typename C> static __device__ __forceinline__ void run(C *v) {
        C a0 = cadd_(v[0], v[2]), a1 = csub_(v[0], v[2]);
        C b0 = cadd_(v[1], v[3]), b1 = rot_<INV>(csub_(v[1], v[3]));
        v[0] = cadd_(a0, b0); v[1] = cadd_(a1, b1); v[2] = csub_(a0, b0); v[3] = csub_(a1, b1);
    }
};
// four-step in registers: N = A*B, m = B*m1 + m2, k = k1 + A*k2
template <int A, int B, bool INV, typename C>
__device__ __forceinline__ void reg_ct(C *v)
{
    constexpr int N = A * B;
    C t[N];
#pragma unroll
    for (int m2 = 0; m2 < B; m2++) {
        C a[A];
#pragma unroll
        for (int m1 = 0; m1 < A; m1++) a[m1] = v[B * m1 + m2];
        RDft<A, INV>::run(a);
#pragma unroll
        for (int k1 = 0; k1 < A; k1++) t[m2 * A + k1] = twc<N, INV>(a[k1], m2 * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) {
        C b[B];
#pragma unroll
        for (int m2 = 0; m2 < B; m2++) b[m2] = t[m2 * A + k1];
        RDft<B, INV>::run(b);
#pragma unroll
        for (int k2 = 0; k2 < B; k2++) v[k1 + A * k2] = b[k2];
    }
}
template <bool INV> struct RDft<8, INV> { template <typename C> static __device__ __forceinline__ void run(C *v) { reg_ct<2, 4, INV>(v); } };
template <bool INV> struct RDft<16, INV> { template <typename C> static __device__ __forceinline__ void run(C *v) { reg_ct<4, 4, INV>(v); } };
template <bool INV> struct RDft<12, INV> { template <typename C> static __device__ __forceinline__ void run(C *v) { reg_ct<4, 3, INV>(v); } };

// ---- the kernel --------------------------------------------------------------------
// DIR 0: x lines (a tile = 2S contiguous rows), DIR 1: y lines (a tile = 2S
// adjacent columns over all ny rows).
//
// WS (x lines with NP dividing 32): the NP threads of a sequence sit in one
// warp, so the exchanges need only warp barriers.  The warps then run
// through their tiles independently; an "empty" mbarrier per tile buffer
// (one arrival per warp once it has read the tile) tells the thread that
// issues the TMA copies when a buffer may be refilled.
// Per-sequence stride of the exchange rows, in complex elements.  The
// forward exchange holds N1 rows of N2 + 1, the inverse one N2 rows of
// N1 + 1, the spectra's separation N + N/32 padded elements: the stride
// covers the largest.  A shared-memory wavefront serves U = 128 /
// sizeof(complex) consecutive elements.  x lines: the threads of a
// half-warp (quarter-warp in FP64) belong to one or two sequences, and a
// stride of 1 mod 16 keeps them on distinct banks.  y lines: thread tid is
// lane tid / S of sequence tid % S, so a wavefront's threads are G = U / S
// lanes of U / G sequences; a stride of G mod U puts them on distinct banks
// (exchange element sidx * stride + lane * 1 or lane * (odd row) + const).
template <typename R, int DIR, int N1, int N2, int S>
__host__ __device__ constexpr int ct_lds()
{
    constexpr int U = 128 / (2 * (int)sizeof(R));
    constexpr int G = U / S > 1 ? U / S : 1;
    constexpr int MF = N1 * (N2 + 1), MI = N2 * (N1 + 1), MS = N1 * N2 + (N1 * N2) / 32 + 1;
    constexpr int M = MF > MI ? (MF > MS ? MF : MS) : (MI > MS ? MI : MS);
    return DIR == 0 ? ((M + 15) / 16) * 16 + 1 : ((M + U - 1) / U) * U + G;
}

// dynamic shared memory of one CTA: two tile buffers, the exchange rows,
// the twiddle table(s) and the three multiplier tables
template <typename R, int DIR, int N1, int N2, int S>
__host__ __device__ constexpr size_t ct_smem_bytes()
{
    constexpr int N = N1 * N2;
    constexpr int LDS = ct_lds<R, DIR, N1, N2, S>();
    return 2 * (size_t)(2 * S * N) * sizeof(R) + ((size_t)S * LDS + (size_t)N) * 2 * sizeof(R);
}
// two CTAs per SM where their shared memory fits (227 KB per SM), else one
// CTA with the whole register file
template <typename R, int DIR, int N1, int N2, int S>
__host__ __device__ constexpr int ct_min_blocks()
{
    return (S * (N1 > N2 ? N1 : N2) <= 256 && 2 * ct_smem_bytes<R, DIR, N1, N2, S>() <= 232448) ? 2 : 1;
}

template <typename R, int DIR, int N1, int N2, int S, bool WSYNC>
__global__ void __launch_bounds__(S * (N1 > N2 ? N1 : N2), (ct_min_blocks<R, DIR, N1, N2, S>()))
line_ct64(JobPackCT<R> jobs, const __grid_constant__ TmapPack tmaps, LineTables<R> tb, int nx, int ny, int nz,
        int tpp, int total, int *err)
{
    PDL_WAIT();
    using C = typename CT<R>::T;
    constexpr int N = N1 * N2;
    constexpr int NP = N1 > N2 ? N1 : N2;
    constexpr int NT = S * NP;
    constexpr int TILE = 2 * S * N;                   // reals per tile
    constexpr int LXF = N2 + 1;                       // padded exchange rows: forward,
    constexpr int LXI = N1 + 1;                       // inverse
    constexpr int LDS = ct_lds<R, DIR, N1, N2, S>();  // per-sequence exchange stride
    constexpr bool WS = WSYNC && DIR == 0 && (32 % NP == 0) && NT % 32 == 0;

    extern __shared__ __align__(128) unsigned char smem[];
    R *tile0 = reinterpret_cast<R *>(smem);
    R *tile1 = tile0 + TILE;
    C *ex = reinterpret_cast<C *>(tile1 + TILE);
    C *twf = ex + (size_t)S * LDS;                    // W_N^e
    __shared__ __align__(8) uint64_t bar[4];          // full[2], empty[2]

    const int tid = threadIdx.x;
    const int sidx = DIR == 0 ? tid / NP : tid % S;
    const int lane = DIR == 0 ? tid % NP : tid / S;
    const size_t np = (size_t)nx * ny;
    auto sync = [&]() {
        if constexpr (WS) __syncwarp();
        else __syncthreads();
    };

    for (int e = tid; e < N; e += NT) {
        twf[e] = tb.tw[e];
    }
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_init(&bar[2], NT / 32);
        mbar_init(&bar[3], NT / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();

    auto issue = [&](int t, R *dst, uint64_t *b) {
        const int job = t / (nz * tpp);
        const int rem = t - job * (nz * tpp);
        const int plane = rem / tpp;
        const int l0 = (rem - plane * tpp) * 2 * S;
        const R *src = jobs.j[job].in + (size_t)plane * np;
        if (DIR == 0) {
            if (tid == 0) {
                mbar_expect_tx(b, TILE * (unsigned)sizeof(R));
                tma_load(dst, src + (size_t)l0 * nx, TILE * (unsigned)sizeof(R), b);
            }
        } else if (tid == 0) {
            // boxes of 2S columns x (up to 256) rows of this plane
            constexpr int BR = ybox_rows(N);
            mbar_expect_tx(b, TILE * (unsigned)sizeof(R));
#pragma unroll
            for (int c = 0; c < N / BR; c++)
                tma_load_3d(dst + (size_t)c * BR * 2 * S, &tmaps.m[job], l0, c * BR, plane, b);
            (void)src;
        }
    };

    if (blockIdx.x < total) issue(blockIdx.x, tile0, &bar[0]);
    int it = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x, it++) {
        R *cur = (it & 1) ? tile1 : tile0;
        R *nxt = (it & 1) ? tile0 : tile1;
        bool issued_next = false;
        if (t + (int)gridDim.x < total) {
            if (WS && it >= 1 && tid == 0) {
                // every warp has read buffer nxt (its use in iteration it - 1)
                if (!mbar_wait(&bar[2 + ((it + 1) & 1)], ((it - 1) >> 1) & 1)) {
                    // report, then let this tile's copy (still in flight)
                    // land before the CTA's shared memory is released
                    atomicExch(err, 1);
                    mbar_wait(&bar[it & 1], (it >> 1) & 1);
                    return;
                }
            }
            if (tid == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(t + gridDim.x, nxt, &bar[(it + 1) & 1]);
            issued_next = true;
        }
        if (!mbar_wait(&bar[it & 1], (it >> 1) & 1)) {
            if (tid == 0) {
                // report, then wait (bounded) for the copies this CTA issued
                atomicExch(err, 1);
                mbar_wait(&bar[it & 1], (it >> 1) & 1);
                if (issued_next) mbar_wait(&bar[(it + 1) & 1], ((it + 1) >> 1) & 1);
            }
            return;
        }
        const int job = t / (nz * tpp);
        const int rem = t - job * (nz * tpp);
        const int plane = rem / tpp;
        const int l0 = (rem - plane * tpp) * 2 * S;
        const LineJob<R> &jb = jobs.j[job];
        const size_t pbase = (size_t)plane * np;
        const int op1 = jb.op1;
        C *ex_s = ex + (size_t)sidx * LDS;

        // element e of sequence sidx in the tile
        auto tile_z = [&](int e) -> C {
            C z;
            if (DIR == 0) { z.x = cur[(2 * sidx) * N + e]; z.y = cur[(2 * sidx + 1) * N + e]; }
            else { z = reinterpret_cast<const C *>(cur)[(size_t)e * S + sidx]; }
            return z;
        };

        C X[N2];   // thread lane = k1 holds X[k1 + N1 k2], k2 = 0..N2-1
        if (op1 != OP_INV) {
            // forward, first level: thread m2 = lane, N1-point DFT over m1
            if (lane < N2) {
                C a[N1];
#pragma unroll
                for (int m1 = 0; m1 < N1; m1++) a[m1] = tile_z(N2 * m1 + lane);
                RDft<N1, false>::run(a);
#pragma unroll
                for (int k1 = 0; k1 < N1; k1++) {
                    const C w = twf[modn<N>(lane * k1)];
                    ex_s[k1 * LXF + lane] = k1 == 0 ? a[k1] : cmul_(a[k1], w);
                }
            }
            sync();
            // second level: thread k1 = lane, N2-point DFT over m2
            if (lane < N1) {
#pragma unroll
                for (int m2 = 0; m2 < N2; m2++) X[m2] = ex_s[lane * LXF + m2];
                RDft<N2, false>::run(X);
            }
            sync();
        } else if (lane < N1) {
            // halfcomplex input lines a (re) and b (im): Z_k = A_k + i B_k
#pragma unroll
            for (int k2 = 0; k2 < N2; k2++) {
                const int k = lane + N1 * k2;
                const int kk = k <= N / 2 ? k : N - k;
                const bool edge = kk == 0 || 2 * kk == N;
                C pa = tile_z(kk);                     // (ha[kk], hb[kk])
                C pb = edge ? C{0, 0} : tile_z(N - kk); // (ha[n-kk], hb[n-kk])
                R ar = pa.x, br = pa.y, ai = k <= N / 2 ? pb.x : -pb.x, bi = k <= N / 2 ? pb.y : -pb.y;
                X[k2].x = ar - bi;
                X[k2].y = ai + br;
            }
        }
        if constexpr (WS) {
            // this warp is done with the tile buffer
            __syncwarp();
            if ((tid & 31) == 0) mbar_arrive(&bar[2 + (it & 1)]);
        }

        if (op1 == OP_FWD) {
            // separate Z into the halfcomplex spectra of the two real lines
            if (lane < N1) {
#pragma unroll
                for (int k2 = 0; k2 < N2; k2++) ex_s[lane + N1 * k2 + ((lane + N1 * k2) >> 5)] = X[k2];
            }
            sync();
            for (int p = lane; p < N; p += NP) {
                const int q = p == 0 ? 0 : N - p;
                C zp = ex_s[p + (p >> 5)], zq = ex_s[q + (q >> 5)];
                R va, vb;
                if (2 * p <= N) { va = (R)0.5 * (zp.x + zq.x); vb = (R)0.5 * (zp.y + zq.y); }
                else { va = (R)0.5 * (zq.y - zp.y); vb = (R)0.5 * (zp.x - zq.x); }
                const int la = l0 + 2 * sidx;
                if (DIR == 0) {
                    R *oa = jb.out1 + pbase + (size_t)la * nx + p, *ob = oa + nx;
                    *oa = va;
                    *ob = vb;
                } else {
                    // the two lines are adjacent columns: one vector store
                    *reinterpret_cast<C *>(jb.out1 + pbase + (size_t)p * nx + la) = C{ va, vb };
                }
            }
            sync();
            continue;
        }

        // inverse transform, store
        if (lane < N1) {
            C Y[N2];
#pragma unroll
            for (int k2 = 0; k2 < N2; k2++) Y[k2] = X[k2];
            // inverse, first level: thread k1 = lane, N2-point DFT over k2
            RDft<N2, true>::run(Y);
#pragma unroll
            for (int m2 = 0; m2 < N2; m2++) {
                C w = twf[modn<N>(m2 * lane)];
                w.y = -w.y;
                ex_s[m2 * LXI + lane] = m2 == 0 ? Y[m2] : cmul_(Y[m2], w);
            }
        }
        sync();
        // second level: thread m2 = lane, N1-point DFT over k1
        if (lane < N2) {
            C a[N1];
#pragma unroll
            for (int k1 = 0; k1 < N1; k1++) a[k1] = ex_s[lane * LXI + k1];
            RDft<N1, true>::run(a);
            const R sc = (R)1 / (R)N;
            const int la = l0 + 2 * sidx;
#pragma unroll
            for (int m1 = 0; m1 < N1; m1++) {
                const int e = lane + N2 * m1;
                const R va = a[m1].x * sc, vb = a[m1].y * sc;
                if (DIR == 0) {
                    R *oa = jb.out1 + pbase + (size_t)la * nx + e, *ob = oa + nx;
                    *oa = va;
                    *ob = vb;
                } else {
                    *reinterpret_cast<C *>(jb.out1 + pbase + (size_t)e * nx + la) = C{ va, vb };
                }
            }
        }
        sync();
    }
}

// ---- host side ------------------------------------------------------------------------
int line_ct64_configure()
{
    double2 td[32];
    for (int q = 0; q < 32; q++) {
        // exp(-2 pi i q/32) with exact quadrant values
        double a = 2.0 * M_PI * (double)q / 32.0;
        double c = cos(a), s = sin(a);
        if (q % 8 == 0) {
            c = (q == 0) ? 1.0 : (q == 16 ? -1.0 : 0.0);
            s = (q == 8) ? 1.0 : (q == 24 ? -1.0 : 0.0);
        }
        td[q].x = c; td[q].y = -s;
    }
    CUDA_TRY(cudaMemcpyToSymbol(c_tw32d, td, sizeof(td)));
    double2 ud[96];
    for (int q = 0; q < 96; q++) {
        double c, s;
        sincos2pi_host(q, 96, &c, &s);
        ud[q].x = c; ud[q].y = -s;
    }
    CUDA_TRY(cudaMemcpyToSymbol(c_tw96d, ud, sizeof(ud)));
    return VEC_OK;
}

// TMA descriptor of a (nx, ny, nz) field read in boxes of 2S columns x BR rows
template <typename R>
static int encode_ymap64(CUtensorMap *m, const R *base, int nx, int ny, int nz, int S, int BR)
{
    const auto enc = (PFN_cuTensorMapEncodeTiled_v12000)tma_encode_fn();
    if (!enc) return VEC_ERR_CUDA;
    cuuint64_t dims[3] = { (cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz };
    cuuint64_t strides[2] = { (cuuint64_t)nx * sizeof(R), (cuuint64_t)nx * ny * sizeof(R) };
    cuuint32_t box[3] = { (cuuint32_t)(2 * S), (cuuint32_t)BR, 1 };
    cuuint32_t es[3] = { 1, 1, 1 };
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, (void *)base, dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        vec_set_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
        return VEC_ERR_CUDA;
    }
    return VEC_OK;
}

template <typename R, int DIR, int N1, int N2, int S, bool WSYNC>
static int run_ct(Engine *E, const LineJob<R> *jobs, int nj, const char *name)
{
    constexpr int N = N1 * N2;
    constexpr int NP = N1 > N2 ? N1 : N2;
    constexpr int LDS = ct_lds<R, DIR, N1, N2, S>();
    static SmemLimit limit;
    const size_t smem = ct_smem_bytes<R, DIR, N1, N2, S>();
    static_assert(ct_smem_bytes<R, DIR, N1, N2, S>() + 128 <= 232448, "tile does not fit one SM's shared memory");
    static_assert(LDS >= N1 * (N2 + 1) && LDS >= N2 * (N1 + 1) && LDS >= N + N / 32 + 1, "exchange rows");
    CUDA_TRY(limit.raise((const void *)line_ct64<R, DIR, N1, N2, S, WSYNC>, (int)smem));
    const int L = DIR == 0 ? E->ny : E->nx;
    const int tpp = L / (2 * S);
    JobPackCT<R> pk;
    memset(&pk, 0, sizeof(pk));
    double fields = 0.0;
    for (int j = 0; j < nj; j++) {
        pk.j[j] = jobs[j];
        fields += 2.0;
    }
    TmapPack tp;
    memset(&tp, 0, sizeof(tp));
    if (DIR == 1) {
        int st;
        constexpr int BR = ybox_rows(N);
        for (int j = 0; j < nj; j++)
            if ((st = encode_ymap64<R>(&tp.m[j], jobs[j].in, E->nx, E->ny, E->nz, S, BR))) return st;
    }
    const int total = nj * E->nz * tpp;
    int per_sm = 1;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, line_ct64<R, DIR, N1, N2, S, WSYNC>, S * NP, smem));
    if (per_sm < 1) per_sm = 1;
    int grid = E->num_sms * per_sm;
    if (grid > total) grid = total;
    E->prof_begin(name, fields * (double)E->n * sizeof(R));
    CUDA_TRY(launch_k(*E, line_ct64<R, DIR, N1, N2, S, WSYNC>, dim3(grid), dim3(S * NP), smem, pk, tp,
                      DIR == 0 ? E->tx64 : E->ty64, E->nx, E->ny, E->nz, tpp, total, E->dev_err));
    E->prof_end();
    CUDA_TRY(cudaGetLastError());
    return VEC_OK;
}

static bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

// up to CT64_JOBS plain forward or inverse jobs: 1 if done, 0 if the lengths or addresses are not its own, < 0
// on error
int launch_lines_ct64(Engine *E, int dir, const LineJob<double> *jobs, int njobs)
{
    constexpr int S = 8;     // sequences per tile
    const int n = dir == 0 ? E->nx : E->ny;
    const int L = dir == 0 ? E->ny : E->nx;
    if (!E->tx64.tw || !E->ty64.tw || njobs > CT64_JOBS || L % (2 * S) != 0) return 0;
    for (int j = 0; j < njobs; j++) {
        if (!aligned16(jobs[j].in) || !aligned16(jobs[j].out1) || (jobs[j].out2 && !aligned16(jobs[j].out2)))
            return 0;
    }
    const bool ws = E->ct_warp;
    const char *name = dir == 0 ? "line_x_f64" : "line_y_f64";
    int st = VEC_ERR_ARG;
#define CT_CASE(NN, A, B)                                                                                \
    if (n == NN)                                                                                         \
        st = dir == 1 ? run_ct<double, 1, A, B, S, false>(E, jobs, njobs, name)                         \
                      : (ws ? run_ct<double, 0, A, B, S, true>(E, jobs, njobs, name)                    \
                            : run_ct<double, 0, A, B, S, false>(E, jobs, njobs, name));
    CT_CASE(64, 8, 8) CT_CASE(128, 16, 8) CT_CASE(256, 16, 16) CT_CASE(96, 8, 12) CT_CASE(192, 16, 12)
#undef CT_CASE
    return st ? (st < 0 ? st : -st) : 1;
}
