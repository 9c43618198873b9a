// pfft.cuh -- register-resident transforms of two neighbouring lines at a
// time, the building block of the Green's function passes.
//
// sm_100a issues two FP32 operations with one instruction (add, mul and fma
// on f32x2 register pairs).  Every value here is such a pair: the same
// element of two neighbouring lines (two x1 wavenumbers, or two rows), real
// parts in one pair and imaginary parts in another, so that a butterfly on
// two lines costs the instructions of one and no operand has to be swapped.
// The pairs run at the rate of the scalar instructions per element (36e12
// per second measured for both), but a pass was bound by instruction issue,
// not by the FP32 pipes, and its shared-memory accesses become 16 bytes wide.
//
// A line of n = N1*N2 values is transformed as
//     X[k1 + N1 k2] = sum_j2 W_N2^(j2 k2) [ W_n^(j2 k1) sum_j1 x[N2 j1 + j2] W_N1^(j1 k1) ]
// Stage A: N2 threads per pair of lines each hold the N1 values x[N2 j1 + j2]
// in registers and transform them; stage B: after one shared-memory
// transpose each thread transforms the groups k1 = t, t + N2, ... of N2
// values.  N1 >= N2; where N2 does not divide N1 the last round of stage B
// leaves threads idle.
#pragma once

#include "common.cuh"

namespace relax {
namespace {

// one complex element of two lines
struct P2 {
    float2 r, i;
};
// a twiddle factor, the same for both lines
struct W2 {
    float2 x, y;
};
// one complex element of one line, for the pass that needs the warps more
// than the instructions (x1 inverse)
struct P1 {
    float r, i;
};
struct W1 {
    float x, y;
};

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

__device__ __forceinline__ float neg2(float a) { return -a; }
__device__ __forceinline__ float add2(float a, float b) { return a + b; }
__device__ __forceinline__ float sub2(float a, float b) { return a - b; }
__device__ __forceinline__ float mul2(float a, float b) { return a * b; }
__device__ __forceinline__ float fma2(float a, float b, float c) { return fmaf(a, b, c); }
// the constant a in the type of the second argument's parts
__device__ __forceinline__ float2 like(float a, float2) { return f2(a); }
__device__ __forceinline__ float like(float a, float) { return a; }

template <class P>
__device__ __forceinline__ P padd(P a, P b) { return {add2(a.r, b.r), add2(a.i, b.i)}; }
template <class P>
__device__ __forceinline__ P psub(P a, P b) { return {sub2(a.r, b.r), sub2(a.i, b.i)}; }
// a + S i b
template <int S, class P>
__device__ __forceinline__ P paddi(P a, P b)
{
    return S > 0 ? P{sub2(a.r, b.i), add2(a.i, b.r)} : P{add2(a.r, b.i), sub2(a.i, b.r)};
}
// a w, or a conj(w) for CONJ
template <bool CONJ, class P, class W>
__device__ __forceinline__ P pmul(P a, W w)
{
    const auto p = mul2(a.r, w.x), q = mul2(a.i, w.x);
    if (CONJ) return {fma2(a.i, w.y, p), fma2(neg2(a.r), w.y, q)};
    return {fma2(neg2(a.i), w.y, p), fma2(a.r, w.y, q)};
}
__device__ __forceinline__ W2 w2(float4 v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }
// two complex values of neighbouring lines that are neighbours in memory
__device__ __forceinline__ P2 pair(float4 v) { return {make_float2(v.x, v.z), make_float2(v.y, v.w)}; }
__device__ __forceinline__ float4 unpair(P2 v) { return make_float4(v.r.x, v.i.x, v.r.y, v.i.y); }

// exp(-2 pi i m / 32) as (cos, cos, sin, sin)
__constant__ float4 c_p32[32] = {
    {1.000000000e+00f, 1.000000000e+00f, 0.000000000e+00f, 0.000000000e+00f}, {9.807852804e-01f, 9.807852804e-01f, -1.950903220e-01f, -1.950903220e-01f},
    {9.238795325e-01f, 9.238795325e-01f, -3.826834324e-01f, -3.826834324e-01f}, {8.314696123e-01f, 8.314696123e-01f, -5.555702330e-01f, -5.555702330e-01f},
    {7.071067812e-01f, 7.071067812e-01f, -7.071067812e-01f, -7.071067812e-01f}, {5.555702330e-01f, 5.555702330e-01f, -8.314696123e-01f, -8.314696123e-01f},
    {3.826834324e-01f, 3.826834324e-01f, -9.238795325e-01f, -9.238795325e-01f}, {1.950903220e-01f, 1.950903220e-01f, -9.807852804e-01f, -9.807852804e-01f},
    {0.000000000e+00f, 0.000000000e+00f, -1.000000000e+00f, -1.000000000e+00f}, {-1.950903220e-01f, -1.950903220e-01f, -9.807852804e-01f, -9.807852804e-01f},
    {-3.826834324e-01f, -3.826834324e-01f, -9.238795325e-01f, -9.238795325e-01f}, {-5.555702330e-01f, -5.555702330e-01f, -8.314696123e-01f, -8.314696123e-01f},
    {-7.071067812e-01f, -7.071067812e-01f, -7.071067812e-01f, -7.071067812e-01f}, {-8.314696123e-01f, -8.314696123e-01f, -5.555702330e-01f, -5.555702330e-01f},
    {-9.238795325e-01f, -9.238795325e-01f, -3.826834324e-01f, -3.826834324e-01f}, {-9.807852804e-01f, -9.807852804e-01f, -1.950903220e-01f, -1.950903220e-01f},
    {-1.000000000e+00f, -1.000000000e+00f, 0.000000000e+00f, 0.000000000e+00f}, {-9.807852804e-01f, -9.807852804e-01f, 1.950903220e-01f, 1.950903220e-01f},
    {-9.238795325e-01f, -9.238795325e-01f, 3.826834324e-01f, 3.826834324e-01f}, {-8.314696123e-01f, -8.314696123e-01f, 5.555702330e-01f, 5.555702330e-01f},
    {-7.071067812e-01f, -7.071067812e-01f, 7.071067812e-01f, 7.071067812e-01f}, {-5.555702330e-01f, -5.555702330e-01f, 8.314696123e-01f, 8.314696123e-01f},
    {-3.826834324e-01f, -3.826834324e-01f, 9.238795325e-01f, 9.238795325e-01f}, {-1.950903220e-01f, -1.950903220e-01f, 9.807852804e-01f, 9.807852804e-01f},
    {0.000000000e+00f, 0.000000000e+00f, 1.000000000e+00f, 1.000000000e+00f}, {1.950903220e-01f, 1.950903220e-01f, 9.807852804e-01f, 9.807852804e-01f},
    {3.826834324e-01f, 3.826834324e-01f, 9.238795325e-01f, 9.238795325e-01f}, {5.555702330e-01f, 5.555702330e-01f, 8.314696123e-01f, 8.314696123e-01f},
    {7.071067812e-01f, 7.071067812e-01f, 7.071067812e-01f, 7.071067812e-01f}, {8.314696123e-01f, 8.314696123e-01f, 5.555702330e-01f, 5.555702330e-01f},
    {9.238795325e-01f, 9.238795325e-01f, 3.826834324e-01f, 3.826834324e-01f}, {9.807852804e-01f, 9.807852804e-01f, 1.950903220e-01f, 1.950903220e-01f},
};

// exp(-2 pi i m / 24) as (cos, cos, sin, sin)
__constant__ float4 c_p24[24] = {
    {1.000000000e+00f, 1.000000000e+00f, 0.000000000e+00f, 0.000000000e+00f}, {9.659258263e-01f, 9.659258263e-01f, -2.588190451e-01f, -2.588190451e-01f},
    {8.660254038e-01f, 8.660254038e-01f, -5.000000000e-01f, -5.000000000e-01f}, {7.071067812e-01f, 7.071067812e-01f, -7.071067812e-01f, -7.071067812e-01f},
    {5.000000000e-01f, 5.000000000e-01f, -8.660254038e-01f, -8.660254038e-01f}, {2.588190451e-01f, 2.588190451e-01f, -9.659258263e-01f, -9.659258263e-01f},
    {0.000000000e+00f, 0.000000000e+00f, -1.000000000e+00f, -1.000000000e+00f}, {-2.588190451e-01f, -2.588190451e-01f, -9.659258263e-01f, -9.659258263e-01f},
    {-5.000000000e-01f, -5.000000000e-01f, -8.660254038e-01f, -8.660254038e-01f}, {-7.071067812e-01f, -7.071067812e-01f, -7.071067812e-01f, -7.071067812e-01f},
    {-8.660254038e-01f, -8.660254038e-01f, -5.000000000e-01f, -5.000000000e-01f}, {-9.659258263e-01f, -9.659258263e-01f, -2.588190451e-01f, -2.588190451e-01f},
    {-1.000000000e+00f, -1.000000000e+00f, 0.000000000e+00f, 0.000000000e+00f}, {-9.659258263e-01f, -9.659258263e-01f, 2.588190451e-01f, 2.588190451e-01f},
    {-8.660254038e-01f, -8.660254038e-01f, 5.000000000e-01f, 5.000000000e-01f}, {-7.071067812e-01f, -7.071067812e-01f, 7.071067812e-01f, 7.071067812e-01f},
    {-5.000000000e-01f, -5.000000000e-01f, 8.660254038e-01f, 8.660254038e-01f}, {-2.588190451e-01f, -2.588190451e-01f, 9.659258263e-01f, 9.659258263e-01f},
    {0.000000000e+00f, 0.000000000e+00f, 1.000000000e+00f, 1.000000000e+00f}, {2.588190451e-01f, 2.588190451e-01f, 9.659258263e-01f, 9.659258263e-01f},
    {5.000000000e-01f, 5.000000000e-01f, 8.660254038e-01f, 8.660254038e-01f}, {7.071067812e-01f, 7.071067812e-01f, 7.071067812e-01f, 7.071067812e-01f},
    {8.660254038e-01f, 8.660254038e-01f, 5.000000000e-01f, 5.000000000e-01f}, {9.659258263e-01f, 9.659258263e-01f, 2.588190451e-01f, 2.588190451e-01f},
};

// exp(-2 pi i m / 27) as (cos, cos, sin, sin)
__constant__ float4 c_p27[27] = {
    {1.000000000e+00f, 1.000000000e+00f, 0.000000000e+00f, 0.000000000e+00f}, {9.730448706e-01f, 9.730448706e-01f, -2.306158707e-01f, -2.306158707e-01f},
    {8.936326403e-01f, 8.936326403e-01f, -4.487991802e-01f, -4.487991802e-01f}, {7.660444431e-01f, 7.660444431e-01f, -6.427876097e-01f, -6.427876097e-01f},
    {5.971585917e-01f, 5.971585917e-01f, -8.021231928e-01f, -8.021231928e-01f}, {3.960797660e-01f, 3.960797660e-01f, -9.182161069e-01f, -9.182161069e-01f},
    {1.736481777e-01f, 1.736481777e-01f, -9.848077530e-01f, -9.848077530e-01f}, {-5.814482891e-02f, -5.814482891e-02f, -9.983081583e-01f, -9.983081583e-01f},
    {-2.868032327e-01f, -2.868032327e-01f, -9.579895123e-01f, -9.579895123e-01f}, {-5.000000000e-01f, -5.000000000e-01f, -8.660254038e-01f, -8.660254038e-01f},
    {-6.862416379e-01f, -6.862416379e-01f, -7.273736416e-01f, -7.273736416e-01f}, {-8.354878114e-01f, -8.354878114e-01f, -5.495089781e-01f, -5.495089781e-01f},
    {-9.396926208e-01f, -9.396926208e-01f, -3.420201433e-01f, -3.420201433e-01f}, {-9.932383577e-01f, -9.932383577e-01f, -1.160929141e-01f, -1.160929141e-01f},
    {-9.932383577e-01f, -9.932383577e-01f, 1.160929141e-01f, 1.160929141e-01f}, {-9.396926208e-01f, -9.396926208e-01f, 3.420201433e-01f, 3.420201433e-01f},
    {-8.354878114e-01f, -8.354878114e-01f, 5.495089781e-01f, 5.495089781e-01f}, {-6.862416379e-01f, -6.862416379e-01f, 7.273736416e-01f, 7.273736416e-01f},
    {-5.000000000e-01f, -5.000000000e-01f, 8.660254038e-01f, 8.660254038e-01f}, {-2.868032327e-01f, -2.868032327e-01f, 9.579895123e-01f, 9.579895123e-01f},
    {-5.814482891e-02f, -5.814482891e-02f, 9.983081583e-01f, 9.983081583e-01f}, {1.736481777e-01f, 1.736481777e-01f, 9.848077530e-01f, 9.848077530e-01f},
    {3.960797660e-01f, 3.960797660e-01f, 9.182161069e-01f, 9.182161069e-01f}, {5.971585917e-01f, 5.971585917e-01f, 8.021231928e-01f, 8.021231928e-01f},
    {7.660444431e-01f, 7.660444431e-01f, 6.427876097e-01f, 6.427876097e-01f}, {8.936326403e-01f, 8.936326403e-01f, 4.487991802e-01f, 4.487991802e-01f},
    {9.730448706e-01f, 9.730448706e-01f, 2.306158707e-01f, 2.306158707e-01f},
};

// exp(-2 pi i m / 18) as (cos, cos, sin, sin)
__constant__ float4 c_p18[18] = {
    {1.000000000e+00f, 1.000000000e+00f, 0.000000000e+00f, 0.000000000e+00f}, {9.396926208e-01f, 9.396926208e-01f, -3.420201433e-01f, -3.420201433e-01f},
    {7.660444431e-01f, 7.660444431e-01f, -6.427876097e-01f, -6.427876097e-01f}, {5.000000000e-01f, 5.000000000e-01f, -8.660254038e-01f, -8.660254038e-01f},
    {1.736481777e-01f, 1.736481777e-01f, -9.848077530e-01f, -9.848077530e-01f}, {-1.736481777e-01f, -1.736481777e-01f, -9.848077530e-01f, -9.848077530e-01f},
    {-5.000000000e-01f, -5.000000000e-01f, -8.660254038e-01f, -8.660254038e-01f}, {-7.660444431e-01f, -7.660444431e-01f, -6.427876097e-01f, -6.427876097e-01f},
    {-9.396926208e-01f, -9.396926208e-01f, -3.420201433e-01f, -3.420201433e-01f}, {-1.000000000e+00f, -1.000000000e+00f, 0.000000000e+00f, 0.000000000e+00f},
    {-9.396926208e-01f, -9.396926208e-01f, 3.420201433e-01f, 3.420201433e-01f}, {-7.660444431e-01f, -7.660444431e-01f, 6.427876097e-01f, 6.427876097e-01f},
    {-5.000000000e-01f, -5.000000000e-01f, 8.660254038e-01f, 8.660254038e-01f}, {-1.736481777e-01f, -1.736481777e-01f, 9.848077530e-01f, 9.848077530e-01f},
    {1.736481777e-01f, 1.736481777e-01f, 9.848077530e-01f, 9.848077530e-01f}, {5.000000000e-01f, 5.000000000e-01f, 8.660254038e-01f, 8.660254038e-01f},
    {7.660444431e-01f, 7.660444431e-01f, 6.427876097e-01f, 6.427876097e-01f}, {9.396926208e-01f, 9.396926208e-01f, 3.420201433e-01f, 3.420201433e-01f},
};

// exp(-2 pi i m / R)
__device__ __forceinline__ W2 wlike(float4 v, P2) { return w2(v); }
__device__ __forceinline__ W1 wlike(float4 v, P1) { return {v.x, v.z}; }
template <int R>
__device__ __forceinline__ float4 pconst(int m)
{
    static_assert(32 % R == 0 || 24 % R == 0 || 27 % R == 0 || 18 % R == 0, "no constants for this length");
    if (32 % R == 0) return c_p32[m * (32 / R) % 32];
    if (24 % R == 0) return c_p24[m * (24 / R) % 24];
    if (27 % R == 0) return c_p27[m * (27 / R) % 27];
    return c_p18[m * (18 / R) % 18];
}

// DFT of R values (P2 or P1) in registers, natural order in and out; the inputs from nz
// on are zero (they are not read), nz a constant after unrolling
template <int R, int S> struct PDft;

template <int S> struct PDft<2, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 2)
    {
        if (nz <= 1) { v[1] = v[0]; return; }
        const P a = v[0], b = v[1];
        v[0] = padd(a, b);
        v[1] = psub(a, b);
    }
};

template <int S> struct PDft<3, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 3)
    {
        if (nz <= 1) { v[1] = v[2] = v[0]; return; }
        const P t = nz <= 2 ? v[1] : padd(v[1], v[2]), d = nz <= 2 ? v[1] : psub(v[1], v[2]);
        const auto h = like(-0.5f, v[0].r), s = like(S * 0.86602540378443864676f, v[0].r), m = neg2(s);
        const P a = {fma2(t.r, h, v[0].r), fma2(t.i, h, v[0].i)};
        v[0] = padd(v[0], t);
        v[1] = {fma2(d.i, m, a.r), fma2(d.r, s, a.i)};
        v[2] = {fma2(d.i, s, a.r), fma2(d.r, m, a.i)};
    }
};

template <int S> struct PDft<4, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 4)
    {
        if (nz <= 1) { v[1] = v[2] = v[3] = v[0]; return; }
        const P a = v[0], b = v[1];
        const P t0 = nz <= 2 ? a : padd(a, v[2]), t1 = nz <= 2 ? a : psub(a, v[2]);
        const P t2 = nz <= 3 ? b : padd(b, v[3]), d = nz <= 3 ? b : psub(b, v[3]);
        v[0] = padd(t0, t2);
        v[2] = psub(t0, t2);
        v[1] = paddi<S>(t1, d);
        v[3] = paddi<-S>(t1, d);
    }
};

template <int S> struct PDft<8, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 8)
    {
        const auto h = like(0.70710678118654752440f, v[0].r), mh = neg2(h);
        P e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        if (nz <= 1) {
#pragma unroll
            for (int k = 1; k < 8; k++) v[k] = v[0];
            return;
        }
        PDft<4, S>::run(e, (nz + 1) / 2);
        PDft<4, S>::run(o, nz / 2);
        const P x1 = paddi<S>(o[1], o[1]), x3 = paddi<-S>(o[3], o[3]);   // (1 + S i) o1, (1 - S i) o3
        v[0] = padd(e[0], o[0]);
        v[4] = psub(e[0], o[0]);
        v[1] = {fma2(x1.r, h, e[1].r), fma2(x1.i, h, e[1].i)};
        v[5] = {fma2(x1.r, mh, e[1].r), fma2(x1.i, mh, e[1].i)};
        v[2] = paddi<S>(e[2], o[2]);
        v[6] = paddi<-S>(e[2], o[2]);
        v[3] = {fma2(x3.r, mh, e[3].r), fma2(x3.i, mh, e[3].i)};
        v[7] = {fma2(x3.r, h, e[3].r), fma2(x3.i, h, e[3].i)};
    }
};

// R = A B: n = n1 + A n2, k = k2 + B k1
template <int A, int B, int S>
struct PDftAB {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz)
    {
        constexpr int R = A * B;
        P a[A][B];
#pragma unroll
        for (int n1 = 0; n1 < A; n1++) {
#pragma unroll
            for (int n2 = 0; n2 < B; n2++) a[n1][n2] = v[n1 + A * n2];
            PDft<B, S>::run(a[n1], nz >= R ? B : (nz - n1 + A - 1) / A);
#pragma unroll
            for (int k2 = 1; k2 < B; k2++) {
                if (n1 == 0) continue;
                if (4 * n1 * k2 == R)
                    a[n1][k2] = S > 0 ? P{neg2(a[n1][k2].i), a[n1][k2].r} : P{a[n1][k2].i, neg2(a[n1][k2].r)};
                else
                    a[n1][k2] = pmul<(S > 0)>(a[n1][k2], wlike(pconst<R>(n1 * k2), P{}));
            }
        }
#pragma unroll
        for (int k2 = 0; k2 < B; k2++) {
            P t[A];
#pragma unroll
            for (int n1 = 0; n1 < A; n1++) t[n1] = a[n1][k2];
            PDft<A, S>::run(t);
#pragma unroll
            for (int k1 = 0; k1 < A; k1++) v[k2 + B * k1] = t[k1];
        }
    }
};
template <int S> struct PDft<6, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 6) { PDftAB<2, 3, S>::run(v, nz); }
};
template <int S> struct PDft<9, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 9) { PDftAB<3, 3, S>::run(v, nz); }
};
template <int S> struct PDft<12, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 12) { PDftAB<3, 4, S>::run(v, nz); }
};
template <int S> struct PDft<16, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 16) { PDftAB<4, 4, S>::run(v, nz); }
};
template <int S> struct PDft<18, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 18) { PDftAB<3, 6, S>::run(v, nz); }
};
template <int S> struct PDft<24, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 24) { PDftAB<3, 8, S>::run(v, nz); }
};
template <int S> struct PDft<27, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 27) { PDftAB<3, 9, S>::run(v, nz); }
};
template <int S> struct PDft<32, S> {
    template <class P>
    __device__ __forceinline__ static void run(P *v, int nz = 32) { PDftAB<4, 8, S>::run(v, nz); }
};

}  // namespace
}  // namespace relax
