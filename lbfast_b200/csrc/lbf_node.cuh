// lbf_node.cuh -- per-node arithmetic of the step kernels: reciprocals, packed
// pairs, the HIGHORDER coefficients, populations from coefficients, sums of the
// populations that a node receives, wall links.
#pragma once
#include "lbf_stream.cuh"

namespace lbf {

// Reciprocal and square root: in FP32 the hardware approximations (about 2 ulp)
// instead of the correctly rounded sequences, which cost several instructions
// and a branch each; FP64 stays correctly rounded.
template <typename R> __device__ __forceinline__ R rcp(R x);
template <> __device__ __forceinline__ float rcp<float>(float x) { return __fdividef(1.0f, x); }
template <> __device__ __forceinline__ double rcp<double>(double x) { return 1.0 / x; }
template <typename R> __device__ __forceinline__ R sqrt_a(R x);
template <> __device__ __forceinline__ float sqrt_a<float>(float x) { return x > 0.0f ? x * rsqrtf(x) : 0.0f; }
template <> __device__ __forceinline__ double sqrt_a<double>(double x) { return sqrt(x); }

// A product that several terms read, rounded on its own: the compiler may
// contract a plain a * b into some of the sums it enters and not into others,
// and which ones depends on the code around it.  The one-component step is two
// compilations of each lattice (with and without HIGHORDER) in four storage
// types; with the products of its collision left to the compiler, D3Q27 runs in
// bfloat16 moved by 4e-4 of the result between one form of the kernel and the next.
template <typename R> __device__ __forceinline__ R mul_rn(R a, R b);
template <> __device__ __forceinline__ float mul_rn<float>(float a, float b) { return __fmul_rn(a, b); }
template <> __device__ __forceinline__ double mul_rn<double>(double a, double b) { return __dmul_rn(a, b); }

// Smagorinsky constant of the reference: the single-precision product 0.053 * 18.0
constexpr double SMAG_C = (double)(0.053f * 18.0f);

// vector of two R (the populations of cz = -1 and 0 of one (cx, cy) group)
template <typename R> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };

// Pairs of independent values in one instruction: FP32 as f32x2 (FFMA2,
// FADD2, FMUL2 of sm_100: two lanes' operations per issue slot, each rounded
// as the scalar instruction), FP64 as two scalar operations
template <typename R> struct PK;
template <> struct PK<float> {
    using T = float2;
    static __device__ __forceinline__ float2 mk(float a, float b) { return make_float2(a, b); }
    static __device__ __forceinline__ float2 fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
    static __device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
    static __device__ __forceinline__ float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
};
template <> struct PK<double> {
    using T = double2;
    static __device__ __forceinline__ double2 mk(double a, double b) { return make_double2(a, b); }
    static __device__ __forceinline__ double2 fma(double2 a, double2 b, double2 c) {
        return make_double2(::fma(a.x, b.x, c.x), ::fma(a.y, b.y, c.y));
    }
    static __device__ __forceinline__ double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
    static __device__ __forceinline__ double2 mul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
};
// d1q3_inv with the second coefficient negated (m2n = -m2), the same
// roundings: scalar and packed
template <typename R> __device__ __forceinline__ void d1q3n(R m0, R m1, R m2n, R& vm, R& v0, R& vp) {
    const R s = fmaf_t(m0, R(1.0 / 6.0), R(-0.5) * m2n);
    const R d = R(0.5) * m1;
    vm = s - d;
    vp = s + d;
    v0 = fmaf_t(m0, R(2.0 / 3.0), m2n);
}
template <typename R, typename T = typename PK<R>::T>
__device__ __forceinline__ void d1q3n2(T m0, T m1, T m2n, T& vm, T& v0, T& vp) {
    using P = PK<R>;
    const T s = P::fma(m0, P::mk(R(1.0 / 6.0), R(1.0 / 6.0)), P::mul(P::mk(R(-0.5), R(-0.5)), m2n));
    const T d = P::mul(P::mk(R(0.5), R(0.5)), m1);
    vm = P::fma(d, P::mk(R(-1), R(-1)), s);
    vp = P::add(s, d);
    v0 = P::fma(m0, P::mk(R(2.0 / 3.0), R(2.0 / 3.0)), m2n);
}

// HIGHORDER coefficients, rows 10..26 of the reference
// (lb_cuda_fused_module.f90:667-703): each the equilibrium monomial + om1 x
// its non-equilibrium projection.  Two forms.  `ho_rows_wide` is the
// reference's own.  `ho_rows` takes out the factors that rows share: about 90
// operations against 160, but longer chains of them, and other roundings.  The
// two-component step with obstacles, which sits at the register limit, takes it
// (512 x 256 x 256 channel: 2.74 -> 2.43 ms); the plain two-component one, which
// waits on latency, is slower with it (256^3: 917 -> 928 us with 5.7 % fewer
// instructions).
template <typename R>
__device__ __forceinline__ void ho_rows_wide(R (&M)[3][3][3], const R u, const R v, const R w, const R om1, const R X,
                                             const R Y, const R Z, const R XY, const R XZ, const R YZ) {
    const R u2 = u * u, v2 = v * v, w2 = w * w;
    M[2][1][0] = u2 * v + om1 * (R(2) * XY * u + X * v);
    M[2][0][1] = u2 * w + om1 * (R(2) * XZ * u + X * w);
    M[1][2][0] = u * v2 + om1 * (Y * u + R(2) * XY * v);
    M[1][0][2] = u * w2 + om1 * (Z * u + R(2) * XZ * w);
    M[0][1][2] = v * w2 + om1 * (Z * v + R(2) * YZ * w);
    M[0][2][1] = v2 * w + om1 * (R(2) * YZ * v + Y * w);
    M[1][1][1] = u * v * w + om1 * (YZ * u + XZ * v + XY * w);
    M[2][2][0] = u2 * v2 + om1 * (Y * u2 + R(2) * v * (R(3) * XY * u + X * v));
    M[2][0][2] = u2 * w2 + om1 * (Z * u2 + R(2) * w * (R(3) * XZ * u + X * w));
    M[0][2][2] = v2 * w2 + om1 * (Z * v2 + R(2) * w * (R(3) * YZ * v + Y * w));
    M[1][1][2] = u * v * w2 + om1 * (Z * u * v + w * (R(3) * YZ * u + R(3) * XZ * v + R(2) * XY * w));
    M[1][2][1] = u * v2 * w + om1 * (R(2) * YZ * u * v + XZ * v2 + R(2) * Y * u * w + R(4) * XY * v * w);
    M[2][1][1] = u2 * v * w + om1 * (YZ * u2 + R(2) * XZ * u * v + R(4) * XY * u * w + R(2) * X * v * w);
    M[2][1][2] = u2 * v * w2 + om1 * (Z * u2 * v + R(3) * w * (YZ * u2 + R(2) * XZ * u * v + R(2) * XY * u * w + X * v * w));
    M[2][2][1] = u2 * v2 * w + om1 * (R(2) * u * v * (YZ * u + XZ * v) + R(2) * Y * u2 * w +
                                      v * (R(10) * XY * u + R(3) * X * v) * w);
    M[1][2][2] = u * v2 * w2 + om1 * (Z * u * v2 + R(3) * w * (R(2) * YZ * u * v + XZ * v2 + Y * u * w + R(2) * XY * v * w));
    M[2][2][2] = u2 * v2 * w2 + om1 * (Z * u2 * v2 + w * (R(6) * u * v * (YZ * u + XZ * v) + R(3) * Y * u2 * w +
                                                          R(2) * v * (R(7) * XY * u + R(2) * X * v) * w));
}
template <typename R>
__device__ __forceinline__ void ho_rows(R (&M)[3][3][3], const R u, const R v, const R w, const R om1, const R Xn,
                                        const R Yn, const R Zn, const R XYn, const R XZn, const R YZn) {
    const R X = om1 * Xn, Y = om1 * Yn, Z = om1 * Zn;
    const R XY = om1 * XYn, XZ = om1 * XZn, YZ = om1 * YZn;
    const R u2 = u * u, v2 = v * v, w2 = w * w, uv = u * v, uw = u * w, vw = v * w;
    const R u2v = u * uv, X2 = X + X, Y2 = Y + Y, XY4 = R(4) * XY;
    const R bxy = fmaf_t(R(2), XY, uv), bxz = fmaf_t(R(2), XZ, uw), byz = fmaf_t(R(2), YZ, vw);
    M[2][1][0] = fmaf_t(u, bxy, X * v);
    M[2][0][1] = fmaf_t(u, bxz, X * w);
    M[1][2][0] = fmaf_t(v, bxy, Y * u);
    M[1][0][2] = fmaf_t(w, bxz, Z * u);
    M[0][1][2] = fmaf_t(w, byz, Z * v);
    M[0][2][1] = fmaf_t(v, byz, Y * w);
    const R g = fmaf_t(YZ, u, XZ * v);  // YZ u + XZ v
    M[1][1][1] = fmaf_t(w, uv + XY, g);
    const R zw = Z + w2;
    M[2][2][0] = fmaf_t(u2, v2 + Y, fmaf_t(R(6) * XY, uv, X2 * v2));
    M[2][0][2] = fmaf_t(u2, zw, fmaf_t(R(6) * XZ, uw, X2 * w2));
    M[0][2][2] = fmaf_t(v2, zw, fmaf_t(R(6) * YZ, vw, Y2 * w2));
    const R yv = v2 + Y2, w3 = R(3) * w;
    const R gu = fmaf_t(YZ, u, g), gv = fmaf_t(XZ, v, g);  // 2 YZ u + XZ v, YZ u + 2 XZ v
    M[1][1][2] = fmaf_t(uv, zw, w * fmaf_t(R(2) * XY, w, R(3) * g));
    M[1][2][1] = fmaf_t(uw, yv, v * fmaf_t(XY4, w, gu));
    M[2][1][1] = fmaf_t(vw, u2 + X2, u * fmaf_t(XY4, w, gv));
    const R hu = fmaf_t(R(2) * XY, w, gv), hv = fmaf_t(R(2) * XY, w, gu);
    M[2][1][2] = fmaf_t(u2v, zw, w3 * fmaf_t(u, hu, X * vw));
    M[1][2][2] = fmaf_t(v * uv, zw, w3 * fmaf_t(v, hv, Y * uw));
    M[2][2][1] = fmaf_t(w, fmaf_t(u2, yv, v * fmaf_t(R(10) * XY, u, R(3) * (X * v))),
                        R(2) * uv * g);
    M[2][2][2] = fmaf_t(v * u2v, zw,
                        w * fmaf_t(w, fmaf_t(R(3) * Y, u2, (v + v) * fmaf_t(R(7) * XY, u, X2 * v)),
                                   R(6) * uv * g));
}

// Populations of a D3Q27 node from its 27 coefficients M[a][b][c] by the three
// one-axis transforms.  The x (a) and y (b) transforms are packed over the pair
// c = 0, 1 of the z coefficient index, c = 2 alone; both take the second
// coefficient negated, carried by the sign (-1)^([a==2] + [b==2]) of the
// coefficients (exact: the values are those of the scalar transforms).
template <typename R> struct XPops {
    typename PK<R>::T p[3][3];  // [cx + 1][b], (c = 0, 1), with the sign (-1)^[b==2]
    R q[3][3];                  // [cx + 1][b], c = 2
};
template <typename R> __device__ __forceinline__ void x_transform27(const R (&M)[3][3][3], XPops<R>& X) {
    using PT = typename PK<R>::T;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        PT P[3];
        R Q[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const R sg = ((a == 2) != (b == 2)) ? R(-1) : R(1);
            P[a] = PK<R>::mk(sg * M[a][b][0], sg * M[a][b][1]);
            Q[a] = sg * M[a][b][2];
        }
        d1q3n2<R>(P[0], P[1], P[2], X.p[0][b], X.p[1][b], X.p[2][b]);
        d1q3n<R>(Q[0], Q[1], Q[2], X.q[0][b], X.q[1][b], X.q[2][b]);
    }
}
// all 27, by link
template <typename R> __device__ __forceinline__ void full_pops27(const R (&M)[3][3][3], R (&fpop)[27]) {
    XPops<R> X;
    x_transform27<R>(M, X);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        typename PK<R>::T MP[3];
        R MQ[3];
        d1q3n2<R>(X.p[a][0], X.p[a][1], X.p[a][2], MP[0], MP[1], MP[2]);
        d1q3n<R>(X.q[a][0], X.q[a][1], X.q[a][2], MQ[0], MQ[1], MQ[2]);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            R vm, v0, vp;
            d1q3_inv<R>(MP[b].x, MP[b].y, MQ[b], vm, v0, vp);
            fpop[LINK(a - 1, b - 1, -1)] = vm;
            fpop[LINK(a - 1, b - 1, 0)] = v0;
            fpop[LINK(a - 1, b - 1, 1)] = vp;
        }
    }
}
// a column ring node streams into the tile along cx = dir only: the x
// transform for that value, then put(b, cz = -1, 0, +1) for cy = b - 1
template <typename R, typename F>
__device__ __forceinline__ void ring_col_pops27(const R (&M)[3][3][3], const R dir, F&& put) {
    R T[3][3];  // [b][c]
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const R sv = fmaf_t(M[0][b][c], R(1.0 / 6.0), R(0.5) * M[2][b][c]);
            T[b][c] = sv + dir * (R(0.5) * M[1][b][c]);
        }
    R Y[3][3];  // [b][c]
#pragma unroll
    for (int c = 0; c < 3; ++c) d1q3_inv<R>(T[0][c], T[1][c], T[2][c], Y[0][c], Y[1][c], Y[2][c]);
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        R vm, v0, vp;
        d1q3_inv<R>(Y[b][0], Y[b][1], Y[b][2], vm, v0, vp);
        put(b, vm, v0, vp);
    }
}
// a row ring node along cy = dir only: put(a, cz = -1, 0, +1) for cx = a - 1
template <typename R, typename F>
__device__ __forceinline__ void ring_row_pops27(const R (&M)[3][3][3], const R dir, F&& put) {
    XPops<R> X;
    x_transform27<R>(M, X);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        R Y[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const R t0 = c == 0 ? X.p[a][0].x : (c == 1 ? X.p[a][0].y : X.q[a][0]);
            const R t1 = c == 0 ? X.p[a][1].x : (c == 1 ? X.p[a][1].y : X.q[a][1]);
            const R t2n = c == 0 ? X.p[a][2].x : (c == 1 ? X.p[a][2].y : X.q[a][2]);
            const R sv = fmaf_t(t0, R(1.0 / 6.0), R(-0.5) * t2n);
            Y[c] = sv + dir * (R(0.5) * t1);
        }
        R vm, v0, vp;
        d1q3_inv<R>(Y[0], Y[1], Y[2], vm, v0, vp);
        put(a, vm, v0, vp);
    }
}

// Second-order populations of D3Q19 / D3Q15 (by D3Q27 link):
// w ((base + 3 m.c) + 4.5 c c:m_diagonal + 9 c c:m_off-diagonal), the terms
// added in this order.  Opposite links differ in the sign of m.c alone and go
// as a pair.  (The even terms first, once for both links, are two operations
// less a pair; but the order of the sums decides which 16-bit stored values
// round up, and that one moved bfloat16 runs by 1.6e-4 of the result.)
template <int LAT, typename R>
__device__ __forceinline__ void low_order_pops(const R m0, const R mx, const R my, const R mz, const R mxx, const R myy,
                                               const R mzz, const R mxy, const R mxz, const R myz, R (&fpop)[27]) {
    using P = PK<R>;
    const R base = m0 - R(1.5) * (mxx + myy + mzz);
    const R m1[3] = {mx, my, mz}, m2[3] = {mxx, myy, mzz}, mc[3] = {mxy, mxz, myz};
    fpop[0] = R(WL<LAT>(0)) * base;
#pragma unroll
    for (int l = 1; l < 27; l += 2) {
        if (!IN<LAT>(l)) continue;
        const int c[3] = {EX(l), EY(l), EZ(l)}, cc[3] = {c[0] * c[1], c[0] * c[2], c[1] * c[2]};
        R odd = R(0), diag = R(0), off = R(0);
        bool first = true, first_off = true;  // the sums start with their first term, not with 0 + it
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (c[d]) {
                const R m = c[d] > 0 ? m1[d] : -m1[d];
                odd = first ? m : odd + m;
                diag = first ? m2[d] : diag + m2[d];
                first = false;
            }
            if (cc[d]) {
                const R m = cc[d] > 0 ? mc[d] : -mc[d];
                off = first_off ? m : off + m;
                first_off = false;
            }
        }
        typename P::T f = P::fma(P::mk(R(3), R(-3)), P::mk(odd, odd), P::mk(base, base));
        f = P::fma(P::mk(R(4.5), R(4.5)), P::mk(diag, diag), f);
        if (!first_off) f = P::fma(P::mk(R(9), R(9)), P::mk(off, off), f);
        f = P::mul(P::mk(R(WL<LAT>(l)), R(WL<LAT>(l))), f);
        fpop[l] = f.x;
        fpop[l + 1] = f.y;
    }
}

// population of link l, 0 for one that the lattice lacks
template <int LAT, typename R> __device__ __forceinline__ R fpop_or0(const R (&fpop)[27], int l) {
    return IN<LAT>(l) ? fpop[l] : R(0);
}

// Adds the D3Q27 populations that a node receives from one plane, by (cy, cx)
// -- gp: cz = -1 and 0, gs: cz = +1 -- to the raw moments {sum g, sum g c,
// sum g c c} of the planes they go to: A2 (cz = -1, 0), ap (cz = +1).
template <typename R>
__device__ __forceinline__ void pull_sums27(const typename PK<R>::T (&gp)[3][3], const R (&gs)[3][3],
                                            typename PK<R>::T (&A2)[10], R (&ap)[10]) {
    {
        using P = PK<R>;
        using PP = typename P::T;
        const PP m1 = P::mk(R(-1), R(-1));
        PP S0[3], S1[3], S2[3];
#pragma unroll
        for (int yc = 0; yc < 3; ++yc) {
            const PP* g = gp[yc];
            S0[yc] = P::add(P::add(g[0], g[1]), g[2]);
            S1[yc] = P::fma(g[0], m1, g[2]);
            S2[yc] = P::add(g[2], g[0]);
        }
        const PP Y00 = P::add(P::add(S0[0], S0[1]), S0[2]);
        const PP Y01 = P::fma(S0[0], m1, S0[2]);
        const PP Y02 = P::add(S0[2], S0[0]);
        const PP Y10 = P::add(P::add(S1[0], S1[1]), S1[2]);
        const PP Y11 = P::fma(S1[0], m1, S1[2]);
        const PP Y20 = P::add(P::add(S2[0], S2[1]), S2[2]);
        const PP cz = P::mk(R(-1), R(0)), cz2 = P::mk(R(1), R(0));
        A2[0] = P::add(A2[0], Y00);
        A2[1] = P::add(A2[1], Y10);
        A2[2] = P::add(A2[2], Y01);
        A2[3] = P::fma(cz, Y00, A2[3]);
        A2[4] = P::add(A2[4], Y20);
        A2[5] = P::add(A2[5], Y02);
        A2[6] = P::fma(cz2, Y00, A2[6]);
        A2[7] = P::add(A2[7], Y11);
        A2[8] = P::fma(cz, Y10, A2[8]);
        A2[9] = P::fma(cz, Y01, A2[9]);
    }
    {
        R S0[3], S1[3], S2[3];
#pragma unroll
        for (int yc = 0; yc < 3; ++yc) {
            const R* g = gs[yc];
            S0[yc] = g[0] + g[1] + g[2];
            S1[yc] = g[2] - g[0];
            S2[yc] = g[2] + g[0];
        }
        const R Y00 = S0[0] + S0[1] + S0[2];
        const R Y01 = S0[2] - S0[0];
        const R Y10 = S1[0] + S1[1] + S1[2];
        ap[0] += Y00;
        ap[1] += Y10;
        ap[2] += Y01;
        ap[3] += Y00;
        ap[4] += S2[0] + S2[1] + S2[2];
        ap[5] += S0[2] + S0[0];
        ap[6] += Y00;
        ap[7] += S1[2] - S1[0];
        ap[8] += Y10;
        ap[9] += Y01;
    }
}

// Output moments of node go from the raw moments of its populations
template <typename S, typename R>
__device__ __forceinline__ void write_moments(const StepParams<S, R>& p, const int go, R (&am)[10]) {
    using CD = Codec<S>;
    using LY = Layout<S>;
    const long long N = p.N;
    const R third = am[0] * R(1.0 / 3.0);
    if constexpr (CD::scaled) {
        am[4] -= am[1] * am[1]; am[5] -= am[2] * am[2]; am[6] -= am[3] * am[3];
        am[7] -= am[1] * am[2]; am[8] -= am[1] * am[3]; am[9] -= am[2] * am[3];
    }
    if constexpr (LY::split) {
#pragma unroll
        for (int f = 0; f < 4; ++f) p.pres_out[f * N + go] = (float)am[f];
    } else {
#pragma unroll
        for (int f = 0; f < 4; ++f) CD::st(p.mout + f * N, go, am[f], p.scale[f]);
    }
#pragma unroll
    for (int f = 4; f < 10; ++f)
        CD::st(p.mout + LY::off(f, N), go, f < 7 ? am[f] - third : am[f], p.scale[f]);
}

// The wall links of the tile row of a warp in one plane: lane `tx` is an
// isfluid = -1 node of the box when `wall`.  row_start is the row's first
// entry of p.links, which holds the -1 nodes' links in the order of the nodes;
// 0 for the other lanes.  `any` tells the warp whether there is one at all.
template <typename S, typename R>
__device__ __forceinline__ unsigned wall_links(const StepParams<S, R>& p, const bool wall, const int row_start,
                                               const int tx, bool& any) {
    const unsigned lanes = __ballot_sync(0xffffffffu, wall);
    any = lanes != 0;
    return wall ? __ldg(p.links + row_start + __popc(lanes & ((1u << tx) - 1))) : 0u;
}

// Obstacle bounce-back of a node (lb_cuda_boundary_module.f90:162-199): the raw
// moments d of the populations w_l P + (1 - omega) fneq of its wall links
// (bit l of `links`: the upstream node x - c_l is solid), from its
// non-equilibrium stress.  The population is even in c, so the links go in
// opposite pairs, and without a branch per link: 165 operations for a warp
// that holds a wall node.  Per link it was 26 loads of isfluid with a wrapped
// index and a divergent branch around 25 operations, which the whole CTA waited
// for at the plane's barrier: the 512 x 256 x 256 channel with 64 spheres 3.25 ms
// a step, 2.42 ms now.
template <int LAT, typename R>
__device__ __forceinline__ void wall_link_sums(const unsigned links, const R P, const R om1, const R Xn, const R Yn,
                                               const R Zn, const R XYn, const R XZn, const R YZn, R (&d)[10]) {
    const R k = R(4.5) * om1;
    const R X = k * Xn, Y = k * Yn, Z = k * Zn;
    const R XY = (k + k) * XYn, XZ = (k + k) * XZn, YZ = (k + k) * YZn;
    const R base = P - R(1.0 / 3.0) * (X + Y + Z);
#pragma unroll
    for (int i = 0; i < 10; ++i) d[i] = R(0);
#pragma unroll
    for (int l = 1; l < 27; l += 2) {
        if (!IN<LAT>(l)) continue;
        const int cx = EX(l), cy = EY(l), cz = EZ(l);
        R f = base;
        if (cx) f += X;
        if (cy) f += Y;
        if (cz) f += Z;
        if (cx * cy) f += cx * cy > 0 ? XY : -XY;
        if (cx * cz) f += cx * cz > 0 ? XZ : -XZ;
        if (cy * cz) f += cy * cz > 0 ? YZ : -YZ;
        f *= R(WL<LAT>(l));
        const R a = (links >> l & 1) ? f : R(0), b = (links >> (l + 1) & 1) ? f : R(0);
        const R e = a + b, o = a - b;
        d[0] += e;
        if (cx) { d[1] += cx > 0 ? o : -o; d[4] += e; }
        if (cy) { d[2] += cy > 0 ? o : -o; d[5] += e; }
        if (cz) { d[3] += cz > 0 ? o : -o; d[6] += e; }
        if (cx * cy) d[7] += cx * cy > 0 ? e : -e;
        if (cx * cz) d[8] += cx * cz > 0 ? e : -e;
        if (cy * cz) d[9] += cy * cz > 0 ? e : -e;
    }
}

}  // namespace lbf
