// ccz4_stencil.cuh -- finite-difference stencils of the CCZ4 operator
// (ccz4.cpp:71-223) and the Kreiss-Oliger operator (ccz4.cpp:871-935).
//
// Two evaluation modes, chosen by the algebra type P:
//
//  P = double (plain FP64): every stencil is evaluated in the reference's
//    operation order with explicitly rounded products and sums, so the
//    derivatives and the KO term are bit-identical to the host code. This
//    matters where a field is O(1) and its RHS is ~1e-6 of that (noisy flat
//    regions): there the rounding of the reference's own stencil sums is the
//    size of the result, and only the same rounding reproduces it.
//
//  P = float (mixed): stencils are evaluated from FP64 pair differences
//    (f[+k] - f[-k], f[+k] + f[-k] - 2 f[0], ...) that cancel exactly, and only
//    the small differences are rounded to FP32; the algebra downstream runs in
//    FP32 without losing the cancellation.
#pragma once

#include <type_traits>

#include "ccz4_common.cuh"

namespace granite_b200 {
namespace {

#define RN_MUL __dmul_rn
#define RN_ADD __dadd_rn
#define RN_SUB __dsub_rn

// Neighbours of one point along one axis: operator()(k) is the value k cells
// away (k = +-1 .. +-3), far() the one four cells away on the upwind side (the
// - side for a shift >= 0, ccz4.cpp:109-152).
template <typename Ld, typename O>
struct StridedAxis {
    Ld l;
    O s, s4;
    __device__ __forceinline__ double operator()(int k) const { return l(k * s); }
    __device__ __forceinline__ double far() const { return l(s4); }
};

// Stencil loaders of one field at one point: operator()(o) is the value o cells
// away in the field's storage, stride(d) the cell offset along axis d, and
// axis<D>(beta) the neighbours along axis D.
// Offsets in int where every stencil is FP64 (EXACT): one wide multiply-add per
// neighbour instead of a 64-bit addition chain, 4 % of the FP64 global-load RHS
// (89x70x61: 331 -> 318 us); the mixed build's pair stencils are 8 % slower so
// (234 -> 253 us) and keep 64-bit offsets. Four planes of cells always fit an
// int: 2^29 cells in one plane are 850 GB for a block's nine planes or more.
template <typename O>
struct GlobalLoad {  // read-only global memory through the non-coherent path
    const double* __restrict__ p;
    O off[3];
    __device__ __forceinline__ double operator()(O o) const { return __ldg(p + o); }
    __device__ __forceinline__ O stride(int d) const { return off[d]; }
    template <int D>
    __device__ __forceinline__ StridedAxis<GlobalLoad, O> axis(double beta) const {
        return {*this, off[D], beta >= 0.0 ? -4 * off[D] : 4 * off[D]};
    }
};
template <bool EXACT>
__device__ __forceinline__ auto global_load(const double* f, int tx, int ty) {
    using O = std::conditional_t<EXACT, int, long long>;
    return GlobalLoad<O>{f, {1, tx, (O)tx * ty}};
}
template <int SY, int SZ>
struct SharedLoad {  // a CTA-staged tile in shared memory, rows of SY and planes of SZ cells
    const double* p;
    __device__ __forceinline__ double operator()(int o) const { return p[o]; }
    __device__ __forceinline__ int stride(int d) const { return d == 0 ? 1 : (d == 1 ? SY : SZ); }
    template <int D>
    __device__ __forceinline__ StridedAxis<SharedLoad, int> axis(double beta) const {
        const int s = stride(D);
        return {*this, s, beta >= 0.0 ? -4 * s : 4 * s};
    }
};
// A tile staged in three boxes (TileBoxes): the tile with its halo in x and y
// and one plane beyond it in z, and the three farther planes on either side
// of it without a halo. The z neighbours two to four cells away have their own
// offsets, which depend on the point's plane only.
struct ArmOffsets {
    int lo[3], hi[3];  // of the neighbours 2, 3, 4 planes below / above: bytes from the slot's start
};
// A shared-memory load by 32-bit address. (Through a pointer the neighbours'
// addresses are formed in 64 bits: twice the integer instructions per field.)
__device__ __forceinline__ double load_shared(unsigned a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(v) : "r"(a));
    return v;
}
template <int SY, int SZ>
struct SplitLoad {
    unsigned slot, p;  // shared addresses of the slot and of the point in it
    const ArmOffsets& z;
    __device__ __forceinline__ double operator()(int o) const { return load_shared(p + o * (int)sizeof(double)); }
    __device__ __forceinline__ double at(int bytes) const { return load_shared(slot + bytes); }
    __device__ __forceinline__ int stride(int d) const { return d == 0 ? 1 : (d == 1 ? SY : SZ); }
    // x and y: the fourth neighbour's address is formed from the selected offset
    struct Axis {
        const SplitLoad& l;
        int s, s4;
        __device__ __forceinline__ double operator()(int k) const { return l(k * s); }
        __device__ __forceinline__ double far() const { return l(s4); }
    };
    struct AxisZ {
        const SplitLoad& l;
        int z4;
        __device__ __forceinline__ double operator()(int k) const {
            return k == 1 || k == -1 ? l(k * SZ) : l.at(k < 0 ? l.z.lo[-k - 2] : l.z.hi[k - 2]);
        }
        __device__ __forceinline__ double far() const { return l.at(z4); }
    };
    template <int D>
    __device__ __forceinline__ auto axis(double beta) const {
        if constexpr (D == 2) {
            return AxisZ{*this, beta >= 0.0 ? z.lo[2] : z.hi[2]};
        } else {
            const int s = stride(D);
            return Axis{*this, s, beta >= 0.0 ? -4 * s : 4 * s};
        }
    }
};

template <typename P>
struct AxisDer {
    P d1;  // 4th-order centred first derivative, ccz4.cpp:71-99
    P up;  // 4th-order one-sided derivative on the upwind side, ccz4.cpp:109-152
    P d2;  // 4th-order second derivative, ccz4.cpp:156-184
};

// Reference-order evaluation (P = double). `ko` accumulates the KO sum across
// the three axes exactly as ccz4.cpp:912-926 does.
//
// The upwind derivative is evaluated without a branch: the side is selected
// (the fourth neighbour is loaded from it). The beta < 0 form of ccz4.cpp:109-152,
// inv12h (-25 f0 + 48 f+1 - 36 f+2 + 16 f+3 - 3 f+4), rounded left to right,
// is bit for bit the negation of the beta >= 0 form applied to the + side
// (round-to-nearest is odd-symmetric; only the sign of an exact zero differs).
template <bool WANT_D2, bool WANT_KO, typename Ax>
__device__ __forceinline__ AxisDer<double> axis_exact(const Ax& f, double f0, double beta, double inv12h, double inv12h2,
                                                     const double* kw, double& ko) {
    const double fm1 = f(-1), fp1 = f(1);
    const double fm2 = f(-2), fp2 = f(2);
    const double fm3 = f(-3), fp3 = f(3);
    const double g4 = f.far();
    AxisDer<double> r;
    // inv12h * (-f[+2] + 8 f[+1] - 8 f[-1] + f[-2])
    r.d1 = RN_MUL(inv12h, RN_ADD(RN_SUB(RN_ADD(-fp2, RN_MUL(8.0, fp1)), RN_MUL(8.0, fm1)), fm2));
    const bool pos = beta >= 0.0;
    const double g1 = pos ? fm1 : fp1, g2 = pos ? fm2 : fp2, g3 = pos ? fm3 : fp3;
    // inv12h * (25 f0 - 48 g1 + 36 g2 - 16 g3 + 3 g4), g = the - side for beta >= 0
    const double up = RN_MUL(inv12h, RN_ADD(RN_SUB(RN_ADD(RN_SUB(RN_MUL(25.0, f0), RN_MUL(48.0, g1)), RN_MUL(36.0, g2)),
                                                   RN_MUL(16.0, g3)),
                                            RN_MUL(3.0, g4)));
    r.up = pos ? up : -up;
    if (WANT_D2) {
        // inv12h2 * (-f[+2] + 16 f[+1] - 30 f0 + 16 f[-1] - f[-2])
        r.d2 = RN_MUL(inv12h2, RN_SUB(RN_ADD(RN_SUB(RN_ADD(-fp2, RN_MUL(16.0, fp1)), RN_MUL(30.0, f0)),
                                             RN_MUL(16.0, fm1)),
                                      fm2));
    } else {
        r.d2 = 0.0;
    }
    if (WANT_KO) {
        // diss += (cf w_s) u(x + s e_d), s = -3..3, w = {1,-6,15,-20,15,-6,1}
        ko = RN_ADD(ko, RN_MUL(kw[0], fm3));
        ko = RN_ADD(ko, RN_MUL(kw[1], fm2));
        ko = RN_ADD(ko, RN_MUL(kw[2], fm1));
        ko = RN_ADD(ko, RN_MUL(kw[3], f0));
        ko = RN_ADD(ko, RN_MUL(kw[2], fp1));
        ko = RN_ADD(ko, RN_MUL(kw[1], fp2));
        ko = RN_ADD(ko, RN_MUL(kw[0], fp3));
    }
    return r;
}

// Pair-difference evaluation (P = float: the mixed form; P = double: the FP64
// pass of the per-tile precision, equal to the reference-order form to
// rounding). The pair differences and their weighted sums stay FP64 (small,
// exactly cancelled numbers) and each derivative the algebra uses is rounded
// to P once. The advection and KO terms are sums over the three axes: they
// are accumulated in FP64 and rounded once per field by the caller (once
// together, where the algebra only adds them: KOSEP false).
//
// The advection term of one axis is w |beta| inv12h e + (1 - w) beta inv12h c
// (ccz4.cpp:567-574). The upwind stencil (ccz4.cpp:109-152) takes the side of
// the shift: for beta >= 0, e = 25 f0 - 48 g1 + 36 g2 - 16 g3 + 3 g4 with g_k =
// f[-k], times beta; for beta < 0 the mirror (g_k = f[+k]) with -e, so the term
// is |beta| e either way and needs no select of e. The fourth neighbour is
// loaded once from the selected side. c is the centred sum d1 is made of. The
// two factors do not depend on the field: au = w beta inv12h (its sign is the
// side) and ac = (1 - w) beta inv12h, computed once per point.
template <bool WANT_D2, typename P, typename Ax>
__device__ __forceinline__ void axis_pairs(const Ax& f, double f0, double au, double ac, P inv12h_p, P inv12h2_p,
                                           double kocf, P& d1, P& d2, double& adv, double& kod) {
    // differences from the centre, a_k = f[-k] - f0 and b_k = f[+k] - f0, shared by
    // every stencil below
    const double a1 = f(-1) - f0, b1 = f(1) - f0;
    const double a2 = f(-2) - f0, b2 = f(2) - f0;
    const double a3 = f(-3) - f0, b3 = f(3) - f0;
    const double c4 = f.far() - f0;
    // 8 (f+1 - f-1) - (f+2 - f-2)
    const double c = 8.0 * (b1 - a1) - (b2 - a2);
    d1 = inv12h_p * (P)c;
    const bool pos = au >= 0.0;
    const double x1 = pos ? a1 : b1, x2 = pos ? a2 : b2, x3 = pos ? a3 : b3;
    // 25 f0 - 48 g1 + 36 g2 - 16 g3 + 3 g4 (g: the upwind side), weights summing to zero
    const double e = -48.0 * x1 + 36.0 * x2 - 16.0 * x3 + 3.0 * c4;
    adv += fabs(au) * e;
    adv += ac * c;
    const double t1 = b1 + a1;
    const double t2 = b2 + a2;
    d2 = WANT_D2 ? inv12h2_p * (P)(16.0 * t1 - t2) : (P)0;
    // (f-3 + f+3) - 6 (f-2 + f+2) + 15 (f-1 + f+1) - 20 f0
    kod += kocf * ((b3 + a3) - 6.0 * t2 + 15.0 * t1);
}

// 2nd-order mixed derivative, ccz4.cpp:185-222: inv4hh * (f++ - f+- - f-+ + f--),
// in the reference's order (EXACT) or from pair differences.
template <typename P, bool EXACT, int DA, int DB, typename L>
__device__ __forceinline__ P dmix(const L& f, P inv4hh) {
    const auto sa = f.stride(DA), sb = f.stride(DB);
    const double pp = f(sa + sb), pm = f(sa - sb);
    const double mp = f(-sa + sb), mm = f(-sa - sb);
    if constexpr (EXACT)
        return RN_MUL(inv4hh, RN_ADD(RN_SUB(RN_SUB(pp, pm), mp), mm));
    else
        return inv4hh * (P)((pp - pm) - (mp - mm));
}

// Everything one field contributes: gradient, blended advection, KO, and
// (optionally) its Hessian.
template <typename P>
struct FieldDer {
    P d[3];
    P adv;  // w sum beta_d up_d + (1-w) sum beta_d d1_d, ccz4.cpp:567-574
    P ko;   // KO term of the field (added after the rest of its RHS)
    P h[6]; // xx xy xz yy yz zz
};

// What the advection of every field at a point shares.
//  EXACT: the shift and the blend weight; else the factors of axis_pairs.
template <typename P, bool EXACT>
struct Advection {
    double beta[3];
    P w;
    __device__ __forceinline__ Advection(const StencilCoef&, const double b[3], double w_) : beta{b[0], b[1], b[2]}, w((P)w_) {}
    __device__ __forceinline__ double side(int d) const { return beta[d]; }
};
template <typename P>
struct Advection<P, false> {
    double au[3], ac[3];
    __device__ __forceinline__ Advection(const StencilCoef& B, const double b[3], double w) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            au[d] = w * (b[d] * B.inv12h[d]);
            ac[d] = (1.0 - w) * (b[d] * B.inv12h[d]);
        }
    }
    __device__ __forceinline__ double side(int d) const { return au[d]; }
};

// The coefficient in the algebra's precision: the double, or its float copy.
template <typename P>
__device__ __forceinline__ P coef_p(double d, float f) {
    if constexpr (sizeof(P) == 8)
        return d;
    else
        return f;
}

// One axis of field_der_l.
template <int D, typename P, bool HESS, bool KO, bool EXACT, typename L>
__device__ __forceinline__ void axis_der(const StencilCoef& B, const L& f, double f0, const Advection<P, EXACT>& A,
                                         FieldDer<P>& r, P up[3], double& adv, double& kod) {
    constexpr int DD = D == 0 ? 0 : (D == 1 ? 3 : 5);
    const auto ax = f.template axis<D>(A.side(D));
    if constexpr (EXACT) {
        const AxisDer<P> a = axis_exact<HESS, KO>(ax, f0, A.beta[D], B.inv12h[D], B.inv12h2[D], B.kow[D], kod);
        r.d[D] = a.d1;
        up[D] = a.up;
        if (HESS) r.h[DD] = a.d2;
    } else {
        static_assert(KO, "the pair form evaluates the KO term");
        P d2;
        axis_pairs<HESS, P>(ax, f0, A.au[D], A.ac[D], coef_p<P>(B.inv12h[D], B.inv12h_f[D]),
                            coef_p<P>(B.inv12h2[D], B.inv12h2_f[D]), B.kocf[D], r.d[D], d2, adv, kod);
        if (HESS) r.h[DD] = d2;
    }
}

// EXACT (P = double only): every stencil in the reference's operation order.
// KOSEP false: the pair form may return advection and KO as one sum in adv.
template <typename P, bool HESS, bool KO, bool EXACT, bool KOSEP = true, typename L>
__device__ __forceinline__ FieldDer<P> field_der_l(const StencilCoef& B, const L& f, const Advection<P, EXACT>& A) {
    static_assert(!EXACT || sizeof(P) == 8, "reference-order stencils are FP64");
    const double f0 = f(0);
    FieldDer<P> r;
    P up[3];                       // EXACT: the upwind derivatives
    double adv = 0.0, kod = 0.0;   // advection (pair form) and KO sums, FP64
    double& ks = EXACT || KOSEP ? kod : adv;
    axis_der<0, P, HESS, KO, EXACT>(B, f, f0, A, r, up, adv, ks);
    axis_der<1, P, HESS, KO, EXACT>(B, f, f0, A, r, up, adv, ks);
    axis_der<2, P, HESS, KO, EXACT>(B, f, f0, A, r, up, adv, ks);
    if constexpr (EXACT) {
        const P b0 = (P)A.beta[0], b1 = (P)A.beta[1], b2 = (P)A.beta[2];
        const P cen_sum = b0 * r.d[0] + b1 * r.d[1] + b2 * r.d[2];
        const P up_sum = b0 * up[0] + b1 * up[1] + b2 * up[2];
        r.adv = A.w * up_sum + ((P)1 - A.w) * cen_sum;
    } else {
        r.adv = (P)adv;
    }
    r.ko = EXACT || KOSEP ? (P)kod : (P)0;
    if (HESS) {
        r.h[1] = dmix<P, EXACT, 0, 1>(f, coef_p<P>(B.inv4hh[0], B.inv4hh_f[0]));
        r.h[2] = dmix<P, EXACT, 0, 2>(f, coef_p<P>(B.inv4hh[1], B.inv4hh_f[1]));
        r.h[4] = dmix<P, EXACT, 1, 2>(f, coef_p<P>(B.inv4hh[2], B.inv4hh_f[2]));
    } else {
#pragma unroll
        for (int a = 0; a < 6; ++a) r.h[a] = (P)0;
    }
    return r;
}

// Field derivatives straight from global memory, without the KO term.
template <typename P, bool HESS>
__device__ __forceinline__ FieldDer<P> field_der_noko(const DevBlock& B, const double* __restrict__ f,
                                                      const double beta[3], P w) {
    return field_der_l<P, HESS, false, true>(B, global_load<true>(f, B.tx, B.ty),
                                             Advection<P, true>(B, beta, w));
}

__device__ __forceinline__ int sy(int a, int b) {
    // symmetric pair -> packed index (types.hpp:52-54)
    return (a <= b) ? (a * 3 - a * (a - 1) / 2 + b - a) : (b * 3 - b * (b - 1) / 2 + a - b);
}

}  // namespace
}  // namespace granite_b200
