// Reconstruction and Riemann fluxes as straight-line code (exact.cuh's divisions
// and square roots, selects instead of branches), included by kernels.cuh. FP64
// results are the bits of reconstruct() and riemann_flux(), which a face takes
// (PlainFace) when an operand is out of the range where that holds.
#pragma once
#include "exact.cuh"

namespace psst {

// Whether a state's values lie where the straight-line operations are exact.
template <typename R, int DIM>
__device__ __forceinline__ bool ordinary(const Prim<R, DIM> &s) {
    constexpr int B = sizeof(R) == 8 ? 60 : 40;
    bool ok = positive_in_range<B, B>(s.p) && positive_in_range<B, B>(s.T) && positive_in_range<B, B>(s.rho);
#pragma unroll
    for (int k = 0; k < DIM; ++k) ok = ok && zero_or_in_range(s.u[k]);
    return ok;
}

// x y + z, the sum's other product exact or rounded: in FP32 one rounding for both
// operations, whatever the code around it is (in FP64 the reference's two). Left to
// the compiler, cp T + vs / 2 became vs (1 / 2) + (cp T rounded) here, which added
// 1.3 to 1.6% to the error of p and T after ten iterations of 54000 tets (passes).
template <typename R>
__device__ __forceinline__ R mul_add(R x, R y, R z) {
    if constexpr (sizeof(R) == 4)
        return fmaf(x, y, z);
    else
        return x * y + z;
}

// limiter_value without branches
template <int LIM, typename R>
__device__ __forceinline__ R lin_limiter(R num, R den, bool &fine) {
    const R eps = (R)1.0e-10;
    const bool flat = fabs(den) < eps;
    const R d = flat ? (R)1 : den;
    R v;
    if constexpr (sizeof(R) == 4) {
        if (LIM == 1) v = lin_div(num * num + num * d, num * num + d * d);
        if (LIM == 2) v = fabsf(num) > fabsf(d) ? (R)1 : lin_div(num, d);
        if (LIM == 3) {
            const R b = num + d;
            v = lin_div((R)2 * num, b != (R)0 ? b : (R)1);
        }
    } else {
        fine = fine && zero_or_in_range(num) && den_ok(d);
        const R r = lin_div(num, d);
        if (LIM == 1) v = lin_div(r * r + r, r * r + (R)1);
        if (LIM == 2) v = r > (R)1 ? (R)1 : r;
        if (LIM == 3) {
            const R b = (R)1 + r;
            fine = fine && zero_or_in_range(r) && (den_ok(b) || b == (R)0);
            v = lin_div((R)2 * r, b != (R)0 ? b : (R)1);
        }
        if (LIM == 1) fine = fine && (r == (R)0 || positive_in_range<100, 100>(fabs(r)));
    }
    if (flat) v = LIM == 3 ? (R)2 : (R)1;
    if ((num > (R)0 && den < (R)0) || (num < (R)0 && den > (R)0)) v = (R)0;
    return v;
}

// reconstruct() without branches
template <typename R, int DIM, int REC, int LIM>
__device__ __forceinline__ void lin_reconstruct(Prim<R, DIM> r[2], const R d0[DIM + 2], const R d1[DIM + 2], R rm,
                                                bool &fine) {
#pragma unroll
    for (int i = 0; i < DIM + 2; ++i) {
        if (REC == 1) {
            const R dl = d1[i], dr = d0[i];
            const R v0 = pvar<R, DIM>(r[0], i), v1 = pvar<R, DIM>(r[1], i);
            const R vlm = v1 - ((R)2 * dl - (v0 - v1));
            const R vrp = v0 + ((R)2 * dr - (v0 - v1));
            const R nl = v0 - v1, dnl = v1 - vlm;
            const R nr = v1 - v0, dnr = v0 - vrp;
            pvar<R, DIM>(r[0], i) += (R)0.5 * lin_limiter<LIM, R>(nr, dnr, fine) * dnr;
            pvar<R, DIM>(r[1], i) += (R)0.5 * lin_limiter<LIM, R>(nl, dnl, fine) * dnl;
        } else {
            pvar<R, DIM>(r[0], i) += d0[i];
            pvar<R, DIM>(r[1], i) += d1[i];
        }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        fine = fine && den_ok(rm * r[j].T);
        r[j].rho = lin_div(r[j].p, rm * r[j].T);
    }
}

// riemann_flux() (edge < 0), or the physical flux of side `edge`
// (boundary_flux), without branches: every value that some wave pattern needs
// is formed, and the pattern selects. `fine` is cleared where an operand is out
// of the straight-line operations' range or the wave speeds cannot be ordered.
template <typename R, int DIM, int FLUX>
__device__ __forceinline__ void lin_flux(const Prim<R, DIM> r[2], const R *nn, const Gas &gas, int edge,
                                         R flow[DIM + 2], bool &fine) {
    const R rm = (R)gas.rm, cp = (R)gas.cp, cv = (R)gas.cv, gamma = (R)gas.gamma;
    fine = fine && ordinary<R, DIM>(r[0]) && ordinary<R, DIM>(r[1]);
    R vn[2], a[2], H[2], vsq[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        vn[j] = (R)0;
        R vs = (R)0;
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            vn[j] += r[j].u[k] * nn[k];
            vs += r[j].u[k] * r[j].u[k];
        }
        vsq[j] = vs;
        a[j] = lin_sqrt(gamma * rm * r[j].T);
        H[j] = mul_add<R>(cp, r[j].T, (R)0.5 * vs);
    }
    if (FLUX == 1) {  // psstConvectiveAUSM::calculate (psstConvectiveFlow.cpp:804-851)
        fine = fine && den_ok(a[0]) && den_ok(a[1]);
        const R M1 = lin_div(vn[1], a[1]), M0 = lin_div(vn[0], a[0]);
        const R Ms1 = M1 >= (R)1 ? M1 : M1 <= (R)-1 ? (R)0 : (R)0.25 * (M1 + (R)1) * (M1 + (R)1);
        const R ps1 = M1 >= (R)1    ? r[1].p
                      : M1 <= (R)-1 ? (R)0
                                    : (R)0.25 * r[1].p * (M1 + (R)1) * (M1 + (R)1) * ((R)2 - M1);
        const R Ms0 = M0 >= (R)1 ? (R)0 : M0 <= (R)-1 ? M0 : (R)-0.25 * (M0 - (R)1) * (M0 - (R)1);
        const R ps0 = M0 >= (R)1    ? (R)0
                      : M0 <= (R)-1 ? r[0].p
                                    : (R)0.25 * r[0].p * (M0 - (R)1) * (M0 - (R)1) * ((R)2 + M0);
        const R Mf = Ms0 + Ms1, pf = ps0 + ps1;
        const bool sd = edge >= 0 ? edge == 1 : Mf > (R)0;  // upwind side: 1 if Mf > 0
        const R rho = sd ? r[1].rho : r[0].rho, h = sd ? H[1] : H[0], p = sd ? r[1].p : r[0].p;
        const R t = Mf * (sd ? a[1] : a[0]) * rho, v = sd ? vn[1] : vn[0];
#pragma unroll
        for (int j = 0; j < DIM; ++j) {
            const R u = sd ? r[1].u[j] : r[0].u[j];
            flow[j] = edge >= 0 ? rho * u * v + p * nn[j] : t * u + pf * nn[j];
        }
        flow[DIM] = edge >= 0 ? rho * v : t;
        flow[DIM + 1] = edge >= 0 ? rho * v * h : t * h;
        return;
    }
    // Roe-averaged wave speeds (psstConvectiveFlow.cpp:13-24, 247-266, 531-550)
    const R sl = lin_sqrt(r[1].rho), sr = lin_sqrt(r[0].rho), sden = sl + sr, y = lin_recip(sden);
    fine = fine && den_ok(sden);
    const R HR = lin_quot(H[1] * sl + H[0] * sr, sden, y);
    R vRn = (R)0, vs = (R)0;
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
        const R vR = lin_quot(r[1].u[k] * sl + r[0].u[k] * sr, sden, y);
        vRn += vR * nn[k];
        vs += vR * vR;
    }
    const R aR2 = (gamma - (R)1) * (HR - (R)0.5 * vs);
    fine = fine && positive_in_range<100, 100>(aR2);
    const R aR = lin_sqrt(aR2);
    R s0, s1, t;
    s1 = vn[1] - a[1];
    t = vRn - aR;
    if (s1 > t) s1 = t;
    s0 = vn[0] + a[0];
    t = vRn + aR;
    if (s0 < t) s0 = t;
    // physical flux f and conserved state w of a side
    auto side = [&](const Prim<R, DIM> &s, R v, R h, R v2, R f[DIM + 2], R w[DIM + 2]) {
        const R E = mul_add<R>(cv, s.T, (R)0.5 * v2);
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            f[k] = mul_add<R>(s.rho * s.u[k], v, s.p * nn[k]);
            w[k] = s.rho * s.u[k];
        }
        w[DIM] = s.rho;
        w[DIM + 1] = s.rho * E;
        f[DIM] = s.rho * v;
        f[DIM + 1] = s.rho * v * h;
    };
    if (FLUX == 2) {  // HLL (psstConvectiveFlow.cpp:268-286)
        R f0[DIM + 2], w0[DIM + 2], f1[DIM + 2], w1[DIM + 2];
        side(r[0], vn[0], H[0], vsq[0], f0, w0);
        side(r[1], vn[1], H[1], vsq[1], f1, w1);
        const bool is1 = edge >= 0 ? edge == 1 : s1 >= (R)0;
        const bool mid = edge < 0 && !is1 && s1 <= (R)0 && s0 >= (R)0;
        fine = fine && (edge >= 0 || is1 || mid || s0 <= (R)0);
        const R den = mid ? s0 - s1 : (R)1, z = lin_recip(den);
        fine = fine && den_ok(den);
#pragma unroll
        for (int j = 0; j < DIM + 2; ++j) {
            const R q = lin_quot(s0 * f1[j] - s1 * f0[j] + s0 * s1 * (w0[j] - w1[j]), den, z);
            flow[j] = mid ? q : is1 ? f1[j] : f0[j];
        }
        return;
    }
    // HLLC (psstConvectiveFlow.cpp:552-585)
    const R p0 = r[0].p, p1 = r[1].p, d0 = r[0].rho, d1 = r[1].rho;
    const R shd = d1 * (s1 - vn[1]) - d0 * (s0 - vn[0]);
    fine = fine && (den_ok(shd) || edge >= 0);
    const R sh = lin_div(p0 - p1 + d1 * vn[1] * (s1 - vn[1]) - d0 * vn[0] * (s0 - vn[0]), shd);
    const bool up1 = s1 >= (R)0, star1 = s1 <= (R)0 && sh >= (R)0;
    const bool star = edge < 0 && !up1 && (star1 || (sh <= (R)0 && s0 >= (R)0));
    fine = fine && (edge >= 0 || up1 || star || s0 <= (R)0);
    const bool sd = edge >= 0 ? edge == 1 : up1 || star1;  // the side whose state is used
    Prim<R, DIM> s;
#pragma unroll
    for (int i = 0; i < DIM + 2; ++i)
        pvar<R, DIM>(s, i) = sd ? pvar<R, DIM>(r[1], i) : pvar<R, DIM>(r[0], i);
    s.rho = sd ? d1 : d0;
    const R vv = sd ? vn[1] : vn[0], ss = sd ? s1 : s0;
    R fs[DIM + 2], ws[DIM + 2];
    side(s, vv, sd ? H[1] : H[0], sd ? vsq[1] : vsq[0], fs, ws);
    const R tt = star ? ss - sh : (R)1, z = lin_recip(tt);
    fine = fine && den_ok(tt);
#pragma unroll
    for (int j = 0; j < DIM + 2; ++j) {
        R top = sh * (ss * ws[j] - fs[j]);
        if (j < DIM) top = top + ss * (s.p + s.rho * (ss - vv) * (sh - vv)) * nn[j];
        if (j == DIM + 1) top = top + ss * (s.p + s.rho * (ss - vv) * (sh - vv)) * sh;
        const R q = lin_quot(top, tt, z);
        flow[j] = star ? q : fs[j];
    }
}

// One face by the plain operators; false where the wave speeds cannot be ordered.
template <typename R, int DIM, int REC, int LIM>
struct PlainFace {
    Prim<R, DIM> r[2];
    R d0[DIM + 2], d1[DIM + 2], n[DIM], flow[DIM + 2];
    int flux, edge;
    static __device__ __noinline__ bool run(PlainFace *f, const Gas *gas) {
        if (f->edge >= 0) {
            boundary_flux<R, DIM>(f->r[f->edge], f->n, *gas, f->flow);
            return true;
        }
        if (REC) reconstruct<R, DIM, REC, LIM>(f->r, f->d0, f->d1, (R)gas->rm);
        return f->flux == 1   ? riemann_flux<R, DIM, 1>(f->r, f->n, *gas, f->flow)
               : f->flux == 2 ? riemann_flux<R, DIM, 2>(f->r, f->n, *gas, f->flow)
                              : riemann_flux<R, DIM, 3>(f->r, f->n, *gas, f->flow);
    }
};

}  // namespace psst
