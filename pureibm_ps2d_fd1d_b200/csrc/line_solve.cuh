// line_solve.cuh -- per-warp solves of the x-line systems of velstep.
//
// Every cyclic system of velstep has constant coefficients (a = c, b on every
// row, periodic coupling), i.e. it is a symmetric circulant matrix; the
// reference solves it with Thomas + Sherman-Morrison (tridiagonal.F90:90-150,
// usteptime.F90:344-349,457-468).  With rho the root of a rho^2 + b rho + a = 0
// inside the unit circle and S the shift x(i) -> x(i-1),
//     a S^-1 + b + a S = c (1 - rho S)(1 - rho S^-1),   c = -a/rho,
// so the exact solution is one forward recurrence y(i) = r(i)/c + rho y(i-1)
// and one backward recurrence x(i) = y(i) + rho x(i+1), both cyclic.  A warp
// holds a line as 32 blocks of R consecutive planes: each lane runs its block,
// the block ends combine by cyclic doubling (after k steps a lane holds the
// sum over 2^k blocks), and 1/(1 - rho^N) closes the period.  Doubling stops
// where rho^(R 2^k) is below the last bit of anything it could be added to:
// about one step for the viscous systems and three for most pressure lines.
//
// Against the eigen-decomposition by warp FFTs used before (10 butterfly
// stages over all R elements of a lane, 4 shuffles each): two shuffles per
// double and step for one element per lane, and 4 R + 10 multiply-adds per
// component instead of about 30 R.  The x-line kernel went from 24 / 45 / 74 /
// 142 / 1860 to 16 / 27 / 56 / 103 / 1209 us at 32 / 64 / 96 / 128 / 256^3 (the two
// small ones mostly by the (0,0) line below).  Both matrices are symmetric, so
// the same solves serve the adjoint step.
//
// The (ky,kz) = (0,0) pressure line is not circulant (nx-1 unknowns, zero at
// either end, b = -2a: poisson.F90:127-142, 309-325) and is solved through its
// Green's function, two prefix sums (dirichlet_solve); the reference's Thomas
// recursion is a serial chain of two divisions per plane that one lane walked
// twice per step while the GPU waited: at 64^3 it was half of the kernel.
#pragma once
#include "step_common.cuh"

namespace pibm {

// Slot of plane i in a line's row: a gap after every 8 planes, so that the 8
// lanes of a shared-memory phase hit distinct 16-byte slots both when they
// walk consecutive planes (i = lane + 32 r) and when they hold consecutive
// blocks (i = R lane + r, R = 1, 2, 4, 8; two of the 8 share a slot for R = 3).
__host__ __device__ __forceinline__ constexpr int row_slot(int i) { return i + (i >> 3); }

__device__ __forceinline__ double2 shfl2(double2 v, int src) {
    return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
__device__ __forceinline__ double2 fma2(double a, double2 x, double2 y) { return make_double2(__fma_rn(a, x.x, y.x), __fma_rn(a, x.y, y.y)); }

// Factors of one line's circulant system: rho, 1/c and rho^k (k <= R), and the
// closures of the forward and backward recurrences.
template <int R> struct Circ {
    double rho, rc, pw[R], invf, invb, hf, hb;
};
// a x(i-1) + b x(i) + a x(i+1), b^2 > 4 a^2.  hw: x(i + N) = x(i)/hw (1 for the
// periodic systems; the scalar's lines carry the heat ratio): the forward
// recurrence picks up hw across the period, the backward one 1/hw.
template <int R, bool kTwist = false>
__device__ __forceinline__ Circ<R> circ_factor(double a, double b, double hw = 1.0) {
    Circ<R> k;
    const double s = __dsqrt_rn(__dmul_rn(__dsub_rn(b, __dmul_rn(2.0, a)), __dadd_rn(b, __dmul_rn(2.0, a))));
    const double c = __dmul_rn(0.5, __dadd_rn(b, copysign(s, b)));
    k.rc = 1.0 / c;
    k.rho = -(a / c);
    k.pw[0] = k.rho;
#pragma unroll
    for (int r = 1; r < R; ++r) k.pw[r] = __dmul_rn(k.pw[r - 1], k.rho);
    double pn = k.pw[R - 1];
#pragma unroll
    for (int h = 1; h < 32; h <<= 1) pn = __dmul_rn(pn, pn);
    k.hf = kTwist ? hw : 1.0;
    k.hb = kTwist ? 1.0 / hw : 1.0;
    k.invf = 1.0 / __dsub_rn(1.0, __dmul_rn(pn, k.hf));
    k.invb = kTwist ? 1.0 / __dsub_rn(1.0, __dmul_rn(pn, k.hb)) : k.invf;
    return k;
}
// Cyclic sum over the lanes' block ends: P(lane) = sum_j q^j P(lane -+ j), the
// period closed by inv; a value that crosses the period's end takes factor hw.
template <bool kBack, bool kTwist>
__device__ __forceinline__ double2 circ_carry(double2 P, double q, double inv, double hw, int lane) {
#pragma unroll 1
    for (int h = 1; h < 32 && fabs(q) > 1e-22; h <<= 1) {   // q is the line's: one branch per warp
        const int src = kBack ? lane + h : lane - h;
        const double2 t = shfl2(P, src & 31);
        P = fma2(kTwist && (src & ~31) ? __dmul_rn(q, hw) : q, t, P);
        q = __dmul_rn(q, q);
    }
    const int src = kBack ? lane + 1 : lane - 1;
    double2 y = shfl2(P, src & 31);
    const double f = kTwist && (src & ~31) ? __dmul_rn(inv, hw) : inv;
    return make_double2(__dmul_rn(f, y.x), __dmul_rn(f, y.y));
}
// The solve on a lane's block: on entry v[r] = right-hand side at plane
// R lane + r, on exit the solution there.
template <int R, bool kTwist = false>
__device__ __forceinline__ void circ_solve(double2 (&v)[R], const Circ<R> &k, int lane) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
        v[r] = make_double2(__dmul_rn(v[r].x, k.rc), __dmul_rn(v[r].y, k.rc));
        if (r > 0) v[r] = fma2(k.rho, v[r - 1], v[r]);
    }
    double2 y = circ_carry<false, kTwist>(v[R - 1], k.pw[R - 1], k.invf, k.hf, lane);
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = fma2(k.pw[r], y, v[r]);
#pragma unroll
    for (int r = R - 2; r >= 0; --r) v[r] = fma2(k.rho, v[r + 1], v[r]);
    y = circ_carry<true, kTwist>(v[0], k.pw[R - 1], k.invb, k.hb, lane);
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = fma2(k.pw[R - 1 - r], y, v[r]);
}
// The (0,0) pressure line: a (x(i-1) - 2 x(i) + x(i+1)) = r(i) for planes
// 0..N-2 with x(-1) = x(N-1) = 0, on the real parts; x(N-1) = 0 and the
// imaginary parts 0.  With f = r/a,
//   x(i) = -( (N-1-i) sum_{k<=i} (k+1) f(k) + (i+1) sum_{k>i} (N-1-k) f(k) )/N.
template <int R>
__device__ __forceinline__ void dirichlet_solve(double2 (&v)[R], double a, int lane) {
    constexpr int N = 32 * R;
    const int i0 = R * lane;
    double A[R], B[R];   // inclusive prefix of (k+1) f, exclusive suffix of (N-1-k) f within the block
    double sa = 0.0, sb = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const double f = i0 + r < N - 1 ? v[r].x / a : 0.0;
        sa = __fma_rn((double)(i0 + r + 1), f, sa);
        A[r] = sa;
        B[r] = __dmul_rn((double)(N - 1 - i0 - r), f);
    }
#pragma unroll
    for (int r = R - 1; r >= 0; --r) {
        const double t = B[r];
        B[r] = sb;
        sb = __dadd_rn(sb, t);
    }
    double pa = sa, pb = sb;
#pragma unroll
    for (int h = 1; h < 32; h <<= 1) {
        const double ta = __shfl_up_sync(0xffffffffu, pa, h), tb = __shfl_down_sync(0xffffffffu, pb, h);
        if (lane >= h) pa = __dadd_rn(pa, ta);
        if (lane + h < 32) pb = __dadd_rn(pb, tb);
    }
    pa = __shfl_up_sync(0xffffffffu, pa, 1);
    pb = __shfl_down_sync(0xffffffffu, pb, 1);
    if (lane == 0) pa = 0.0;
    if (lane == 31) pb = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = i0 + r;
        const double t = __fma_rn((double)(N - 1 - i), __dadd_rn(A[r], pa), __dmul_rn((double)(i + 1), __dadd_rn(B[r], pb)));
        v[r] = make_double2(i < N - 1 ? -(t / (double)N) : 0.0, 0.0);
    }
}
// Solve on a row in shared memory (plane i at row[row_slot(i)]; one warp, in
// place): the (0,0) line's Dirichlet problem or the circulant one.
template <int R, bool kTwist = false>
__device__ __forceinline__ void circ_solve_row(double2 *row, const Circ<R> &k, int lane) {
    double2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = row[row_slot(R * lane + r)];
    circ_solve<R, kTwist>(v, k, lane);
#pragma unroll
    for (int r = 0; r < R; ++r) row[row_slot(R * lane + r)] = v[r];
    __syncwarp();
}
template <int R>
__device__ __forceinline__ void dirichlet_solve_row(double2 *row, double a, int lane) {
    double2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = row[row_slot(R * lane + r)];
    dirichlet_solve<R>(v, a, lane);
#pragma unroll
    for (int r = 0; r < R; ++r) row[row_slot(R * lane + r)] = v[r];
    __syncwarp();
}

// Pressure-source and explicit ustep terms of the x-line kernels with every
// rounding written out (no multiply-add contraction), so that a kernel which
// accumulates them one input field at a time forms bitwise the values of one
// that has every field at hand.
__device__ __forceinline__ double2 cadd_rn(double2 a, double2 b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
__device__ __forceinline__ double2 cscale_rn(double2 a, double c) { return make_double2(__dmul_rn(c, a.x), __dmul_rn(c, a.y)); }
// Term of component n of one field (coefficient c when coef, none for ff) in
// the pressure source at plane i (poisson.F90:97-116): x0, x1 the field at
// planes i and i+1; n = 0: c (x1 - x0)/dx; n = 1, 2: c i k (x1 + x0)/2, k = ky, kz.
__device__ __forceinline__ double2 psrc_term_rt(int n, bool coef, double c, double2 x0, double2 x1, double ky, double kz, double dx,
                                                double rdx) {
    if (n == 0) {
        double2 d = make_double2(__dsub_rn(x1.x, x0.x), __dsub_rn(x1.y, x0.y));
        if (coef) d = cscale_rn(d, c);
        return make_double2(qdiv(d.x, dx, rdx), qdiv(d.y, dx, rdx));
    }
    const double k = n == 1 ? ky : kz;
    double2 d = make_double2(__dmul_rn(-k, __dadd_rn(x1.y, x0.y)), __dmul_rn(k, __dadd_rn(x1.x, x0.x)));
    if (coef) d = cscale_rn(d, c);
    return cscale_rn(d, 0.5);
}
template <bool kCoef>
__device__ __forceinline__ double2 psrc_term(int n, double c, double2 x0, double2 x1, double ky, double kz, double dx, double rdx) {
    return psrc_term_rt(n, kCoef, c, x0, x1, ky, kz, dx, rdx);
}
// Per-line coefficients of velstep's three systems and right-hand sides,
// every rounding written out (poisson.F90:118-161, usteptime.F90:73-300).
struct LineCoef {
    double pa, pb;         // pressure and divcorr systems: a (= c), b
    double ua, ub;         // ustep system: a (= c), b
    double fy, gd, alp;    // ustep right-hand side: 1 - dt vis c1 w2, dt vis c1, dt (c1 + c2)
    double c2dtv;          // divcorr pressure update: c2 dt vis
};
__device__ __forceinline__ LineCoef line_coef(double dt, double vis, double c1, double c2, double dx2, double w2) {
    LineCoef k;
    const double r1 = 1.0 / dx2, r2 = -2.0 / dx2, dtv = __dmul_rn(dt, vis);
    k.pa = __dsub_rn(r1, __dmul_rn(0.25, w2));
    k.pb = __dsub_rn(r2, __dmul_rn(0.5, w2));
    const double dvc2 = __dmul_rn(dtv, c2);
    k.ua = -(dvc2 / dx2);
    k.ub = __dadd_rn(1.0, __dmul_rn(dvc2, __dadd_rn(2.0 / dx2, w2)));
    k.gd = __dmul_rn(dtv, c1);
    k.fy = __dsub_rn(1.0, __dmul_rn(k.gd, w2));
    k.alp = __dmul_rn(dt, __dadd_rn(c1, c2));
    k.c2dtv = __dmul_rn(__dmul_rn(c2, dt), vis);
    return k;
}
// p + (phi - p): the pressure estimate of poisson.F90:163-175 with relaxation 1.
__device__ __forceinline__ double2 p_update(double2 po, double2 tp) {
    return make_double2(__dadd_rn(po.x, __dsub_rn(tp.x, po.x)), __dadd_rn(po.y, __dsub_rn(tp.y, po.y)));
}
// ustep right-hand side of component n at one plane (usteptime.F90:73-300):
// u fy + ex - alp grad_n p + gd lap(u)/dx^2, ex the explicit part, pm and p0
// the pressure at planes i-1 and i; the plane i = 0 forms the Laplacian as
// (u(i+1) - 2u) + u(i-1), the others as (u(i-1) + u(i+1)) - 2u.
__device__ __forceinline__ double2 ustep_rhs(int n, const LineCoef &k, double2 ui, double2 um, double2 up, double2 ex, double2 pm,
                                             double2 p0, bool i0, double ky, double kz, double dx, double rdx, double dx2,
                                             double rdx2) {
    double2 rv = make_double2(__dadd_rn(__dmul_rn(ui.x, k.fy), ex.x), __dadd_rn(__dmul_rn(ui.y, k.fy), ex.y));
    double2 gp;
    if (n == 0) {
        gp = make_double2(qdiv(__dmul_rn(k.alp, __dsub_rn(p0.x, pm.x)), dx, rdx), qdiv(__dmul_rn(k.alp, __dsub_rn(p0.y, pm.y)), dx, rdx));
    } else {
        const double ah = __dmul_rn(k.alp, 0.5), kk = n == 1 ? ky : kz;
        const double2 sp = make_double2(__dmul_rn(ah, __dadd_rn(pm.x, p0.x)), __dmul_rn(ah, __dadd_rn(pm.y, p0.y)));
        gp = make_double2(__dmul_rn(-kk, sp.y), __dmul_rn(kk, sp.x));
    }
    rv = make_double2(__dsub_rn(rv.x, gp.x), __dsub_rn(rv.y, gp.y));
    double2 lap;
    if (i0) lap = make_double2(__dadd_rn(__dsub_rn(up.x, __dmul_rn(2.0, ui.x)), um.x), __dadd_rn(__dsub_rn(up.y, __dmul_rn(2.0, ui.y)), um.y));
    else lap = make_double2(__dsub_rn(__dadd_rn(um.x, up.x), __dmul_rn(2.0, ui.x)), __dsub_rn(__dadd_rn(um.y, up.y), __dmul_rn(2.0, ui.y)));
    return make_double2(__dadd_rn(rv.x, qdiv(__dmul_rn(k.gd, lap.x), dx2, rdx2)), __dadd_rn(rv.y, qdiv(__dmul_rn(k.gd, lap.y), dx2, rdx2)));
}
// Divergence of u at plane i (poisson.F90:260-300, steptheflow.F90:219-240):
// (u1(i+1) - u1(i))/dx + i ky (u2(i) + u2(i+1))/2 + i kz (u3(i) + u3(i+1))/2.
__device__ __forceinline__ double2 div_term(double2 u1i, double2 u1p, double2 u2i, double2 u2p, double2 u3i, double2 u3p, double ky,
                                            double kz, double dx, double rdx) {
    double2 t = make_double2(qdiv(__dsub_rn(u1p.x, u1i.x), dx, rdx), qdiv(__dsub_rn(u1p.y, u1i.y), dx, rdx));
    const double2 sy = make_double2(__dmul_rn(__dadd_rn(u2i.x, u2p.x), 0.5), __dmul_rn(__dadd_rn(u2i.y, u2p.y), 0.5));
    const double2 sz = make_double2(__dmul_rn(__dadd_rn(u3i.x, u3p.x), 0.5), __dmul_rn(__dadd_rn(u3i.y, u3p.y), 0.5));
    t = make_double2(__dadd_rn(t.x, __dmul_rn(-ky, sy.y)), __dadd_rn(t.y, __dmul_rn(ky, sy.x)));
    return make_double2(__dadd_rn(t.x, __dmul_rn(-kz, sz.y)), __dadd_rn(t.y, __dmul_rn(kz, sz.x)));
}
__device__ __forceinline__ double cabs_rn(double2 t) { return __dsqrt_rn(__dadd_rn(__dmul_rn(t.x, t.x), __dmul_rn(t.y, t.y))); }
// divcorr's correction at plane i (poisson.F90:330-508): phi d0 at i, dm at
// i-1, dp at i+1; u -= alpc grad phi, p += phi - c2 dt vis lap(phi).
__device__ __forceinline__ void divcorr_update(const LineCoef &k, double2 d0, double2 dm, double2 dp, bool i0, double2 U1, double2 U2,
                                               double2 U3, double2 Pw, double ky, double kz, double w2, double dx, double rdx,
                                               double dx2, double rdx2, double2 &nu1, double2 &nu2, double2 &nu3, double2 &np) {
    const double alpc = k.alp;
    const double2 s = make_double2(__dadd_rn(dm.x, d0.x), __dadd_rn(dm.y, d0.y));
    double2 gy, gz;
    if (i0) {
        gy = make_double2(__dmul_rn(__dmul_rn(-ky, 0.0), 0.5), __dmul_rn(__dmul_rn(ky, alpc), 0.5));
        gz = make_double2(__dmul_rn(__dmul_rn(-kz, 0.0), 0.5), __dmul_rn(__dmul_rn(kz, alpc), 0.5));
    } else {
        const double ah = __dmul_rn(alpc, 0.5);
        gy = make_double2(__dmul_rn(-ky, 0.0), __dmul_rn(ky, ah));
        gz = make_double2(__dmul_rn(-kz, 0.0), __dmul_rn(kz, ah));
    }
    nu1 = make_double2(__dsub_rn(U1.x, qdiv(__dmul_rn(alpc, __dsub_rn(d0.x, dm.x)), dx, rdx)),
                       __dsub_rn(U1.y, qdiv(__dmul_rn(alpc, __dsub_rn(d0.y, dm.y)), dx, rdx)));
    nu2 = make_double2(__dsub_rn(U2.x, __dsub_rn(__dmul_rn(gy.x, s.x), __dmul_rn(gy.y, s.y))),
                       __dsub_rn(U2.y, __dadd_rn(__dmul_rn(gy.x, s.y), __dmul_rn(gy.y, s.x))));
    nu3 = make_double2(__dsub_rn(U3.x, __dsub_rn(__dmul_rn(gz.x, s.x), __dmul_rn(gz.y, s.y))),
                       __dsub_rn(U3.y, __dadd_rn(__dmul_rn(gz.x, s.y), __dmul_rn(gz.y, s.x))));
    const double2 lap = make_double2(__dsub_rn(qdiv(__dadd_rn(__dsub_rn(dm.x, __dmul_rn(2.0, d0.x)), dp.x), dx2, rdx2), __dmul_rn(w2, d0.x)),
                                     __dsub_rn(qdiv(__dadd_rn(__dsub_rn(dm.y, __dmul_rn(2.0, d0.y)), dp.y), dx2, rdx2), __dmul_rn(w2, d0.y)));
    np = make_double2(__dsub_rn(__dadd_rn(Pw.x, d0.x), __dmul_rn(k.c2dtv, lap.x)), __dsub_rn(__dadd_rn(Pw.y, d0.y), __dmul_rn(k.c2dtv, lap.y)));
}

}  // namespace pibm
