// sweep.cuh -- plane transforms of 256^2 planes as separate sweeps over the
// columns (z) and the rows (y) of a plane, with the (z, ky) planes in between
// kept in device memory.
//
// A 256^2 plane needs a cluster of 8 SMs in the plane kernels of plane_cl.cuh,
// which pay for every element that crosses SMs.  A column or a row is 4 KB:
// blocks of 32 KB, four to six to an SM, stream them.  The planes in between
// cost a write and a read of L2 / HBM; in return
// the columns' kernels do everything that is local to a (kx-plane, ky) column:
//   k_cz  inverse z of 7 fields: u(3), p, i kz u1, i kz u2, i kz p, from which
//         k_ry forms the 10 real fields' rows (vorticity and pressure gradient
//         combine in (z, ky) space: 7 z transforms serve 10 fields)
//   k_rp  rows of the 5 products and 3 x-flux differences, forward y
//   k_cn  per component: forward z of i ky F(u1 uc) + F(D_c) (one transform) and
//         of F(u2 uc), nl from them
//   k_cq, k_rq  Q's spectrum from nl, onl and u, inverse z, inverse y
//   k_rf, k_cf  forward y and z of the forcing
// The items (fields, components) of one block of planes run side by side
// (blockIdx.x), so what they share comes from L2.
// Measured (us per step at 256^3, plane kernels -> sweeps): fields to real space
// 1521 -> 958, nonlinear term 2037 -> 1220, forcing 412 -> 311.  At 128, where a
// plane fits one SM or two, blocks of 8 columns take 132 against 140, 185
// against 192 and 48 against 44 us, 1% of a step, for 5 launches more: it keeps
// the plane kernels.
#pragma once
#include "step_common.cuh"

namespace pibm {

template <int N> struct Sweep {
    static constexpr int AZ = Plan<N>::AZ, BZ = Plan<N>::BZ, M = N / 2, my2 = M + 1, PS = my2 * N;
    static_assert(N == 256, "the only grid that transforms by sweeps (kSweepMin)");
    static constexpr int QC = 8;                      // columns of a block: 128 contiguous bytes per kz
    static constexpr int NS = M / QC;                 // blocks of a plane (without column M)
    static constexpr int CT = QC * BZ;                // threads of a column block: AZ points of a column each
    static constexpr int GC = N * NS + N / QC;        // blocks of a field: its planes' columns < M, then column M of QC planes each
    static constexpr int CSM = (N * QC + N) * 16;     // shared memory of one column buffer and the twiddles
    static constexpr int RC = 16;                     // rows of a block
    static constexpr int RT = 128, RB = N / RC;       // threads, blocks of a plane
    static constexpr int RSM = (RC * my2 + N) * 16;
    static constexpr int RBLK = 6;                    // row blocks per SM the register budget is sized for
    static constexpr uint32_t RBYTES = RC * my2 * 16; // rows of a block, spectral or real: N (N+2) doubles = my2 N complex
    static_assert(M % QC == 0 && N % QC == 0 && QC * AZ % CT == 0, "column blocks");
    // 228 KB per SM, of which each block takes 1 KB beside its own (a barrier is its only static memory)
    static_assert(RBLK * (RSM + 128 + 1024) <= 228 * 1024, "row blocks");
};
// A thread's column: its plane, ky index and offset in a field's planes.
struct ColPos { int i, j; size_t off; };
template <int N> __device__ __forceinline__ ColPos col_pos(int b, int q) {
    using W = Sweep<N>;
    ColPos c;
    if (b < N * W::NS) { c.i = b / W::NS; c.j = (b % W::NS) * W::QC + q; }
    else { c.i = (b - N * W::NS) * W::QC + q; c.j = W::M; }   // column M: one of QC planes per lane
    c.off = (size_t)c.i * W::PS + c.j;
    return c;
}
// Inverse z of a column whose points kz = BZ*n1 + n2 this thread holds in
// v[n1]; out(R, X) gets row R of the transform order (R = BZ*k1 + k2, z = k1 + AZ*k2).
// The buffer may be rewritten after the call's last barrier by its own thread only.
template <int N, class F>
__device__ __forceinline__ void col_c2r(double2 (&v)[Plan<N>::AZ], double2 *sm, const double2 *tw, F out) {
    using W = Sweep<N>;
    constexpr int AZ = W::AZ, BZ = W::BZ, QC = W::QC;
    const int q = threadIdx.x % QC, n2 = threadIdx.x / QC;
    Dft<AZ, 1>::run(v);
    sm[n2 * QC + q] = v[0];
#pragma unroll
    for (int k1 = 1; k1 < AZ; ++k1) sm[(BZ * k1 + n2) * QC + q] = cmul(v[k1], tw_get<1>(tw, n2 * k1));
    __syncthreads();
#pragma unroll
    for (int u0 = 0; u0 < QC * AZ; u0 += W::CT) {
        const int k1 = (u0 + (int)threadIdx.x) / QC;
        double2 x[BZ];
#pragma unroll
        for (int n = 0; n < BZ; ++n) x[n] = sm[(BZ * k1 + n) * QC + q];
        Dft<BZ, 1>::run(x);
#pragma unroll
        for (int k2 = 0; k2 < BZ; ++k2) out(BZ * k1 + k2, x[k2]);
    }
}
// Forward z of a column: in(R) reads row R of the transform order; on return
// v[k1] = X[kz = BZ*k1 + k2] with k2 = thread / QC.  Starts and ends with the
// buffer in use by every thread of the column.
template <int N, class F>
__device__ __forceinline__ void col_r2c(double2 (&v)[Plan<N>::AZ], double2 *sm, const double2 *tw, F in) {
    using W = Sweep<N>;
    constexpr int AZ = W::AZ, BZ = W::BZ, QC = W::QC;
    const int q = threadIdx.x % QC;
#pragma unroll
    for (int u0 = 0; u0 < QC * AZ; u0 += W::CT) {
        const int n1 = (u0 + (int)threadIdx.x) / QC;
        double2 x[BZ];
#pragma unroll
        for (int n = 0; n < BZ; ++n) x[n] = in(BZ * n1 + n);
        Dft<BZ, -1>::run(x);
        sm[BZ * n1 * QC + q] = x[0];
#pragma unroll
        for (int k2 = 1; k2 < BZ; ++k2) sm[(BZ * n1 + k2) * QC + q] = cmul(x[k2], tw_get<-1>(tw, n1 * k2));
    }
    __syncthreads();
    const int k2 = threadIdx.x / QC;
#pragma unroll
    for (int n1 = 0; n1 < AZ; ++n1) v[n1] = sm[(BZ * n1 + k2) * QC + q];
    Dft<AZ, -1>::run(v);
}

// k_cz: inverse z of field t: u1, u2, u3, p, i kz u1, i kz u2, i kz p -> zf[t].
template <int N>
__device__ __forceinline__ void b_cz(const Geo &g, const double2 *__restrict__ u, const double2 *__restrict__ p, double2 *__restrict__ zf) {
    using W = Sweep<N>;
    constexpr int AZ = W::AZ, BZ = W::BZ, QC = W::QC, my2 = W::my2;
    extern __shared__ double2 sm[];
    double2 *tws = sm + N * QC;
    for (int t = threadIdx.x; t < N; t += W::CT) tws[t] = g.tw[t];
    grid_dep_wait();   // the twiddles above are set-up data; the fields come from earlier kernels
    const int t = blockIdx.x, q = threadIdx.x % QC, n2 = threadIdx.x / QC;
    const ColPos c = col_pos<N>(blockIdx.y, q);
    const double2 *src = (t == 3 || t == 6 ? p : u + (size_t)(t < 3 ? t : t - 4) * N * W::PS) + c.off + (size_t)n2 * my2;
    double2 v[AZ];
#pragma unroll
    for (int n1 = 0; n1 < AZ; ++n1) v[n1] = src[BZ * n1 * my2];
    if (t >= 4)
#pragma unroll
        for (int n1 = 0; n1 < AZ; ++n1) { const double k = g.kz[BZ * n1 + n2]; v[n1] = make_double2(-k * v[n1].y, k * v[n1].x); }
    __syncthreads();   // the twiddles are in place
    double2 *dst = zf + (size_t)t * N * W::PS + c.off;
    col_c2r<N>(v, sm, tws, [&](int R, double2 x) { dst[R * my2] = x; });
}

// k_ry: the rows of the 10 real fields from k_cz's planes (b_a0's items, the
// products with i ky and the x differences taken in (z, ky) space);
// part[(i*RB + block)*12 + q] as in b_a0.
template <int N>
__device__ __forceinline__ void b_ry(const Geo &g, const double2 *__restrict__ zf, double *__restrict__ ubcp, double *__restrict__ pbcp,
                                     double *__restrict__ omega, double *__restrict__ pgr, Scal *__restrict__ sc,
                                     double *__restrict__ part) {
    using W = Sweep<N>;
    constexpr int my2 = W::my2, PS = W::PS, RSP = RP<N>::RSP, nx = N;
    extern __shared__ double2 sm[];
    double2 *buf = sm, *tws = sm + W::RC * my2;
    __shared__ uint64_t mb;
    if (threadIdx.x == 0) mbar_init(&mb, 1);
    for (int t = threadIdx.x; t < N; t += W::RT) tws[t] = g.tw[t];
    __syncthreads();
    grid_dep_wait();
    const int t = blockIdx.x, i = blockIdx.y / W::RB, rb = blockIdx.y % W::RB;
    const int im = i == 0 ? nx - 1 : i - 1, ip = i == nx - 1 ? 0 : i + 1;
    auto Z = [&](int f, int pl) { return zf + ((size_t)f * nx + pl) * PS + (size_t)rb * W::RC * my2; };
    if (t < 4 || t == 9) {
        if (threadIdx.x == 0) { fence_async_smem(); bulk_load(buf, Z(t < 4 ? t : 6, i), W::RBYTES, &mb); }
        uint32_t phase = 0;
        load_wait(&mb, phase, sc);
    } else {
        const double tdx = 2.0 * g.dx, rtdx = 1.0 / tdx;   // divisor and reciprocal for qdiv
        // i ky a + s b + (hp - hm)/2dx with the sources of the item
        const int fa = t == 4 ? 2 : t == 6 ? 0 : 3, fb = t == 4 ? 5 : 4, fd = t == 5 ? 2 : t == 6 ? 1 : 3;
        const double2 *A = Z(fa, i), *B = Z(fb, i), *Hp = Z(fd, ip), *Hm = Z(fd, im);
#pragma unroll 4
        for (int e = threadIdx.x; e < W::RC * my2; e += W::RT) {
            double2 f;
            if (t == 4) {          // i ky u3 - (i kz u2)
                const double ky = g.ky[e % my2];
                const double2 a = A[e], b = B[e];
                f = make_double2(-ky * a.y - b.x, ky * a.x - b.y);
            } else if (t == 8) {   // i ky p
                const double ky = g.ky[e % my2];
                const double2 a = A[e];
                f = make_double2(-ky * a.y, ky * a.x);
            } else {
                const double2 hp = Hp[e], hm = Hm[e];
                f = make_double2(qdiv(hp.x - hm.x, tdx, rtdx), qdiv(hp.y - hm.y, tdx, rtdx));
                if (t == 5) {          // i kz u1 - d(u3)/dx
                    const double2 b = B[e];
                    f = make_double2(b.x - f.x, b.y - f.y);
                } else if (t == 6) {   // d(u2)/dx - i ky u1
                    const double ky = g.ky[e % my2];
                    const double2 a = A[e];
                    f = make_double2(f.x + ky * a.y, f.y - ky * a.x);
                }
            }
            buf[e] = f;
        }
    }
    __syncthreads();
    rows_c2r<N, W::RC, W::RT, false>(buf, tws);
    const size_t roff = (size_t)i * RSP + (size_t)rb * W::RC * (N + 2);
    if (t < 3) {
        // u + umean; fluid, solid and total sums and max |u| of this block's rows.
        // Scratch of its own left room for five blocks per SM (fields to real space 1031 -> 958 us).
        double *scr = (double *)tws;   // the transform's last barrier is behind every thread
        static_assert(N * sizeof(double2) >= 32 * 3 * sizeof(double), "reduction scratch");
        const double um = sc->umean[t];
        double *b = (double *)buf;
        const uint8_t *fl = g.fluid + roff;
        double sf = 0.0, ss = 0.0, sa = 0.0, mx = kSmallD;
        for (int e = threadIdx.x; e < W::RC * (N + 2); e += W::RT) {
            if (e % (N + 2) >= N) continue;
            const double x = b[e] + um;
            b[e] = x;
            if (fl[e]) sf += x; else ss += x;
            sa += x;
            mx = fmax(mx, fabs(x));
        }
        double v3[3] = {sf, ss, sa};
        block_reduce_k<3>(v3, scr);
        mx = block_max(mx, scr);
        const size_t slot = (size_t)blockIdx.y * 12;
        if (threadIdx.x == 0) { part[slot + t] = v3[0]; part[slot + 3 + t] = v3[1]; part[slot + 6 + t] = v3[2]; part[slot + 9 + t] = mx; }
    }
    double *dst = (t < 3 ? ubcp + (size_t)t * nx * RSP : t == 3 ? pbcp : t < 7 ? omega + (size_t)(t - 4) * nx * RSP : pgr + (size_t)(t - 7) * nx * RSP) + roff;
    if (threadIdx.x == 0) { bulk_store(dst, buf, W::RBYTES); bulk_wait_read(); }
}

// k_rp: forward y of the rows of item t: the products u0u1, u0u2, u1u1, u1u2,
// u2u2, then the x-flux differences D_c -> pz[t] (unscaled).
template <int N>
__device__ __forceinline__ void b_rp(const Geo &g, const double *__restrict__ ubcp, const double *__restrict__ Dx, double2 *__restrict__ pz,
                                     Scal *__restrict__ sc) {
    using W = Sweep<N>;
    constexpr int RSP = RP<N>::RSP, nx = N;
    extern __shared__ double2 sm[];
    double2 *buf = sm, *tws = sm + W::RC * W::my2;
    __shared__ uint64_t mb;
    if (threadIdx.x == 0) mbar_init(&mb, 1);
    for (int t = threadIdx.x; t < N; t += W::RT) tws[t] = g.tw[t];
    __syncthreads();
    grid_dep_wait();
    const int t = blockIdx.x, i = blockIdx.y / W::RB, rb = blockIdx.y % W::RB;
    const size_t roff = (size_t)i * RSP + (size_t)rb * W::RC * (N + 2);
    const int na = t < 2 ? 0 : t < 4 ? 1 : 2, nb = t == 0 || t == 2 ? 1 : 2;   // the product's factors
    if (threadIdx.x == 0) {
        fence_async_smem();
        bulk_load(buf, (t < 5 ? ubcp + (size_t)na * nx * RSP : Dx + (size_t)(t - 5) * nx * RSP) + roff, W::RBYTES, &mb);
    }
    uint32_t phase = 0;
    if (t < 5 && na != nb) {
        const double2 *B2 = (const double2 *)(ubcp + (size_t)nb * nx * RSP + roff);
        constexpr int E = W::RC * W::my2, K = 8, EB = K * W::RT;
        bool waited = false;
        for (int e0 = threadIdx.x; e0 < E; e0 += EB) {   // the second factor's loads start before the first is waited for
            double2 y[K];
#pragma unroll
            for (int k = 0; k < K; ++k) if (e0 + k * W::RT < E) y[k] = B2[e0 + k * W::RT];
            if (!waited) { load_wait(&mb, phase, sc); waited = true; }
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (e0 + k * W::RT < E) { const double2 x = buf[e0 + k * W::RT]; buf[e0 + k * W::RT] = make_double2(x.x * y[k].x, x.y * y[k].y); }
        }
    } else {
        load_wait(&mb, phase, sc);
        if (t < 5)
            for (int e = threadIdx.x; e < W::RC * W::my2; e += W::RT) { const double2 x = buf[e]; buf[e] = make_double2(x.x * x.x, x.y * x.y); }
    }
    __syncthreads();
    rows_r2c_1<N, W::RC, W::RT>(buf, tws);
    rows_r2c_2<N, W::RC, W::RT, false>(buf, tws);
    if (threadIdx.x == 0) { bulk_store(pz + ((size_t)t * nx + i) * W::PS + (size_t)rb * W::RC * W::my2, buf, W::RBYTES); bulk_wait_read(); }
}

// k_cn: component c of the nonlinear term (b_nl) from k_rp's rows.  The first
// transform waits in its place of nl_new while the second runs in the
// registers it used (a second shared buffer, or all of Q's loads in this
// kernel, left three blocks to an SM).
template <int N>
__device__ __forceinline__ void b_cn(const Geo &g, const double2 *__restrict__ pz, double2 *nl_new) {
    using W = Sweep<N>;
    constexpr int AZ = W::AZ, BZ = W::BZ, QC = W::QC, my2 = W::my2, nx = N;
    extern __shared__ double2 sm[];
    double2 *tws = sm + N * QC;
    for (int t = threadIdx.x; t < N; t += W::CT) tws[t] = g.tw[t];
    __syncthreads();
    grid_dep_wait();
    const int c = blockIdx.x, q = threadIdx.x % QC, k2 = threadIdx.x / QC;
    const ColPos cp = col_pos<N>(blockIdx.y, q);
    const double ky = g.ky[cp.j];
    const size_t FS = (size_t)nx * W::PS;
    const double2 *A = pz + (c == 0 ? 0 : c + 1) * FS + cp.off, *B = pz + (c == 0 ? 1 : c + 2) * FS + cp.off, *Dc = pz + (5 + c) * FS + cp.off;
    double2 *dst = nl_new + c * FS + cp.off;
    double2 v[AZ];
    col_r2c<N>(v, sm, tws, [&](int R) {
        const double2 a = A[R * my2], d = Dc[R * my2];
        return make_double2(d.x - ky * a.y, d.y + ky * a.x);
    });
#pragma unroll
    for (int k1 = 0; k1 < AZ; ++k1) dst[(BZ * k1 + k2) * my2] = v[k1];   // read back by this thread
    __syncthreads();   // every thread has read the buffer
    col_r2c<N>(v, sm, tws, [&](int R) { return B[R * my2]; });
    constexpr int G = 4;
#pragma unroll
    for (int g0 = 0; g0 < AZ; g0 += G) {
        double2 s[G];
#pragma unroll
        for (int k = 0; k < G; ++k) s[k] = dst[(BZ * (g0 + k) + k2) * my2];
#pragma unroll
        for (int k = 0; k < G; ++k) {
            const int kz = BZ * (g0 + k) + k2;
            const double kzv = g.kz[kz];
            const double2 s1 = r2c_norm<N>(s[k], g.nrm), s2 = r2c_norm<N>(v[g0 + k], g.nrm);
            dst[kz * my2] = make_double2(-(s1.x - kzv * s2.y), -(s1.y + kzv * s2.x));
        }
    }
}
// k_cq: inverse z of Q's spectrum, -c3 nl - c4 onl - c12 diffn.
template <int N>
__device__ __forceinline__ void b_cq(const Geo &g, const double2 *__restrict__ nl, const double2 *__restrict__ u, const double2 *__restrict__ onl,
                                     double2 *__restrict__ qz) {
    using W = Sweep<N>;
    constexpr int AZ = W::AZ, BZ = W::BZ, QC = W::QC, my2 = W::my2, nx = N;
    extern __shared__ double2 sm[];
    double2 *tws = sm + N * QC;
    for (int t = threadIdx.x; t < N; t += W::CT) tws[t] = g.tw[t];
    __syncthreads();
    grid_dep_wait();
    const int c = blockIdx.x, q = threadIdx.x % QC, n2 = threadIdx.x / QC;
    const ColPos cp = col_pos<N>(blockIdx.y, q);
    const double c12 = g.c1 + g.c2;
    const size_t F = c * (size_t)nx * W::PS;
    const int im = cp.i == 0 ? nx - 1 : cp.i - 1, ip = cp.i == nx - 1 ? 0 : cp.i + 1;
    const double2 *nn = nl + F + cp.off, *on = onl + F + cp.off, *u0 = u + F + cp.off;
    const double2 *um = u + F + (size_t)im * W::PS + cp.j, *up = u + F + (size_t)ip * W::PS + cp.j;
    double2 v[AZ];
    constexpr int G = 2;   // points whose loads are in flight together
#pragma unroll
    for (int g0 = 0; g0 < AZ; g0 += G) {
        double2 x[G], o[G], a[G], b[G], d[G];
        double w2[G];
#pragma unroll
        for (int k = 0; k < G; ++k) {
            const int e = (BZ * (g0 + k) + n2) * my2;
            x[k] = nn[e]; o[k] = on[e]; a[k] = um[e]; b[k] = u0[e]; d[k] = up[e]; w2[k] = g.w2[e + cp.j];
        }
#pragma unroll
        for (int k = 0; k < G; ++k) {
            double2 df = make_double2(g.rdx2 * ((a[k].x - 2.0 * b[k].x) + d[k].x), g.rdx2 * ((a[k].y - 2.0 * b[k].y) + d[k].y));
            df = make_double2((df.x - w2[k] * b[k].x) * g.vis, (df.y - w2[k] * b[k].y) * g.vis);
            v[g0 + k] = make_double2((-g.c3 * x[k].x - g.c4 * o[k].x) - c12 * df.x, (-g.c3 * x[k].y - g.c4 * o[k].y) - c12 * df.y);
        }
    }
    double2 *qd = qz + F + cp.off;
    col_c2r<N>(v, sm, tws, [&](int R, double2 x) { qd[R * my2] = x; });
}

// k_rq: inverse y of the rows of Q.
template <int N>
__device__ __forceinline__ void b_rq(const Geo &g, const double2 *__restrict__ qz, double *__restrict__ Q, Scal *__restrict__ sc) {
    using W = Sweep<N>;
    extern __shared__ double2 sm[];
    double2 *buf = sm, *tws = sm + W::RC * W::my2;
    __shared__ uint64_t mb;
    if (threadIdx.x == 0) mbar_init(&mb, 1);
    for (int t = threadIdx.x; t < N; t += W::RT) tws[t] = g.tw[t];
    __syncthreads();
    grid_dep_wait();
    const size_t off = ((size_t)blockIdx.x * N + blockIdx.y / W::RB) * W::PS + (size_t)(blockIdx.y % W::RB) * W::RC * W::my2;
    if (threadIdx.x == 0) { fence_async_smem(); bulk_load(buf, qz + off, W::RBYTES, &mb); }
    uint32_t phase = 0;
    load_wait(&mb, phase, sc);
    rows_c2r<N, W::RC, W::RT, false>(buf, tws);
    if (threadIdx.x == 0) { bulk_store(Q + 2 * off, buf, W::RBYTES); bulk_wait_read(); }
}

// k_rf, k_cf: ff = r2c(fr - frmean) (b_ff).
template <int N>
__device__ __forceinline__ void b_rf(const Geo &g, const double *__restrict__ fr, double2 *__restrict__ fz, Scal *__restrict__ sc) {
    using W = Sweep<N>;
    extern __shared__ double2 sm[];
    double2 *buf = sm, *tws = sm + W::RC * W::my2;
    __shared__ uint64_t mb;
    if (threadIdx.x == 0) mbar_init(&mb, 1);
    for (int t = threadIdx.x; t < N; t += W::RT) tws[t] = g.tw[t];
    __syncthreads();
    grid_dep_wait();
    const size_t off = ((size_t)blockIdx.x * N + blockIdx.y / W::RB) * W::PS + (size_t)(blockIdx.y % W::RB) * W::RC * W::my2;
    if (threadIdx.x == 0) { fence_async_smem(); bulk_load(buf, fr + 2 * off, W::RBYTES, &mb); }
    uint32_t phase = 0;
    load_wait(&mb, phase, sc);
    const double fmn = sc->frmean[blockIdx.x];
    for (int e = threadIdx.x; e < W::RC * W::my2; e += W::RT) { const double2 x = buf[e]; buf[e] = make_double2(x.x - fmn, x.y - fmn); }
    __syncthreads();
    rows_r2c_1<N, W::RC, W::RT>(buf, tws);
    rows_r2c_2<N, W::RC, W::RT, false>(buf, tws);
    if (threadIdx.x == 0) { bulk_store(fz + off, buf, W::RBYTES); bulk_wait_read(); }
}
template <int N>
__device__ __forceinline__ void b_cf(const Geo &g, const double2 *__restrict__ fz, double2 *__restrict__ ff) {
    using W = Sweep<N>;
    extern __shared__ double2 sm[];
    double2 *tws = sm + N * W::QC;
    for (int t = threadIdx.x; t < N; t += W::CT) tws[t] = g.tw[t];
    __syncthreads();
    grid_dep_wait();
    const ColPos c = col_pos<N>(blockIdx.y, threadIdx.x % W::QC);
    const size_t FS = (size_t)N * W::PS;
    const double2 *src = fz + blockIdx.x * FS + c.off;
    double2 *dst = ff + blockIdx.x * FS + c.off;
    double2 v[W::AZ];
    col_r2c<N>(v, sm, tws, [&](int R) { return src[R * W::my2]; });
#pragma unroll
    for (int k1 = 0; k1 < W::AZ; ++k1) dst[(W::BZ * k1 + threadIdx.x / W::QC) * W::my2] = r2c_norm<N>(v[k1], g.nrm);
}

}  // namespace pibm
