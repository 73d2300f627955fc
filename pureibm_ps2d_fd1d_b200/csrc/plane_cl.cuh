// plane_cl.cuh -- y-z plane transforms of one plane held in shared memory.
//
// A plane is N rows kz x (N/2+1) columns ky of complex FP64: 133 KB at N = 128.
// Up to 96 one CTA holds the whole plane and two or more CTAs share an SM, so
// their loads, stores and barriers overlap.  At 128 and 256 a cluster of C
// CTAs shares a plane, each holding 1/C of it:
//
//   column phase (z transforms)  CTA r holds columns ky in [r*MC, (r+1)*MC) of
//                                all N rows at pitch PZ = MC+1; CTA 0 also
//                                keeps column ky = M = N/2 in slot MC.
//   row phase (y transforms)     CTA r holds rows [r*NR, (r+1)*NR) of the plane
//                                in z-transform output order at pitch P = M+1:
//                                a real plane keeps its HBM layout and CTA r
//                                moves its rows with one contiguous bulk copy.
//
// With one CTA both layouts coincide (PZ = P) and also equal the plane's image
// in HBM, so a plane moves with a single bulk copy either way.
//
// A transform is four passes, each one read and one write of the plane:
//   c2r   z over AZ + twiddle | z over BZ, stored in the row owner's rows |
//         half-length real reconstruction + y over AY + twiddle | y over BY
//   r2c   y over BY + twiddle | y over AY + real split, stored in the column
//         owner's columns | z over BZ + twiddle | z over AZ
// The half-length step pairs column n with M-n.  A thread of the AY pass owns
// the residue classes g and BY-g (0 and BY/2) of one row, which contain both
// members of every such pair, so the step needs no pass of its own.  Between
// CTAs the elements cross by 16-byte stores into the owner's shared memory
// (distributed shared memory) between two cluster barriers; the pass that
// sends them holds its outputs in registers over the first one.
// The radix twiddles are immediates (cos48); the pass twiddles come from a
// table of e^{-2 pi i m/N}.
//
// Bound: no unit is saturated.  At 128^3 k_a0 and k_nl keep the shared-memory pipe
// (4 x 2 plane traversals) 54 and 48% busy, FP64 and DRAM 22%, and their warps
// wait for global loads most of all, in k_nl with one CTA to an SM and nothing
// to run meanwhile.  The step's kernels (us per launch at 32 / 64 / 96 / 128^3;
// before: five passes, clusters of 2 CTAs at 64-128, radix twiddles from the
// table; at 256^3 the step transforms by the sweeps of sweep.cuh):
//   k_a0  11.2 / 29.2 / 101 / 150  ->  10.6 / 21.2 / 56.5 / 141
//   k_nl  14.8 / 40.8 / 119 / 226  ->  16.7 / 33.1 / 78.7 / 194
//   k_ff   8.6 / 14.7 / 33.0 / 50.3 ->   8.5 / 12.6 / 22.6 / 43.8
// (One launch of 1280 planes c2r at 128 with its load and store from HBM: 119 ->
// 105 us, 53 us at the copy rate; 960 at 96: 78 -> 38 us; 640 at 64: 20.8 -> 12.6 us.)
#pragma once
#include <cooperative_groups.h>

#include <type_traits>

#include "fft2d.cuh"

namespace pibm {

// CTAs per plane (C), threads per CTA (T) and CTAs per SM the register budget
// is sized for (MINB).
template <int N_, int C_, int T_, int MINB_> struct PlaneCfg {
    static constexpr int N = N_, C = C_, T = T_, MINB = MINB_;
    static constexpr int M = N / 2, P = M + 1;          // row-phase pitch (complex slots)
    static constexpr int MC = M / C, PZ = MC + 1;       // columns per CTA, column-phase pitch
    static constexpr int NR = N / C;                    // rows per CTA in the row phase
    static constexpr int BUF = (N * PZ > NR * P) ? N * PZ : NR * P;   // complex slots of the buffer
    static constexpr int ROWS = NR * (N + 2);           // doubles of one CTA's real rows
    static constexpr uint32_t RBYTES = ROWS * 8;
    static constexpr int NOUT = N * PZ;                 // column-phase slots (slot MC: rank 0 only)
    static constexpr size_t SMEM = (size_t)(BUF + N) * sizeof(double2);   // buffer + twiddle table
    static_assert(M % C == 0 && N % C == 0, "plane split");
    static_assert(RBYTES % 16 == 0, "bulk copies move 16-byte multiples");
};
// The kernels' shapes, chosen by measurement per size.  PL: the step's c2r
// kernels.  RL: r2c.  NL: the nonlinear terms (r2c and c2r of one plane in
// turn: one or two items per SM, so more threads each).  SL: the scalar's c2r.
// At 128 a plane on one CTA of 512 threads beats the cluster of two where
// the loads are bulk copies (k_nl 203 -> 194, k_ff 48 -> 44 us; with the
// scalar's kernels too the scalar step takes 0.916 against 1.02 ms), and
// loses where a CTA gathers its input with plain loads that a second CTA of
// the SM would hide (k_a0 141 -> 165 us).
template <int N> struct PlaneSel;
template <> struct PlaneSel<32>  { using PL = PlaneCfg<32, 1, 128, 4>;  using RL = PL; using NL = PlaneCfg<32, 1, 256, 2>;  using SL = PL; };
template <> struct PlaneSel<64>  { using PL = PlaneCfg<64, 1, 128, 6>;  using RL = PL; using NL = PlaneCfg<64, 1, 256, 2>;  using SL = PL; };
template <> struct PlaneSel<96>  { using PL = PlaneCfg<96, 1, 384, 2>;  using RL = PL; using NL = PL; using SL = PL; };
template <> struct PlaneSel<128> { using PL = PlaneCfg<128, 2, 256, 3>; using RL = PlaneCfg<128, 1, 512, 1>; using NL = RL; using SL = RL; };
template <> struct PlaneSel<256> { using PL = PlaneCfg<256, 8, 256, 3>; using RL = PlaneCfg<256, 8, 128, 5>; using NL = PL; using SL = PL; };
template <int N> using PL = typename PlaneSel<N>::PL;
template <int N> using RL = typename PlaneSel<N>::RL;
template <int N> using NL = typename PlaneSel<N>::NL;
template <int N> using SL = typename PlaneSel<N>::SL;

// Physical z of shared-memory row R (inverse of zrow).
template <int N> __device__ __forceinline__ int zinv(int R) { return (R % Plan<N>::BZ) * Plan<N>::AZ + R / Plan<N>::BZ; }

// Global column ky of column-phase slot jl of CTA `rank`.
template <class L> __device__ __forceinline__ int cl_col(int jl, int rank) { return jl == L::MC ? L::M : rank * L::MC + jl; }

// 32-bit shared::cluster address of element `slot` of CTA `rank`'s buffer,
// and a 16-byte store through it (distributed shared memory).
__device__ __forceinline__ uint32_t cl_addr(const double2 *buf, int slot, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(buf + slot)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_st(uint32_t addr, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}
// Barrier over the CTAs of a plane.
template <class L> __device__ __forceinline__ void cl_sync() {
    if constexpr (L::C > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
}

// Columns 0 and M of rank 0 packed into column 0 (see herm_pack).  Every
// thread of the CTA calls it; ends with a block barrier.
template <class L>
__device__ __forceinline__ void cl_pack_col0(double2 *buf, int rank) {
    constexpr int K0 = (L::N + L::T - 1) / L::T;
    double2 y[K0];
    if (rank == 0) {
#pragma unroll
        for (int k = 0; k < K0; ++k) {
            const int kz = (int)threadIdx.x + k * L::T;
            if (kz < L::N) {
                const int km = (L::N - kz) % L::N;
                y[k] = herm_pack(buf[kz * L::PZ], buf[km * L::PZ], buf[kz * L::PZ + L::MC], buf[km * L::PZ + L::MC]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < K0; ++k) {
            const int kz = (int)threadIdx.x + k * L::T;
            if (kz < L::N) buf[kz * L::PZ] = y[k];
        }
    }
    __syncthreads();
}

// Spectral value of column-phase slot (kz, jl) after cl_r2c (unscaled).
// CTA 0 reads ky = 0 (jl = 0) and ky = M (jl = MC) from the packed column 0.
template <class L>
__device__ __forceinline__ double2 cl_unpack(const double2 *buf, int kz, int jl, int rank) {
    if (rank != 0 || (jl != 0 && jl != L::MC)) return buf[kz * L::PZ + jl];
    const double2 y = buf[kz * L::PZ], ym = buf[((L::N - kz) % L::N) * L::PZ];
    if (jl == 0) return make_double2(0.5 * (y.x + ym.x), 0.5 * (y.y - ym.y));
    return make_double2(0.5 * (y.y + ym.y), -0.5 * (y.x - ym.x));
}

// Half-length real step of one column pair (n, M-n).
// c2r: Z[n] = E + i w D, Z[M-n] = conj(E) + i conj(w D), with
// E = X[n] + conj X[M-n], D = X[n] - conj X[M-n], w = e^{+i pi n/M}.
__device__ __forceinline__ void c2r_pre_pair(double2 &a, double2 &b, double2 w) {
    const double2 e = make_double2(a.x + b.x, a.y - b.y), d = make_double2(a.x - b.x, a.y + b.y), od = cmul(d, w);
    a = make_double2(e.x - od.y, e.y + od.x);
    b = make_double2(e.x + od.y, od.x - e.y);
}
// r2c: X[n] = e + w o, X[M-n] = conj(e - w o), with e = (Z[n] + conj Z[M-n])/2,
// o = (Z[n] - conj Z[M-n])/(2i), w = e^{-i pi n/M}.
__device__ __forceinline__ void r2c_post_pair(double2 &a, double2 &b, double2 w) {
    const double2 e = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y)), o = make_double2(0.5 * (a.y + b.y), -0.5 * (a.x - b.x));
    const double2 t = cmul(w, o);
    a = make_double2(e.x + t.x, e.y + t.y);
    b = make_double2(e.x - t.x, t.y - e.y);
}
// e^{S 2 pi i m/N} from the table tw of e^{-2 pi i m/N}, 0 <= m < N.
template <int S> __device__ __forceinline__ double2 tw_get(const double2 *tw, int m) {
    const double2 v = tw[m];
    return S > 0 ? make_double2(v.x, -v.y) : v;
}

// ---- y passes over NR rows at pitch M+1 held by T threads ----
// c2r: rows of spectral values (natural column order; ky = 0 and M both in
// slot 0 when kPacked, else in slots 0 and M, of which the real parts count)
// -> rows of real pairs, pair m = k1 + AY*k2 in slot BY*k1 + k2.
template <int N, int NR, int T, bool kPacked>
__device__ __forceinline__ void rows_c2r(double2 *buf, const double2 *tw) {
    constexpr int AY = Plan<N>::AY, BY = Plan<N>::BY, H = BY / 2, M = N / 2, P = M + 1;
    const int tid = threadIdx.x;
    // real reconstruction and y over AY (slot BY*n1 + n2), twiddle w_M^{n2 k1}
#pragma unroll
    for (int u0 = 0; u0 < NR * H; u0 += T) {
        const int u = u0 + tid;
        if (NR * H % T == 0 || u < NR * H) {
            const int g = u / NR, ca = g, cb = g == 0 ? H : BY - g;
            double2 *row = buf + (u % NR) * P;
            double2 a[AY], b[AY];
#pragma unroll
            for (int n = 0; n < AY; ++n) { a[n] = row[ca + BY * n]; b[n] = row[cb + BY * n]; }
            if (g == 0) {   // classes 0 (with ky = 0, M and M/2) and BY/2 mirror onto themselves
                const double xm = kPacked ? a[0].y : row[M].x;
                a[0] = make_double2(a[0].x + xm, a[0].x - xm);
#pragma unroll
                for (int n = 1; n < AY / 2; ++n) c2r_pre_pair(a[n], a[AY - n], tw_get<1>(tw, BY * n));
                a[AY / 2] = make_double2(2.0 * a[AY / 2].x, -2.0 * a[AY / 2].y);
#pragma unroll
                for (int n = 0; n < AY / 2; ++n) c2r_pre_pair(b[n], b[AY - 1 - n], tw_get<1>(tw, H + BY * n));
            } else {
#pragma unroll
                for (int n = 0; n < AY; ++n) c2r_pre_pair(a[n], b[AY - 1 - n], tw_get<1>(tw, g + BY * n));
            }
            Dft<AY, 1>::run(a);
            row[ca] = a[0];
#pragma unroll
            for (int k1 = 1; k1 < AY; ++k1) row[ca + BY * k1] = cmul(a[k1], tw_get<1>(tw, 2 * ca * k1));
            Dft<AY, 1>::run(b);
            row[cb] = b[0];
#pragma unroll
            for (int k1 = 1; k1 < AY; ++k1) row[cb + BY * k1] = cmul(b[k1], tw_get<1>(tw, 2 * cb * k1));
        }
    }
    __syncthreads();
    // y over BY
#pragma unroll
    for (int u0 = 0; u0 < NR * AY; u0 += T) {
        const int u = u0 + tid;
        if (NR * AY % T == 0 || u < NR * AY) {
            double2 *base = buf + (u % NR) * P + BY * (u / NR);
            double2 v[BY];
#pragma unroll
            for (int n2 = 0; n2 < BY; ++n2) v[n2] = base[n2];
            Dft<BY, 1>::run(v);
#pragma unroll
            for (int k2 = 0; k2 < BY; ++k2) base[k2] = v[k2];
        }
    }
    __syncthreads();
}
// r2c, first pass: y over BY (slot BY*n1 + n2 holds the pair n1 + AY*n2),
// twiddle w_M^{n1 k2}.
template <int N, int NR, int T>
__device__ __forceinline__ void rows_r2c_1(double2 *buf, const double2 *tw) {
    constexpr int AY = Plan<N>::AY, BY = Plan<N>::BY, P = N / 2 + 1;
#pragma unroll
    for (int u0 = 0; u0 < NR * AY; u0 += T) {
        const int u = u0 + (int)threadIdx.x;
        if (NR * AY % T == 0 || u < NR * AY) {
            const int n1 = u / NR;
            double2 *base = buf + (u % NR) * P + BY * n1;
            double2 v[BY];
#pragma unroll
            for (int n2 = 0; n2 < BY; ++n2) v[n2] = base[n2];
            Dft<BY, -1>::run(v);
            base[0] = v[0];
#pragma unroll
            for (int k2 = 1; k2 < BY; ++k2) base[k2] = cmul(v[k2], tw_get<-1>(tw, 2 * n1 * k2));
        }
    }
    __syncthreads();
}
// Unit u of the second pass, y over AY (column BY*k1 + k2) and the real split:
// columns ca + BY*k (a) and cb + BY*k (b) of row u % NR; a[0] = X[0] + i X[M].
template <int N, int NR>
__device__ __forceinline__ void row_unit_r2c(const double2 *buf, const double2 *tw, int u, double2 (&a)[Plan<N>::AY],
                                             double2 (&b)[Plan<N>::AY]) {
    constexpr int AY = Plan<N>::AY, BY = Plan<N>::BY, H = BY / 2, P = N / 2 + 1;
    const int g = u / NR, ca = g, cb = g == 0 ? H : BY - g;
    const double2 *row = buf + (u % NR) * P;
#pragma unroll
    for (int n = 0; n < AY; ++n) { a[n] = row[ca + BY * n]; b[n] = row[cb + BY * n]; }
    Dft<AY, -1>::run(a);
    Dft<AY, -1>::run(b);
    if (g == 0) {   // ky = 0 and M, both real, stay packed as ky = 0 + i ky = M
        a[0] = make_double2(a[0].x + a[0].y, a[0].x - a[0].y);
#pragma unroll
        for (int n = 1; n < AY / 2; ++n) r2c_post_pair(a[n], a[AY - n], tw_get<-1>(tw, BY * n));
        a[AY / 2].y = -a[AY / 2].y;
#pragma unroll
        for (int n = 0; n < AY / 2; ++n) r2c_post_pair(b[n], b[AY - 1 - n], tw_get<-1>(tw, H + BY * n));
    } else {
#pragma unroll
        for (int n = 0; n < AY; ++n) r2c_post_pair(a[n], b[AY - 1 - n], tw_get<-1>(tw, g + BY * n));
    }
}
// r2c, second pass in place; ky = 0 and M packed in slot 0, or in slots 0 and M.
template <int N, int NR, int T, bool kPacked>
__device__ __forceinline__ void rows_r2c_2(double2 *buf, const double2 *tw) {
    constexpr int AY = Plan<N>::AY, BY = Plan<N>::BY, H = BY / 2, TOT = NR * H, M = N / 2, P = M + 1;
#pragma unroll
    for (int u0 = 0; u0 < TOT; u0 += T) {
        const int u = u0 + (int)threadIdx.x;
        if (TOT % T == 0 || u < TOT) {
            double2 a[AY], b[AY];
            row_unit_r2c<N, NR>(buf, tw, u, a, b);
            const int g = u / NR, ca = g, cb = g == 0 ? H : BY - g;
            double2 *row = buf + (u % NR) * P;
            if (!kPacked && g == 0) { row[M] = make_double2(a[0].y, 0.0); a[0].y = 0.0; }
#pragma unroll
            for (int n = 0; n < AY; ++n) { row[ca + BY * n] = a[n]; row[cb + BY * n] = b[n]; }
        }
    }
    __syncthreads();
}

// c2r of the CTA's columns (natural kz, column-phase layout; CTA 0 with
// ky = M in slot MC).  Call after a __syncthreads.  On return the CTA holds
// rows [rank*NR, (rank+1)*NR) of the real plane image: real value (z, y) of
// such a row R = zrow(z) is ((double*)buf)[(R - rank*NR)*(N+2) + 2*yslot(y/2) + (y&1)].
template <class L>
__device__ __forceinline__ void cl_c2r(double2 *buf, const double2 *tw, int rank) {
    using PN = Plan<L::N>;
    constexpr int T = L::T, AZ = PN::AZ, BZ = PN::BZ;
    constexpr int MC = L::MC, PZ = L::PZ, NR = L::NR, P = L::P;
    const int tid = threadIdx.x;
    cl_pack_col0<L>(buf, rank);
    // z over AZ (kz = BZ*n1 + n2), twiddle w_N^{n2 k1}
#pragma unroll
    for (int u0 = 0; u0 < MC * BZ; u0 += T) {
        const int u = u0 + tid;
        if (MC * BZ % T == 0 || u < MC * BZ) {
            const int q = u % MC, n2 = u / MC;
            double2 *base = buf + n2 * PZ + q;
            double2 v[AZ];
#pragma unroll
            for (int n1 = 0; n1 < AZ; ++n1) v[n1] = base[BZ * n1 * PZ];
            Dft<AZ, 1>::run(v);
            base[0] = v[0];
#pragma unroll
            for (int k1 = 1; k1 < AZ; ++k1) base[BZ * k1 * PZ] = cmul(v[k1], tw_get<1>(tw, n2 * k1));
        }
    }
    __syncthreads();
    // z over BZ: row BZ*k1 + k2 holds z = k1 + AZ*k2
    constexpr int TOT = MC * AZ, K2 = (TOT + T - 1) / T;
    auto z2_load = [&](int u, double2 (&v)[BZ]) {
        const double2 *base = buf + BZ * (u / MC) * PZ + u % MC;
#pragma unroll
        for (int n2 = 0; n2 < BZ; ++n2) v[n2] = base[n2 * PZ];
        Dft<BZ, 1>::run(v);
    };
    if constexpr (L::C == 1) {
#pragma unroll
        for (int u0 = 0; u0 < TOT; u0 += T) {
            const int u = u0 + tid;
            if (TOT % T == 0 || u < TOT) {
                double2 v[BZ];
                z2_load(u, v);
                double2 *base = buf + BZ * (u / MC) * PZ + u % MC;
#pragma unroll
                for (int k2 = 0; k2 < BZ; ++k2) base[k2 * PZ] = v[k2];
            }
        }
        __syncthreads();
    } else {
        double2 v[K2][BZ];
#pragma unroll
        for (int k = 0; k < K2; ++k)
            if (TOT % T == 0 || tid + k * T < TOT) z2_load(tid + k * T, v[k]);
        cl_sync<L>();   // every CTA of the plane has read its columns: buffers may be rewritten
#pragma unroll
        for (int k = 0; k < K2; ++k) {
            const int u = tid + k * T;
            if (TOT % T == 0 || u < TOT) {
                const int q = u % MC, k1 = u / MC;
#pragma unroll
                for (int k2 = 0; k2 < BZ; ++k2) {
                    const int R = BZ * k1 + k2;
                    cl_st(cl_addr(buf, (R % NR) * P + rank * MC + q, R / NR), v[k][k2]);
                }
            }
        }
        cl_sync<L>();   // every row of the plane is in place
    }
    rows_c2r<L::N, NR, T, true>(buf, tw);
}

// The passes of cl_r2c before the last one (z over AZ).
template <class L>
__device__ __forceinline__ void cl_r2c_head(double2 *buf, const double2 *tw, int rank) {
    using PN = Plan<L::N>;
    constexpr int T = L::T, AZ = PN::AZ, BZ = PN::BZ, AY = PN::AY, BY = PN::BY;
    constexpr int MC = L::MC, PZ = L::PZ, NR = L::NR;
    const int tid = threadIdx.x;
    rows_r2c_1<L::N, NR, T>(buf, tw);
    if constexpr (L::C == 1) {
        rows_r2c_2<L::N, NR, T, true>(buf, tw);
    } else {
        constexpr int H = BY / 2, TOT = NR * H, K2 = (TOT + T - 1) / T;
        double2 a[K2][AY], b[K2][AY];
#pragma unroll
        for (int k = 0; k < K2; ++k)
            if (TOT % T == 0 || tid + k * T < TOT) row_unit_r2c<L::N, NR>(buf, tw, tid + k * T, a[k], b[k]);
        cl_sync<L>();   // every CTA of the plane has read its rows: buffers may be rewritten
#pragma unroll
        for (int k = 0; k < K2; ++k) {
            const int u = tid + k * T;
            if (TOT % T == 0 || u < TOT) {
                const int g = u / NR, ca = g, cb = g == 0 ? H : BY - g, R = (rank * NR + u % NR) * PZ;
#pragma unroll
                for (int n = 0; n < AY; ++n) {
                    const int ja = ca + BY * n, jb = cb + BY * n;
                    cl_st(cl_addr(buf, R + ja % MC, ja / MC), a[k][n]);
                    cl_st(cl_addr(buf, R + jb % MC, jb / MC), b[k][n]);
                }
            }
        }
        cl_sync<L>();   // every column of the plane is in place
    }
    // z over BZ (row BZ*n1 + n2 holds z = n1 + AZ*n2), twiddle w_N^{n1 k2}
#pragma unroll
    for (int u0 = 0; u0 < MC * AZ; u0 += T) {
        const int u = u0 + tid;
        if (MC * AZ % T == 0 || u < MC * AZ) {
            const int n1 = u / MC;
            double2 *base = buf + BZ * n1 * PZ + u % MC;
            double2 v[BZ];
#pragma unroll
            for (int n2 = 0; n2 < BZ; ++n2) v[n2] = base[n2 * PZ];
            Dft<BZ, -1>::run(v);
            base[0] = v[0];
#pragma unroll
            for (int k2 = 1; k2 < BZ; ++k2) base[k2 * PZ] = cmul(v[k2], tw_get<-1>(tw, n1 * k2));
        }
    }
    __syncthreads();
}

// r2c of the CTA's real rows (row-phase layout, as cl_c2r leaves them).  Call
// after a __syncthreads.  On return the CTA holds its columns, natural in kz,
// unscaled; read them with cl_unpack.
template <class L>
__device__ __forceinline__ void cl_r2c(double2 *buf, const double2 *tw, int rank) {
    constexpr int T = L::T, AZ = Plan<L::N>::AZ, BZ = Plan<L::N>::BZ, MC = L::MC, PZ = L::PZ;
    cl_r2c_head<L>(buf, tw, rank);
#pragma unroll
    for (int u0 = 0; u0 < MC * BZ; u0 += T) {
        const int u = u0 + (int)threadIdx.x;
        if (MC * BZ % T == 0 || u < MC * BZ) {
            double2 *base = buf + (u / MC) * PZ + u % MC;
            double2 v[AZ];
#pragma unroll
            for (int n1 = 0; n1 < AZ; ++n1) v[n1] = base[BZ * n1 * PZ];
            Dft<AZ, -1>::run(v);
#pragma unroll
            for (int k1 = 0; k1 < AZ; ++k1) base[BZ * k1 * PZ] = v[k1];
        }
    }
    __syncthreads();
}
// cl_r2c whose last pass hands the spectral values of the CTA's columns from
// registers to out(kz, step, jl, X, n): column slot jl, X[k] at kz + step*k,
// k < n (n an integral_constant).  Each element comes exactly once and to the
// same thread in every call; rank 0's columns 0 and M go through shared
// memory (packed).  The buffer may be rewritten after a barrier.
template <class L, class F>
__device__ __forceinline__ void cl_r2c_out(double2 *buf, const double2 *tw, int rank, F out) {
    constexpr int T = L::T, AZ = Plan<L::N>::AZ, BZ = Plan<L::N>::BZ, MC = L::MC, PZ = L::PZ, N = L::N;
    cl_r2c_head<L>(buf, tw, rank);
#pragma unroll
    for (int u0 = 0; u0 < MC * BZ; u0 += T) {
        const int u = u0 + (int)threadIdx.x;
        if (MC * BZ % T == 0 || u < MC * BZ) {
            const int q = u % MC, k2 = u / MC;
            double2 *base = buf + k2 * PZ + q;
            double2 v[AZ];
#pragma unroll
            for (int n1 = 0; n1 < AZ; ++n1) v[n1] = base[BZ * n1 * PZ];
            Dft<AZ, -1>::run(v);
            if (q == 0 && rank == 0) {
#pragma unroll
                for (int k1 = 0; k1 < AZ; ++k1) base[BZ * k1 * PZ] = v[k1];
            } else {
                out(k2, BZ, q, v, std::integral_constant<int, AZ>());
            }
        }
    }
    __syncthreads();
    if (rank == 0)
        for (int kz = threadIdx.x; kz < N; kz += T) {
            const double2 x0 = cl_unpack<L>(buf, kz, 0, 0), xm = cl_unpack<L>(buf, kz, MC, 0);
            out(kz, 0, 0, &x0, std::integral_constant<int, 1>());
            out(kz, 0, MC, &xm, std::integral_constant<int, 1>());
        }
}
// dst[n0 + stride*k] = f(k, dst[n0 + stride*k]) over a column piece, k < n: the
// values are read four at a time before the first is written (a read behind
// a write of the same array starts its trip to L2 only after it).
template <class I, class F>
__device__ __forceinline__ void update_piece(double2 *dst, int n0, int stride, I n, F f) {
    constexpr int B = I::value < 4 ? I::value : 4;
#pragma unroll
    for (int k0 = 0; k0 < I::value; k0 += B) {
        double2 d[B];
#pragma unroll
        for (int k = 0; k < B; ++k) d[k] = dst[n0 + stride * (k0 + k)];
#pragma unroll
        for (int k = 0; k < B; ++k) dst[n0 + stride * (k0 + k)] = f(k0 + k, d[k]);
    }
}

}  // namespace pibm
