// fft2d.cuh -- FP64 2-D plane transforms for one y-z plane held in shared
// memory, with the conventions of the reference's ff2rc / ff2cr
// (SRC/FLO/fftw_interface.F90:48-133):
//   r2c: real (my,mz) -> complex (my2,mz), y halved, e^{-i}, scaled 1/float(my*mz)
//   c2r: complex (my2,mz) -> real (my,mz), e^{+i}, unscaled; after the z pass
//        the imaginary parts of the ky=0 and ky=my/2 columns are ignored
//        (the real-to-complex reconstruction below forces them to zero).
//
// Layout: the plane is rows of an odd number of complex slots (pitch*16 B is
// 4 banks mod 32, so accesses that walk across rows or columns are
// conflict-free).  A real row of my values occupies the first my/2 slots as
// pairs (x[2m], x[2m+1]).
//
// 1-D transforms of length A*B are two in-place passes (four-step): c2r takes
// natural input and leaves X[k1 + A*k2] in slot B*k1+k2, r2c takes that order
// and leaves a natural one.  A thread owns whole A- or B-point sub-transforms
// in registers; the digit permutation perm(m) = B*(m % A) + m / A is absorbed
// into the loads and stores of the calling kernels, so no pass needs a second
// buffer.
#pragma once
#include <cuda_runtime.h>
#include "fft_plane.cuh"

namespace pibm {

template <int A, int B> __device__ __host__ __forceinline__ int perm_ab(int m) { return B * (m % A) + m / A; }

// ---------------------------------------------------------------------------
// In-register DFTs of R points (e^{S 2 pi i}), natural order in and out, with
// the twiddles of the composite radices as immediates: a table read costs two
// shared-memory cycles per warp even when every lane reads the same entry.
// ---------------------------------------------------------------------------
// cos(2 pi m/48): every twiddle of the radices up to 16 and 12.
__host__ __device__ constexpr double cos48(int m) {
    m %= 48;
    if (m < 0) m += 48;
    if (m > 24) m = 48 - m;
    const bool neg = m > 12;
    if (neg) m = 24 - m;
    const double v = m == 0 ? 1.0 : m == 1 ? 0.9914448613738104111445575 : m == 2 ? 0.9659258262890682867497432
                   : m == 3 ? 0.9238795325112867561281832 : m == 4 ? 0.8660254037844386467637232
                   : m == 5 ? 0.7933533402912351645797770 : m == 6 ? 0.7071067811865475244008444
                   : m == 7 ? 0.6087614290087206394160975 : m == 8 ? 0.5 : m == 9 ? 0.3826834323650897717284600
                   : m == 10 ? 0.2588190451025207623488988 : m == 11 ? 0.1305261922200515915484062 : 0.0;
    return neg ? -v : v;
}
// v e^{S 2 pi i m/R}
template <int R, int m, int S> __device__ __forceinline__ double2 cmul_root(double2 v) {
    static_assert(48 % R == 0, "radix");
    constexpr int k = (m * (48 / R)) % 48;
    if constexpr (k == 0) return v;
    else if constexpr (k == 12) return make_double2(-S * v.y, S * v.x);
    else if constexpr (k == 24) return make_double2(-v.x, -v.y);
    else if constexpr (k == 36) return make_double2(S * v.y, -S * v.x);
    else if constexpr (k == 6) return make_double2(cos48(6) * (v.x - S * v.y), cos48(6) * (v.y + S * v.x));
    else if constexpr (k == 18) return make_double2(-cos48(6) * (v.x + S * v.y), cos48(6) * (S * v.x - v.y));
    else return cmul(v, make_double2(cos48(k), S * cos48(k - 12)));
}
template <int R, int S> struct Dft;
template <int S> struct Dft<2, S> {
    __device__ __forceinline__ static void run(double2 *v) {
        const double2 a = v[0], b = v[1];
        v[0] = cadd(a, b); v[1] = csub(a, b);
    }
};
template <int S> struct Dft<3, S> {
    __device__ __forceinline__ static void run(double2 *v) {
        constexpr double h = S * cos48(4);   // S sin(2 pi/3)
        const double2 a0 = v[0], t1 = cadd(v[1], v[2]), t2 = csub(v[1], v[2]);
        const double2 c = make_double2(a0.x - 0.5 * t1.x, a0.y - 0.5 * t1.y);
        v[0] = cadd(a0, t1);
        v[1] = make_double2(c.x - h * t2.y, c.y + h * t2.x);
        v[2] = make_double2(c.x + h * t2.y, c.y - h * t2.x);
    }
};
template <int S> struct Dft<4, S> {
    __device__ __forceinline__ static void run(double2 *v) {
        const double2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]), t2 = cadd(v[1], v[3]), t3 = csub(v[1], v[3]);
        v[0] = cadd(t0, t2); v[2] = csub(t0, t2);
        v[1] = make_double2(t1.x - S * t3.y, t1.y + S * t3.x);
        v[3] = make_double2(t1.x + S * t3.y, t1.y - S * t3.x);
    }
};
// composite R = P*Q by the four-step in registers
template <int P, int Q, int S> struct DftComp {
    template <int n2, int k1> __device__ __forceinline__ static void twiddle(const double2 *a, double2 *t) {
        if constexpr (k1 < P) { t[Q * k1 + n2] = cmul_root<P * Q, n2 * k1, S>(a[k1]); twiddle<n2, k1 + 1>(a, t); }
    }
    template <int n2> __device__ __forceinline__ static void columns(const double2 *v, double2 *t) {
        if constexpr (n2 < Q) {
            double2 a[P];
#pragma unroll
            for (int n1 = 0; n1 < P; ++n1) a[n1] = v[Q * n1 + n2];
            Dft<P, S>::run(a);
            twiddle<n2, 0>(a, t);
            columns<n2 + 1>(v, t);
        }
    }
    __device__ __forceinline__ static void run(double2 *v) {
        double2 t[P * Q];
        columns<0>(v, t);
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) {
            Dft<Q, S>::run(t + Q * k1);
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) v[k1 + P * k2] = t[Q * k1 + k2];
        }
    }
};
template <int S> struct Dft<8, S> : DftComp<4, 2, S> {};
template <int S> struct Dft<12, S> : DftComp<4, 3, S> {};
template <int S> struct Dft<16, S> : DftComp<4, 4, S> {};

// ---------------------------------------------------------------------------
// Per-size plans: z length N = AZ*BZ, y half length M = N/2 = AY*BY.  A thread
// of the AY pass holds two AY-point classes, so AY is the smaller factor; BY
// is even (its classes pair up).
// ---------------------------------------------------------------------------
template <int N> struct Plan;
template <> struct Plan<32>  { static constexpr int AZ = 4,  BZ = 8,  AY = 4, BY = 4; };
template <> struct Plan<64>  { static constexpr int AZ = 8,  BZ = 8,  AY = 4, BY = 8; };
template <> struct Plan<96>  { static constexpr int AZ = 12, BZ = 8,  AY = 4, BY = 12; };
template <> struct Plan<128> { static constexpr int AZ = 8,  BZ = 16, AY = 8, BY = 8; };
template <> struct Plan<256> { static constexpr int AZ = 16, BZ = 16, AY = 8, BY = 16; };

// smem row of physical z after an inverse z pass (the c2r's output order), and
// the slot of real pair index m in a row (c2r output, r2c input order).
template <int N> __device__ __forceinline__ int zrow(int z) { return perm_ab<Plan<N>::AZ, Plan<N>::BZ>(z); }
template <int N> __device__ __forceinline__ int yslot(int m) { return perm_ab<Plan<N>::AY, Plan<N>::BY>(m); }

// ---------------------------------------------------------------------------
// Packed ky = 0 / ky = M columns.  The two columns share one complex z
// transform held in column 0:
//  c2r: only Re of their inverse z transforms is used (the y reconstruction
//       drops the imaginary parts of ky = 0 and ky = M), and
//       Re(IFFT X) = IFFT(Herm X), Herm X[k] = (X[k] + conj X[-k])/2, so
//       column 0 <- Herm X0 + i Herm XM; the y reconstruction reads
//       Re -> ky = 0 and Im -> ky = M back from column 0.
//  r2c: both columns are real after the y pass, column 0 <- X0 + i XM; the
//       spectrum is read back with cl_unpack (A = (Y[k] + conj Y[-k])/2,
//       B = (Y[k] - conj Y[-k])/(2i)).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 herm_pack(double2 a, double2 am, double2 b, double2 bm) {
    const double2 h0 = make_double2(0.5 * (a.x + am.x), 0.5 * (a.y - am.y));
    const double2 hm = make_double2(0.5 * (b.x + bm.x), 0.5 * (b.y - bm.y));
    return make_double2(h0.x - hm.y, h0.y + hm.x);
}
// Offset of real node (z, y) inside one physical plane of the HBM real fields,
// which are stored exactly as the c2r plane transform leaves its rows in
// shared memory (rows of my+2 doubles), so plane loads and stores are bulk copies.
template <int N> __device__ __host__ __forceinline__ int real_off(int z, int y) {
    return (Plan<N>::BZ * (z % Plan<N>::AZ) + z / Plan<N>::AZ) * (N + 2) + 2 * (Plan<N>::BY * ((y >> 1) % Plan<N>::AY) + (y >> 1) / Plan<N>::AY) + (y & 1);
}

}  // namespace pibm
