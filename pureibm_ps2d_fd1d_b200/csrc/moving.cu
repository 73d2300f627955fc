// moving.cu -- moving particles (IMOVE = 1): the soft-sphere DEM of
// des_time_march (SRC/FLO/collision_mod.F90, soft_sphere_coll.F90) and the
// per-step rebuild of the immersed-boundary geometry that bcset does after it
// (grid_nodes_insphere, update_nrpr_array: dependent_functions.F90:783-1051).
//
// Compiled with --fmad=false: every expression is evaluated with the
// reference's operation order and no contraction, so positions, cell
// indices, contact and neighbour lists and the solid mask come out bit-equal
// to a serial evaluation of the same expressions.
//
// The reference keeps the contact lists with one sequential loop over the
// particles.  Here all sub-steps of a flow step run in one launch of one
// thread-block cluster (k_dem_march), up to kMarchMax particles; larger
// systems, which need the whole GPU, and larger ones with few sub-steps take
// three launches per sub-step:
//   k_dem_update  one thread per particle L: every pair (J, L) is evaluated by
//                 both its threads with the same arithmetic; L applies what the
//                 serial loop does to L's list at J's turn (J < L), then at
//                 its own turn (compaction, own pairs), forms FC(L) in the
//                 serial order (lower partners ascending, then its own pairs in
//                 NEIGHBOURS order) and advances L (CFNEWVALUES)
//   k_dem_bin     one CTA: particles per coarse cell, ascending
//   k_dem_search  one warp per particle: GRID_BASED_NEIGHBOR_SEARCH's list of L
//                 (entries appended by lower particles' searches, L itself,
//                 L's own finds in cell-scan order), then CFUPDATEOLD
// What makes this exact: within a sub-step the reference changes L's entries
// for a partner P > L only at L's own turn and its entries for P < L only at
// P's turn, so every decision reads lists as they were at the sub-step start.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "step_common.cuh"

namespace pibm {

namespace {

constexpr double kPiD = 3.14159265358979323846;
// Squared distances beyond this factor of a squared radius (below its inverse)
// are decided without the square root: far outside the roundings of either.
constexpr double kFar = 1.0 + 1e-9;

// One contact pair as CALC_FORCE_DES evaluates it at LL = A's turn, I = B
// (soft_sphere_coll.F90:300-420, CFRELVEL :728-776): periodic unwrap of B,
// overlap test, normal spring-dashpot force on A.  Reads the sub-step's
// starting positions and velocities.
__device__ __forceinline__ bool pair_force(const Mov &m, const double *pos, const double *vel, int A, int B, double fn[3], Scal *sc) {
    const double L3[3] = {m.XL, m.YL, m.ZL};
    double pB[3], dist[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double a = pos[3 * A + d], b = pos[3 * B + d];
        pB[d] = b;
        if (fabs(a - b) > 4.0 * m.max_radius) pB[d] = b > a ? b - L3[d] : b + L3[d];
        dist[d] = pB[d] - a;
    }
    double dd = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) dd = dd + dist[d] * dist[d];
    const double rlm = m.rad + m.rad;
    if (dd > rlm * rlm * kFar) return false;   // apart whatever the roundings of the test below
    const double distmod = sqrt(dd);
    if (!(rlm - distmod > kSmallD)) return false;
    if (distmod == 0.0) { atomicCAS(&sc->status, 0, PIBM_ERR_DEM_MOVE); return false; }
    double nrm[3], vrel[3], osum[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        nrm[d] = dist[d] / distmod;
        vrel[d] = vel[3 * A + d] - vel[3 * B + d];
        osum[d] = 0.0 * m.rad + 0.0 * m.rad;   // OMEGA stays zero (rotation update disabled)
    }
    const double vrot[3] = {osum[1] * nrm[2] - osum[2] * nrm[1], osum[2] * nrm[0] - osum[0] * nrm[2],
                            osum[0] * nrm[1] - osum[1] * nrm[0]};
    double vrn = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) { vrel[d] = vrel[d] + vrot[d]; vrn = vrn + vrel[d] * nrm[d]; }
    const double ov_n = rlm - distmod;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double fns1 = -(m.kn * ov_n) * nrm[d];
        const double fns2 = -(m.eta_n * vrn) * nrm[d];
        fn[d] = fns1 + fns2;
    }
    return true;
}

// Sub-step count of this flow step (des_time_march :272-279) and the reset of
// the geometry counters rebuilt after the DEM.
__global__ void k_dem_start(Mov m, Scal *sc) {
    if (threadIdx.x != 0) return;
    sc->count_solid = 0;
    if (sc->status) return;
    const double dt = sc->dt;
    int factor = 1;
    double dts = dt;
    if (m.soft) {
        factor = (int)(dt / m.dtsolid);
        dts = m.dtsolid;
        if (factor < 1) { factor = 1; dts = dt; }
    }
    if (factor > m.max_factor) { sc->status = PIBM_ERR_ARG; factor = 0; }
    m.factor[0] = factor;
    m.dts[0] = dts;
    sc->dem_substeps = factor;
}

// CALC_FORCE_DES + CFNEWVALUES for particle L (see the file comment), one warp
// per particle: the lanes evaluate L's pairs (every entry of NEIGHBOURS(L)
// other than L), lane 0 then applies them in the serial order.
constexpr int kUpdWarps = 4;
constexpr int kMaxList = 40;   // >= MAXNEIGHBORS
__global__ void __launch_bounds__(32 * kUpdWarps) k_dem_update(Mov m, Scal *sc, const double *__restrict__ pres,
                                                               const double *__restrict__ visc, int ifac) {
    if (ifac > m.factor[0] || sc->status) return;
    __shared__ double fn_s[kUpdWarps][kMaxList][3];
    __shared__ int cf_s[kUpdWarps][kMaxList], wl_s[kUpdWarps][kMaxList], wv_s[kUpdWarps][kMaxList];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int L = blockIdx.x * kUpdWarps + wid;
    if (L >= m.N) return;
    const int MX = m.maxn, nc = m.ncnt[L];
    // pair (J, L) for J < L as at J's turn (flag bit 0 contact, bit 1 "already
    // in J's contact list"), pair (L, I) for I > L as at L's turn
    for (int q = lane; q < nc; q += 32) {
        const int P = m.neigh[L * MX + q];
        int f = 0;
        double fn[3] = {0.0, 0.0, 0.0};
        if (P < L) {
            if (pair_force(m, m.pos_old, m.vel_old, P, L, fn, sc)) {
                f = 1;
                for (int p = 0; p < m.pncnt[P]; ++p)
                    if (m.pn[P * MX + p] == L) { if (m.pv[P * MX + p] == 1) f |= 2; break; }
            }
        } else if (P > L) {
            if (pair_force(m, m.pos_old, m.vel_old, L, P, fn, sc)) f = 1;
        }
        cf_s[wid][q] = f;
#pragma unroll
        for (int d = 0; d < 3; ++d) fn_s[wid][q][d] = fn[d];
    }
    __syncwarp();
    if (lane != 0) return;
    int *wl = wl_s[wid], *wv = wv_s[wid];
    int wc = m.pncnt[L];
    for (int q = 0; q < wc; ++q) { wl[q] = m.pn[L * MX + q]; wv[q] = m.pv[L * MX + q]; }
    double fc[3] = {0.0, 0.0, 0.0};
    bool over = false;
    // turns of the lower partners J (ascending: they precede L in NEIGHBOURS(L))
    for (int q = 0; q < nc; ++q) {
        const int J = m.neigh[L * MX + q];
        if (J >= L || !(cf_s[wid][q] & 1)) continue;
        if (cf_s[wid][q] & 2) {
            for (int p = 0; p < wc; ++p) if (wl[p] == J) { wv[p] = 1; break; }
        } else if (wc + 1 < MX) {
            wl[wc] = J; wv[wc] = 1; ++wc;
        } else {
            over = true;
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) fc[d] = fc[d] - fn_s[wid][q][d];
    }
    // L's turn: drop the entries whose contact ended, clear the flags, own pairs
    int w = 0;
    for (int p = 0; p < wc; ++p) if (wv[p]) { wl[w] = wl[p]; ++w; }
    wc = w;
    for (int p = 0; p < wc; ++p) wv[p] = 0;
    for (int q = 0; q < nc; ++q) {
        const int I = m.neigh[L * MX + q];
        if (I <= L || !(cf_s[wid][q] & 1)) continue;
        int found = -1;
        for (int p = 0; p < wc; ++p) if (wl[p] == I) { found = p; break; }
        if (found >= 0) {
            wv[found] = 1;
        } else if (wc + 1 < MX) {
            wl[wc] = I; wv[wc] = 1; ++wc;
        } else {
            over = true;
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) fc[d] = fc[d] + fn_s[wid][q][d];
    }
    if (over) atomicCAS(&sc->status, 0, PIBM_ERR_NEIGH_OVERFLOW);
    m.pncnt2[L] = wc;
    for (int p = 0; p < wc; ++p) { m.pn2[L * MX + p] = wl[p]; m.pv2[L * MX + p] = wv[p]; }
    // CFNEWVALUES (collision_mod.F90:1335-1462), softsphere coupled to the flow
    const double dts = m.dts[0];
    const int N = m.N;
    double pn[3], dd = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const size_t q = (size_t)L + (size_t)N * d;
        double a = fc[d] / m.pmass + (m.rhof * (pres[q] + visc[q])) / m.pmass;
        a = a - sc->frame_accln[d];
        a = a - (sc->mpg[d] * m.pvol) / m.pmass;
        const double v = m.vel_old[3 * L + d] + a * dts;
        m.vel[3 * L + d] = v;
        pn[d] = m.pos_old[3 * L + d] + v * dts;
        const double t = pn[d] - m.pos_old[3 * L + d];
        dd = dd + t * t;
    }
    if (sqrt(dd) >= m.rad) atomicCAS(&sc->status, 0, PIBM_ERR_DEM_MOVE);
    const double L3[3] = {m.XL, m.YL, m.ZL};
    const double dc[3] = {m.dxc, m.dyc, m.dzc};
    const int cmax[3] = {m.cx, m.cy, m.cz};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (pn[d] > L3[d]) pn[d] = pn[d] - (L3[d] - 0.0);
        else if (pn[d] < 0.0) pn[d] = pn[d] + (L3[d] - 0.0);
        m.pos[3 * L + d] = pn[d];
        m.pijk[3 * L + d] = min((int)(pn[d] / dc[d]) + 2, cmax[d]);   // FIND_CELL_INDEX (:743-762)
    }
}

// 'none' collision type (des_time_march :295-328): velocities kept, positions
// advanced over dt; the neighbour lists are not rebuilt.
__global__ void k_dem_none(Mov m, Scal *sc) {
    const int L = blockIdx.x * blockDim.x + threadIdx.x;
    if (L >= m.N || sc->status) return;
    const double dt = sc->dt;
    const double L3[3] = {m.XL, m.YL, m.ZL};
    double pn[3], dd = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double v = m.vel_old[3 * L + d];
        m.vel[3 * L + d] = v;
        pn[d] = m.pos_old[3 * L + d] + v * dt;
        const double t = pn[d] - m.pos_old[3 * L + d];
        dd = dd + t * t;
    }
    if (sqrt(dd) >= m.rad) atomicCAS(&sc->status, 0, PIBM_ERR_DEM_MOVE);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (pn[d] > L3[d]) pn[d] = pn[d] - (L3[d] - 0.0);
        else if (pn[d] < 0.0) pn[d] = pn[d] + (L3[d] - 0.0);
        m.pos[3 * L + d] = pn[d];
        m.pos_old[3 * L + d] = pn[d];
    }
}

__device__ __forceinline__ int cell_id(const Mov &m, int i, int j, int k) {
    return (i - 2) + (m.cx - 1) * ((j - 2) + (m.cy - 1) * (k - 2));
}

// PARTICLES_IN_CELL (collision_mod.F90:764-805): particles of every coarse
// cell in ascending order.  One CTA of 1024 threads; smem holds ncell counts,
// starts and fill counters and N particle slots.
__global__ void __launch_bounds__(1024) k_dem_bin(Mov m, Scal *sc, int ifac) {
    if (ifac > m.factor[0] || sc->status) return;
    extern __shared__ int sh[];
    int *cnt = sh, *start = sh + m.ncell, *fill = start + m.ncell + 1, *tmp = fill + m.ncell;
    __shared__ int wsum[32];
    const int T = blockDim.x, t = threadIdx.x, N = m.N, NC = m.ncell;
    for (int c = t; c < NC; c += T) { cnt[c] = 0; fill[c] = 0; }
    __syncthreads();
    for (int l = t; l < N; l += T) atomicAdd(&cnt[cell_id(m, m.pijk[3 * l], m.pijk[3 * l + 1], m.pijk[3 * l + 2])], 1);
    __syncthreads();
    // exclusive scan of cnt: each thread a contiguous chunk, then a block scan of the chunk sums
    const int per = (NC + T - 1) / T, c0 = min(t * per, NC), c1 = min(c0 + per, NC);
    int s = 0;
    for (int c = c0; c < c1; ++c) s += cnt[c];
    int x = s;
    const int lane = t & 31, wid = t >> 5;
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int v = lane < (T >> 5) ? wsum[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += y; }
        wsum[lane] = v;
    }
    __syncthreads();
    int run = x - s + (wid > 0 ? wsum[wid - 1] : 0);
    for (int c = c0; c < c1; ++c) { start[c] = run; run += cnt[c]; }
    if (t == 0) start[NC] = N;
    __syncthreads();
    for (int l = t; l < N; l += T) {
        const int c = cell_id(m, m.pijk[3 * l], m.pijk[3 * l + 1], m.pijk[3 * l + 2]);
        tmp[start[c] + atomicAdd(&fill[c], 1)] = l;
    }
    __syncthreads();
    for (int l = t; l < N; l += T) {
        const int c = cell_id(m, m.pijk[3 * l], m.pijk[3 * l + 1], m.pijk[3 * l + 2]);
        int rank = 0;
        for (int e = start[c]; e < start[c + 1]; ++e) rank += tmp[e] < l ? 1 : 0;
        m.clist[start[c] + rank] = l;
    }
    for (int c = t; c <= NC; c += T) m.cstart[c] = start[c];
}

// Neighbourhood cell `o` (0..26, the reference's kk/jj/ii scan order) of a
// particle in cell (ci, cj, ck): wrapped cell and periodic image factors
// (collision_mod.F90:866-945).
__device__ __forceinline__ int nb_cell(const Mov &m, int ci, int cj, int ck, int o, double sh[3]) {
    int ii = ci + (o % 3) - 1, jj = cj + (o / 3) % 3 - 1, kk = ck + o / 9 - 1;
    sh[0] = sh[1] = sh[2] = 0.0;
    if (ii > m.cx) { ii = 2; sh[0] = 1.0; }
    if (ii < 2) { ii = m.cx; sh[0] = -1.0; }
    if (jj > m.cy) { jj = 2; sh[1] = 1.0; }
    if (jj < 2) { jj = m.cy; sh[1] = -1.0; }
    if (kk > m.cz) { kk = 2; sh[2] = 1.0; }
    if (kk < 2) { kk = m.cz; sh[2] = -1.0; }
    return cell_id(m, ii, jj, kk);
}
// The search's distance test of PNO seen from LL through image sh.
__device__ __forceinline__ bool near_img(const Mov &m, int LL, int PNO, const double sh[3]) {
    const double rlm = 1.2 * (m.rad + m.rad);
    const double c0 = m.pos[3 * PNO + 0] + sh[0] * m.LXs;
    const double c1 = m.pos[3 * PNO + 1] + sh[1] * m.LYs;
    const double c2 = m.pos[3 * PNO + 2] + sh[2] * m.LZs;
    const double d0 = c0 - m.pos[3 * LL + 0], d1 = c1 - m.pos[3 * LL + 1], d2 = c2 - m.pos[3 * LL + 2];
    double dd = 0.0;
    dd = dd + d0 * d0;
    dd = dd + d1 * d1;
    dd = dd + d2 * d2;
    return rlm - sqrt(dd) > kSmallD;
}

// The image factor through which a search from cell cJ sees cell cL along one
// direction when the coarse grid has at least 3 cells there (then exactly one
// of the offsets -1, 0, +1 wraps onto cL).
__device__ __forceinline__ double img_dir(int cJ, int cL, int cmax) {
    if (cJ - 1 >= 2 && cJ - 1 == cL) return 0.0;
    if (cJ + 1 <= cmax && cJ + 1 == cL) return 0.0;
    if (cJ == cL) return 0.0;
    return cJ + 1 > cmax ? 1.0 : -1.0;   // the wrapped neighbour: across the upper or the lower boundary
}

// GRID_BASED_NEIGHBOR_SEARCH (collision_mod.F90:807-1062) for one particle per
// warp, then CFUPDATEOLD and the contact lists of the next sub-step.
//  - coarse grids with >= 3 cells per direction: the 27 neighbourhood cells
//    are distinct, so lane o < 27 scans cell o; finds are placed by a prefix
//    sum over the lanes, which keeps the reference's cell-scan order
//  - smaller grids (cells repeat through the periodic wrap): lane 0 follows
//    the serial loop, first accepted image of a particle only
constexpr int kSearchWarps = 4;
__global__ void __launch_bounds__(32 * kSearchWarps) k_dem_search(Mov m, Scal *sc, int ifac) {
    if (ifac > m.factor[0] || sc->status) return;
    __shared__ int own_s[kSearchWarps][64], mir_s[kSearchWarps][64];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int L = blockIdx.x * kSearchWarps + wid;
    if (L >= m.N) return;
    const int MX = m.maxn;
    int *own = own_s[wid], *mir = mir_s[wid];
    const int ci = m.pijk[3 * L], cj = m.pijk[3 * L + 1], ck = m.pijk[3 * L + 2];
    const int cL = cell_id(m, ci, cj, ck);
    int nown = 0, nmir = 0;
    const bool fast = m.cx >= 4 && m.cy >= 4 && m.cz >= 4;
    if (fast) {
        double sh[3] = {0.0, 0.0, 0.0};
        int c = 0, s0 = 0, s1 = 0;
        if (lane < 27) { c = nb_cell(m, ci, cj, ck, lane, sh); s0 = m.cstart[c]; s1 = m.cstart[c + 1]; }
        // own finds P > L of this lane's cell
        int cnt = 0;
        for (int e = s0; e < s1; ++e) { const int P = m.clist[e]; if (P > L && near_img(m, L, P, sh)) ++cnt; }
        int x = cnt;
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
        nown = __shfl_sync(0xffffffffu, x, 31);
        int pos = x - cnt;
        for (int e = s0; e < s1; ++e) {
            const int P = m.clist[e];
            if (P > L && near_img(m, L, P, sh)) { if (pos < 64) own[pos] = P; ++pos; }
        }
        // lower particles J whose search accepts L: J sees cell cL through one image
        cnt = 0;
        for (int e = s0; e < s1; ++e) {
            const int J = m.clist[e];
            if (J >= L) continue;
            const double shj[3] = {img_dir(m.pijk[3 * J], ci, m.cx), img_dir(m.pijk[3 * J + 1], cj, m.cy),
                                   img_dir(m.pijk[3 * J + 2], ck, m.cz)};
            if (near_img(m, J, L, shj)) ++cnt;
        }
        x = cnt;
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
        nmir = __shfl_sync(0xffffffffu, x, 31);
        pos = x - cnt;
        for (int e = s0; e < s1; ++e) {
            const int J = m.clist[e];
            if (J >= L) continue;
            const double shj[3] = {img_dir(m.pijk[3 * J], ci, m.cx), img_dir(m.pijk[3 * J + 1], cj, m.cy),
                                   img_dir(m.pijk[3 * J + 2], ck, m.cz)};
            if (near_img(m, J, L, shj)) { if (pos < 64) mir[pos] = J; ++pos; }
        }
        __syncwarp();
    } else if (lane == 0) {
        for (int o = 0; o < 27; ++o) {
            double sh[3];
            const int c = nb_cell(m, ci, cj, ck, o, sh);
            for (int e = m.cstart[c]; e < m.cstart[c + 1]; ++e) {
                const int P = m.clist[e];
                if (P <= L || !near_img(m, L, P, sh)) continue;
                bool already = false;
                for (int q = 0; q < nown && q < 64; ++q) if (own[q] == P) { already = true; break; }
                if (!already) { if (nown < 64) own[nown] = P; ++nown; }
            }
        }
        for (int o = 0; o < 27; ++o) {
            double sh[3];
            const int c = nb_cell(m, ci, cj, ck, o, sh);
            bool seen = false;
            for (int o2 = 0; o2 < o; ++o2) { double t[3]; if (nb_cell(m, ci, cj, ck, o2, t) == c) { seen = true; break; } }
            if (seen) continue;
            for (int e = m.cstart[c]; e < m.cstart[c + 1]; ++e) {
                const int J = m.clist[e];
                if (J >= L) continue;
                const int ji = m.pijk[3 * J], jj = m.pijk[3 * J + 1], jk = m.pijk[3 * J + 2];
                bool acc = false;
                for (int oj = 0; oj < 27 && !acc; ++oj) {
                    double shj[3];
                    if (nb_cell(m, ji, jj, jk, oj, shj) == cL && near_img(m, J, L, shj)) acc = true;
                }
                if (acc) { if (nmir < 64) mir[nmir] = J; ++nmir; }
            }
        }
    }
    if (!fast) {   // counts of the serial path are in lane 0
        nown = __shfl_sync(0xffffffffu, nown, 0);
        nmir = __shfl_sync(0xffffffffu, nmir, 0);
    }
    __syncwarp();
    const bool over = nmir > 64 || nown > 64 || nmir + 1 + nown + 1 > MX;
    if (lane == 0 && !over) {
        for (int a = 1; a < nmir; ++a) {   // ascending J
            const int v = mir[a];
            int b = a - 1;
            while (b >= 0 && mir[b] > v) { mir[b + 1] = mir[b]; --b; }
            mir[b + 1] = v;
        }
    }
    __syncwarp();
    if (over) {
        if (lane == 0) atomicCAS(&sc->status, 0, PIBM_ERR_NEIGH_OVERFLOW);
        return;
    }
    const int tot = nmir + 1 + nown;
    for (int q = lane; q < tot; q += 32)
        m.neigh[L * MX + q] = q < nmir ? mir[q] : (q == nmir ? L : own[q - nmir - 1]);
    if (lane == 0) m.ncnt[L] = tot;
    // CFUPDATEOLD and the contact lists written by this sub-step
    if (lane < 3) { m.pos_old[3 * L + lane] = m.pos[3 * L + lane]; m.vel_old[3 * L + lane] = m.vel[3 * L + lane]; }
    const int pc = m.pncnt2[L];
    for (int q = lane; q < pc; q += 32) { m.pn[L * MX + q] = m.pn2[L * MX + q]; m.pv[L * MX + q] = m.pv2[L * MX + q]; }
    if (lane == 0) m.pncnt[L] = pc;
}

// ============================================================================
// k_dem_march: every sub-step of one flow step (CALC_FORCE_DES, CFNEWVALUES,
// the neighbour search and CFUPDATEOLD, as k_dem_update / k_dem_bin /
// k_dem_search run them) in one launch: one cluster of up to 8 CTAs, a warp
// per particle (in turn when there are more), one cluster barrier per
// sub-step.  Every CTA keeps all positions, velocities and cells in shared
// memory, in two buffers that ping-pong: the warp that advances a particle
// stores them into each CTA's copy, and may search with the new positions and
// start its next update while others still search.  Neighbour lists stay in
// the shared memory of their particle's CTA; contact lists, which are mostly
// empty and read by a partner only in contact, ping-pong in global memory.
//
// The search needs no bins: a warp keeps the particles within the search
// radius plus a skin (kSkin radii) of its own as candidates, rebuilt from all
// pairs when any particle has moved half the skin since (a flow step moves
// them by a small fraction of a cell).  Each candidate is put through the
// reference's test for every one of the 27 neighbourhood cells that its cell
// matches, and the finds are ordered as the cell scan finds them, so the
// lists are those of the serial loop whatever the coarse grid.
//
// Bound: a chain of dependent shared-memory reads and FP64 arithmetic per
// particle, and the barrier: 1.9 us of update, 1.4 us of search and 1.7 us of
// barrier per sub-step with 43 particles on eight SMs, 4.9 us against 16.5 us
// for the three launches.
// ============================================================================
// Where one launch per flow step is the shorter one (dem_march).  Eight SMs take
// 41 us per sub-step with 1202 particles (their FP64 pipes are full), the three
// launches over the whole GPU 33; with 512 it is 23 against 33, and fewer gain
// more.  But the march forms all candidates once per flow step, which takes
// eight SMs longer than it takes the GPU, and from 256 particles on needs more
// sub-steps to share it.  Steps of a suspension at 64^3, d = 6, by launches / by
// the march: 512 particles 1.16 at 26 sub-steps, 1.07 at 11, 1.02 at 6, 0.97 at 4 and 1;
// 448: 1.05 at 7, 0.98 at 5; 384: 1.02 at 5, 0.98 at 3; 320: 1.02 at 4, 1.00 at 3, 0.96 at 1;
// 256: 1.14 at 5, 1.00 at 1; 128^3, d = 12, 400 particles: 1.04 at 13, 0.99 at 6.
constexpr int kMarchMax = 512, kMarchAny = 256, kMarchPerSubStep = 32;
constexpr int kMarchCtas = 8;      // portable cluster size
constexpr int kMaxCand = 48;
constexpr double kSkin = 0.4;      // in particle radii, on top of 2.4 (the search radius)
struct MarchWarp {
    double fn[kMaxList][3], fc[4];
    int wl[kMaxList], wv[kMaxList];
    unsigned short id[kMaxList], own[kMaxList], mir[kMaxList], key[kMaxList];
    unsigned char cf[kMaxList];
};
// Shared-memory layout of a CTA (the same in every CTA of the cluster).
struct MarchMem {
    double *P[2], *V[2], *pcand, *hyd;   // [3*l + d] of all particles; of the CTA's own: candidates' base, fluid force / mass
    int *cell[2], *flags, *pcs;          // packed cells of all; 3 rotating flag words and the sub-step count; contact counts held in either global buffer
    unsigned short *nb, *cand;
    unsigned char *nbc, *cdc;
    MarchWarp *w;
    __host__ __device__ static size_t bytes(int N, int slots, int maxn, int warps) {
        return (size_t)N * (12 * 8 + 8) + (size_t)slots * (6 * 8 + 8 + (maxn + kMaxCand) * 2 + 2) + 64 + warps * sizeof(MarchWarp);
    }
    __device__ MarchMem(unsigned char *base, int N, int slots, int maxn, int warps) {
        w = (MarchWarp *)base;
        double *d = (double *)(base + warps * sizeof(MarchWarp));
        for (int b = 0; b < 2; ++b) { P[b] = d; d += 3 * N; }
        for (int b = 0; b < 2; ++b) { V[b] = d; d += 3 * N; }
        pcand = d; d += 3 * slots;
        hyd = d; d += 3 * slots;
        int *q = (int *)d;
        for (int b = 0; b < 2; ++b) { cell[b] = q; q += N; }
        pcs = q; q += 2 * slots;
        flags = q; q += 4;
        nb = (unsigned short *)q;
        cand = nb + (size_t)slots * maxn;
        nbc = (unsigned char *)(cand + (size_t)slots * kMaxCand);
        cdc = nbc + slots;
    }
};
__device__ __forceinline__ int pack_cell(int i, int j, int k) { return i | (j << 10) | (k << 20); }
__device__ __forceinline__ int cell_dir(int c, int d) { return (c >> (10 * d)) & 1023; }
// Offset d in {-1, 0, 1} of one direction from cell c: whether it leads to
// `target`, and the image factor through which the search sees it (nb_cell).
__device__ __forceinline__ bool nb_dir(int c, int d, int cmax, int target, double &sh) {
    int ii = c + d;
    sh = 0.0;
    if (ii > cmax) { ii = 2; sh = 1.0; }
    if (ii < 2) { ii = cmax; sh = -1.0; }
    return ii == target;
}
// First of the 27 offsets, in the reference's scan order, through which the
// search from a particle at A (cell cA) accepts the particle at B (cell cB); 27 if none.
__device__ __forceinline__ int first_image(const Mov &m, const double *A, int cA, const double *B, int cB) {
    const double rlm = 1.2 * (m.rad + m.rad);
    for (int dz = -1; dz <= 1; ++dz) {
        double sz;
        if (!nb_dir(cell_dir(cA, 2), dz, m.cz, cell_dir(cB, 2), sz)) continue;
        for (int dy = -1; dy <= 1; ++dy) {
            double sy;
            if (!nb_dir(cell_dir(cA, 1), dy, m.cy, cell_dir(cB, 1), sy)) continue;
            for (int dx = -1; dx <= 1; ++dx) {
                double sx;
                if (!nb_dir(cell_dir(cA, 0), dx, m.cx, cell_dir(cB, 0), sx)) continue;
                const double c0 = B[0] + sx * m.LXs, c1 = B[1] + sy * m.LYs, c2 = B[2] + sz * m.LZs;
                const double d0 = c0 - A[0], d1 = c1 - A[1], d2 = c2 - A[2];
                double dd = 0.0;
                dd = dd + d0 * d0;
                dd = dd + d1 * d1;
                dd = dd + d2 * d2;
                if (dd > rlm * rlm * kFar) continue;
                if (dd * kFar < rlm * rlm || rlm - sqrt(dd) > kSmallD) return (dx + 1) + 3 * (dy + 1) + 9 * (dz + 1);
            }
        }
    }
    return 27;
}
// Squared distance between two points of the periodic box.
__device__ __forceinline__ double box_dist2(const Mov &m, const double *A, const double *B) {
    const double t0 = fabs(A[0] - B[0]), t1 = fabs(A[1] - B[1]), t2 = fabs(A[2] - B[2]);
    const double u0 = fmin(t0, fabs(m.XL - t0)), u1 = fmin(t1, fabs(m.YL - t1)), u2 = fmin(t2, fabs(m.ZL - t2));
    return u0 * u0 + u1 * u1 + u2 * u2;
}

__global__ void __launch_bounds__(1024, 1) k_dem_march(Mov m, Scal *sc, const double *__restrict__ pres,
                                                       const double *__restrict__ visc) {
    extern __shared__ __align__(16) unsigned char march_s[];
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int ctas = gridDim.x, rank = blockIdx.x;
    const int N = m.N, MX = m.maxn, slots = (N + ctas - 1) / ctas;   // particle L: CTA L % ctas, slot L / ctas
    MarchMem S(march_s, N, slots, MX, nw);
    MarchWarp &W = S.w[wid];
    const double dts = m.dts[0];
    const int d3 = lane % 3;               // this lane's direction in CFNEWVALUES
    const double fa = sc->frame_accln[d3], gm = (sc->mpg[d3] * m.pvol) / m.pmass;
    const double Ld = d3 == 0 ? m.XL : d3 == 1 ? m.YL : m.ZL, dcd = d3 == 0 ? m.dxc : d3 == 1 ? m.dyc : m.dzc;
    const double rdcd = 1.0 / dcd;
    const int cmd = d3 == 0 ? m.cx : d3 == 1 ? m.cy : m.cz;
    for (int q = threadIdx.x; q < 3 * N; q += blockDim.x) { S.P[0][q] = m.pos_old[q]; S.V[0][q] = m.vel_old[q]; }
    for (int k = wid; k < slots; k += nw) {
        const int L = k * ctas + rank;
        if (L >= N) continue;
        const int nc = m.ncnt[L];
        for (int q = lane; q < nc; q += 32) S.nb[k * MX + q] = (unsigned short)m.neigh[L * MX + q];
        if (lane < 3) {
            const size_t q = (size_t)L + (size_t)N * lane;
            S.hyd[3 * k + lane] = (m.rhof * (pres[q] + visc[q])) / m.pmass;
        }
        if (lane == 0) { S.nbc[k] = (unsigned char)nc; S.pcs[k] = m.pncnt[L]; S.pcs[slots + k] = -1; }
    }
    if (threadIdx.x < 3) S.flags[threadIdx.x] = 0;
    // The sub-steps to take, none after a failure: every thread must come to the
    // cluster's barriers equally often, so one thread reads the status for all
    // (a kernel beside this one may set it at any time).
    if (rank == 0 && threadIdx.x == 3) S.flags[3] = sc->status != 0 ? 0 : m.factor[0];
    cl.sync();
    const int F = cl.map_shared_rank(S.flags, 0)[3];
    auto raise = [&](int f, int word) {   // in every CTA's copy of the flag word
        for (int r = 0; r < ctas; ++r) atomicOr(cl.map_shared_rank(S.flags, r) + word, f);
    };
    int s = 0, c = 0;
    for (; s < F; ++s, c ^= 1) {
        double *const Pc = S.P[c], *const Vc = S.V[c], *const Pn = S.P[c ^ 1], *const Vn = S.V[c ^ 1];
        int *const Cn = S.cell[c ^ 1];
        int *const gl = c ? m.pn2 : m.pn, *const gv = c ? m.pv2 : m.pv, *const gc = c ? m.pncnt2 : m.pncnt;
        int *const gln = c ? m.pn : m.pn2, *const gvn = c ? m.pv : m.pv2, *const gcn = c ? m.pncnt : m.pncnt2;
        const int w3 = s % 3;
        // ---- forces on and advance of every particle (k_dem_update) ----
        for (int k = wid; k < slots; k += nw) {
            const int L = k * ctas + rank;
            if (L >= N) continue;
            const int nc = S.nbc[k];
            int wc = S.pcs[c * slots + k];
            for (int q = lane; q < wc; q += 32) { W.wl[q] = __ldcg(gl + L * MX + q); W.wv[q] = __ldcg(gv + L * MX + q); }
            bool touch = false;
            for (int q = lane; q < nc; q += 32) {
                const int P = S.nb[k * MX + q];
                int f = 0;
                double fn[3] = {0.0, 0.0, 0.0};
                if (P < L) {
                    if (pair_force(m, Pc, Vc, P, L, fn, sc)) {
                        f = 1;
                        const int np = __ldcg(gc + P);
                        for (int p = 0; p < np; ++p)
                            if (__ldcg(gl + P * MX + p) == L) { if (__ldcg(gv + P * MX + p) == 1) f |= 2; break; }
                    }
                } else if (P > L) {
                    if (pair_force(m, Pc, Vc, L, P, fn, sc)) f = 1;
                }
                W.id[q] = (unsigned short)P;
                W.cf[q] = (unsigned char)f;
                touch = touch || f;
#pragma unroll
                for (int d = 0; d < 3; ++d) W.fn[q][d] = fn[d];
            }
            touch = __any_sync(0xffffffffu, touch);
            __syncwarp();
            if (lane == 0) {
                int *wl = W.wl, *wv = W.wv;
                double fc[3] = {0.0, 0.0, 0.0};
                bool over = false;
                if (touch)
                    for (int q = 0; q < nc; ++q) {
                        const int J = W.id[q];
                        if (J >= L || !(W.cf[q] & 1)) continue;
                        if (W.cf[q] & 2) {
                            for (int p = 0; p < wc; ++p) if (wl[p] == J) { wv[p] = 1; break; }
                        } else if (wc + 1 < MX) {
                            wl[wc] = J; wv[wc] = 1; ++wc;
                        } else {
                            over = true;
                        }
#pragma unroll
                        for (int d = 0; d < 3; ++d) fc[d] = fc[d] - W.fn[q][d];
                    }
                int w = 0;
                for (int p = 0; p < wc; ++p) if (wv[p]) { wl[w] = wl[p]; ++w; }
                wc = w;
                for (int p = 0; p < wc; ++p) wv[p] = 0;
                if (touch)
                    for (int q = 0; q < nc; ++q) {
                        const int I = W.id[q];
                        if (I <= L || !(W.cf[q] & 1)) continue;
                        int found = -1;
                        for (int p = 0; p < wc; ++p) if (wl[p] == I) { found = p; break; }
                        if (found >= 0) {
                            wv[found] = 1;
                        } else if (wc + 1 < MX) {
                            wl[wc] = I; wv[wc] = 1; ++wc;
                        } else {
                            over = true;
                        }
#pragma unroll
                        for (int d = 0; d < 3; ++d) fc[d] = fc[d] + W.fn[q][d];
                    }
                if (over) { atomicCAS(&sc->status, 0, PIBM_ERR_NEIGH_OVERFLOW); raise(2, w3); }
#pragma unroll
                for (int d = 0; d < 3; ++d) W.fc[d] = fc[d];
            }
            wc = __shfl_sync(0xffffffffu, wc, 0);
            __syncwarp();
            if (wc > 0 || S.pcs[(c ^ 1) * slots + k] != 0) {   // else the global buffer holds the empty list already
                for (int q = lane; q < wc; q += 32) { gln[L * MX + q] = W.wl[q]; gvn[L * MX + q] = W.wv[q]; }
                if (lane == 0) gcn[L] = wc;
            }
            // CFNEWVALUES (collision_mod.F90:1335-1462), softsphere coupled to the flow: every lane its direction
            const double fcd = W.fc[d3];
            double a = (fcd == 0.0 ? fcd : fcd / m.pmass) + S.hyd[3 * k + d3];
            a = a - fa;
            a = a - gm;
            const double po = Pc[3 * L + d3];
            const double v = Vc[3 * L + d3] + a * dts;
            double pn = po + v * dts;
            const double t = pn - po;
            double dd = 0.0;
#pragma unroll
            for (int e = 0; e < 3; ++e) { const double te = __shfl_sync(0xffffffffu, t, e); dd = dd + te * te; }
            if (pn > Ld) pn = pn - (Ld - 0.0);
            else if (pn < 0.0) pn = pn + (Ld - 0.0);
            // FIND_CELL_INDEX (:743-762); the division only near a cell boundary
            const double cq = pn * rdcd;
            const int cn = (int)cq;
            const int ci = min((cq - (double)cn > 1e-9 && (double)cn + 1.0 - cq > 1e-9 ? cn : (int)(pn / dcd)) + 2, cmd);
            const int cell = pack_cell(__shfl_sync(0xffffffffu, ci, 0), __shfl_sync(0xffffffffu, ci, 1), __shfl_sync(0xffffffffu, ci, 2));
            double A[3];
#pragma unroll
            for (int e = 0; e < 3; ++e) A[e] = __shfl_sync(0xffffffffu, pn, e);
            if (lane < 3 * ctas) {   // lane 3 r + d: direction d into CTA r's copy
                const int r = lane / 3;
                cl.map_shared_rank(Pn, r)[3 * L + d3] = pn;
                cl.map_shared_rank(Vn, r)[3 * L + d3] = v;
                if (d3 == 0) cl.map_shared_rank(Cn, r)[L] = cell;
            }
            if (lane == 0) {
                S.pcs[(c ^ 1) * slots + k] = wc;
                int fl = 0;
                if (dd * kFar >= m.rad * m.rad && sqrt(dd) >= m.rad) { atomicCAS(&sc->status, 0, PIBM_ERR_DEM_MOVE); fl |= 2; }
                if (s > 0 && !(box_dist2(m, A, S.pcand + 3 * k) < (0.49 * kSkin * m.rad) * (0.49 * kSkin * m.rad))) fl |= 1;
                if (fl) raise(fl, w3);
            }
            __syncwarp();
        }
        cl.sync();
        const int flags = *(volatile int *)(S.flags + w3);   // complete: set before the barrier
        if (threadIdx.x == 0) S.flags[(s + 2) % 3] = 0;       // last read before this barrier, next set after the next one
        if (flags & 2) { ++s; c ^= 1; break; }
        // ---- GRID_BASED_NEIGHBOR_SEARCH at the new positions (k_dem_search) ----
        for (int k = wid; k < slots; k += nw) {
            const int L = k * ctas + rank;
            if (L >= N) continue;
            const double A[3] = {Pn[3 * L], Pn[3 * L + 1], Pn[3 * L + 2]};
            const int cA = Cn[L];
            int ncand = S.cdc[k];
            if (s == 0 || (flags & 1)) {
                ncand = 0;
                const double cut = (2.4 + kSkin) * m.rad;
                for (int b = 0; b < N; b += 32) {
                    const int P = b + lane;
                    const bool in = P < N && P != L && box_dist2(m, A, Pn + 3 * P) < cut * cut;
                    const unsigned bal = __ballot_sync(0xffffffffu, in);
                    const int at = ncand + __popc(bal & ((1u << lane) - 1u));
                    if (in && at < kMaxCand) S.cand[k * kMaxCand + at] = (unsigned short)P;
                    ncand += __popc(bal);
                }
                if (ncand > kMaxCand) ncand = 255;   // too many to keep: every particle is a candidate
                if (lane == 0) S.cdc[k] = (unsigned char)ncand;
                if (lane < 3) S.pcand[3 * k + lane] = Pn[3 * L + lane];
                __syncwarp();
            }
            const bool all = ncand == 255;
            const int n = all ? N : ncand;
            int nown = 0, nmir = 0;
            for (int b = 0; b < n; b += 32) {
                const int at = b + lane;
                int P = -1, o = 27;
                if (at < n) P = all ? at : S.cand[k * kMaxCand + at];
                if (P >= 0 && P != L)
                    o = P > L ? first_image(m, A, cA, Pn + 3 * P, Cn[P]) : first_image(m, Pn + 3 * P, Cn[P], A, cA);
                const unsigned bo = __ballot_sync(0xffffffffu, o < 27 && P > L), bm = __ballot_sync(0xffffffffu, o < 27 && P < L);
                const unsigned below = (1u << lane) - 1u;
                if (o < 27 && P > L) { const int q = nown + __popc(bo & below); if (q < kMaxList) { W.own[q] = (unsigned short)P; W.key[q] = (unsigned short)o; } }
                if (o < 27 && P < L) { const int q = nmir + __popc(bm & below); if (q < kMaxList) W.mir[q] = (unsigned short)P; }
                nown += __popc(bo);
                nmir += __popc(bm);
            }
            __syncwarp();
            if (nmir + 1 + nown + 1 > MX) {   // MX < kMaxList: the scratch lists were long enough
                if (lane == 0) { atomicCAS(&sc->status, 0, PIBM_ERR_NEIGH_OVERFLOW); raise(2, (s + 1) % 3); }
                continue;
            }
            for (int q = lane; q < nmir; q += 32) S.nb[k * MX + q] = W.mir[q];   // ascending
            for (int q = lane; q < nown; q += 32) {   // by scan offset, ascending within a cell
                const int o = W.key[q];
                int r = 0;
                for (int e = 0; e < nown; ++e) r += W.key[e] < o || (W.key[e] == o && e < q) ? 1 : 0;
                S.nb[k * MX + nmir + 1 + r] = W.own[q];
            }
            if (lane == 0) { S.nb[k * MX + nmir] = (unsigned short)L; S.nbc[k] = (unsigned char)(nmir + 1 + nown); }
            __syncwarp();
        }
    }
    // the last sub-step's state back to global memory, where the other kernels and the next step read it
    for (int k = wid; k < slots && s > 0; k += nw) {
        const int L = k * ctas + rank;
        if (L >= N) continue;
        if (lane < 3) {
            m.pos[3 * L + lane] = m.pos_old[3 * L + lane] = S.P[c][3 * L + lane];
            m.vel[3 * L + lane] = m.vel_old[3 * L + lane] = S.V[c][3 * L + lane];
            m.pijk[3 * L + lane] = cell_dir(S.cell[c][L], lane);
        }
        const int nc = S.nbc[k], pc = S.pcs[c * slots + k];
        for (int q = lane; q < nc; q += 32) m.neigh[L * MX + q] = S.nb[k * MX + q];
        if (c)
            for (int q = lane; q < pc; q += 32) { m.pn[L * MX + q] = __ldcg(m.pn2 + L * MX + q); m.pv[L * MX + q] = __ldcg(m.pv2 + L * MX + q); }
        if (lane == 0) { m.ncnt[L] = nc; m.pncnt[L] = pc; }
    }
    cl.sync();   // no CTA leaves while another may still store into its copy
}

// IBMUPDATE (collision_mod.F90:1464-1474): grid-unit centres and velocities.
__global__ void k_dem_ibm(Mov m, Scal *sc, double dx) {
    const int L = blockIdx.x * blockDim.x + threadIdx.x;
    if (L >= m.N || sc->status) return;
    const int N = m.N;
    m.xc[L] = m.pos[3 * L + 0] / dx + 1.0 - 0.0;
    m.xc[L + N] = m.pos[3 * L + 1] / dx + 1.0;
    m.xc[L + 2 * N] = m.pos[3 * L + 2] / dx + 1.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) m.vel_ibm[L + (size_t)N * d] = m.vel[3 * L + d];
}

// grid_nodes_insphere (dependent_functions.F90:783-963): one CTA per sphere
// clears the nodes of its bounding box that lie in the sphere (nodes covered
// by two spheres are counted twice, as in the reference).
template <int N>
__global__ void __launch_bounds__(256) k_mask(Geo g, Mov m, Scal *sc) {
    __shared__ double scr[32];
    if (block_failed(sc)) return;
    const int s = blockIdx.x, NB = g.nbody, nx = g.nx;
    const double cx = m.xc[s], cy = m.xc[s + NB], cz = m.xc[s + 2 * NB], r = g.rb;
    const int i0 = (int)ceil(cx - r), i1 = (int)floor(cx + r);
    const int j0 = (int)ceil(cy - r), j1 = (int)floor(cy + r);
    const int k0 = (int)ceil(cz - r), k1 = (int)floor(cz + r);
    const int ni = i1 - i0 + 1, nj = j1 - j0 + 1, nk = k1 - k0 + 1;
    double cnt = 0.0;
    for (int e = threadIdx.x; e < ni * nj * nk; e += blockDim.x) {
        const int k = k0 + e / (ni * nj), j = j0 + (e / ni) % nj, i = i0 + e % ni;
        const double a = (double)i - cx, b = (double)j - cy, c = (double)k - cz;
        double d2 = a * a;
        d2 = d2 + b * b + c * c;
        if (sqrt(d2) - r <= kSmallD) {
            const int ii = wrapi(i, nx), jj = wrapi(j, N), kk = wrapi(k, N);
            m.fluid[(size_t)(ii - 1) * RP<N>::RSP + real_off<N>(kk - 1, jj - 1)] = 0;
            cnt += 1.0;
        }
    }
    cnt = block_sum(cnt, scr);
    if (threadIdx.x == 0) atomicAdd((unsigned long long *)&sc->count_solid, (unsigned long long)cnt);
}

// update_nrpr_array + check_external_pt (dependent_functions.F90:966-1051):
// one CTA per sphere flags its reversal points whose outer point lies in a
// neighbour sphere, counts the active ones and sets da(2) of bcset.
__global__ void __launch_bounds__(256) k_nrpr(Geo g, Mov m, Scal *sc) {
    __shared__ double scr[32];
    if (block_failed(sc)) return;
    const int s = blockIdx.x, NB = g.nbody, nb = g.nbnd;
    const double px = (double)(g.nx + 1), py = (double)g.my, pz = (double)g.mz;
    const int nc = m.ncnt[s];
    double act = 0.0;
    for (int l = threadIdx.x; l < nb; l += blockDim.x) {
        double xo[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) xo[d] = m.xc[s + d * NB] + g.bnd[3 * l + d] * g.ro;
        if (xo[0] < 1.0) xo[0] = px + xo[0];
        if (xo[0] > px) xo[0] = xo[0] - px;
        if (xo[1] < 1.0) xo[1] = py + 1.0 + xo[1];
        if (xo[1] > py) xo[1] = xo[1] - py - 1.0;
        if (xo[2] < 1.0) xo[2] = pz + 1.0 + xo[2];
        if (xo[2] > pz) xo[2] = xo[2] - pz - 1.0;
        bool active = true;
        if (nc > 1) {
            for (int q = 0; q < nc; ++q) {
                const int P = m.neigh[s * m.maxn + q];
                double d2 = 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) { const double a = m.xc[P + d * NB] - xo[d]; d2 = d2 + a * a; }
                if (sqrt(d2) < g.rb) { active = false; break; }
            }
        }
        m.revflag[(size_t)s * nb + l] = active ? 1 : 0;
        act += active ? 1.0 : 0.0;
    }
    act = block_sum(act, scr);
    if (threadIdx.x == 0) {
        const int n = (int)act;
        m.nrpr[s] = n;
        m.da2[s] = 4.0 * kPiD * ((g.ri * g.dx) * (g.ri * g.dx)) / (double)n;
    }
}

// Offsets of every sphere's active points in the (sphere, point) list, the
// point count, and the solid/fluid counts of the new mask.
__global__ void __launch_bounds__(1024) k_pts_scan(Geo g, Mov m, Scal *sc) {
    __shared__ int wsum[32];
    if (block_failed(sc)) return;
    const int T = blockDim.x, t = threadIdx.x, NB = g.nbody;
    const int per = (NB + T - 1) / T, c0 = min(t * per, NB), c1 = min(c0 + per, NB);
    int s = 0;
    for (int c = c0; c < c1; ++c) s += m.nrpr[c];
    int x = s;
    const int lane = t & 31, wid = t >> 5;
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int v = lane < (T >> 5) ? wsum[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += y; }
        wsum[lane] = v;
    }
    __syncthreads();
    int run = x - s + (wid > 0 ? wsum[wid - 1] : 0);
    for (int c = c0; c < c1; ++c) { m.ptoff[c] = run; run += m.nrpr[c]; }
    if (t == T - 1) {
        sc->npts = run;
        sc->count_fluid = g.ncell - sc->count_solid;
        sc->maxvolfrac = (double)sc->count_solid / (double)g.ncell;
    }
}

// Active points of one sphere written in point order at its offset.
__global__ void __launch_bounds__(256) k_pts_write(Geo g, Mov m, Scal *sc) {
    __shared__ int wsum[8];
    __shared__ int base;
    if (block_failed(sc)) return;
    const int s = blockIdx.x, nb = g.nbnd, t = threadIdx.x, lane = t & 31, wid = t >> 5;
    if (t == 0) base = m.ptoff[s];
    __syncthreads();
    for (int l0 = 0; l0 < nb; l0 += blockDim.x) {
        const int l = l0 + t;
        const int f = l < nb ? m.revflag[(size_t)s * nb + l] : 0;
        const unsigned bal = __ballot_sync(0xffffffffu, f);
        if (lane == 0) wsum[wid] = __popc(bal);
        __syncthreads();
        int before = 0;
        for (int w = 0; w < wid; ++w) before += wsum[w];
        if (f) {
            const int p = base + before + __popc(bal & ((1u << lane) - 1u));
            m.pt_m[p] = s;
            m.pt_l[p] = l;
        }
        __syncthreads();
        if (t == 0) { int a = 0; for (int w = 0; w < (int)(blockDim.x >> 5); ++w) a += wsum[w]; base += a; }
        __syncthreads();
    }
}

// Spreading targets (boundary_condition.F90:1379-1462): every (point, corner)
// whose node receives force goes into that node's bucket.
template <int N>
__global__ void __launch_bounds__(256) k_sp_count(Geo g, Mov m, Scal *sc) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (sc->status || p >= sc->npts) return;
    const int s = m.pt_m[p], l = m.pt_l[p], NB = g.nbody;
    int base[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) base[d] = cell_of(m.xc[s + d * NB] + g.bnd[3 * l + d] * g.ri);
    for (int ck = 0; ck < 2; ++ck)
        for (int cj = 0; cj < 2; ++cj)
            for (int ci = 0; ci < 2; ++ci) {
                const int i = wrapi(base[0] + ci, g.nx), j = wrapi(base[1] + cj, N), k = wrapi(base[2] + ck, N);
                const size_t node = (size_t)(i - 1) * RP<N>::RSP + real_off<N>(k - 1, j - 1);
                if (!g.include_frmeanfluid && m.fluid[node]) continue;
                const int slot = atomicAdd(&m.spcnt[node], 1);
                if (slot < m.kmax) m.spbuf[node * m.kmax + slot] = p * 8 + ci + 2 * cj + 4 * ck;
                else atomicCAS(&sc->status, 0, PIBM_ERR_SPREAD_OVERFLOW);
            }
}

// A node's bucket in ascending entry order, the reference's accumulation
// order ((point, corner) or (evaluation, corner)): buckets of up to 8 entries
// (nearly all) through a 19-comparator sorting network in registers, longer
// ones by insertion sort.  f(entry) is called in that order.
template <class F>
__device__ __forceinline__ void bucket_in_order(const int *bucket, int c, F f) {
    if (c <= 8) {
        // whole 16-byte loads (a bucket holds kmax >= 8 slots at a 64-byte multiple)
        const int4 lo = *(const int4 *)bucket, hi = c > 4 ? *(const int4 *)(bucket + 4) : make_int4(0, 0, 0, 0);
        int v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = q < c ? v[q] : 0x7fffffff;
        auto ce = [&](int a, int b) { const int x = min(v[a], v[b]), y = max(v[a], v[b]); v[a] = x; v[b] = y; };
        ce(0, 1); ce(2, 3); ce(4, 5); ce(6, 7);
        ce(0, 2); ce(1, 3); ce(4, 6); ce(5, 7);
        ce(1, 2); ce(5, 6);
        ce(0, 4); ce(1, 5); ce(2, 6); ce(3, 7);
        ce(2, 4); ce(3, 5);
        ce(1, 2); ce(3, 4); ce(5, 6);
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (q < c) f(v[q]);
    } else {
        int e[64];
        const int cc = min(c, 64);
        for (int q = 0; q < cc; ++q) {
            const int x = bucket[q];
            int b = q - 1;
            while (b >= 0 && e[b] > x) { e[b + 1] = e[b]; --b; }
            e[b + 1] = x;
        }
        for (int q = 0; q < cc; ++q) f(e[q]);
    }
}

// The forced nodes of a block's window of kSpreadWin consecutive nodes, dense
// over its threads.  Forced nodes are a shell around each sphere, and the
// transform order deals neighbouring nodes to different warps, so one thread
// per node left a warp with a few forced lanes that the others waited for.
// none(node) is called for every node without entries, by consecutive threads;
// some(node, entries) for the others.  Nodes are independent: their order
// among the threads does not matter.
// 256^3, 1202 spheres: k_spread_dyn 1.49 -> 0.81 ms.
constexpr int kSpreadWin = 1024;
template <class F0, class F1>
__device__ __forceinline__ void for_forced_nodes(const int *cnt, size_t nodes, int kmax, F0 none, F1 some) {
    __shared__ unsigned short list[kSpreadWin], num[kSpreadWin];
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * kSpreadWin;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < kSpreadWin; k += 256) {
        const size_t node = base + k + threadIdx.x;
        const int c = node < nodes ? cnt[node] : 0;
        if (node < nodes && c == 0) none(node);
        const unsigned bal = __ballot_sync(0xffffffffu, c > 0);
        int at = 0;
        if (lane == 0 && bal) at = atomicAdd(&total, __popc(bal));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(bal & ((1u << lane) - 1u));
        if (c > 0) { list[at] = (unsigned short)(k + threadIdx.x); num[at] = (unsigned short)min(c, kmax); }
    }
    __syncthreads();
    for (int q = threadIdx.x; q < total; q += blockDim.x) some(base + list[q], (int)num[q]);
}

// fr at every node: the bucket's contributions in ascending (point, corner)
// order, the reference's accumulation order; nodes without force get zero.
__global__ void __launch_bounds__(256) k_spread_dyn(Geo g, Mov m, const double *__restrict__ rec,
                                                    const double *__restrict__ rz, double *__restrict__ fr, Scal *sc) {
    const size_t CR = (size_t)g.nx * g.RS;
    if (block_failed(sc)) return;
    const double rdx3 = 1.0 / g.dx3;
    for_forced_nodes(
        m.spcnt, CR, m.kmax,
        [&](size_t node) {
#pragma unroll
            for (int n = 0; n < 3; ++n) fr[n * CR + node] = 0.0;
        },
        [&](size_t node, int c) {
            double acc[3] = {0.0, 0.0, 0.0};
            bucket_in_order(m.spbuf + node * m.kmax, c, [&](int ent) {
                double t[3];
                corner_contrib(rz, rec, ent, g.dx3, rdx3, t);
                if (g.include_frmeanfluid) {
#pragma unroll
                    for (int n = 0; n < 3; ++n) acc[n] = acc[n] + t[n];
                } else {
                    const double *r = rec + (size_t)(ent >> 3) * 6 + 3;
#pragma unroll
                    for (int n = 0; n < 3; ++n) acc[n] = (acc[n] + t[n]) + r[n];
                }
            });
#pragma unroll
            for (int n = 0; n < 3; ++n) fr[n * CR + node] = acc[n];
        });
}

// ---------------------------------------------------------------------------
// Passive scalar with moving particles: the reversal-point evaluations of
// calc_inner_rev_data (SRC/SCALAR/bc_scalar.F90:558-932, serial branch) for
// the step's active points.  Inner point x = xc + bnd*radibdy, its cell
// wrapped into 1..nx (WEST/EAST_PERIODIC_IMAGE, ibm.h:148-149); a point in
// cell nx is evaluated a second time one period west (EAST_PERIODIC_IMAGE_MOD,
// ibm.h:150).  Evaluations are ordered (sphere, point, evaluation).
// ---------------------------------------------------------------------------
struct ScalEval {
    double x[3];
    int c[3], nev;
};
__device__ __forceinline__ ScalEval scal_eval(const Geo &g, const Mov &m, int s, int l) {
    ScalEval e;
    const int NB = g.nbody, nx = g.nx, mxf = g.nx + 1;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        e.x[d] = m.xc[s + d * NB] + g.bnd[3 * l + d] * g.ri;
        e.c[d] = cell_of(e.x[d]);
    }
    int pct = e.c[0];
    double xlt = e.x[0];
    if (!(1 <= pct && pct <= nx)) {
        if (e.c[0] < 1) { pct = mxf + e.c[0] - 1; xlt = mxf + e.x[0] - 1; }
        else if (e.c[0] >= mxf) { pct = e.c[0] - (mxf - 1); xlt = e.x[0] - (mxf - 1); }
    }
    e.nev = pct == nx ? 2 : 1;
    e.c[0] = pct;
    e.x[0] = xlt;
    return e;
}

// Evaluations per sphere.
__global__ void __launch_bounds__(256) k_sev_count(Geo g, Mov m, Scal *sc) {
    __shared__ double scr[32];
    if (block_failed(sc)) return;
    const int s = blockIdx.x, nb = g.nbnd;
    double n = 0.0;
    for (int l = threadIdx.x; l < nb; l += blockDim.x)
        if (m.revflag[(size_t)s * nb + l]) n += (double)scal_eval(g, m, s, l).nev;
    n = block_sum(n, scr);
    if (threadIdx.x == 0) m.sev_cnt[s] = (int)n;
}

// Offsets of every sphere's evaluations and their total.
__global__ void __launch_bounds__(1024) k_sev_scan(Geo g, Mov m, Scal *sc) {
    __shared__ int wsum[32];
    if (block_failed(sc)) return;
    const int T = blockDim.x, t = threadIdx.x, NB = g.nbody;
    const int per = (NB + T - 1) / T, c0 = min(t * per, NB), c1 = min(c0 + per, NB);
    int s = 0;
    for (int c = c0; c < c1; ++c) s += m.sev_cnt[c];
    int x = s;
    const int lane = t & 31, wid = t >> 5;
    for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int v = lane < (T >> 5) ? wsum[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += y; }
        wsum[lane] = v;
    }
    __syncthreads();
    int run = x - s + (wid > 0 ? wsum[wid - 1] : 0);
    for (int c = c0; c < c1; ++c) { m.sev_off[c] = run; run += m.sev_cnt[c]; }
    if (t == T - 1) sc->nsev = run;
}

// One sphere's evaluations written in (point, evaluation) order at its offset,
// and for every active point the index of its first one (negated: ~index, when it has two).
__global__ void __launch_bounds__(256) k_sev_write(Geo g, Mov m, Scal *sc) {
    __shared__ int wsum[8], wact[8];
    __shared__ int base, pbase;
    if (block_failed(sc)) return;
    const int s = blockIdx.x, nb = g.nbnd, t = threadIdx.x, lane = t & 31, wid = t >> 5, mxf = g.nx + 1;
    if (t == 0) { base = m.sev_off[s]; pbase = m.ptoff[s]; }
    __syncthreads();
    for (int l0 = 0; l0 < nb; l0 += blockDim.x) {
        const int l = l0 + t;
        ScalEval e;
        int n = 0;
        if (l < nb && m.revflag[(size_t)s * nb + l]) { e = scal_eval(g, m, s, l); n = e.nev; }
        const unsigned act = __ballot_sync(0xffffffffu, n > 0);
        int x = n;
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
        if (lane == 31) { wsum[wid] = x; wact[wid] = __popc(act); }
        __syncthreads();
        int before = 0, pbefore = 0;
        for (int w = 0; w < wid; ++w) { before += wsum[w]; pbefore += wact[w]; }
        int q = base + before + x - n;
        if (n > 0) m.sev_of[pbase + pbefore + __popc(act & ((1u << lane) - 1u))] = n == 2 ? ~q : q;
        for (int ev = 1; ev <= n; ++ev, ++q) {
            if (ev == 2 && e.c[0] >= mxf - 1) { e.c[0] = e.c[0] - (mxf - 1); e.x[0] = e.x[0] - (mxf - 1); }
            m.sev_m[q] = s;
            m.sev_l[q] = l;
#pragma unroll
            for (int d = 0; d < 3; ++d) { m.sev_x[3 * (size_t)q + d] = e.x[d]; m.sev_c[3 * (size_t)q + d] = e.c[d]; }
        }
        __syncthreads();
        if (t == 0)
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { base += wsum[w]; pbase += wact[w]; }
        __syncthreads();
    }
}

// Scalar forcing at every node of planes 1..nx in (evaluation, corner) order,
// from the flow's buckets: a point's evaluations put its 8 stencil corners on
// the nodes its point force goes to (the corners of cell nx's second plane come
// from the second evaluation, one period west; corners off planes 1..nx are
// dropped by one evaluation and covered by the other), and evaluations are
// numbered in point order, so a bucket in (point, corner) order is in
// (evaluation, corner) order too.  Buckets of its own (k_ssp_count) took 0.33 ms
// per step and 2.1 GB at 256^3.
__global__ void __launch_bounds__(256) k_sspread_dyn(Geo g, Mov m, const double *__restrict__ sctb,
                                                     const double *__restrict__ sfd, double *__restrict__ sfr, Scal *sc) {
    if (block_failed(sc)) return;
    for_forced_nodes(
        m.spcnt, (size_t)g.nx * g.RS, m.kmax, [&](size_t node) { sfr[node] = 0.0; },
        [&](size_t node, int c) {
            double v = 0.0;
            bucket_in_order(m.spbuf + node * m.kmax, c, [&](int ent) {
                const int f = m.sev_of[ent >> 3];
                const size_t e = (size_t)(f >= 0 ? f : ~f + (ent & 1));   // corner bit 0: the second x plane
                v = v + sctb[8 * e + (ent & 7)];
                if (!g.include_frmeanfluid) v = v + sfd[e];
            });
            sfr[node] = v;
        });
}

template <int N>
void enqueue_moving_scalar_t(const Geo &g, const Mov &m, Scal *sc, cudaStream_t s) {
    k_sev_count<<<g.nbody, 256, 0, s>>>(g, m, sc);
    k_sev_scan<<<1, 1024, 0, s>>>(g, m, sc);
    k_sev_write<<<g.nbody, 256, 0, s>>>(g, m, sc);
}

// Shape of the sub-step kernel: CTAs of few warps each up to the cluster's 8
// (FP64 instructions of one SM's warps queue on its pipes: 43 particles on two
// CTAs took 6.3 us per sub-step), and a warp per particle as far as shared
// memory holds the warps' scratch.
struct MarchShape { int ctas, warps; size_t smem; };
MarchShape march_shape(const Mov &m) {
    MarchShape t;
    t.ctas = std::min(kMarchCtas, (m.N + 3) / 4);
    const int slots = (m.N + t.ctas - 1) / t.ctas;
    t.warps = std::min(32, slots);
    while (t.warps > 1 && MarchMem::bytes(m.N, slots, m.maxn, t.warps) > 227 * 1024) --t.warps;
    t.smem = MarchMem::bytes(m.N, slots, m.maxn, t.warps);
    return t;
}
void launch_march(const Mov &m, Scal *sc, const double *pres, const double *visc, cudaStream_t s) {
    const MarchShape t = march_shape(m);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)t.ctas, 1, 1);
    cfg.blockDim = dim3((unsigned)(32 * t.warps), 1, 1);
    cfg.dynamicSmemBytes = t.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)t.ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_dem_march, m, sc, pres, visc);
}

template <int N>
void enqueue_moving_t(const Geo &g, const Mov &m, Scal *sc, const double *pres, const double *visc, cudaStream_t s) {
    const int pb = (m.N + 127) / 128;
    k_dem_start<<<1, 32, 0, s>>>(m, sc);
    if (m.soft) {
        const size_t bin_smem = (size_t)(3 * m.ncell + 1 + m.N) * sizeof(int);
        if (m.march) launch_march(m, sc, pres, visc, s);
        else for (int ifac = 1; ifac <= m.max_factor; ++ifac) {
            k_dem_update<<<(m.N + kUpdWarps - 1) / kUpdWarps, 32 * kUpdWarps, 0, s>>>(m, sc, pres, visc, ifac);
            k_dem_bin<<<1, 1024, bin_smem, s>>>(m, sc, ifac);
            k_dem_search<<<(m.N + kSearchWarps - 1) / kSearchWarps, 32 * kSearchWarps, 0, s>>>(m, sc, ifac);
        }
    } else {
        k_dem_none<<<pb, 128, 0, s>>>(m, sc);
    }
    k_dem_ibm<<<pb, 128, 0, s>>>(m, sc, g.dx);
    cudaMemsetAsync(m.fluid, 1, (size_t)g.nx * RP<N>::RSP, s);
    cudaMemsetAsync(m.spcnt, 0, (size_t)g.nx * RP<N>::RSP * sizeof(int), s);
    k_mask<N><<<g.nbody, 256, 0, s>>>(g, m, sc);
    k_nrpr<<<g.nbody, 256, 0, s>>>(g, m, sc);
    k_pts_scan<<<1, 1024, 0, s>>>(g, m, sc);
    k_pts_write<<<g.nbody, 256, 0, s>>>(g, m, sc);
    k_sp_count<N><<<(g.npts + 255) / 256, 256, 0, s>>>(g, m, sc);
}

}  // namespace

// The DEM of one flow step and the geometry rebuild that follows it
// (bcset, boundary_condition.F90:539-554), enqueued after compute_mpg_at_n.
void enqueue_moving(const Geo &g, const Mov &m, Scal *sc, const double *pres, const double *visc, cudaStream_t s) {
    switch (g.my) {
        case 32: enqueue_moving_t<32>(g, m, sc, pres, visc, s); break;
        case 64: enqueue_moving_t<64>(g, m, sc, pres, visc, s); break;
        case 96: enqueue_moving_t<96>(g, m, sc, pres, visc, s); break;
        case 128: enqueue_moving_t<128>(g, m, sc, pres, visc, s); break;
        case 256: enqueue_moving_t<256>(g, m, sc, pres, visc, s); break;
    }
}
int moving_kernels_per_step(const Mov &m) { return 1 + (m.soft && !m.march ? 3 * m.max_factor : 1) + 6; }

// Scalar geometry of the step (before calc_inner_rev_data) and its spreading.
void enqueue_moving_scalar(const Geo &g, const Mov &m, Scal *sc, cudaStream_t s) {
    switch (g.my) {
        case 32: enqueue_moving_scalar_t<32>(g, m, sc, s); break;
        case 64: enqueue_moving_scalar_t<64>(g, m, sc, s); break;
        case 96: enqueue_moving_scalar_t<96>(g, m, sc, s); break;
        case 128: enqueue_moving_scalar_t<128>(g, m, sc, s); break;
        case 256: enqueue_moving_scalar_t<256>(g, m, sc, s); break;
    }
}
void enqueue_sspread_dyn(const Geo &g, const Mov &m, const double *sctb, const double *sfd, double *sfr, Scal *sc, cudaStream_t s) {
    const size_t CR = (size_t)g.nx * g.RS;
    k_sspread_dyn<<<(unsigned)((CR + kSpreadWin - 1) / kSpreadWin), 256, 0, s>>>(g, m, sctb, sfd, sfr, sc);
}
int moving_scalar_kernels_per_step() { return 3; }

void enqueue_spread_dyn(const Geo &g, const Mov &m, const double *rec, const double *rz, double *fr, Scal *sc, cudaStream_t s) {
    const size_t CR = (size_t)g.nx * g.RS;
    k_spread_dyn<<<(unsigned)((CR + kSpreadWin - 1) / kSpreadWin), 256, 0, s>>>(g, m, rec, rz, fr, sc);
}

// Set-up: cells and the first neighbour search of des_time_march(.TRUE.)
// (initialize_flo.F90:631-639) on the uploaded positions.
void enqueue_dem_init(const Mov &m, Scal *sc, cudaStream_t s) {
    k_dem_start<<<1, 32, 0, s>>>(m, sc);   // also sets factor >= 1 for the two launches below
    const size_t bin_smem = (size_t)(3 * m.ncell + 1 + m.N) * sizeof(int);
    k_dem_bin<<<1, 1024, bin_smem, s>>>(m, sc, 1);
    k_dem_search<<<(m.N + kSearchWarps - 1) / kSearchWarps, 32 * kSearchWarps, 0, s>>>(m, sc, 1);
}

// Whether a run's sub-steps go in one launch per flow step (kMarchMax).
bool dem_march(const Mov &m) {
    return m.soft && m.N <= kMarchMax && m.N <= kMarchAny + kMarchPerSubStep * (m.max_factor - 1) && m.maxn < kMaxList &&
           m.cx < 1024 && m.cy < 1024 && m.cz < 1024;
}

cudaError_t configure_moving_kernels(const Mov &m) {
    const int smem = (int)((size_t)(3 * m.ncell + 1 + m.N) * sizeof(int));
    const cudaError_t e = cudaFuncSetAttribute(k_dem_march, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_dem_bin, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

}  // namespace pibm
