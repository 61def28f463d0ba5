// mp_split.cuh -- the harmonic walk of a few points split over the warps of a block.
//
// With one thread per point a call of a few thousand points leaves most of the GPU idle
// while each thread walks every harmonic in turn: 1000 points are 32 warps on 148 SMs, each
// with a chain of 289 steps at lmax 32.  Here a block takes a tile of at most 32 points
// (lane = point) and its warps share the |m| groups; all lanes of a warp walk the same (l, m),
// so there is no divergence and the recurrence constants stay uniform.  A group's sums are
// formed by the operations of mp_harmonics_reg and one warp adds the groups in their order and
// finishes the leaf, so a point's result is that of one thread per point, bit for bit.
// Consecutive leaves take turns between two buffers and between finishing warps, so a leaf is
// finished while the next one is walked.
#pragma once
#include "multipole.cuh"

// sums of a point that each group adds to
__host__ __device__ constexpr int split_sums(int mode) { return mode == AGB_MODE_POT ? 1 : 4; }
// and, with Hessians, the values kept per |m| group: six of each trig column
#define AGB_SPLIT_HESS_COLS 12
// values of a leaf's result
__host__ __device__ constexpr int split_out(int mode)
{
    return mode == AGB_MODE_HESS ? 10 : mode == AGB_MODE_GRAD ? 4 : 1;
}

// bytes of a tile's results, 16-byte aligned
__host__ __device__ constexpr int split_results(int mode, int T, int n_leaves)
{
    return (n_leaves * split_out(mode) * T * (int)sizeof(double) + 15) & ~15;
}

// most threads of a block: 128 registers a thread, 255 with Hessians
__host__ __device__ constexpr int split_threads(int mode)
{
    return (mode == AGB_MODE_POT || mode == AGB_MODE_GRAD || mode == AGB_MODE_DENS) ? 512 : 256;
}

// first column of |m| group m in a regular table (column 0 is the monopole)
template <int PAR>
__device__ __forceinline__ int mp_group_start(int m, int lmax)
{
    if (m == 0) return 1;
    if (PAR == 2) {
        const int h = lmax >> 1;
        return 1 + h + 2 * ((m - 1) * (h + 1) - ((m * m) >> 2));
    }
    return 1 + lmax + 2 * ((m - 1) * (lmax + 1) - ((m * (m - 1)) >> 1));
}

// The sums of one |m| group: the body of mp_harmonics_reg's loop over m.
template <int MODE, typename R, int PAR>
__device__ __forceinline__ void mp_group(const R* rec, int m, int lmax, R s, double cth_d,
                                         double sth_d, double sinpow, double sinpow_m1,
                                         MPCol<R>& gc, MPCol<R>& gs)
{
    constexpr bool NEED_ANG = MODE == AGB_MODE_GRAD || MODE == AGB_MODE_HESS;
    const bool near_pole = sth_d < 1.0e-10;
    R sp[6];
    sp[0] = R(1); sp[1] = s; sp[2] = s * s; sp[3] = sp[2] * s; sp[4] = sp[2] * sp[2]; sp[5] = sp[4] * s;
    const R cth = (R)cth_d, sth = (R)sth_d;
    const R c2 = (R)__dmul_rn(cth_d, cth_d), w2 = (R)(-2.0 * cth_d * sth_d);
    int l0 = (PAR == 2) ? (m + (m & 1)) : m;
    if (m == 0) l0 = PAR;
    gc.zero();
    gs.zero();
    if (l0 > lmax) return;
    R Pc = (R)(AGB_SEED[m] * sinpow), Pp = R(0), dPc = R(0), dPp = R(0);
    if (NEED_ANG && m > 0)
        dPc = (m == 1) ? (R)(AGB_SEED[1] * cth_d)
                       : (near_pole ? R(0) : (R)((double)m * AGB_SEED[m] * sinpow_m1 * cth_d));
    const int tb = m * AGB_LEG_N;
    auto step = [&](int L) {
        const R nb = MPConst<R>::nbetaq(tb + L);
        const R Pn = fma(cth, Pc, nb * Pp);
        if (NEED_ANG) {
            const R dPn = fma(cth, dPc, fma(-sth, Pc, nb * dPp));
            dPp = dPc;
            dPc = dPn;
        }
        Pp = Pc;
        Pc = Pn;
    };
    auto acc = [&](int L, auto has_sin) {
        R ac[6], as[6];
        if (has_sin) MPPtr<R>::load_cs(rec, ac, as);
        else MPPtr<R>::load(rec, ac);
        rec += has_sin ? 2 * MPPtr<R>::REC : MPPtr<R>::REC;
        const R ll1 = R(L * (L + 1));
        mp_col_acc<MODE, R>(gc, ac, sp, Pc, dPc, ll1);
        if (has_sin) mp_col_acc<MODE, R>(gs, as, sp, Pc, dPc, ll1);
    };
    const int ts = m * AGB_SKIP_N;
    auto skip2 = [&](int L) {
        const auto ab = MPConst<R>::skip(ts + (L >> 1));
        const R t = mp_cos2_add<MODE, R>(cth, c2, (R)ab.x);
        const R Pn = fma(t, Pc, (R)ab.y * Pp);
        if (NEED_ANG) {
            const R dPn = fma(w2, Pc, fma(t, dPc, (R)ab.y * dPp));
            dPp = dPc;
            dPc = dPn;
        }
        Pp = Pc;
        Pc = Pn;
    };
    const R seed = Pc;
    auto walk = [&](auto has_sin) {
        int l = m;
        while (l < l0) step(++l);
        acc(l, has_sin);
        if (PAR == 2) {
            Pp = (m == 0) ? seed : R(0);
            dPp = R(0);
            #pragma unroll 4
            for (l = l0 + 2; l <= lmax; l += 2) {
                skip2(l);
                acc(l, has_sin);
            }
        } else {
            #pragma unroll 4
            for (l = l0 + 1; l <= lmax; ++l) {
                step(l);
                acc(l, has_sin);
            }
        }
    };
    if (m == 0) walk(std::false_type());
    else walk(std::true_type());
}

// The sums of a point (split_sums), in this order.
template <int MODE, typename F>
__device__ __forceinline__ void mp_each_sum(MPSums& t, F f)
{
    f(0, t.A);
    if (MODE != AGB_MODE_POT) f(1, t.B);
    if (MODE == AGB_MODE_DENS) { f(2, t.D); f(3, t.L); }
    if (MODE == AGB_MODE_GRAD) { f(2, t.Th); f(3, t.Pos); }
}

// The |m| groups are dealt out to the block's S warps in snake order: warp w takes m = p S + w
// on even passes p and p S + S-1-w on odd ones, which gives every warp about the same number
// of (l, m) steps.  What a group adds to each of the point's sums (with Hessians its columns,
// see mp_combine_hess) is kept in out [m][value][point] and added up in ascending m, as
// mp_harmonics_reg adds it: the same bits as one thread per point, whatever S is.
template <int MODE, typename R, int PAR>
__device__ __forceinline__ void mp_split_walk(const DevComp& c, int k, double s, double cth_d,
                                              double sth_d, double cph, double sph, int w, int S,
                                              void* out, int T)
{
    constexpr bool HESS = MODE == AGB_MODE_HESS;
    const bool near_pole = sth_d < 1.0e-10;
    const R inv_sth = near_pole ? R(0) : (R)(1.0 / sth_d);
    const int lmax = c.lmax;
    double cm = 1.0, sm = 0.0, sinpow = 1.0, sinpow_m1 = 0.0;
    int at = 0;
    for (int p = 0; p * S <= lmax; ++p) {
        const int m = p * S + ((p & 1) ? S - 1 - w : w);
        if (m > lmax) continue;
        for (; at < m; ++at) {
            if (!HESS) mp_rotate(cm, sm, cph, sph);
            sinpow_m1 = sinpow;
            sinpow *= sth_d;
        }
        MPCol<R> gc, gs;
        mp_group<MODE, R, PAR>(MPPtr<R>::base(c, k) + mp_group_start<PAR>(m, lmax) * MPPtr<R>::REC,
                               m, lmax, (R)s, cth_d, sth_d, sinpow, sinpow_m1, gc, gs);
        if (HESS) {
            R* o = static_cast<R*>(out) + m * AGB_SPLIT_HESS_COLS * T;
            auto put = [&](int q, R a, R b) { o[2 * q * T] = a; o[(2 * q + 1) * T] = b; };
            put(0, gc.V, gs.V);
            put(1, gc.VR, gs.VR);
            put(2, gc.VT, gs.VT);
            put(3, gc.VRR, gs.VRR);
            put(4, gc.VRT, gs.VRT);
            put(5, gc.L, gs.L);
            continue;
        }
        const R q1 = (near_pole && m == 1) ? R(1) : R(0);
        mp_col_finish<MODE, R>(gc, inv_sth, q1, R(0), R(0), R(0));
        mp_col_finish<MODE, R>(gs, inv_sth, q1, R(0), R(0), R(0));
        MPSums t = {};
        mp_combine<MODE, R>(t, gc, gs, m, cm, sm);
        double* o = static_cast<double*>(out) + m * split_sums(MODE) * T;
        mp_each_sum<MODE>(t, [&](int q, double& u) { o[q * T] = u; });
    }
}

// the sums of a point from its groups' shares, in ascending m
template <int MODE>
__device__ __forceinline__ void mp_split_total(int lmax, const double* shares, int T, MPSums& t)
{
    constexpr int NS = split_sums(MODE);
    #pragma unroll 4
    for (int m = 0; m <= lmax; ++m)
        mp_each_sum<MODE>(t, [&](int q, double& u) { u += shares[(m * NS + q) * T]; });
}

// the groups of a Hessian leaf in ascending m, as mp_harmonics_reg adds them
template <typename R, int PAR>
__device__ __forceinline__ void mp_split_hess(int lmax, double cth_d, double sth_d, double cph,
                                              double sph, const R* cols, int T, MPSums& tot)
{
    const bool near_pole = sth_d < 1.0e-10;
    const R inv_sth = near_pole ? R(0) : (R)(1.0 / sth_d);
    const R cot = near_pole ? R(0) : (R)(cth_d / sth_d);
    const R np1 = near_pole ? R(0) : R(1);
    double cm = 1.0, sm = 0.0;
    for (int m = 0; m <= lmax; ++m) {
        if (m > 0) mp_rotate(cm, sm, cph, sph);
        if ((m == 0 ? PAR : (PAR == 2) ? (m + (m & 1)) : m) > lmax) continue;
        const R q1 = (near_pole && m == 1) ? R(1) : R(0);
        const R m2 = R(m * m) * inv_sth * inv_sth;
        MPCol<R> gc, gs;
        gc.zero();
        gs.zero();
        const R* o = cols + (long long)m * AGB_SPLIT_HESS_COLS * T;
        auto get = [&](int q, R& a, R& b) { a = o[2 * q * T]; b = o[(2 * q + 1) * T]; };
        get(0, gc.V, gs.V);
        get(1, gc.VR, gs.VR);
        get(2, gc.VT, gs.VT);
        get(3, gc.VRR, gs.VRR);
        get(4, gc.VRT, gs.VRT);
        get(5, gc.L, gs.L);
        mp_col_finish<AGB_MODE_HESS, R>(gc, inv_sth, q1, np1, cot, m2);
        mp_col_finish<AGB_MODE_HESS, R>(gs, inv_sth, q1, np1, cot, m2);
        mp_combine_hess<R>(tot, gc, gs, m, cm, sm);
    }
}

// A point's place in a Multipole's radial grid: interval k and offset s (as multipole_point
// finds them); false at the origin and beyond the grid.
__device__ __forceinline__ bool mp_place(const DevComp& c, double r, int& k, double& s)
{
    const double logr_min = c.p[0], dlogr = c.p[1], inv_dlogr = c.p[2];
    if (r < 1.0e-300) return false;
    const double logr = log(r);
    if (logr < logr_min) return false;
    k = (int)((logr - logr_min) * inv_dlogr);
    if (k < 0) k = 0;
    if (k >= c.n_int) return false;
    s = (logr - (logr_min + k * dlogr)) * inv_dlogr;
    s = fmin(fmax(s, 0.0), 1.0);
    return true;
}
