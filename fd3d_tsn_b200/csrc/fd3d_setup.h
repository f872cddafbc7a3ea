// fd3d_setup.h -- host-side set-up shared by the single-model context and the batch:
// parameter checks, the padded layout, the PML boxes/profiles (init_pml) and the
// per-step scalars in the field type.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>
#include "../../include/fd3d_gpu.h"
#include "fd3d_common.cuh"
#include "fd3d_kernels.cuh"

namespace fd3d {

inline
int validate_params(const fd3d_params* p) {
    if (!p) return FD3D_ERR_ARG;
    if (p->nabc < 3 || (p->fspace != 0 && p->fspace != 1)) return FD3D_ERR_ARG;
    if (p->nfs != (p->fspace ? p->nabc : 2)) return FD3D_ERR_ARG;  // fd3d_init.f90:161-165
    if (p->nxt < 2 * p->nabc + 4 || p->nyt < p->nabc + 4 || p->nzt < p->nabc + p->nfs + 4) return FD3D_ERR_ARG;
    if (!(p->dh > 0) || !(p->dt > 0)) return FD3D_ERR_ARG;
    if (p->law != FD3D_LAW_SW && p->law != FD3D_LAW_FVW) return FD3D_ERR_ARG;
    if (p->precision != FD3D_PREC_F32 && p->precision != FD3D_PREC_F64) return FD3D_ERR_ARG;
    if (p->nstations < 0 || p->nstations > FD3D_MAX_STATIONS) return FD3D_ERR_ARG;
    for (int s = 0; s < p->nstations; ++s)
        if (p->staX[s] < 1 || p->staX[s] > p->nxt || p->staY[s] < 1 || p->staY[s] > p->nyt || p->staZ[s] < 1 ||
            p->staZ[s] > p->nzt)
            return FD3D_ERR_ARG;
    if (p->history_stride < 0 || p->history_capacity < 0) return FD3D_ERR_ARG;
    if (p->vp_max > 0 && p->vp_max * p->dt / p->dh > 0.25) return FD3D_ERR_CFL;  // fd3d_init.f90:274-278
    return FD3D_OK;
}

inline Grid make_grid(const fd3d_params& p) {
    Grid g;
    g.nxt = p.nxt; g.nyt = p.nyt; g.nzt = p.nzt; g.nabc = p.nabc; g.nfs = p.nfs;
    g.fspace = p.fspace;
    g.off = (32 - (p.nabc % 32)) % 32;
    g.px = ((p.nxt + g.off + 31) / 32) * 32;
    g.plane = (long long)g.px * p.nyt;
    g.klo = 1; g.khi = p.nzt; g.kofs = 0; g.nzl = p.nzt;
    g.n3 = g.plane * p.nzt + 64;
    return g;
}

// Halo planes a z-slab stores on each side of the planes it owns: the 4th-order sweeps
// read two planes beyond their own, one more is kept as a margin.
constexpr int SLAB_HALO = 3;

// The grid of the z-slab that owns planes klo..khi of the model
inline Grid make_slab_grid(const fd3d_params& p, int klo, int khi) {
    Grid g = make_grid(p);
    g.klo = klo; g.khi = khi;
    const int kb = std::max(1, klo - SLAB_HALO), ke = std::min(p.nzt, khi + SLAB_HALO);
    g.kofs = kb - 1;
    g.nzl = ke - kb + 1;
    g.n3 = g.plane * g.nzl + 64;
    return g;
}

// A valid slab range: at least SLAB_MIN planes, and the top slab of a model with a free
// surface owns the two planes below it (the free-surface rows its fres and fuvw write stay
// out of every neighbour's halo).
constexpr int SLAB_MIN = 4;
inline bool slab_range_ok(const fd3d_params& p, int klo, int khi) {
    if (klo < 1 || khi > p.nzt || khi - klo + 1 < SLAB_MIN) return false;
    const int ks = p.nzt - p.nfs;
    if (khi >= ks && klo > ks - 2) return false;
    if (khi < p.nzt && khi >= ks - 2) return false;  // the slab above would not own ks-2 .. nzt
    return true;
}

// The pair (h, l) of div_by for the divisor b: see there for the method.  With b's significand
// Y and x's significand X as integers in [2^23, 2^24), x/b sits at a midpoint up to
// R / (Y (2Q+1)) relative, where 2^s X = Y (2Q+1) + R (s = 24 if X >= Y, else 25).  The error
// of the sum is at most 6*2^-48 (h nearest to 1/b, l within two units of 1/b - h), |R| <= 12, or
// 36*2^-48 (h up to three units below 1/b), |R| <= 72; RM is a little above that.  For each R
// the X that satisfy the congruence are a residue class mod Y, a few values at most.
inline bool div_pair_holds(float b, float h, float l, int64_t RM) {
    int e;
    const uint64_t Y = (uint64_t)std::ldexp((double)std::frexp(b, &e), 24);
    int t = 0;
    while (!((Y >> t) & 1)) ++t;
    const int64_t Yo = (int64_t)(Y >> t);
    if (Yo == 1) return l == 0x1p-149f;  // a power of two: x*h is exact, l only keeps x*l finite
    for (int s = 24; s <= 25; ++s) {
        int64_t p2 = 1;  // 2^(s-t) mod Yo and its inverse
        for (int k = 0; k < s - t; ++k) p2 = p2 * 2 % Yo;
        int64_t t0 = 0, t1 = 1, r0 = Yo, r1 = p2;
        while (r1) {
            const int64_t q = r0 / r1;
            int64_t x = t0 - q * t1; t0 = t1; t1 = x;
            x = r0 - q * r1; r0 = r1; r1 = x;
        }
        const int64_t inv = (t0 % Yo + Yo) % Yo;
        for (int64_t R = -RM; R <= RM; ++R) {
            if (R == 0 || R % ((int64_t)1 << t) != 0) continue;
            const int64_t Rm = ((R >> t) % Yo + Yo) % Yo;
            const int64_t lo = (int64_t)1 << 23;
            int64_t X = inv * Rm % Yo;  // both below 2^24
            if (X < lo) X += (lo - X + Yo - 1) / Yo * Yo;
            for (; X < 2 * lo; X += Yo) {
                if ((s == 24) != (X >= (int64_t)Y)) continue;
                const float x = (float)X, xl = x * l;
                if (std::fmaf(x, h, xl) != x / b) return false;
                // the sum's distance from the midpoint next to it must be more than what an
                // underflow of x*l could add for |x| >= 2^-70 (2^-66 relative)
                const double q = (double)x / (double)b;
                int qe;
                std::frexp(q, &qe);
                const double unit = std::ldexp(1.0, qe - 25);  // half a unit in the last place
                const double mid = (2.0 * std::floor(q / unit / 2.0) + 1.0) * unit;
                const double d = ((double)x * (double)h - mid) + (double)xl;
                if (std::fabs(d) < std::ldexp(q, -57)) return false;
            }
        }
    }
    return true;
}
// nonneg: only pairs with l >= 0 (the sign of a zero dividend is kept without more work); otherwise h
// is RN(1/b), with or without a pair.  false: no pair found (see PmlForm), or b out of range.
inline bool div_in_range(float b) { return b >= 0x1p-20f && b <= 0x1p20f; }
inline bool div_pair(float b, bool nonneg, float& h, float& l) {
    h = l = 0.f;
    if (!div_in_range(b)) return false;
    const double z = 1.0 / (double)b;
    h = (float)z;
    if (nonneg && (double)h > z) h = std::nextafterf(h, 0.f);
    for (int k = 0; k < (nonneg ? 3 : 1); ++k, h = std::nextafterf(h, 0.f)) {
        const float l0 = (float)(std::fma(-(double)b, (double)h, 1.0) / (double)b);
        for (int o = 0; o < 5; ++o) {  // the nearest l, then up to two units either way
            l = l0 == 0.f ? 0x1p-149f : l0;
            for (int u = 0; u < (o + 1) / 2; ++u) l = std::nextafterf(l, (o & 1) ? INFINITY : -INFINITY);
            if (div_pair_holds(b, h, l, nonneg ? 80 : 16)) return true;
        }
    }
    h = (float)z;
    return false;
}
// The PmlForm that one divisor asks for; h, l its pair if it has one, y = RN(1/b) (0 out of range).
// signed_ok: a pair of either sign serves as well as one with l >= 0 (1 + omega)
inline int div_form(float b, bool signed_ok, float& h, float& l, float& y) {
    y = div_in_range(b) ? (float)(1.0 / (double)b) : 0.f;
    if (div_pair(b, !signed_ok, h, l)) return PML_PAIR;
    if (!signed_ok && div_pair(b, false, h, l)) return PML_SIGNED;
    return div_in_range(b) ? PML_STEPS : PML_EXACT;
}
inline int div_form(double, bool, double& h, double& l, double& y) { h = l = y = 0; return PML_PAIR; }  // divides directly
// The scale of div_by's dividends for divisors up to b: a scaled dividend of 2^-70 or more has a
// quotient by b that is a normal number when it is scaled back, 2^-70 / S / b >= 2^-126.
inline double div_scale(double b) { return std::ldexp(1.0, std::min(56, 56 - (int)std::ceil(std::log2(b)))); }

// init_pml (fd3d_deriv.f90:1319-1493): strip boxes and damping profiles, in T.
template <class T>
void make_pml(const fd3d_params& p, PmlDesc& D, std::vector<Damp<T>>& prof) {
    const int nxt = p.nxt, nyt = p.nyt, nzt = p.nzt, nabc = p.nabc, nfs = p.nfs;
    const int bx[PML_MAXS][6] = {{2, nabc, nabc + 1, nyt - 1, nabc + 1, nzt - nfs},
                                 {nxt - nabc + 1, nxt - 1, nabc + 1, nyt - 1, nabc + 1, nzt - nfs},
                                 {2, nxt - 1, 2, nabc, nabc + 1, nzt - nfs},
                                 {2, nxt - 1, 2, nyt - 1, 2, nabc},
                                 {2, nxt - 1, 2, nyt - 1, nzt - nabc + 1, nzt - 1}};  // FSPACE top strip
    long long base = 0;
    prof.clear();
    D.ns = p.fspace ? 5 : 4;
    D.klo = 1;
    D.khi = p.nzt;
    D.cum[0] = 0;
    std::vector<std::vector<T>> ox(PML_MAXS), oxS(PML_MAXS), oy(PML_MAXS), oyS(PML_MAXS), oz(PML_MAXS), ozS(PML_MAXS);
    for (int s = 0; s < PML_MAXS; ++s) {
        if (s >= D.ns) {  // absent strip: empty range
            D.s[s] = D.s[s - 1];
            D.s[s].ncells = 0;
            D.cnt[s] = 0;
            D.cum[s + 1] = D.cum[s];
            continue;
        }
        Strip& S = D.s[s];
        S.nxb = bx[s][0]; S.nxe = bx[s][1]; S.nyb = bx[s][2]; S.nye = bx[s][3]; S.nzb = bx[s][4]; S.nze = bx[s][5];
        S.ni = S.nxe - S.nxb + 1; S.nk = S.nze - S.nzb + 1; S.nj1 = S.nye - S.nyb + 2;
        S.jend_uw = (s == 2) ? S.nye : S.nye + 1;
        S.ncells = (long long)S.ni * S.nj1 * S.nk;
        S.base = base;
        base += S.ncells;
        // every strip starts on a tile boundary, so a tile's cells share a strip
        D.cnt[s] = (long long)S.ni * (S.jend_uw - S.nyb + 1) * S.nk;
        D.cum[s + 1] = D.cum[s] + (D.cnt[s] + PML_TILE - 1) / PML_TILE * PML_TILE;
        S.rni = 1.0f / (float)S.ni;
        S.rnj = 1.0f / (float)(S.jend_uw - S.nyb + 1);
        S.fastdiv = D.cnt[s] < (1LL << 24);
        ox[s].assign(S.ni, (T)0); oxS[s].assign(S.ni, (T)0);
        oy[s].assign(S.nj1, (T)0); oyS[s].assign(S.nj1, (T)0);
        oz[s].assign(S.nk, (T)0); ozS[s].assign(S.nk, (T)0);
    }
    const T dt = (T)p.dt, dh = (T)p.dh;
    const T omegaM = (T)p.pml_fact * (T)p.pml_vp / ((T)2 * dh * (T)(nabc - 1));
    const int n = nabc - 1;
    std::vector<T> om(n), omR(n), omM(n), omRM(n);
    for (int i = 1; i <= n; ++i) {
        T r = (T)i / (T)n, rM = ((T)i - (T)0.5) / (T)n;
        om[i - 1] = (T)0.5 * dt * omegaM * ((r * r) * (r * r));
        omR[nabc - i - 1] = om[i - 1];
        omM[i - 1] = (T)0.5 * dt * omegaM * ((rM * rM) * (rM * rM));
        omRM[nabc - i - 1] = omM[i - 1];
    }
    for (int i = 1; i <= n; ++i) {  // 1-based reference index i -> 0-based i-1
        ox[0][i - 1] = omR[i - 1];  oxS[0][i - 1] = omRM[i - 1];
        ox[1][i - 1] = omM[i - 1];  oxS[1][i - 1] = om[i - 1];
        oy[2][i - 1] = omR[i - 1];  ox[2][i - 1] = omR[i - 1];  ox[2][nxt - i - 2] = omM[i - 1];
        oyS[2][i - 1] = omRM[i - 1]; oxS[2][i - 1] = omRM[i - 1]; oxS[2][nxt - i - 2] = om[i - 1];
        oz[3][i - 1] = omR[i - 1];  ox[3][i - 1] = omR[i - 1];  ox[3][nxt - i - 2] = omM[i - 1];
        oy[3][i - 1] = omR[i - 1];
        ozS[3][i - 1] = omRM[i - 1]; oxS[3][i - 1] = omRM[i - 1]; oxS[3][nxt - i - 2] = om[i - 1];
        oyS[3][i - 1] = omRM[i - 1];
        if (D.ns == 5) {  // fd3d_deriv.f90:1481-1490
            oz[4][i - 1] = omM[i - 1];  ox[4][i - 1] = omR[i - 1];  ox[4][nxt - i - 2] = omM[i - 1];
            oy[4][i - 1] = omR[i - 1];
            ozS[4][i - 1] = om[i - 1];  oxS[4][i - 1] = omRM[i - 1]; oxS[4][nxt - i - 2] = om[i - 1];
            oyS[4][i - 1] = omRM[i - 1];
        }
    }
    for (int s = 0; s <= PML_MAXS; ++s) D.tile0[s] = (int)(D.cum[s] / PML_TILE);
    std::vector<Damp<T>> pairs;  // the strips share their divisors: one search for each
    D.form = PML_PAIR;
    D.bmax = 1.0;
    for (int s = 0; s < D.ns; ++s) {
        Strip& S = D.s[s];
        auto put = [&](const std::vector<T>& v) {
            const int o = (int)prof.size();
            int last = -1;
            for (T om : v) {
                Damp<T> e;
                e.m = (T)1 - om;
                e.p = (T)1 + om;
                D.bmax = std::max(D.bmax, (double)e.p);
                if (last < 0 || pairs[last].p != e.p) {
                    for (last = 0; last < (int)pairs.size() && pairs[last].p != e.p;) ++last;
                    if (last == (int)pairs.size()) {
                        T y;
                        D.form = std::max(D.form, div_form(e.p, true, e.h, e.l, y));
                        e.h = y;  // (the pair's, if there is one)
                        pairs.push_back(e);
                    }
                }
                e.h = pairs[last].h;
                e.l = pairs[last].l;
                prof.push_back(e);
            }
            return o;
        };
        S.ox_off = put(ox[s]); S.oxS_off = put(oxS[s]);
        S.oy_off = put(oy[s]); S.oyS_off = put(oyS[s]);
        S.oz_off = put(oz[s]); S.ozS_off = put(ozS[s]);
    }
}

// The PML sweeps update a split direction as p + inc where its strip class says the
// direction is never damped (split_mode, fd3d_kernels.cuh), and where a warp's cells lie
// outside the damped ends of a SPLIT_MAYBE direction; that is exact only if every omega there
// is zero.  Checked once per set-up.
template <class T>
bool pml_modes_hold(const PmlDesc& D, const std::vector<Damp<T>>& prof, int nabc) {
    const int n = nabc - 1;
    for (int s = 0; s < D.ns; ++s) {
        const Strip& S = D.s[s];
        const int C = pml_class(s);
        const int offs[3][2] = {{S.ox_off, S.oxS_off}, {S.oy_off, S.oyS_off}, {S.oz_off, S.ozS_off}};
        const int len[3] = {S.ni, S.nj1, S.nk};
        for (int dir = 0; dir < 3; ++dir) {
            const int mode = split_mode(C, dir);
            if (mode == SPLIT_ALWAYS) continue;
            const int q0 = mode == SPLIT_NEVER ? 0 : n;
            const int q1 = mode == SPLIT_MAYBE && dir == 0 ? len[dir] - n : len[dir];
            for (int v = 0; v < 2; ++v)
                for (int q = q0; q < q1; ++q) {
                    const Damp<T>& e = prof[(size_t)offs[dir][v] + q];
                    if (e.m != (T)1 || e.p != (T)1) return false;
                }
        }
    }
    return true;
}

template <class T>
StepConst<T> make_const(const fd3d_params& p, const PmlDesc& D) {
    StepConst<T> c;
    c.dt = (T)p.dt; c.dh = (T)p.dh;
    c.dth = c.dt / c.dh;
    c.dth2 = (T)0.5 * c.dt / c.dh;
    c.dht = c.dh / c.dt;
    c.damp_s = (T)p.damp_s;
    c.c1 = (T)9 / (T)8;
    c.c2 = (T)-1 / (T)24;
    const double scale = div_scale(std::max(D.bmax, (double)c.dh));
    c.ds = (T)scale;
    c.dsi = (T)(1.0 / scale);
    c.pml_form = std::max(D.form, div_form(c.dh, false, c.rdh, c.rdl, c.ydh));
    c.dtA = p.dt;
    c.dhA = (double)c.dh;
    c.dthA = c.dtA / c.dhA;
    return c;
}

}  // namespace fd3d
