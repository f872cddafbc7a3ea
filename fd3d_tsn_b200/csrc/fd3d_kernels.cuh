// fd3d_kernels.cuh -- sm_100a kernels of one FD3D_TSN time step (templated on the
// field type T: float for the production build, double for the FP64 build).
//
// The step is eight launches, or four on a small grid (small_step, fd3d_opt.cuh: 1-3 share a launch and
// 5-7 another), each a set of reference regions whose write sets are
// disjoint and which read nothing another thread of the same launch writes (the fused
// fault boundary condition forms what its fres CTAs write from what they read):
//   1 vel_interior  uxx1/vyy1/wzz1 (fd3d_deriv.f90:50-193)
//   2 vel_fault     uxx0a/vyy0a/wzz0a at j=nyt-1 + v mirror (fd3d_deriv.f90:198-508),
//                   tasu1/tasw1 at j=nyt (fd3d_deriv.f90:1109-1234)
//   3 vel_pml       pml_uvw, 4 strips, 5 under FSPACE (fd3d_deriv.f90:1927-2299)
//   4 vel_fs        fuvw (fd3d_deriv.f90:1018-1062)
//   5 str_interior  dstres (fd3d_deriv.f90:513-622)
//   6 str_fault     sxx/sxy0/sxz0/syz0 at j=nyt-1 + xy/yz mirror, sxz1, tasii
//                   (fd3d_deriv.f90:677-1012,1239-1314)
//   7 str_pml       pml_xyz (fd3d_deriv.f90:2304-2992)
//   8 fault_bc      fres (fd3d_deriv.f90:1067-1104) and the fault boundary condition
//                   (fd3d_theo.f90:225-467): trial traction, |T| at the staggered nodes,
//                   friction law with slip and rupture time, output planes, fused per
//                   tile (fault_bc_body)
// and, for rate-and-state runs with a nucleation ramp, the ramp (fd3d_theo.f90:487-542).
// The fault boundary condition also exists as separate launches (str_fs, traction,
// friction, output), which fd3d_run_noalloc uses.
//
// Operation order inside every expression follows the reference so that, with
// contraction of multiply-add switched off (--fmad=false), the FP32 and FP64
// builds reproduce the CPU restatement's arithmetic exactly for slip weakening.
#pragma once
#include "fd3d_async.cuh"
#include "fd3d_common.cuh"

namespace fd3d {

// ---------------------------------------------------------------- velocity
// Interior 4th-order velocity: one thread per (i,j), marching a chunk of k.
template <class T>
__global__ void __launch_bounds__(256) k_vel_interior(Grid g, Fields<T> f, StepConst<T> c, int kchunk) {
    const int i = g.nabc + 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = g.nabc + 1 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > g.nxt - g.nabc || j > g.nyt - 2) return;
    const int kb = g.kin_lo() + blockIdx.z * kchunk;
    const int ke = min(kb + kchunk - 1, g.kin_hi());
    const long long sy = g.px, sz = g.plane;
    const T c1 = c.c1, c2 = c.c2;
    const T* __restrict__ xx = f.xx; const T* __restrict__ yy = f.yy; const T* __restrict__ zz = f.zz;
    const T* __restrict__ xy = f.xy; const T* __restrict__ yz = f.yz; const T* __restrict__ xz = f.xz;
    for (int k = kb; k <= ke; ++k) {
        const long long p = g.at(i, j, k);
        const T r = c.dth / f.d[p];
        f.u[p] = f.u[p] + r * (c1 * (xx[p] - xx[p - 1]) + c2 * (xx[p + 1] - xx[p - 2]) +
                               c1 * (xy[p] - xy[p - sy]) + c2 * (xy[p + sy] - xy[p - 2 * sy]) +
                               c1 * (xz[p] - xz[p - sz]) + c2 * (xz[p + sz] - xz[p - 2 * sz]));
        f.v[p] = f.v[p] + r * (c1 * (xy[p + 1] - xy[p]) + c2 * (xy[p + 2] - xy[p - 1]) +
                               c1 * (yy[p + sy] - yy[p]) + c2 * (yy[p + 2 * sy] - yy[p - sy]) +
                               c1 * (yz[p] - yz[p - sz]) + c2 * (yz[p + sz] - yz[p - 2 * sz]));
        f.w[p] = f.w[p] + r * (c1 * (xz[p + 1] - xz[p]) + c2 * (xz[p + 2] - xz[p - 1]) +
                               c1 * (yz[p] - yz[p - sy]) + c2 * (yz[p + sy] - yz[p - 2 * sy]) +
                               c1 * (zz[p + sz] - zz[p]) + c2 * (zz[p + 2 * sz] - zz[p - sz]));
    }
}

// FVW Newton solve of one node (fd3d_deriv.f90:1148-1161), FP64, bounded.
__device__ __forceinline__ double fvw_newton(double vtilde, double cdelta, double uw, double psi, double a,
                                             double v0, int* status) {
    const double e = v0 * exp(-psi / a);
    double ferr = 10.0;
    int it = 0;
    while (fabs(ferr) > 1e-10) {
        ++it;
        const double fwv = vtilde + cdelta * uw + sinh(uw) * e;
        const double dfw = cdelta + cosh(uw) * e;
        ferr = fwv / dfw;
        uw = uw - ferr;
        if (it > FD3D_NEWTON_MAXIT) { atomicOr(status, ST_NEWTON); break; }
    }
    return uw;
}

// Band j=nyt-1 (2nd order + damping, v mirror) and split-node fault velocity at j=nyt.  The
// parts are independent and go to CTAs of their own (bz_): 0 the band (and the step counter), 1
// u and 2 w on the fault.  Bound by latency on a few hundred CTAs or less, so every part loads
// all it needs before it stores (a store to one field holds back a load from the next).
// One launch, us (before: one thread for all parts, each field loaded after the store to the one
// before): rate-and-state 11 K fault nodes 8.4 (13.8), slip weakening 19 K nodes 4.7 (7.1);
// the stress band of 11 K nodes 4.1 (8.8).
constexpr int VEL_FAULT_PARTS = 3;
template <class T>
__device__ __forceinline__ void vel_fault_body(const Grid& g, const Fields<T>& f, const Fault<T>& q,
                                               const StepConst<T>& c, int law, const FvwScalars& s, int* it_dev,
                                               int* status, int bx_, int by_, int bz_) {
    const int ii = bx_ * blockDim.x + threadIdx.x;
    const int kk = by_ * blockDim.y + threadIdx.y;
    const int ks = g.ks();
    const long long sy = g.px, sz = g.plane;
    const int i = g.nabc + 1 + ii, k = g.kin_lo() + kk;
    const bool in = i <= g.nxt - g.nabc && k <= g.kin_hi();
    const int n2 = g.at2(i, k);
    if (bz_ == 0) {
        if (ii == 0 && kk == 0) atomicAdd(it_dev, 1);  // step counter read by the fault BC launches
        // ghost row k=ks+1: v(:,nyt,ks+1) = v(:,nyt-1,ks+1)  (bnd2d mirror, fd3d_deriv.f90:225-232);
        // under FSPACE that row belongs to the top PML strip, whose tiles mirror it
        if (!g.fspace && kk == 0 && ii < g.nxt && g.owns(ks + 1)) {
            const long long p = g.at(ii + 1, g.nyt - 1, ks + 1);
            f.v[p + sy] = f.v[p];
        }
        if (!in) return;
        // uxx0a / vyy0a / wzz0a  (fd3d_deriv.f90:284-508)
        const long long p = g.at(i, g.nyt - 1, k);
        const T d = f.d[p], u = f.u[p], v = f.v[p], w = f.w[p], au1 = q.au1[n2], av1 = q.av1[n2], aw1 = q.aw1[n2];
        const T pdx = (f.xx[p] - f.xx[p - 1]) + (f.xy[p] - f.xy[p - sy]) + (f.xz[p] - f.xz[p - sz]);
        const T pdy = (f.xy[p + 1] - f.xy[p]) + (f.yy[p + sy] - f.yy[p]) + (f.yz[p] - f.yz[p - sz]);
        const T pdz = (f.xz[p + 1] - f.xz[p]) + (f.yz[p] - f.yz[p - sy]) + (f.zz[p + sz] - f.zz[p]);
        const T r = c.dth / d;
        const T au = pdx - au1, av = pdy - av1, aw = pdz - aw1;
        const T vn = v + r * (pdy + c.damp_s * av);
        f.u[p] = u + r * (pdx + c.damp_s * au);
        f.v[p] = vn;
        f.v[p + sy] = vn;  // mirror into the fault plane
        f.w[p] = w + r * (pdz + c.damp_s * aw);
        q.au1[n2] = pdx;
        q.av1[n2] = pdy;
        q.aw1[n2] = pdz;
        return;
    }
    if (!in) return;
    const long long pf = g.at(i, g.nyt, k);
    if (law == 0) {  // tasu1/tasw1 slip weakening
        const T d = f.d[pf];
        if (bz_ == 1) {
            const T u = f.u[pf], t = q.tx[n2], rf = q.RFx[n2], r = c.dth / d;
            f.u[pf] = u + r * (T)2 * (t + rf);
        } else {
            const T w = f.w[pf], t = q.tz[n2], rf = q.RFz[n2], r = c.dth / d;
            f.w[pf] = w + r * ((T)2 * (t + rf));
        }
        return;
    }
    // FVW (fd3d_deriv.f90:1141-1162, 1204-1226), FP64
    const double d = (double)f.d[pf];
    const double rr = c.dthA / d;
    if (bz_ == 1) {
        const double u = (double)f.u[pf];
        const double a = (double)q.aX[n2];
        const double s1 = 2.0 * (fabs((double)q.wX[n2]) + fabs(s.wini)), s2 = 2.0 * (fabs(u) + fabs(s.uini));
        const double sr = sqrt(s1 * s1 + s2 * s2);
        const double cdelta = 2.0 * rr * s.Sn * a;
        double uw = asinh(exp(q.psiX[n2] / a) * sr / (2.0 * s.v0));
        const double rfz = ((double)q.RFz[n2] + (double)q.RFz[g.at2(i - 1, k)] + (double)q.RFz[g.at2(i, k - 1)] +
                            (double)q.RFz[g.at2(i - 1, k - 1)]) / 4.0;
        const double q1 = (double)q.wX[n2] + 2.0 * rr * (rfz - (double)q.T0Z[n2]);
        const double q2 = u + 2.0 * rr * ((double)q.RFx[n2] - (double)q.T0X[n2]);
        const double vt = -sqrt(q1 * q1 + q2 * q2);
        uw = fvw_newton(vt, cdelta, uw, q.psiX[n2], a, s.v0, status);
        f.u[pf] = (T)(((double)q.tx[n2] + (double)q.T0X[n2]) * (-sinh(uw)) * s.v0 * exp(-q.psiX[n2] / a) /
                      (double)q.tabsX[n2] + s.uini);
    } else {
        const double w = (double)f.w[pf];
        const double a = (double)q.aZ[n2];
        const double s1 = 2.0 * (w - s.wini), s2 = 2.0 * ((double)q.uZ[n2] - s.uini);
        const double sr = sqrt(s1 * s1 + s2 * s2);
        const double cdelta = 2.0 * rr * s.Sn * a;
        double uw = asinh(exp(q.psiZ[n2] / a) * sr / (2.0 * s.v0));
        const int e1 = g.at2(i + 1, k), e2 = g.at2(i, k + 1), e3 = g.at2(i + 1, k + 1);
        const double rfx = ((double)q.RFx[n2] + (double)q.RFx[e1] + (double)q.RFx[e2] + (double)q.RFx[e3]) / 4.0;
        const double t0x = ((double)q.T0X[n2] + (double)q.T0X[e1] + (double)q.T0X[e2] + (double)q.T0X[e3]) / 4.0;
        const double q1 = w + 2.0 * rr * ((double)q.RFz[n2] - (double)q.T0Z[n2]);
        const double q2 = (double)q.uZ[n2] + 2.0 * rr * (rfx - t0x);
        const double vt = -sqrt(q1 * q1 + q2 * q2);
        uw = fvw_newton(vt, cdelta, uw, q.psiZ[n2], a, s.v0, status);
        f.w[pf] = (T)(((double)q.tz[n2] + (double)q.T0Z[n2]) * (-sinh(uw) * s.v0 * exp(-q.psiZ[n2] / a)) /
                      (double)q.tabsZ[n2] + s.wini);
    }
}

constexpr int PML_MAXS = 5;  // strips 1-4, and 5 (the top) under FSPACE
struct PmlDesc {
    Strip s[PML_MAXS];
    long long cum[PML_MAXS + 1];  // first compact index of each strip (a multiple of PML_TILE); cum[PML_MAXS] = end
    long long cnt[PML_MAXS];      // cells of each strip's u/w loop range (0 for an absent strip)
    int ns;                       // strips present: 4, or 5 under FSPACE
    int klo, khi;                 // planes updated (Grid::klo, khi)
    int tile0[PML_MAXS + 1];      // cum in tiles
    int form;                     // the PmlForm that the divisors 1 + omega ask for
    double bmax;                  // the largest of them
};

// PML auxiliary components (the 24 split fields that init_pml allocates per strip,
// fd3d_deriv.f90:1330-1406, 1413-1437) are indexed by the compact cell index t of the
// u/w loop ranges of the strips (strip s holds t in [cum[s], cum[s] + cnt[s]); each strip
// starts on a PML_TILE boundary, so every tile lies in one strip) and stored in blocks of
// 32 cells: inside a block the 32 values of one component are contiguous and the
// components of a group follow each other.  The velocity group (u,v,w splits, 9
// components) and the stress group (xx,yy,zz,xy,xz,yz splits, 15) are separate spans,
// so the auxiliaries of PML_TILE consecutive cells are one contiguous range per group:
// one bulk copy brings a tile's range into shared memory.
constexpr int AUX_NV = 9, AUX_NS = 15;
constexpr int PML_TILE = 256;
inline long long pml_aux_cells(const PmlDesc& D) { return (D.cum[PML_MAXS] + PML_TILE - 1) / PML_TILE * PML_TILE; }
inline size_t pml_aux_elems(const PmlDesc& D) { return (size_t)pml_aux_cells(D) * (AUX_NV + AUX_NS); }

// One entry of a damping profile (init_pml's omega at one index): the factors
// 1 - omega and 1 + omega of the split-field update, formed on the host with the same IEEE
// operations the reference performs, and the pair of 1 + omega for div_by_signed (h = RN(1/(1 +
// omega)) always, for div_steps).
template <class T>
struct alignas(4 * sizeof(T)) Damp {
    T m, p, h, l;  // 1 - omega, 1 + omega, pair
};

// Damping of one split direction over a strip, from where init_pml leaves the profiles
// zero (fd3d_deriv.f90:1436-1490): the x strips are damped in x only, the y strip in y
// and, in its corners, in x; the z strips in z and, in their corners and edges, in x and
// y.  SPLIT_NEVER: omega = 0 over the whole strip, the update is p + inc.  SPLIT_ALWAYS:
// the general form (p*(1-omega) + inc)/(1+omega), which is also exact where omega = 0
// (a*1 = a, x/1 = x).  SPLIT_MAYBE: the general form where any lane of the warp lies in the
// direction's nabc-1 outer cells, p + inc where none does (a warp-uniform branch, so no lane
// loads a profile entry or forms a quotient it discards).  The host checks the undamped
// ranges against the profiles (pml_modes_hold).
enum { SPLIT_NEVER = 0, SPLIT_MAYBE = 1, SPLIT_ALWAYS = 2 };
// strip class: 0 the x strips (1, 2), 1 the y strip (3), 2 the z strips (4, and 5 under FSPACE)
__host__ __device__ constexpr int pml_class(int s) { return s <= 1 ? 0 : (s == 2 ? 1 : 2); }
// mode of direction DIR (0 x, 1 y, 2 z) in strip class C
__host__ __device__ constexpr int split_mode(int C, int DIR) {
    return DIR == C ? SPLIT_ALWAYS : (DIR < C ? SPLIT_MAYBE : SPLIT_NEVER);
}

// The two divisions of a split-field update, by dh and by 1 + omega.
//   DIV_FAST: the quotients of div_by on dividends scaled by c.ds; `key` tells whether
//             all of them are right.  The quotient by dh stays scaled: its only use is an
//             addition, where a multiply-add takes the factor out without a rounding.
//   DIV_TINY: right for finite operands of any size, DIV_FULL: for all
// FORM (PML_PAIR, PML_SIGNED, PML_STEPS): the quotients of the first two.
enum { DIV_FAST = 0, DIV_TINY = 1, DIV_FULL = 2 };
template <class T, int HOW, int FORM>
struct PmlDiv {
    const StepConst<T>& c;
    unsigned key = 0xffffffffu;
    __device__ __forceinline__ T scaled(T r) const {
        if constexpr (HOW == DIV_FAST) return r * c.ds;
        else return r;
    }
    // x / dh (of a scaled x: scaled)
    __device__ __forceinline__ T by_dh(T x) {
        if constexpr (HOW == DIV_FAST && FORM == PML_STEPS) return div_steps(x, c.dh, c.ydh, key);
        else if constexpr (HOW == DIV_FAST && FORM == PML_SIGNED) return div_by_signed(x, c.rdh, c.rdl, key);
        else if constexpr (HOW == DIV_FAST) return div_by(x, c.rdh, c.rdl, key);
        else if constexpr (HOW == DIV_TINY && FORM == PML_STEPS) return div_small<true>(x, c.dh, c.ydh, (T)0);
        else if constexpr (HOW == DIV_TINY) return div_small<false>(x, c.dh, c.rdh, c.rdl);
        else return div_exact(x, c.dh);
    }
    __device__ __forceinline__ T plus(T a, T q) const {  // a + x / dh
        if constexpr (HOW == DIV_FAST) return __fmaf_rn(q, c.dsi, a);
        else return a + q;
    }
    // the new split component: p old, q = by_dh(...) of its increment
    template <int MODE>
    __device__ __forceinline__ T split(T p, T q, const Damp<T>& o, bool warp_damped) {
        if (MODE == SPLIT_NEVER || (MODE == SPLIT_MAYBE && !warp_damped)) return plus(p, q);
        const T x = plus(p * o.m, q);
        if constexpr (HOW == DIV_FAST && FORM == PML_STEPS) return div_steps(x * c.ds, o.p, o.h, key) * c.dsi;
        else if constexpr (HOW == DIV_FAST) return div_by_signed(x * c.ds, o.h, o.l, key) * c.dsi;
        else if constexpr (HOW == DIV_TINY) return div_small<FORM == PML_STEPS>(x, o.p, o.h, o.l);
        else return div_exact(x, o.p);
    }
};
// false for a sum of magnitudes with one that is not finite (a sum that overflows only sends
// the cell to the exact form)
__device__ __forceinline__ bool pml_finite(float s) { return fabsf(s) <= 3.402823466e38f; }

template <class T>
struct PmlAux {
    T* vel;              // velocity group, pml_aux_cells * AUX_NV elements
    T* str;              // stress group, pml_aux_cells * AUX_NS elements
    const Damp<T>* prof; // damping profiles
};

// carve the two groups out of one pool of pml_aux_elems(D) elements
template <class T>
inline void pml_aux_bind(PmlAux<T>& X, T* pool, const PmlDesc& D) {
    X.vel = pool;
    X.str = pool + pml_aux_cells(D) * AUX_NV;
}

// first component of the cell with compact index t in a group of ncomp components; the others
// follow at steps of 32 elements
__device__ __forceinline__ long long aux_at(long long t, int ncomp) { return (t >> 5) * (32 * ncomp) + (t & 31); }

// strip of the tile that starts at compact index t0
__device__ __forceinline__ int pml_tile_strip(const PmlDesc& D, long long t0) {
    const int tile = (int)(t0 / PML_TILE);
    return (tile >= D.tile0[1]) + (tile >= D.tile0[2]) + (tile >= D.tile0[3]) + (tile >= D.tile0[4]);
}

// (i,j,k) of compact cell index t of strip s; false past the strip's last cell and, for
// a z-slab (SLAB), outside its planes
template <bool SLAB>
__device__ __forceinline__ bool pml_cell(const PmlDesc& D, int s, long long t, int& i, int& j, int& k) {
    const long long r0 = t - D.cum[s];
    if (r0 >= D.cnt[s]) return false;
    const Strip& S = D.s[s];
    // strip-local index fits 32 bits (a strip is ni*nj*nk cells)
    const unsigned r = (unsigned)r0;
    const unsigned ni = (unsigned)S.ni, nj = (unsigned)(S.jend_uw - S.nyb + 1);
    unsigned q1, k2, ri, rj;
    if (S.fastdiv) {
        q1 = udiv_small(r, ni, S.rni, ri);
        k2 = udiv_small(q1, nj, S.rnj, rj);
    } else {
        q1 = r / ni; ri = r - q1 * ni;
        k2 = q1 / nj; rj = q1 - k2 * nj;
    }
    i = S.nxb + (int)ri; j = S.nyb + (int)rj; k = S.nzb + (int)k2;
    return !SLAB || (k >= D.klo && k <= D.khi);
}

// The PML sweeps.  A tile's split components come by one bulk copy into shared memory while each
// thread loads its cell's neighbours, profile entries and medium (all before the wait); the new
// components go straight back from registers, one full line per warp and component (a bulk
// copy back had to drain before the CTA could leave: 25% slower at 0.5 M cells, 3% at 12 M).
// Bound by memory latency at 4 CTAs per SM (64 registers): on 2.3 M PML cells the velocity / stress sweep
// moves 5.0 / 4.5 TB/s of DRAM (61 / 55% of peak) and issues in 51 / 42% of cycles, 430 / 528 instructions
// a cell (546 / 702 with the five-operation quotients), its warps waiting for memory in 5.4 / 7.6 of the
// cycles between two instructions.
// Measured, velocity / stress, in us, against five-operation quotients with a branch each and
// partly written sectors in the x strips (pml_sector_rest): 11.9 M PML cells 279 / 381 (340 /
// 543), 13 M cells of 64 models 375 / 526 (446 / 638), 0.5 M cells 14.3 / 18.9 (15.5 / 22.7).
// Left out, measured: the components by plain loads (the registers hold a third of the inputs
// at a time); all inputs through shared memory by bulk copies of row pieces (a copy is issued
// by one lane, 30 a tile); u, v, w and the normal and shear stresses in CTAs of their own.
//
// Starts the copy of a tile's range of a group (bytes); every thread calls it.
__device__ __forceinline__ void pml_tile_begin(uint32_t sm, const void* src, uint32_t bytes, uint32_t bar) {
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
        fence_proxy_async_global();
        mbar_expect_tx(bar, bytes);
        bulk_load(sm, src, bytes, bar);
    }
}
// Waits (bounded) for the tile's load; false on every thread if any thread gave up
// (ST_TIMEOUT recorded after one more bounded wait for the copy in flight).
__device__ __forceinline__ bool pml_tile_wait(uint32_t bar, int* status) {
    const bool ok = mbar_wait(bar, 0u);
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0 && threadIdx.y == 0) atomicOr(status, ST_TIMEOUT);
        mbar_wait(bar, 0u);
        return false;
    }
    return true;
}
// whether any of a warp's cells lies in the damped ends of the strip in x / y (SPLIT_MAYBE);
// every lane of the warp calls it
template <int C>
__device__ __forceinline__ void pml_damped(const Grid& g, const Strip& S, bool act, int i, int j, bool& wx, bool& wy) {
    const int i2 = i - S.nxb, n = g.nabc - 1;
    wx = wy = true;
    if (split_mode(C, 0) == SPLIT_MAYBE) wx = __any_sync(0xffffffffu, act && (i2 < n || i2 >= S.ni - n));
    if (split_mode(C, 1) == SPLIT_MAYBE) wy = __any_sync(0xffffffffu, act && j - S.nyb < n);
}

// The x strips' rows are nabc-1 cells, one of them (the outermost) alone in its 32-byte sector:
// a store of 4 bytes that the L2 has to merge with the rest of the sector from memory, a third of
// the stress sweep's time at 18 M cells.  The rest of that sector is the boundary cell (i = 1 or
// nxt, which nothing updates) and the row's padding, both 0: the strip's other lanes store
// the zeros, so the sector is written whole.  o: the field; returns the element of this lane
// (i2 cells into the strip), or -1.
template <class T>
__device__ __forceinline__ int pml_sector_rest(const Grid& g, const Strip& S, int i2) {
    constexpr int N = 32 / (int)sizeof(T);
    if (S.nxb == 2) {
        const int e = g.off + 1, q = (e & ~(N - 1)) + i2;
        return q < e ? q : -1;
    }
    const int e = g.off + S.nxe - 1, q = e + 1 + i2;
    return q <= (e | (N - 1)) ? q : -1;
}

// inputs of a velocity cell, loaded while its split components fly
template <class T, int C>
struct VelPmlIn {
    T xx0, xx1, xy0, xy1, xy2, xz0, xz1, xz2, yz0, yz1, yz2, yy0, yy1, zz0, zz1, r;  // r = dt / d
    Damp<T> ox, oxS, oy, oz;
    __device__ __forceinline__ void load(const Grid& g, const Fields<T>& f, const PmlAux<T>& X, const StepConst<T>& c,
                                         const Strip& S, int i, int j, int k, bool wx, bool wy) {
        const long long p = g.at(i, j, k), sy = g.px, sz = g.plane;
        const int i2 = i - S.nxb, j2 = j - S.nyb, k2 = k - S.nzb;
        if (f.lay) r = f.lay[4 * g.nzt + k - 1];  // dt/d of the plane (1-D medium)
        else r = f.d[p];
        xx0 = f.xx[p]; xx1 = f.xx[p - 1]; xy0 = f.xy[p]; xy1 = f.xy[p - sy]; xz0 = f.xz[p]; xz1 = f.xz[p - sz];
        xz2 = f.xz[p + 1]; yz0 = f.yz[p]; yz1 = f.yz[p - sy]; zz0 = f.zz[p]; zz1 = f.zz[p + sz];
        xy2 = yy0 = yy1 = yz2 = 0;
        if (j <= S.nye) { xy2 = f.xy[p + 1]; yy0 = f.yy[p + sy]; yy1 = f.yy[p]; yz2 = f.yz[p - sz]; }
        constexpr int MX = split_mode(C, 0), MY = split_mode(C, 1), MZ = split_mode(C, 2);
        ox = oxS = oy = oz = Damp<T>{1, 1, 1, 0};
        if (MX == SPLIT_ALWAYS || (MX == SPLIT_MAYBE && wx)) { ox = X.prof[S.ox_off + i2]; oxS = X.prof[S.oxS_off + i2]; }
        if (MY == SPLIT_ALWAYS || (MY == SPLIT_MAYBE && wy)) oy = X.prof[S.oy_off + j2];
        if (MZ == SPLIT_ALWAYS) oz = X.prof[S.oz_off + k2];
        if (!f.lay) r = c.dt / r;
    }
};

// pml_uvw at one cell of strip S (fd3d_deriv.f90:1927-2293); a: its first split component in
// shared memory.  Returns HOW, or the form that the cell needs, with nothing stored.
template <class T, int C, int HOW, int FORM>
__device__ __forceinline__ int vel_pml_cell(const Grid& g, const Fields<T>& f, const StepConst<T>& c, const Strip& S,
                                            const VelPmlIn<T, C>& q, const T* a, T* ga, int i, int j,
                                            int k, bool wx, bool wy) {
    constexpr int MX = split_mode(C, 0), MY = split_mode(C, 1), MZ = split_mode(C, 2);
    const bool dov = j <= S.nye;
    // p = (p*(1 - omega) + (dt/d)*diff/dh) / (1 + omega), every division rounded as IEEE
    PmlDiv<T, HOW, FORM> dv{c};
    const T r = dv.scaled(q.r);
    auto inc = [&](T diff) { return dv.by_dh(r * diff); };
    auto at = [&](int n) { return a[32 * n]; };
    auto put = [&](int n) -> T& { return ga[32 * n]; };
    const T u0 = dv.template split<MX>(at(AX_U0), inc(q.xx0 - q.xx1), q.ox, wx);
    const T u1 = dv.template split<MY>(at(AX_U1), inc(q.xy0 - q.xy1), q.oy, wy);
    const T u2 = dv.template split<MZ>(at(AX_U2), inc(q.xz0 - q.xz1), q.oz, true);
    const T w0 = dv.template split<MX>(at(AX_W0), inc(q.xz2 - q.xz0), q.oxS, wx);
    const T w1 = dv.template split<MY>(at(AX_W1), inc(q.yz0 - q.yz1), q.oy, wy);
    const T w2 = dv.template split<MZ>(at(AX_W2), inc(q.zz1 - q.zz0), q.oz, true);
    // (on the fault row, which has no v: the components are 0 and stay so)
    const T v0 = dv.template split<MX>(at(AX_V0), inc(q.xy2 - (dov ? q.xy0 : (T)0)), q.oxS, wx);
    const T v1 = dv.template split<MY>(at(AX_V1), inc(q.yy0 - q.yy1), q.oy, wy);
    const T v2 = dv.template split<MZ>(at(AX_V2), inc((dov ? q.yz0 : (T)0) - q.yz2), q.oz, true);
    const T u = u0 + u1 + u2, w = w0 + w1 + w2, v = v0 + v1 + v2;
    if constexpr (HOW == DIV_FAST) {
        if (!pml_finite(fabsf(u) + fabsf(v) + fabsf(w))) return DIV_FULL;
        if (dv.key < DIV_KEY) return DIV_TINY;
    }
    put(AX_U0) = u0; put(AX_U1) = u1; put(AX_U2) = u2; put(AX_W0) = w0; put(AX_W1) = w1; put(AX_W2) = w2;
    const long long p = g.at(i, j, k), sy = g.px;
    f.u[p] = u;
    f.w[p] = w;
    if (dov) {
        put(AX_V0) = v0; put(AX_V1) = v1; put(AX_V2) = v2;
        if (j == g.nyt - 1) f.v[p + sy] = f.v[p];  // bnd2d mirror of the value before this update
        f.v[p] = v;
    }
    if (C == 0) {
        const int e = pml_sector_rest<T>(g, S, i - S.nxb);
        if (e >= 0) {
            const long long z = p - (g.off + i - 1) + e;
            f.u[z] = (T)0;
            f.w[z] = (T)0;
            if (dov) f.v[z] = (T)0;
        }
    }
    return HOW;
}

// The cells that need another form than DIV_FAST, out of line.
template <class T, int C, int HOW>
__device__ __noinline__ void vel_pml_redo(const Grid* g, const Fields<T>* f, const PmlAux<T>* X, const StepConst<T>* c,
                                          const Strip* S, const T* a, T* ga, int i, int j, int k, bool wx, bool wy) {
    VelPmlIn<T, C> q;
    q.load(*g, *f, *X, *c, *S, i, j, k, wx, wy);
    vel_pml_cell<T, C, HOW, PML_STEPS>(*g, *f, *c, *S, q, a, ga, i, j, k, wx, wy);
}

// pml_uvw in one tile of strip class C, one cell per thread.  false if the copy timed out.  ANY: the
// model's quotients may take any form (PmlForm; those of a pair with l >= 0 are also div_by_signed's).
template <class T, int C, bool SLAB, bool ANY>
__device__ __forceinline__ bool vel_pml_tile_c(const Grid& g, const Fields<T>& f, const PmlDesc& D, const PmlAux<T>& X,
                                               const StepConst<T>& c, int s, long long t0, T* sm, uint32_t bar, int* status) {
    constexpr uint32_t BYTES = PML_TILE * AUX_NV * sizeof(T);
    pml_tile_begin(smem_addr(sm), X.vel + t0 * AUX_NV, BYTES, bar);
    const Strip& S = D.s[s];
    const int l = threadIdx.y * blockDim.x + threadIdx.x;
    int i = 0, j = 0, k = 0;
    bool wx, wy;
    const bool act = pml_cell<SLAB>(D, s, t0 + l, i, j, k);
    pml_damped<C>(g, S, act, i, j, wx, wy);
    VelPmlIn<T, C> q;
    if (act) q.load(g, f, X, c, S, i, j, k, wx, wy);
    __syncthreads();  // the barrier is initialised
    if (!pml_tile_wait(bar, status)) return false;
    if (act) {
        const T* a = sm + aux_at(l, AUX_NV);
        T* ga = X.vel + aux_at(t0 + l, AUX_NV);
        if constexpr (sizeof(T) == 8) {
            vel_pml_cell<T, C, DIV_FULL, PML_PAIR>(g, f, c, S, q, a, ga, i, j, k, wx, wy);
        } else {
            int how = DIV_FAST;
            if (!ANY) how = vel_pml_cell<T, C, DIV_FAST, PML_PAIR>(g, f, c, S, q, a, ga, i, j, k, wx, wy);
            else if (c.pml_form <= PML_SIGNED) how = vel_pml_cell<T, C, DIV_FAST, PML_SIGNED>(g, f, c, S, q, a, ga, i, j, k, wx, wy);
            else if (c.pml_form == PML_STEPS) how = vel_pml_cell<T, C, DIV_FAST, PML_STEPS>(g, f, c, S, q, a, ga, i, j, k, wx, wy);
            else vel_pml_cell<T, C, DIV_FULL, PML_EXACT>(g, f, c, S, q, a, ga, i, j, k, wx, wy);
            if (how == DIV_TINY) {  // the same again: nothing is stored yet
                if (ANY) {
                    vel_pml_redo<T, C, DIV_TINY>(&g, &f, &X, &c, &S, a, ga, i, j, k, wx, wy);
                } else {
                    asm volatile("" ::: "memory");  // (the inputs are loaded anew, not kept in registers)
                    q.load(g, f, X, c, S, i, j, k, wx, wy);
                    vel_pml_cell<T, C, DIV_TINY, PML_PAIR>(g, f, c, S, q, a, ga, i, j, k, wx, wy);
                }
            } else if (how == DIV_FULL) {
                vel_pml_redo<T, C, DIV_FULL>(&g, &f, &X, &c, &S, a, ga, i, j, k, wx, wy);
            }
        }
    }
    return true;
}

// pml_uvw: split-field PML velocity in the strips (fd3d_deriv.f90:1927-2293), one tile of
// PML_TILE consecutive cells per CTA (a tile lies in one strip).
template <class T, bool SLAB, bool ANY>
__device__ __forceinline__ bool vel_pml_tile(const Grid& g, const Fields<T>& f, const PmlDesc& D, const PmlAux<T>& X,
                                             const StepConst<T>& c, int tile, T* sm, uint32_t bar, int* status) {
    const long long t0 = (long long)tile * PML_TILE;
    const int s = pml_tile_strip(D, t0);
    switch (pml_class(s)) {
        case 0: return vel_pml_tile_c<T, 0, SLAB, ANY>(g, f, D, X, c, s, t0, sm, bar, status);
        case 1: return vel_pml_tile_c<T, 1, SLAB, ANY>(g, f, D, X, c, s, t0, sm, bar, status);
        default: return vel_pml_tile_c<T, 2, SLAB, ANY>(g, f, D, X, c, s, t0, sm, bar, status);
    }
}

// fuvw at the ghost row k=ks+1 (fd3d_deriv.f90:1018-1062).  w needs u and v of the
// ghost row at (i+1,j) and (i,j-1); they are recomputed with the same formula
// (identical operands and order), so no second launch is needed.
template <class T>
__device__ __forceinline__ void vel_fs_body(Grid g, Fields<T> f, int bx_, int by_, int bz_) {
    const int i = 1 + bx_ * blockDim.x + threadIdx.x;
    const int j = 1 + by_ * blockDim.y + threadIdx.y;
    if (i > g.nxt || j > g.nyt) return;
    const int n = g.ks();
    const long long sy = g.px, sz = g.plane;
    auto ug = [&](int ii, int jj) -> T {  // loop 1: j=1..nyt, i=2..nxt-1
        const long long p = g.at(ii, jj, n);
        return f.u[p] - (f.w[p] - f.w[p - 1]);
    };
    auto vg = [&](int ii, int jj) -> T {  // loop 2: j=2..nyt-1, i=2..nxt-1; else existing value
        const long long p = g.at(ii, jj, n);
        if (jj >= 2 && jj <= g.nyt - 1 && ii >= 2 && ii <= g.nxt - 1) return f.v[p] - (f.w[p + sy] - f.w[p]);
        return f.v[p + sz];
    };
    T un = (T)0, vn = (T)0, wn = (T)0;
    const bool du = (i >= 2 && i <= g.nxt - 1);
    const bool dv = (j >= 2 && j <= g.nyt - 1 && du);
    const bool dw = (j >= 2 && i >= 2 && i <= g.nxt - 2);
    if (du) un = ug(i, j);
    if (dv) vn = vg(i, j);
    if (dw) {
        const long long p = g.at(i, j, n);
        const T xl = f.lam[p + sz], xm = f.mu[p + sz];
        const T a = (T)2 * xl, b = xl + (T)2 * xm;
        const T u_i1 = ug(i + 1, j);
        const T u_i = du ? un : f.u[p + sz];
        const T v_j = vg(i, j);
        const T v_jm = vg(i, j - 1);
        wn = +(f.w[p - sz] - (a / b) * (f.u[p + 1] - f.u[p] + u_i1 - u_i + f.v[p] - f.v[p - sy] + v_j - v_jm));
    }
    // The ghost-row values read above (v at j=1 and j=nyt) are never written by this
    // launch, so the writes below cannot race with them.
    const long long pg = g.at(i, j, n + 1);
    if (du) f.u[pg] = un;
    if (dv) f.v[pg] = vn;
    if (dw) f.w[pg] = wn;
}

// ---------------------------------------------------------------- stress
template <class T>
__global__ void __launch_bounds__(256) k_str_interior(Grid g, Fields<T> f, StepConst<T> c, int kchunk) {
    const int i = g.nabc + 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = g.nabc + 1 + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > g.nxt - g.nabc || j > g.nyt - 2) return;
    const int kb = g.kin_lo() + blockIdx.z * kchunk;
    const int ke = min(kb + kchunk - 1, g.kin_hi());
    const long long sy = g.px, sz = g.plane;
    const T c1 = c.c1, c2 = c.c2, dth = c.dth;
    const T* __restrict__ u = f.u; const T* __restrict__ v = f.v; const T* __restrict__ w = f.w;
    const T* __restrict__ mu = f.mu;
    for (int k = kb; k <= ke; ++k) {
        const long long p = g.at(i, j, k);
        const T xl = f.lam[p], xm = mu[p];
        const T a = xl + (T)2 * xm, b = xl;
        const T dxu1 = c1 * (u[p + 1] - u[p]), dxu2 = c2 * (u[p + 2] - u[p - 1]);
        const T dyv1 = c1 * (v[p] - v[p - sy]), dyv2 = c2 * (v[p + sy] - v[p - 2 * sy]);
        const T dzw1 = c1 * (w[p] - w[p - sz]), dzw2 = c2 * (w[p + sz] - w[p - 2 * sz]);
        f.xx[p] = f.xx[p] + dth * a * (dxu1 + dxu2) + dth * b * (dyv1 + dyv2 + dzw1 + dzw2);
        f.yy[p] = f.yy[p] + dth * a * (dyv1 + dyv2) + dth * b * (dxu1 + dxu2 + dzw1 + dzw2);
        f.zz[p] = f.zz[p] + dth * a * (dzw1 + dzw2) + dth * b * (dxu1 + dxu2 + dyv1 + dyv2);
        T xmu = (T)0.5 * (xm + mu[p + sy]);
        f.xy[p] = f.xy[p] + dth * xmu * (c1 * (u[p + sy] - u[p]) + c2 * (u[p + 2 * sy] - u[p - sy]) +
                                         c1 * (v[p] - v[p - 1]) + c2 * (v[p + 1] - v[p - 2]));
        xmu = (T)0.5 * (xm + mu[p + sz]);
        f.xz[p] = f.xz[p] + dth * xmu * (c1 * (u[p + sz] - u[p]) + c2 * (u[p + 2 * sz] - u[p - sz]) +
                                         c1 * (w[p] - w[p - 1]) + c2 * (w[p + 1] - w[p - 2]));
        xmu = (T)0.5 * (xm + mu[p + 1 + sy + sz]);
        f.yz[p] = f.yz[p] + dth * xmu * (c1 * (v[p + sz] - v[p]) + c2 * (v[p + 2 * sz] - v[p - sz]) +
                                         c1 * (w[p + sy] - w[p]) + c2 * (w[p + 2 * sy] - w[p - sy]));
    }
}

// Band j=nyt-1 stresses (2nd order) + xy/yz mirror (bz_ = 0); sxz1 and tasii at j=nyt (bz_ = 1):
// CTAs of their own, loads before stores, as vel_fault_body.
constexpr int STR_FAULT_PARTS = 2;
template <class T>
__device__ __forceinline__ void str_fault_body(const Grid& g, const Fields<T>& f, const Fault<T>& q,
                                               const StepConst<T>& c, int bx_, int by_, int bz_) {
    const int i = g.nabc + 1 + bx_ * blockDim.x + threadIdx.x;
    const int k = g.kin_lo() + by_ * blockDim.y + threadIdx.y;
    if (i > g.nxt - g.nabc || k > g.kin_hi()) return;
    const long long sy = g.px, sz = g.plane;
    const T dth = c.dth, dth2 = c.dth2, c1 = c.c1, c2 = c.c2;
    if (bz_ == 0) {   // sxx, sxy0, sxz0, syz0 at j=nyt-1 (fd3d_deriv.f90:818-1012)
        const long long p = g.at(i, g.nyt - 1, k);
        const T xl = f.lam[p], xm = f.mu[p], my = f.mu[p + sy], mz = f.mu[p + sz], md = f.mu[p + 1 + sy + sz];
        const T up = f.u[p], vp = f.v[p], wp = f.w[p];
        const T ux = f.u[p + 1], vy = f.v[p - sy], wz = f.w[p - sz];
        const T uy = f.u[p + sy], vx = f.v[p - 1], uz = f.u[p + sz], wx = f.w[p - 1], vz = f.v[p + sz], wy = f.w[p + sy];
        const T xx = f.xx[p], yy = f.yy[p], zz = f.zz[p], xy = f.xy[p], xz = f.xz[p], yz = f.yz[p];
        const T a = xl + (T)2 * xm, b = xl;
        f.xx[p] = xx + dth * a * (ux - up) + dth * b * (vp - vy + wp - wz);
        f.yy[p] = yy + dth * a * (vp - vy) + dth * b * (ux - up + wp - wz);
        f.zz[p] = zz + dth * a * (wp - wz) + dth * b * (ux - up + vp - vy);
        T xmu = xm + my;
        const T xyn = xy + dth2 * xmu * (uy - up + vp - vx);
        f.xy[p] = xyn; f.xy[p + sy] = xyn;
        xmu = xm + mz;
        f.xz[p] = xz + dth2 * xmu * (uz - up + wp - wx);
        xmu = xm + md;
        const T yzn = yz + dth2 * xmu * (vz - vp + wy - wp);
        f.yz[p] = yzn; f.yz[p + sy] = yzn;
    } else {   // sxz1 (tasxz) and tasii at j=nyt (fd3d_deriv.f90:677-722, 1263-1314)
        const long long p = g.at(i, g.nyt, k);
        const T* u = f.u; const T* w = f.w;
        const T xl = f.lam[p], xm = f.mu[p], mz = f.mu[p + sz];
        const T xx = f.xx[p], yy = f.yy[p], zz = f.zz[p], xz = f.xz[p], vb = f.v[p - sy];
        const T duz = c1 * (u[p + sz] - u[p]) + c2 * (u[p + 2 * sz] - u[p - sz]);
        const T diff1 = c1 * (u[p + 1] - u[p]) + c2 * (u[p + 2] - u[p - 1]);
        const T diff3 = c1 * (w[p] - w[p - sz]) + c2 * (w[p + sz] - w[p - 2 * sz]);
        const T dwx1 = c1 * (w[p] - w[p - 1]), dwx2 = c2 * (w[p + 1] - w[p - 2]);
        const T xmu = xm + mz;
        f.xz[p] = xz + dth2 * xmu * (duz + dwx1 + dwx2);
        const T a = xl + (T)2 * xm, b = xl;
        const T v1t = vb - b * (diff1 + diff3) / ((T)2 * a);
        q.v1t[g.at2(i, k)] = v1t;
        const T dv = v1t - vb;
        f.xx[p] = xx + dth * a * (diff1) + dth * b * ((T)2 * dv + diff3);
        f.yy[p] = yy + dth * a * (T)2 * dv + dth * b * (diff1 + diff3);
        f.zz[p] = zz + dth * a * (diff3) + dth * b * (diff1 + (T)2 * dv);
    }
}

// inputs of a stress cell
template <class T, int C>
struct StrPmlIn {
    T up, ux, uy, uz, vp, vx, vy, vz, wp, wx, wy, wz, xl, xm, my, mz, md;
    Damp<T> ox, oxS, oy, oyS, oz, ozS;
    __device__ __forceinline__ void load(const Grid& g, const Fields<T>& f, const PmlAux<T>& X, const Strip& S, int i,
                                         int j, int k, bool damped_x, bool damped_y) {
        const long long p = g.at(i, j, k), sy = g.px, sz = g.plane;
        const int i2 = i - S.nxb, j2 = j - S.nyb, k2 = k - S.nzb;
        const bool dxy = j <= S.nye;
        my = md = uy = vx = vz = wy = 0;
        if (f.lay) {  // 1-D medium: mu(i,j+1,k) = mu(i,j,k), mu(i+1,j+1,k+1) = mu(i,j,k+1)
            xl = f.lay[k - 1]; xm = f.lay[g.nzt + k - 1]; mz = f.lay[g.nzt + k];
            my = xm; md = mz;
        } else {
            xl = f.lam[p]; xm = f.mu[p]; mz = f.mu[p + sz];
            if (dxy) { my = f.mu[p + sy]; md = f.mu[p + 1 + sy + sz]; }
        }
        up = f.u[p]; ux = f.u[p + 1]; uz = f.u[p + sz]; vp = f.v[p]; vy = f.v[p - sy];
        wp = f.w[p]; wz = f.w[p - sz]; wx = f.w[p - 1];
        if (dxy) { uy = f.u[p + sy]; vx = f.v[p - 1]; vz = f.v[p + sz]; wy = f.w[p + sy]; }
        // xy and yz take omegayS in strips 3-5 and xz, yz omegazS in strips 4-5; in the other
        // strips those directions are undamped (SPLIT_NEVER), so oyS / ozS serve every class
        constexpr int MX = split_mode(C, 0), MY = split_mode(C, 1), MZ = split_mode(C, 2);
        ox = oxS = oy = oyS = oz = ozS = Damp<T>{1, 1, 1, 0};
        if (MX == SPLIT_ALWAYS || (MX == SPLIT_MAYBE && damped_x)) { ox = X.prof[S.ox_off + i2]; oxS = X.prof[S.oxS_off + i2]; }
        if (MY == SPLIT_ALWAYS || (MY == SPLIT_MAYBE && damped_y)) { oy = X.prof[S.oy_off + j2]; oyS = X.prof[S.oyS_off + j2]; }
        if (MZ == SPLIT_ALWAYS) { oz = X.prof[S.oz_off + k2]; ozS = X.prof[S.ozS_off + k2]; }
    }
};

// pml_xyz at one cell of a strip (fd3d_deriv.f90:2304-3143), as vel_pml_cell; free_top: the
// strip's xz and yz components are zeroed at its top row (strips 1-3, not FSPACE)
template <class T, int C, int HOW, int FORM>
__device__ __forceinline__ int str_pml_cell(const Grid& g, const Fields<T>& f, const StepConst<T>& c, const Strip& S,
                                            bool free_top, const StrPmlIn<T, C>& q, const T* a, T* ga, int i, int j,
                                            int k, bool wx, bool wy) {
    constexpr int MX = split_mode(C, 0), MY = split_mode(C, 1), MZ = split_mode(C, 2);
    const bool dxy = j <= S.nye;
    // p = (p*(1 - omega) + dt*modulus*diff/dh) / (1 + omega), every division rounded as IEEE
    PmlDiv<T, HOW, FORM> dv{c};
    auto at = [&](int comp) { return a[32 * (comp - AUX_NV)]; };
    auto put = [&](int comp) -> T& { return ga[32 * (comp - AUX_NV)]; };
    const T dt = c.dt;
    const T ma = dv.scaled(dt * (q.xl + (T)2 * q.xm)), mb = dv.scaled(dt * q.xl);
    // the six products of the normal stresses
    const T diff1 = q.ux - q.up, diff2 = q.vp - q.vy, diff3 = q.wp - q.wz;
    const T qa1 = dv.by_dh(ma * diff1), qb1 = dv.by_dh(mb * diff1);
    const T x0 = dv.template split<MX>(at(AX_XX0), qa1, q.oxS, wx);
    const T y0 = dv.template split<MX>(at(AX_YY0), qb1, q.oxS, wx);
    const T z0 = dv.template split<MX>(at(AX_ZZ0), qb1, q.oxS, wx);
    const T qa2 = dv.by_dh(ma * diff2), qb2 = dv.by_dh(mb * diff2);
    const T x1 = dv.template split<MY>(at(AX_XX1), qb2, q.oy, wy);
    const T y1 = dv.template split<MY>(at(AX_YY1), qa2, q.oy, wy);
    const T z1 = dv.template split<MY>(at(AX_ZZ1), qb2, q.oy, wy);
    const T qa3 = dv.by_dh(ma * diff3), qb3 = dv.by_dh(mb * diff3);
    const T x2 = dv.template split<MZ>(at(AX_XX2), qb3, q.oz, true);
    const T y2 = dv.template split<MZ>(at(AX_YY2), qb3, q.oz, true);
    const T z2 = dv.template split<MZ>(at(AX_ZZ2), qa3, q.oz, true);
    const T xx = x0 + x1 + x2, yy = y0 + y1 + y2, zz = z0 + z1 + z2;
    const T mxz = dv.scaled(dt * ((q.xm + q.mz) / (T)2));
    T q0 = dv.template split<MZ>(at(AX_XZ0), dv.by_dh(mxz * (q.uz - q.up)), q.ozS, true);
    T q1 = dv.template split<MX>(at(AX_XZ1), dv.by_dh(mxz * (q.wp - q.wx)), q.ox, wx);
    const T xz = q0 + q1;
    T e0 = 0, e1 = 0, h0 = 0, h1 = 0;
    if (dxy) {
        const T mxy = dv.scaled(dt * ((q.xm + q.my) / (T)2)), myz = dv.scaled(dt * ((q.xm + q.md) / (T)2));
        e0 = dv.template split<MY>(at(AX_XY0), dv.by_dh(mxy * (q.uy - q.up)), q.oyS, wy);
        e1 = dv.template split<MX>(at(AX_XY1), dv.by_dh(mxy * (q.vp - q.vx)), q.ox, wx);
        h0 = dv.template split<MZ>(at(AX_YZ0), dv.by_dh(myz * (q.vz - q.vp)), q.ozS, true);
        h1 = dv.template split<MY>(at(AX_YZ1), dv.by_dh(myz * (q.wy - q.wp)), q.oyS, wy);
    }
    const T xy = e0 + e1, yz = h0 + h1;
    if constexpr (HOW == DIV_FAST) {
        if (!pml_finite(fabsf(xx) + fabsf(yy) + fabsf(zz) + fabsf(xy) + fabsf(xz) + fabsf(yz))) return DIV_FULL;
        if (dv.key < DIV_KEY) return DIV_TINY;
    }
    if (free_top && k == S.nze) q0 = q1 = h0 = h1 = (T)0;
    put(AX_XX0) = x0; put(AX_XX1) = x1; put(AX_XX2) = x2; put(AX_YY0) = y0; put(AX_YY1) = y1; put(AX_YY2) = y2;
    put(AX_ZZ0) = z0; put(AX_ZZ1) = z1; put(AX_ZZ2) = z2; put(AX_XZ0) = q0; put(AX_XZ1) = q1;
    const long long p = g.at(i, j, k), sy = g.px;
    f.xx[p] = xx;
    f.yy[p] = yy;
    f.zz[p] = zz;
    f.xz[p] = xz;
    if (dxy) {
        put(AX_XY0) = e0; put(AX_XY1) = e1; put(AX_YZ0) = h0; put(AX_YZ1) = h1;
        if (j == g.nyt - 1) {  // strbnd mirror of the values before this update
            f.xy[p + sy] = f.xy[p];
            f.yz[p + sy] = f.yz[p];
        }
        f.xy[p] = xy;
        f.yz[p] = yz;
    }
    if (C == 0) {
        const int e = pml_sector_rest<T>(g, S, i - S.nxb);
        if (e >= 0) {
            const long long z = p - (g.off + i - 1) + e;
            f.xx[z] = (T)0;
            f.yy[z] = (T)0;
            f.zz[z] = (T)0;
            f.xz[z] = (T)0;
            if (dxy) {
                f.xy[z] = (T)0;
                f.yz[z] = (T)0;
            }
        }
    }
    return HOW;
}

template <class T, int C, int HOW>
__device__ __noinline__ void str_pml_redo(const Grid* g, const Fields<T>* f, const PmlAux<T>* X, const StepConst<T>* c,
                                          const Strip* S, bool free_top, const T* a, T* ga, int i, int j, int k,
                                          bool wx, bool wy) {
    StrPmlIn<T, C> q;
    q.load(*g, *f, *X, *S, i, j, k, wx, wy);
    str_pml_cell<T, C, HOW, PML_STEPS>(*g, *f, *c, *S, free_top, q, a, ga, i, j, k, wx, wy);
}

template <class T, int C, bool SLAB, bool ANY>
__device__ __forceinline__ bool str_pml_tile_c(const Grid& g, const Fields<T>& f, const PmlDesc& D, const PmlAux<T>& X,
                                               const StepConst<T>& c, int s, long long t0, T* sm, uint32_t bar, int* status) {
    constexpr uint32_t BYTES = PML_TILE * AUX_NS * sizeof(T);
    pml_tile_begin(smem_addr(sm), X.str + t0 * AUX_NS, BYTES, bar);
    const Strip& S = D.s[s];
    const bool free_top = C <= 1 && !g.fspace;
    const int l = threadIdx.y * blockDim.x + threadIdx.x;
    int i = 0, j = 0, k = 0;
    bool wx, wy;
    const bool act = pml_cell<SLAB>(D, s, t0 + l, i, j, k);
    pml_damped<C>(g, S, act, i, j, wx, wy);
    StrPmlIn<T, C> q;
    if (act) q.load(g, f, X, S, i, j, k, wx, wy);
    __syncthreads();  // the barrier is initialised
    if (!pml_tile_wait(bar, status)) return false;
    if (act) {
        const T* a = sm + aux_at(l, AUX_NS);
        T* ga = X.str + aux_at(t0 + l, AUX_NS);
        if constexpr (sizeof(T) == 8) {
            str_pml_cell<T, C, DIV_FULL, PML_PAIR>(g, f, c, S, free_top, q, a, ga, i, j, k, wx, wy);
        } else {
            int how = DIV_FAST;
            if (!ANY) how = str_pml_cell<T, C, DIV_FAST, PML_PAIR>(g, f, c, S, free_top, q, a, ga, i, j, k, wx, wy);
            else if (c.pml_form <= PML_SIGNED) how = str_pml_cell<T, C, DIV_FAST, PML_SIGNED>(g, f, c, S, free_top, q, a, ga, i, j, k, wx, wy);
            else if (c.pml_form == PML_STEPS) how = str_pml_cell<T, C, DIV_FAST, PML_STEPS>(g, f, c, S, free_top, q, a, ga, i, j, k, wx, wy);
            else str_pml_cell<T, C, DIV_FULL, PML_EXACT>(g, f, c, S, free_top, q, a, ga, i, j, k, wx, wy);
            if (how == DIV_TINY) {  // the same again: nothing is stored yet
                if (ANY) {
                    str_pml_redo<T, C, DIV_TINY>(&g, &f, &X, &c, &S, free_top, a, ga, i, j, k, wx, wy);
                } else {
                    asm volatile("" ::: "memory");  // (the inputs are loaded anew, not kept in registers)
                    q.load(g, f, X, S, i, j, k, wx, wy);
                    str_pml_cell<T, C, DIV_TINY, PML_PAIR>(g, f, c, S, free_top, q, a, ga, i, j, k, wx, wy);
                }
            } else if (how == DIV_FULL) {
                str_pml_redo<T, C, DIV_FULL>(&g, &f, &X, &c, &S, free_top, a, ga, i, j, k, wx, wy);
            }
        }
    }
    return true;
}

// pml_xyz in the strips (fd3d_deriv.f90:2304-3143), one tile per CTA as vel_pml_tile
template <class T, bool SLAB, bool ANY>
__device__ __forceinline__ bool str_pml_tile(const Grid& g, const Fields<T>& f, const PmlDesc& D, const PmlAux<T>& X,
                                             const StepConst<T>& c, int tile, T* sm, uint32_t bar, int* status) {
    const long long t0 = (long long)tile * PML_TILE;
    const int s = pml_tile_strip(D, t0);
    switch (pml_class(s)) {
        case 0: return str_pml_tile_c<T, 0, SLAB, ANY>(g, f, D, X, c, s, t0, sm, bar, status);
        case 1: return str_pml_tile_c<T, 1, SLAB, ANY>(g, f, D, X, c, s, t0, sm, bar, status);
        default: return str_pml_tile_c<T, 2, SLAB, ANY>(g, f, D, X, c, s, t0, sm, bar, status);
    }
}

// fres (fd3d_deriv.f90:1067-1104), all loads before the stores
template <class T>
__device__ __forceinline__ void str_fs_body(const Grid& g, const Fields<T>& f, int i, int j) {
    if (i > g.nxt || j > g.nyt) return;
    const long long p = g.at(i, j, g.ks()), sz = g.plane;
    const T z0 = f.zz[p], z1 = f.zz[p - sz], x1 = f.xz[p - sz], x2 = f.xz[p - 2 * sz], y1 = f.yz[p - sz], y2 = f.yz[p - 2 * sz];
    f.zz[p + sz] = -z0;
    f.zz[p + 2 * sz] = -z1;
    f.xz[p + sz] = -x1;
    f.xz[p + 2 * sz] = -x2;
    f.yz[p + sz] = -y1;
    f.yz[p + 2 * sz] = -y2;
    f.xz[p] = (T)0;
    f.yz[p] = (T)0;
}

// ---------------------------------------------------------------- fault BC
// trial traction, damping, RF (fd3d_theo.f90:233-308).  Under FSPACE the top row k = ks
// takes the interior formula and no ghost row is written (fd3d_theo.f90:260-283).
template <class T>
__device__ __forceinline__ void traction_body(Grid g, Fields<T> f, Fault<T> q, StepConst<T> c, const int* it_dev,
                                              int bx_, int by_, int bz_) {
    const int i = g.nabc + 1 + bx_ * blockDim.x + threadIdx.x;
    const int k = g.kin_lo() + by_ * blockDim.y + threadIdx.y;
    const int ks = g.ks();
    if (i > g.nxt - g.nabc || k > g.kin_hi()) return;
    const long long sy = g.px, sz = g.plane;
    const long long p = g.at(i, g.nyt, k);
    const int n2 = g.at2(i, k);
    const T c1 = c.c1, c2 = c.c2, dht = c.dht, ds = c.damp_s;
    const T* xx = f.xx; const T* xz = f.xz; const T* zz = f.zz;
    const int it = *it_dev;
    const T* avdz_rd = pp_rd(q.avdz, it, q.n2); T* avdz_wr = pp_wr(q.avdz, it, q.n2);
    const T* avdx_rd = pp_rd(q.avdx, it, q.n2); T* avdx_wr = pp_wr(q.avdx, it, q.n2);
    const bool inner = (k < ks) || g.fspace;
    T pdz;
    if (inner)
        pdz = (c1 * (xz[p + 1] - xz[p]) + c2 * (xz[p + 2] - xz[p - 1])) / (T)2 +
              (c1 * (zz[p + sz] - zz[p]) + c2 * (zz[p + 2 * sz] - zz[p - sz])) / (T)2 - f.yz[p - sy];
    else
        pdz = ((xz[p + 1 - sz] - xz[p - sz]) / ((T)2 * (T)4) + (zz[p + sz] - zz[p]) / ((T)2 * (T)2) -
               f.yz[p - sy - sz] / (T)4);
    T av = ds * (pdz - avdz_rd[n2]);
    T rf = pdz + av;
    q.RFz[n2] = rf;
    T tzv;
    if (inner) tzv = -rf - (T)0.5 * f.d[p] * dht * f.w[p];
    else        tzv = -rf - (T)0.5 * f.d[p] * dht * f.w[p] / (T)2;
    q.tzt[n2] = tzv;
    avdz_wr[n2] = pdz;
    const T pdx = (c1 * (xx[p] - xx[p - 1]) + c2 * (xx[p + 1] - xx[p - 2])) / (T)2 +
                  (c1 * (xz[p] - xz[p - sz]) + c2 * (xz[p + sz] - xz[p - 2 * sz])) / (T)2 - f.xy[p - sy];
    av = ds * (pdx - avdx_rd[n2]);
    rf = pdx + av;
    q.RFx[n2] = rf;
    const T txv = -rf - (T)0.5 * f.d[p] * dht * f.u[p];
    q.txt[n2] = txv;
    avdx_wr[n2] = pdx;
    // ghost row nzt-1 (fd3d_theo.f90:304-307); with nfs=2: nzt-1 = ks+1, nzt-2 = ks, nzt-3 = ks-1
    if (!g.fspace && k == ks) q.txt[g.at2(i, ks + 1)] = +txv;
    if (!g.fspace && k == ks - 1) q.tzt[g.at2(i, ks + 1)] = -tzv;
}

// |T| at staggered nodes, friction law, slip, rupture time (fd3d_theo.f90:313-410)
template <class T>
__device__ __forceinline__ void friction_body(Grid g, Fields<T> f, Fault<T> q, StepConst<T> c, int law, FvwScalars s,
                           const int* it_dev, int bx_, int by_, int bz_) {
    const int i = g.nabc + 1 + bx_ * blockDim.x + threadIdx.x;
    const int k = g.kin_lo() + by_ * blockDim.y + threadIdx.y;
    if (i > g.nxt - g.nabc || k > g.kin_hi()) return;
    const int it = *it_dev;
    const double time = (double)it * c.dtA;
    const double* distX_rd = pp_rd(q.distX, it, q.n2);
    double* distX_wr = pp_wr(q.distX, it, q.n2);
    const double dtA = c.dtA, rup = 1.e-3;
    const long long sy = g.px, sz = g.plane;
    (void)sy;
    const int n2 = g.at2(i, k);
    const int e1 = g.at2(i + 1, k), e2 = g.at2(i, k + 1), e3 = g.at2(i + 1, k + 1);
    const int w1i = g.at2(i - 1, k), w2i = g.at2(i, k - 1), w3i = g.at2(i - 1, k - 1);
    const T* txt = q.txt; const T* tzt = q.tzt; const T* T0X = q.T0X; const T* T0Z = q.T0Z;
    T tint = (txt[n2] + T0X[n2] + txt[e1] + T0X[e1] + txt[e2] + T0X[e2] + txt[e3] + T0X[e3]) / (T)4;
    const T szv = tzt[n2] + T0Z[n2];
    const T tabsZ = sqrt(tint * tint + szv * szv);
    tint = (tzt[n2] + T0Z[n2] + tzt[w1i] + T0Z[w1i] + tzt[w2i] + T0Z[w2i] + tzt[w3i] + T0Z[w3i]) / (T)4;
    const T sxv = txt[n2] + T0X[n2];
    const T tabsX = sqrt(sxv * sxv + tint * tint);
    q.tabsZ[n2] = tabsZ;
    q.tabsX[n2] = tabsX;
    const long long p = g.at(i, g.nyt, k);
    const T U = f.u[p], W = f.w[p];
    // Z nodes (fd3d_theo.f90:326-373)
    {
        const T uZ = (U + f.u[p + 1] + f.u[p + sz] + f.u[p + 1 + sz]) / (T)4;
        q.uZ[n2] = uZ;
        const T u1out = -sqrt(W * W + uZ * uZ);
        T tzn = tzt[n2];
        if (law == 1) {
            const double a = (double)q.aZ[n2];
            const double s1 = 2.0 * (fabs((double)W) + fabs(s.wini)), s2 = 2.0 * (fabs((double)uZ) + fabs(s.uini));
            const double sr = sqrt(s1 * s1 + s2 * s2);
            const double flv = s.f0 - ((double)q.bZ[n2] - a) * log(sr / s.v0);
            const double fw = (double)q.fwZ[n2];
            const double fss = fw + (flv - fw) / pow(1.0 + pow(sr / (double)q.vwZ[n2], 8.0), 1.0 / 8.0);
            const double psiss = a * (log(sinh(fss / a)) + log(2.0 * s.v0 / sr));
            const double psi = (q.psiZ[n2] - psiss) * exp(-sr * dtA / (double)q.Dc[n2]) + psiss;
            q.psiZ[n2] = psi;
            const double fric = s.Sn * a * asinh(sr * exp(psi / a) / (2.0 * s.v0));
            q.distZ[n2] = q.distZ[n2] - 2.0 * (double)u1out * dtA;
            q.schangeZ[n2] = (T)fric;
            if (fabs(2.0 * (double)u1out) > rup) {
                if (q.ruptime[n2] != 1.e4) q.rise[n2] = time;
                if (q.ruptime[n2] == 1.e4) q.ruptime[n2] = time;
            }
        } else {
            const double dz = q.distZ[n2], dcz = (double)q.DcZ[n2];
            double fric;
            if (dz <= dcz) fric = (double)q.peakZ[n2] * (1.0 - dz / dcz) + (double)q.dynZ[n2] * dz / dcz + (double)q.coh[n2];
            else           fric = (double)q.dynZ[n2] + (double)q.coh[n2];
            if ((double)tabsZ >= fric) {
                q.distZ[n2] = dz - 2.0 * (double)u1out * dtA;
                tzn = (T)(((double)tzn + (double)T0Z[n2]) * fric / (double)tabsZ - (double)T0Z[n2]);
                if (-2.0 * (double)u1out > rup) {
                    if (q.ruptime[n2] != 1.e4) q.rise[n2] = time;
                    if (q.ruptime[n2] == 1.e4) q.ruptime[n2] = time;
                }
            }
        }
        q.tz[n2] = tzn;
        q.slipZ[n2] = q.slipZ[n2] - 2.0 * (double)W * dtA;
        q.slipX[n2] = q.slipX[n2] - 2.0 * (double)uZ * dtA;
        if (q.sliptime[n2] == 1.e4 && q.distZ[n2] > (double)q.Dc[n2]) q.sliptime[n2] = time;
    }
    // X nodes (fd3d_theo.f90:375-410)
    {
        const T wX = (W + f.w[p - 1] + f.w[p - sz] + f.w[p - 1 - sz]) / (T)4;
        q.wX[n2] = wX;
        const T u1out = -sqrt(wX * wX + U * U);
        T txn = txt[n2];
        if (law == 1) {
            const double a = (double)q.aX[n2];
            const double s1 = 2.0 * (fabs((double)wX) + fabs(s.wini)), s2 = 2.0 * (fabs((double)U) + fabs(s.uini));
            const double sr = sqrt(s1 * s1 + s2 * s2);
            const double flv = s.f0 - ((double)q.bX[n2] - a) * log(sr / s.v0);
            const double fw = (double)q.fwX[n2];
            const double fss = fw + (flv - fw) / pow(1.0 + pow(sr / (double)q.vwX[n2], 8.0), 1.0 / 8.0);
            const double psiss = a * (log(sinh(fss / a)) + log(2.0 * s.v0 / sr));
            const double psi = (q.psiX[n2] - psiss) * exp(-sr * dtA / (double)q.Dc[n2]) + psiss;
            q.psiX[n2] = psi;
            const double fric = s.Sn * a * asinh(sr * exp(psi / a) / (2.0 * s.v0));
            distX_wr[n2] = distX_rd[n2] - 2.0 * (double)u1out * dtA;
            q.schangeX[n2] = (T)fric;
        } else {
            const double dx = distX_rd[n2], dcx = (double)q.DcX[n2];
            double fric;
            if (dx <= (double)q.Dc[n2]) fric = (double)q.peakX[n2] * (1.0 - dx / dcx) + (double)q.dynX[n2] * dx / dcx + (double)q.coh[n2];
            else                        fric = (double)q.dynX[n2] + (double)q.coh[n2];
            if ((double)tabsX >= fric) {
                distX_wr[n2] = dx - 2.0 * (double)u1out * dtA;
                txn = (T)(((double)txn + (double)T0X[n2]) * fric / (double)tabsX - (double)T0X[n2]);
            } else {
                distX_wr[n2] = dx;  // carried into this step's plane
            }
        }
        q.tx[n2] = txn;
    }
    if (k == g.ks()) {  // the reference's tx/tz arrays also carry the ghost row nzt-1
        const int gh = g.at2(i, k + 1);
        q.tx[gh] = txt[gh];
        q.tz[gh] = tzt[gh];
    }
}

struct HistDesc {
    void* ring;         // [cap][nf][nzT][nxT] of T
    int cap, stride, nf;
    int nst;
    int sta[3 * 10];    // station (i,j,k)
    void* seis;         // [cap][nst*3] of T
};

// output planes, stations, history ring (fd3d_theo.f90:413-467); non-finite check
template <class T>
__device__ __forceinline__ void output_body(Grid g, Fields<T> f, Fault<T> q, int law, const int* it_dev, const HistDesc& h, int* status, int bx_, int by_, int bz_) {
    const int ii = bx_ * blockDim.x + threadIdx.x;
    const int kk = by_ * blockDim.y + threadIdx.y;
    const int it = *it_dev;
    const bool rec = (it % h.stride) == 0;
    const long long slot = (long long)((it / h.stride - 1) % h.cap);
    const int nxT = g.nxt - 2 * g.nabc, nzT = g.ks() - g.nabc;
    if (rec && ii < h.nst && kk == 0 && g.owns(h.sta[3 * ii + 2])) {
        const long long p = g.at(h.sta[3 * ii], h.sta[3 * ii + 1], h.sta[3 * ii + 2]);
        T* sp = (T*)h.seis + slot * (3 * h.nst) + 3 * ii;
        sp[0] = f.u[p]; sp[1] = f.v[p]; sp[2] = f.w[p];
    }
    const int i = g.nabc + 1 + ii, k = g.kin_lo() + kk;
    if (ii >= nxT || k > g.kin_hi()) return;
    const bool top = (k == g.ks());
    const long long p = g.at(i, g.nyt, k), sz = g.plane;
    const int n2 = g.at2(i, k), e1 = g.at2(i + 1, k), e2 = g.at2(i, k + 1), e3 = g.at2(i + 1, k + 1);
    const T U = f.u[p], U2 = f.u[p + 1], W = f.w[p];
    T srx, srz, scx, scz;
    srz = (T)-2 * W;
    if (!top) {
        const T U3 = f.u[p + sz], U4 = f.u[p + 1 + sz];
        srx = ((T)-2 * U - (T)2 * U2 - (T)2 * U3 - (T)2 * U4) / (T)4;
        if (law == 0) {
            scz = q.tz[n2] + q.T0Z[n2];
            scx = (q.tx[n2] + q.T0X[n2] + q.tx[e1] + q.T0X[e1] + q.tx[e2] + q.T0X[e2] + q.tx[e3] + q.T0X[e3]) / (T)4;
        }
    } else {
        if (law == 1) {
            srx = ((T)-2 * U - (T)2 * U2) / (T)4;
        } else {
            scz = q.tz[n2] + q.T0Z[n2];
            scx = (q.tx[n2] + q.T0X[n2] + q.tx[e1] + q.T0X[e1]) / (T)2;
            srx = ((T)-2 * U - (T)2 * U2) / (T)2;
        }
    }
    if (law == 1) { scx = q.schangeX[n2]; scz = q.schangeZ[n2]; }
    else { q.schangeX[n2] = scx; q.schangeZ[n2] = scz; }
    if (!(isfinite((double)srx) && isfinite((double)srz) && isfinite((double)scx) && isfinite((double)scz)))
        atomicOr(status, ST_NONFINITE);
    if (rec) {
        const long long plane = (long long)nxT * nzT;
        T* r = (T*)h.ring + slot * h.nf * plane + (long long)(k - g.nabc - 1) * nxT + ii;
        r[0] = srx;
        r[plane] = srz;
        r[2 * plane] = scx;
        r[3 * plane] = scz;
        if (h.nf > 4) r[4 * plane] = (T)q.psiZ[n2];
    }
}

// ---------------------------------------------------------------- fused fault BC
// The fault boundary condition of one step in one launch (fd3d_theo.f90:225-467): fres, the
// trial traction, |T| at the staggered nodes, the friction law with slip and rupture time,
// and the output planes.  A CTA owns a FBC_TX x FBC_TZ tile of fault nodes and computes the
// trial tractions of the tile and a one-node ring around it, and the post-friction
// tractions of the X nodes of the tile plus one column and one row beyond, into shared
// memory; the ring values it only reads, so the state it needs from neighbouring nodes is
// the state before this step (the two-plane avdx, avdz and distX of Fault) and nothing
// another CTA writes in the same launch.  fres runs in separate CTAs of the same launch:
// the three stresses it writes that the trial traction reads (zz at ks+1, xz at ks and
// ks+1, fd3d_deriv.f90:1087-1102) are formed from the values fres reads, with the same
// operation (a negation, or the zero it stores).
constexpr int FBC_TX = 32, FBC_TZ = 8;                   // owned nodes of a tile (CTA of 32 x 8 threads)
constexpr int FBC_HX = FBC_TX + 2, FBC_HZ = FBC_TZ + 2;  // trial tractions: the tile and a one-node ring
constexpr int FBC_PX = FBC_TX + 1, FBC_PZ = FBC_TZ + 1;  // post-friction X-node tractions: tile + 1 in +i, +k
constexpr int FBC_SMEM = 2 * FBC_HX * FBC_HZ + FBC_PX * FBC_PZ;  // elements of T

template <class T>
struct TrialTraction { T pdz, pdx, rfz, rfx, tzv, txv; };

// trial traction at fault node (i,k) (fd3d_theo.f90:233-308), in the operation order of
// traction_body; VIRT: fres has not run yet, its stores are formed here
template <class T, bool VIRT>
__device__ __forceinline__ TrialTraction<T> trial_traction(const Grid& g, const Fields<T>& f, const StepConst<T>& c,
                                                           const T* avdz_rd, const T* avdx_rd, int i, int k) {
    const int ks = g.ks();
    const bool virt = VIRT && !g.fspace;
    const long long sy = g.px;
    auto XZ = [&](int ii, int kk) -> T {
        if (virt && kk == ks) return (T)0;                                 // xz(i,nyt,nzt-nfs) = 0
        if (virt && kk == ks + 1) return -f.xz[g.at(ii, g.nyt, ks - 1)];   // xz(ks+1) = -xz(ks-1)
        return f.xz[g.at(ii, g.nyt, kk)];
    };
    auto ZZ = [&](int kk) -> T {
        if (virt && kk == ks + 1) return -f.zz[g.at(i, g.nyt, ks)];        // zz(ks+1) = -zz(ks)
        return f.zz[g.at(i, g.nyt, kk)];
    };
    const long long p = g.at(i, g.nyt, k);
    const int n2 = g.at2(i, k);
    const T c1 = c.c1, c2 = c.c2, dht = c.dht, ds = c.damp_s;
    const T* xx = f.xx;
    const bool inner = (k < ks) || g.fspace;
    TrialTraction<T> t;
    if (inner)
        t.pdz = (c1 * (XZ(i + 1, k) - XZ(i, k)) + c2 * (XZ(i + 2, k) - XZ(i - 1, k))) / (T)2 +
                (c1 * (ZZ(k + 1) - ZZ(k)) + c2 * (ZZ(k + 2) - ZZ(k - 1))) / (T)2 - f.yz[p - sy];
    else
        t.pdz = ((XZ(i + 1, k - 1) - XZ(i, k - 1)) / ((T)2 * (T)4) + (ZZ(k + 1) - ZZ(k)) / ((T)2 * (T)2) -
                 f.yz[p - sy - g.plane] / (T)4);
    T av = ds * (t.pdz - avdz_rd[n2]);
    t.rfz = t.pdz + av;
    if (inner) t.tzv = -t.rfz - (T)0.5 * f.d[p] * dht * f.w[p];
    else       t.tzv = -t.rfz - (T)0.5 * f.d[p] * dht * f.w[p] / (T)2;
    t.pdx = (c1 * (xx[p] - xx[p - 1]) + c2 * (xx[p + 1] - xx[p - 2])) / (T)2 +
            (c1 * (XZ(i, k) - XZ(i, k - 1)) + c2 * (XZ(i, k + 1) - XZ(i, k - 2))) / (T)2 - f.xy[p - sy];
    av = ds * (t.pdx - avdx_rd[n2]);
    t.rfx = t.pdx + av;
    t.txv = -t.rfx - (T)0.5 * f.d[p] * dht * f.u[p];
    return t;
}

// What the friction law reads at a node beside the trial tractions, loaded before them where the
// CTA has a thread for every node (fault_bc_body).  p0..p3: the law's parameters, slip weakening
// peak, dynamic, Dc (DcX) and cohesion; rate-and-state a, b, vw and fw.
template <class T>
struct FricZ {  // Z node
    T t0z, t0x, t0x1, t0x2, t0x3, U, U1, U2, U3, W, p0, p1, p2, p3, Dc;
    double dist, slipZ, slipX, rt, st, psi;
    __device__ __forceinline__ void load(const Grid& g, const Fields<T>& f, const Fault<T>& q, int law, int i, int k) {
        const int n2 = g.at2(i, k), e1 = g.at2(i + 1, k), e2 = g.at2(i, k + 1), e3 = g.at2(i + 1, k + 1);
        const long long p = g.at(i, g.nyt, k), sz = g.plane;
        t0z = q.T0Z[n2]; t0x = q.T0X[n2]; t0x1 = q.T0X[e1]; t0x2 = q.T0X[e2]; t0x3 = q.T0X[e3];
        U = f.u[p]; U1 = f.u[p + 1]; U2 = f.u[p + sz]; U3 = f.u[p + 1 + sz]; W = f.w[p];
        if (law == 1) { p0 = q.aZ[n2]; p1 = q.bZ[n2]; p2 = q.vwZ[n2]; p3 = q.fwZ[n2]; psi = q.psiZ[n2]; }
        else { p0 = q.peakZ[n2]; p1 = q.dynZ[n2]; p2 = q.DcZ[n2]; p3 = q.coh[n2]; }
        Dc = q.Dc[n2];
        dist = q.distZ[n2]; slipZ = q.slipZ[n2]; slipX = q.slipX[n2]; rt = q.ruptime[n2]; st = q.sliptime[n2];
    }
};
template <class T>
struct FricX {  // X node
    T t0x, t0z, t0z1, t0z2, t0z3, U, W, W1, W2, W3, p0, p1, p2, p3, Dc;
    double dist, psi;
    __device__ __forceinline__ void load(const Grid& g, const Fields<T>& f, const Fault<T>& q, int law,
                                         const double* distX_rd, int i, int k) {
        const int n2 = g.at2(i, k), w1 = g.at2(i - 1, k), w2 = g.at2(i, k - 1), w3 = g.at2(i - 1, k - 1);
        const long long p = g.at(i, g.nyt, k), sz = g.plane;
        t0x = q.T0X[n2]; t0z = q.T0Z[n2]; t0z1 = q.T0Z[w1]; t0z2 = q.T0Z[w2]; t0z3 = q.T0Z[w3];
        U = f.u[p]; W = f.w[p]; W1 = f.w[p - 1]; W2 = f.w[p - sz]; W3 = f.w[p - 1 - sz];
        if (law == 1) { p0 = q.aX[n2]; p1 = q.bX[n2]; p2 = q.vwX[n2]; p3 = q.fwX[n2]; psi = q.psiX[n2]; }
        else { p0 = q.peakX[n2]; p1 = q.dynX[n2]; p2 = q.DcX[n2]; p3 = q.coh[n2]; }
        Dc = q.Dc[n2];
        dist = distX_rd[n2];
    }
};

// strength and new state variable of the rate-and-state law (fd3d_theo.f90:333-350): v1, v2 the
// two velocity components at the node
__device__ __forceinline__ double fvw_strength(const FvwScalars& s, double v1, double v2, double a, double b, double vw,
                                               double fw, double Dc, double dtA, double psi0, double& psi) {
    const double s1 = 2.0 * (fabs(v1) + fabs(s.wini)), s2 = 2.0 * (fabs(v2) + fabs(s.uini));
    const double sr = sqrt(s1 * s1 + s2 * s2);
    const double flv = s.f0 - (b - a) * log(sr / s.v0);
    const double fss = fw + (flv - fw) / pow(1.0 + pow(sr / vw, 8.0), 1.0 / 8.0);
    const double psiss = a * (log(sinh(fss / a)) + log(2.0 * s.v0 / sr));
    psi = (psi0 - psiss) * exp(-sr * dtA / Dc) + psiss;
    return s.Sn * a * asinh(sr * exp(psi / a) / (2.0 * s.v0));
}

// Friction at the X node (i,k) (fd3d_theo.f90:375-410): returns the traction after friction;
// own: also the node's state (tabsX, wX, slip path, psi, strength).
template <class T>
__device__ __forceinline__ T friction_x(const Grid& g, const Fault<T>& q, const StepConst<T>& c, int law,
                                        const FvwScalars& s, const FricX<T>& x, double* distX_wr, T txt0, T tint, bool own,
                                        int i, int k) {
    const int n2 = g.at2(i, k);
    const double dtA = c.dtA;
    const T sxv = txt0 + x.t0x;
    const T tabsX = sqrt(sxv * sxv + tint * tint);
    const T wX = (x.W + x.W1 + x.W2 + x.W3) / (T)4;
    const T u1out = -sqrt(wX * wX + x.U * x.U);
    T txn = txt0;
    if (own) { q.tabsX[n2] = tabsX; q.wX[n2] = wX; }
    if (law == 1) {
        if (own) {
            double psi;
            const double fric = fvw_strength(s, (double)wX, (double)x.U, (double)x.p0, (double)x.p1, (double)x.p2,
                                             (double)x.p3, (double)x.Dc, dtA, x.psi, psi);
            q.psiX[n2] = psi;
            distX_wr[n2] = x.dist - 2.0 * (double)u1out * dtA;
            q.schangeX[n2] = (T)fric;
        }
    } else {
        const double dx = x.dist, dcx = (double)x.p2;
        double fric;
        if (dx <= (double)x.Dc) fric = (double)x.p0 * (1.0 - dx / dcx) + (double)x.p1 * dx / dcx + (double)x.p3;
        else                    fric = (double)x.p1 + (double)x.p3;
        double dnew = dx;
        if ((double)tabsX >= fric) {
            dnew = dx - 2.0 * (double)u1out * dtA;
            txn = (T)(((double)txn + (double)x.t0x) * fric / (double)tabsX - (double)x.t0x);
        }
        if (own) distX_wr[n2] = dnew;
    }
    if (own) q.tx[n2] = txn;
    return txn;
}

// Friction at the Z node (i,k) (fd3d_theo.f90:326-373): state, slip, rupture time; returns tz and,
// rate-and-state, the strength.
template <class T>
__device__ __forceinline__ T friction_z(const Grid& g, const Fault<T>& q, const StepConst<T>& c, int law,
                                        const FvwScalars& s, const FricZ<T>& z, double time, T tzt0, T tint, int i, int k,
                                        T& strength, T& psi_out) {
    const int n2 = g.at2(i, k);
    const double dtA = c.dtA, rup = 1.e-3;
    const T szv = tzt0 + z.t0z;
    const T tabsZ = sqrt(tint * tint + szv * szv);
    q.tabsZ[n2] = tabsZ;
    const T uZ = (z.U + z.U1 + z.U2 + z.U3) / (T)4;
    q.uZ[n2] = uZ;
    const T u1out = -sqrt(z.W * z.W + uZ * uZ);
    T tzn = tzt0;
    double dist = z.dist;
    bool moving;
    if (law == 1) {
        double psi;
        const double fric = fvw_strength(s, (double)z.W, (double)uZ, (double)z.p0, (double)z.p1, (double)z.p2,
                                         (double)z.p3, (double)z.Dc, dtA, z.psi, psi);
        q.psiZ[n2] = psi;
        dist = z.dist - 2.0 * (double)u1out * dtA;
        strength = (T)fric;
        psi_out = (T)psi;
        q.schangeZ[n2] = strength;
        moving = fabs(2.0 * (double)u1out) > rup;
    } else {
        const double dz = z.dist, dcz = (double)z.p2;
        double fric;
        if (dz <= dcz) fric = (double)z.p0 * (1.0 - dz / dcz) + (double)z.p1 * dz / dcz + (double)z.p3;
        else           fric = (double)z.p1 + (double)z.p3;
        const bool slips = (double)tabsZ >= fric;
        if (slips) {
            dist = dz - 2.0 * (double)u1out * dtA;
            tzn = (T)(((double)tzn + (double)z.t0z) * fric / (double)tabsZ - (double)z.t0z);
        }
        moving = slips && -2.0 * (double)u1out > rup;
    }
    q.distZ[n2] = dist;
    if (moving) {
        if (z.rt != 1.e4) q.rise[n2] = time;
        else q.ruptime[n2] = time;
    }
    q.tz[n2] = tzn;
    q.slipZ[n2] = z.slipZ - 2.0 * (double)z.W * dtA;
    q.slipX[n2] = z.slipX - 2.0 * (double)uZ * dtA;
    if (z.st == 1.e4 && dist > (double)z.Dc) q.sliptime[n2] = time;
    return tzn;
}

// One tile of the fused fault boundary condition (without fres) on a CTA of NT threads (thread
// tid); sm holds FBC_SMEM elements.
//
// Bound by latency: a small grid has one tile per SM or less.  With FBC_THREADS each trial
// traction of the tile and its ring, each Z node and each X node has a thread of its own, and what
// the friction law reads is loaded before the trial tractions, so a tile is two rounds of memory
// latency and one friction law long.  With 256 threads the same parts run one after the other.
// One launch, us (before: 256 threads, loads in the law): slip weakening, 50 tiles 11.3 (17.1), 1250
// tiles 69 (72).
constexpr int FBC_THREADS = 576;  // >= 256 Z nodes + 297 X nodes, and the 340 trial tractions
template <class T, int NT>
__device__ __forceinline__ void fault_bc_body(const Grid& g, const Fields<T>& f, const Fault<T>& q,
                                              const StepConst<T>& c, int law, const FvwScalars& s, const int* it_dev,
                                              const HistDesc& h, int* status, int bx_, int by_, T* sm, int tid) {
    constexpr int NZ = FBC_TX * FBC_TZ, NXH = FBC_PX * FBC_PZ - NZ;  // own nodes; X nodes of the column and row beyond
    constexpr bool ALL = NT >= NZ + NZ + NXH;
    const int i0 = g.nabc + 1 + bx_ * FBC_TX, k0 = g.nabc + 1 + by_ * FBC_TZ;
    const int ie = g.nxt - g.nabc, ks = g.ks();
    const int it = *it_dev;
    const T* avdz_rd = pp_rd(q.avdz, it, q.n2); T* avdz_wr = pp_wr(q.avdz, it, q.n2);
    const T* avdx_rd = pp_rd(q.avdx, it, q.n2); T* avdx_wr = pp_wr(q.avdx, it, q.n2);
    const double* distX_rd = pp_rd(q.distX, it, q.n2); double* distX_wr = pp_wr(q.distX, it, q.n2);
    T* s_txt = sm;                        // [FBC_HZ][FBC_HX], node (i,k) at (i-i0+1) + (k-k0+1)*FBC_HX
    T* s_tzt = sm + FBC_HX * FBC_HZ;
    T* s_tx = sm + 2 * FBC_HX * FBC_HZ;   // [FBC_PZ][FBC_PX], node (i,k) at (i-i0) + (k-k0)*FBC_PX

    // the Z node of a thread below NZ, and the n-th X node: the tile's, then the column
    // i0+FBC_TX (k0..k0+FBC_TZ), then the row k0+FBC_TZ (i0..i0+FBC_TX-1)
    const int i = i0 + tid % FBC_TX, k = k0 + tid / FBC_TX;
    const bool own = tid < NZ && i <= ie && k <= ks;
    auto x_node = [&](int n, int& xi, int& xk) {
        if (n < NZ) { xi = i0 + n % FBC_TX; xk = k0 + n / FBC_TX; }
        else if (n < NZ + FBC_PZ) { xi = i0 + FBC_TX; xk = k0 + n - NZ; }
        else { xi = i0 + n - NZ - FBC_PZ; xk = k0 + FBC_TZ; }
        return n < NZ + NXH && xi <= ie && xk <= ks;
    };
    FricZ<T> z;
    FricX<T> x;
    int xi = 0, xk = 0;
    bool has_x = false;
    if (ALL) {
        if (own) z.load(g, f, q, law, i, k);
        has_x = tid >= NZ && x_node(tid - NZ, xi, xk);
        if (has_x) x.load(g, f, q, law, distX_rd, xi, xk);
    }

    // 1. trial tractions of the tile and its ring; the owner stores a node's state
    for (int n = tid; n < FBC_HX * FBC_HZ; n += NT) {
        const int ri = n % FBC_HX, rk = n / FBC_HX;
        const int ti = i0 - 1 + ri, tk = k0 - 1 + rk;
        T tx_ = 0, tz_ = 0;   // outside the traction loops the reference's tx, tz stay 0
        if (ti >= g.nabc + 1 && ti <= ie) {
            if (tk >= g.nabc + 1 && tk <= ks) {
                const TrialTraction<T> t = trial_traction<T, true>(g, f, c, avdz_rd, avdx_rd, ti, tk);
                tx_ = t.txv;
                tz_ = t.tzv;
                if (ri >= 1 && ri <= FBC_TX && rk >= 1 && rk <= FBC_TZ) {
                    const int n2 = g.at2(ti, tk);
                    q.RFz[n2] = t.rfz;
                    q.RFx[n2] = t.rfx;
                    avdz_wr[n2] = t.pdz;
                    avdx_wr[n2] = t.pdx;
                }
            } else if (!g.fspace && tk == ks + 1) {  // ghost row: tx(nzt-1) = tx(nzt-2), tz(nzt-1) = -tz(nzt-3)
                tx_ = +trial_traction<T, true>(g, f, c, avdz_rd, avdx_rd, ti, ks).txv;
                tz_ = -trial_traction<T, true>(g, f, c, avdz_rd, avdx_rd, ti, ks - 1).tzv;
            }
        }
        s_txt[n] = tx_;
        s_tzt[n] = tz_;
    }
    __syncthreads();
    auto TXT = [&](int ii, int kk) { return s_txt[(ii - i0 + 1) + (kk - k0 + 1) * FBC_HX]; };
    auto TZT = [&](int ii, int kk) { return s_tzt[(ii - i0 + 1) + (kk - k0 + 1) * FBC_HX]; };

    // 2. friction at the Z nodes of the tile and at its X nodes with those of the column and row
    //    beyond it (their tractions after friction, for the output)
    T tzn = 0, strength = 0, psi = 0;
    if (own) {
        if (!ALL) z.load(g, f, q, law, i, k);
        const T tint = (TXT(i, k) + z.t0x + TXT(i + 1, k) + z.t0x1 + TXT(i, k + 1) + z.t0x2 + TXT(i + 1, k + 1) +
                        z.t0x3) / (T)4;
        tzn = friction_z<T>(g, q, c, law, s, z, (double)it * c.dtA, TZT(i, k), tint, i, k, strength, psi);
        if (k == ks) {  // the reference's tx/tz arrays also carry the ghost row nzt-1
            const int gh = g.at2(i, k + 1);
            q.tx[gh] = TXT(i, k + 1);
            q.tz[gh] = TZT(i, k + 1);
        }
    }
    auto do_x = [&](int n) {
        T t = 0;   // beyond the interior plane the reference's tx stays 0
        if (has_x) {
            if (law == 1 && n >= NZ) {
                t = TXT(xi, xk);
            } else {
                const T tint = (TZT(xi, xk) + x.t0z + TZT(xi - 1, xk) + x.t0z1 + TZT(xi, xk - 1) + x.t0z2 +
                                TZT(xi - 1, xk - 1) + x.t0z3) / (T)4;
                t = friction_x<T>(g, q, c, law, s, x, distX_wr, TXT(xi, xk), tint, n < NZ, xi, xk);
            }
        }
        s_tx[(xi - i0) + (xk - k0) * FBC_PX] = t;
    };
    if (ALL) {
        if (tid >= NZ && tid < NZ + NZ + NXH) do_x(tid - NZ);
    } else {
        for (int n = tid; n < NZ + NXH; n += NT) {
            has_x = x_node(n, xi, xk);
            if (has_x) x.load(g, f, q, law, distX_rd, xi, xk);
            do_x(n);
        }
    }
    __syncthreads();

    // 3. output planes, stations, history ring (fd3d_theo.f90:413-467) of the tile's nodes
    if (bx_ == 0 && by_ == 0 && tid < h.nst && it % h.stride == 0) {
        const long long slot = (long long)((it / h.stride - 1) % h.cap);
        const long long p = g.at(h.sta[3 * tid], h.sta[3 * tid + 1], h.sta[3 * tid + 2]);
        T* sp = (T*)h.seis + slot * (3 * h.nst) + 3 * tid;
        sp[0] = f.u[p]; sp[1] = f.v[p]; sp[2] = f.w[p];
    }
    if (!own) return;
    auto TX = [&](int ii, int kk) { return s_tx[(ii - i0) + (kk - k0) * FBC_PX]; };
    const bool top = (k == ks);
    const int n2 = g.at2(i, k);
    T srx, srz, scx, scz;
    srz = (T)-2 * z.W;
    if (!top) {
        srx = ((T)-2 * z.U - (T)2 * z.U1 - (T)2 * z.U2 - (T)2 * z.U3) / (T)4;
        if (law == 0) {
            scz = tzn + z.t0z;
            scx = (TX(i, k) + z.t0x + TX(i + 1, k) + z.t0x1 + TX(i, k + 1) + z.t0x2 + TX(i + 1, k + 1) + z.t0x3) / (T)4;
        }
    } else {
        if (law == 1) {
            srx = ((T)-2 * z.U - (T)2 * z.U1) / (T)4;
        } else {
            scz = tzn + z.t0z;
            scx = (TX(i, k) + z.t0x + TX(i + 1, k) + z.t0x1) / (T)2;
            srx = ((T)-2 * z.U - (T)2 * z.U1) / (T)2;
        }
    }
    if (law == 1) { scx = q.schangeX[n2]; scz = strength; }  // (schangeX: this CTA's X node, before the barrier)
    else { q.schangeX[n2] = scx; q.schangeZ[n2] = scz; }
    if (!(isfinite((double)srx) && isfinite((double)srz) && isfinite((double)scx) && isfinite((double)scz)))
        atomicOr(status, ST_NONFINITE);
    if (it % h.stride == 0) {
        const int nxT = g.nxt - 2 * g.nabc, nzT = ks - g.nabc;
        const long long slot = (long long)((it / h.stride - 1) % h.cap);
        const long long plane = (long long)nxT * nzT;
        T* r = (T*)h.ring + slot * h.nf * plane + (long long)(k - g.nabc - 1) * nxT + (i - g.nabc - 1);
        r[0] = srx;
        r[plane] = srz;
        r[2 * plane] = scx;
        r[3 * plane] = scz;
        if (h.nf > 4) r[4 * plane] = psi;
    }
}

// grid of the fused fault BC: fres CTAs (32 x rows (i,j) each), then the fault tiles
inline void fault_bc_grid(const Grid& g, int rows, int& nfres, int& tiles_x, int& tiles) {
    nfres = g.fspace ? 0 : ((g.nxt + 31) / 32) * ((g.nyt + rows - 1) / rows);
    const int nxT = g.nxt - 2 * g.nabc, nzT = g.ks() - g.nabc;
    tiles_x = (nxT + FBC_TX - 1) / FBC_TX;
    tiles = tiles_x * ((nzT + FBC_TZ - 1) / FBC_TZ);
}

// TPV103/104 smooth nucleation of T0X (fd3d_theo.f90:487-542)
template <class T>
__device__ __forceinline__ void nucleation_body(Grid g, Fault<T> q, StepConst<T> c, FvwScalars s, const int* it_dev, int bx_, int by_, int bz_) {
    const int i = g.nabc - 1 + bx_ * blockDim.x + threadIdx.x;
    const int k = g.nabc - 1 + by_ * blockDim.y + threadIdx.y;
    if (i > g.nxt - g.nabc || k > g.ks()) return;
    const double time = (double)(*it_dev) * c.dtA;
    const double th = time - c.dtA / 2.0;
    if (!(th <= s.TT2)) return;
    const double GT = (th < s.TT2) ? exp((th - s.TT2) * (th - s.TT2) / (th * (th - 2.0 * s.TT2))) : 1.0;
    const double hx = (double)i * c.dhA, hz = (double)k * c.dhA;
    const double rr = (hx - s.hx0) * (hx - s.hx0) + (hz - s.hz0) * (hz - s.hz0);
    const double FXZ = (rr < s.RR2 - c.dhA) ? exp(rr / (rr - s.RR2 - c.dhA)) : 0.0;
    const double base = s.nucleation == 2 ? (double)q.T0Xb[g.at2(i, k)] : s.strinixI;
    q.T0X[g.at2(i, k)] = (T)(base + s.perturb * FXZ * GT);
}

// ---------------------------------------------------------------- set-up
// A 1-D layered medium (lam, mu, d per plane in lay, nzt values each) into the padded 3-D
// arrays, whose row padding stays 0; a CTA per row, bound by the stores.  The whole upload call of
// a 0.9 M cell model takes 0.07 ms (5.5 ms with planes filled on the host and copied one by one).
template <class T>
__global__ void k_fill_layers(Grid g, T* lam, T* mu, T* d, const T* lay) {
    const int nrows = g.nyt * g.nzl;  // rows of the stored planes, from kofs+1
    for (int r = blockIdx.x; r < nrows; r += gridDim.x) {
        const int k = g.kofs + 1 + r / g.nyt, j = 1 + r % g.nyt;
        const long long row = g.at(1, j, k) - g.off;
        const T l = lay[k - 1], m = lay[g.nzt + k - 1], dd = lay[2 * g.nzt + k - 1];
        for (int x = threadIdx.x; x < g.px; x += blockDim.x) {
            const bool in = x >= g.off && x < g.off + g.nxt;
            lam[row + x] = in ? l : (T)0;
            mu[row + x] = in ? m : (T)0;
            d[row + x] = in ? dd : (T)0;
        }
    }
}

// ---------------------------------------------------------------- launch wrappers
// A launch, with programmatic stream serialization when pdl is set: the kernel's CTAs may be
// scheduled while the kernel before it drains, and wait in pdl_wait (which such a kernel starts
// with) for its completion.
template <class... K, class... A>
inline cudaError_t launch_kernel(bool pdl, void (*kern)(K...), dim3 grid, dim3 blk, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = blk;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

template <class T>
__global__ void __launch_bounds__(256)
k_vel_fault(const __grid_constant__ Grid g, const __grid_constant__ Fields<T> f, const __grid_constant__ Fault<T> q,
            const __grid_constant__ StepConst<T> c, int law, const __grid_constant__ FvwScalars s, int* it_dev, int* status) {
    vel_fault_body<T>(g, f, q, c, law, s, it_dev, status, blockIdx.x, blockIdx.y, blockIdx.z);
}

// One PML tile per CTA of PML_TILE threads.  MINB: CTAs that must fit one SM
// (register cap); 1 leaves it free.
template <class T, int MINB, bool SLAB, bool ANY>
__global__ void __launch_bounds__(PML_TILE, MINB)
k_vel_pml(const __grid_constant__ Grid g, const __grid_constant__ Fields<T> f, const __grid_constant__ PmlDesc D,
          const __grid_constant__ PmlAux<T> X, const __grid_constant__ StepConst<T> c, int* status, long long tile0) {
    __shared__ __align__(128) T sm[PML_TILE * AUX_NV];
    __shared__ __align__(8) uint64_t bar;
    vel_pml_tile<T, SLAB, ANY>(g, f, D, X, c, tile0 + blockIdx.x, sm, smem_addr(&bar), status);
}

template <class T>
__global__ void k_vel_fs(Grid g, Fields<T> f) {
    pdl_wait();
    pdl_launch_dependents();
    vel_fs_body<T>(g, f, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <class T>
__global__ void __launch_bounds__(256)
k_str_fault(const __grid_constant__ Grid g, const __grid_constant__ Fields<T> f, const __grid_constant__ Fault<T> q,
            const __grid_constant__ StepConst<T> c) {
    str_fault_body<T>(g, f, q, c, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <class T, int MINB, bool SLAB, bool ANY>
__global__ void __launch_bounds__(PML_TILE, MINB)
k_str_pml(const __grid_constant__ Grid g, const __grid_constant__ Fields<T> f, const __grid_constant__ PmlDesc D,
          const __grid_constant__ PmlAux<T> X, const __grid_constant__ StepConst<T> c, int* status, long long tile0) {
    __shared__ __align__(128) T sm[PML_TILE * AUX_NS];
    __shared__ __align__(8) uint64_t bar;
    str_pml_tile<T, SLAB, ANY>(g, f, D, X, c, tile0 + blockIdx.x, sm, smem_addr(&bar), status);
}

// The tiles of strip s that hold cells of planes klo..khi: [t0, t1) (k is the slowest
// index of a strip's compact range)
inline void pml_strip_tiles(const PmlDesc& D, int s, long long& t0, long long& t1) {
    const Strip& S = D.s[s];
    const int kb = std::max(S.nzb, D.klo), ke = std::min(S.nze, D.khi);
    t0 = t1 = D.cum[s] / PML_TILE;
    if (D.cnt[s] == 0 || kb > ke) return;
    const long long per_k = D.cnt[s] / S.nk;
    t0 = (D.cum[s] + (long long)(kb - S.nzb) * per_k) / PML_TILE;
    t1 = (D.cum[s] + (long long)(ke - S.nzb + 1) * per_k + PML_TILE - 1) / PML_TILE;
}

// CTAs per SM that the PML sweeps are compiled for, measured fastest.  0.214 G cells, us: velocity 293
// at 4 (330 at 3, 72 registers), stress 389 at 4 (424 at 3; 5 spills, 399); FP64 (0.6 M cells) 20 at 3, 30
// at 2 (no spills).  A z-slab (us a step of two slabs of 14 M and 68 M cells: 519 and 1641 against 539 and
// 1684 without a cap) and quotients of a form of their own always take these.
template <class T>
constexpr int pml_minb(bool stress) { return sizeof(T) == 4 ? 4 : stress ? 2 : 3; }
template <class T>
using PmlKernel = void (*)(Grid, Fields<T>, PmlDesc, PmlAux<T>, StepConst<T>, int*, long long);
template <class T, bool STRESS, bool SLAB, bool ANY, int MINB = pml_minb<T>(STRESS)>
constexpr PmlKernel<T> pml_kernel_of() {
    if constexpr (STRESS) return k_str_pml<T, MINB, SLAB, ANY>;
    else return k_vel_pml<T, MINB, SLAB, ANY>;
}
// the kernels of quotients with a form of their own, in a module of their own (fd3d_forms.cu): a
// program whose models do not take them does not load them
PmlKernel<float> pml_kernel_forms(bool stress, bool slab);
template <class T, bool STRESS>
inline PmlKernel<T> pml_kernel(int minb, bool slab, bool any) {
    if constexpr (sizeof(T) == 4)  // (FP64 divides directly: one form)
        if (any) return pml_kernel_forms(STRESS, slab);
    if (slab) return pml_kernel_of<T, STRESS, true, false>();
    switch (minb) {
        case 2: return pml_kernel_of<T, STRESS, false, false, 2>();
        case 3: return pml_kernel_of<T, STRESS, false, false, 3>();
        case 4: return pml_kernel_of<T, STRESS, false, false, 4>();
        case 5: return pml_kernel_of<T, STRESS, false, false, 5>();
        default: return pml_kernel_of<T, STRESS, false, false, 1>();
    }
}
template <class T>
inline PmlKernel<T> pml_kernel(bool stress, int minb, bool slab, bool any) {
    return stress ? pml_kernel<T, true>(minb, slab, any) : pml_kernel<T, false>(minb, slab, any);
}
inline bool pml_slab(const Grid& g, const PmlDesc& D) { return D.klo > 1 || D.khi < g.nzt; }

// launch of a PML sweep: one launch over every tile for a whole model (with a register
// cap picked at run time), one per strip over the tiles of its planes for a z-slab
template <class T>
inline void launch_pml(bool stress, int minb, cudaStream_t st, const Grid& g, const Fields<T>& f, const PmlDesc& D,
                       const PmlAux<T>& X, const StepConst<T>& c, int* status) {
    const bool slab = pml_slab(g, D);
    const PmlKernel<T> k = pml_kernel<T>(stress, minb, slab, c.pml_form != PML_PAIR);
    if (!slab) {
        const unsigned n = (unsigned)(D.cum[PML_MAXS] / PML_TILE);
        if (n) k<<<n, PML_TILE, 0, st>>>(g, f, D, X, c, status, 0);
        return;
    }
    for (int s = 0; s < D.ns; ++s) {
        long long t0, t1;
        pml_strip_tiles(D, s, t0, t1);
        if (t1 > t0) k<<<(unsigned)(t1 - t0), PML_TILE, 0, st>>>(g, f, D, X, c, status, t0);
    }
}

template <class T>
__global__ void k_str_fs(Grid g, Fields<T> f) {
    str_fs_body<T>(g, f, 1 + blockIdx.x * blockDim.x + threadIdx.x, 1 + blockIdx.y * blockDim.y + threadIdx.y);
}

template <class T>
__global__ void k_traction(Grid g, Fields<T> f, Fault<T> q, StepConst<T> c, const int* it_dev) {
    traction_body<T>(g, f, q, c, it_dev, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <class T>
__global__ void k_friction(Grid g, Fields<T> f, Fault<T> q, StepConst<T> c, int law, FvwScalars s,
                           const int* it_dev) {
    friction_body<T>(g, f, q, c, law, s, it_dev, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <class T>
__global__ void k_output(Grid g, Fields<T> f, Fault<T> q, int law, const int* it_dev, const __grid_constant__ HistDesc h,
                         int* status) {
    output_body<T>(g, f, q, law, it_dev, h, status, blockIdx.x, blockIdx.y, blockIdx.z);
}

// The fused fault boundary condition of one step: nfres CTAs of fres, then the fault tiles
// (tiles_x per row of tiles); CTA of NT threads.  LAW is a template argument for its registers:
// slip weakening in FP32 fits two CTAs of FBC_THREADS per SM (56 registers, 100 B spilled), the others one.
template <class T, int LAW, int NT>
__global__ void __launch_bounds__(NT, NT == 256 ? (sizeof(T) == 4 ? 3 : 2) : LAW == 0 && sizeof(T) == 4 ? 2 : 1)
k_fault_bc(const __grid_constant__ Grid g, const __grid_constant__ Fields<T> f, const __grid_constant__ Fault<T> q,
           const __grid_constant__ StepConst<T> c, const __grid_constant__ FvwScalars s, const int* it_dev,
           const __grid_constant__ HistDesc h, int* status, int nfres, int tiles_x) {
    __shared__ T sm[FBC_SMEM];
    const int b = blockIdx.x;
    pdl_wait();
    pdl_launch_dependents();
    if (b < nfres) {
        const int sx = (g.nxt + 31) / 32;
        str_fs_body<T>(g, f, 1 + b % sx * 32 + threadIdx.x % 32, 1 + b / sx * (NT / 32) + threadIdx.x / 32);
        return;
    }
    const int t = b - nfres;
    fault_bc_body<T, NT>(g, f, q, c, LAW, s, it_dev, h, status, t % tiles_x, t / tiles_x, sm, threadIdx.x);
}

template <class T, int LAW, int NT>
inline void launch_fault_bc_n(bool pdl, cudaStream_t st, const Grid& g, const Fields<T>& f, const Fault<T>& q, const StepConst<T>& c,
                              const FvwScalars& s, const int* it_dev, const HistDesc& h, int* status) {
    int nfres, tiles_x, tiles;
    fault_bc_grid(g, NT / 32, nfres, tiles_x, tiles);
    launch_kernel(pdl, k_fault_bc<T, LAW, NT>, dim3(nfres + tiles), dim3(NT), 0, st, g, f, q, c, s, it_dev, h, status, nfres, tiles_x);
}
// FBC_THREADS threads a tile where two tiles fit an SM (slip weakening, FP32), and elsewhere where
// there are no more tiles than SMs; 256 threads beyond that, since the kernel is then bound by
// the warps it has in flight (rate-and-state, us: 50 tiles 13.9 against 20.5, 950 tiles 78
// against 48.6).
template <class T>
inline void launch_fault_bc(bool pdl, int law, int nsm, cudaStream_t st, const Grid& g, const Fields<T>& f, const Fault<T>& q,
                            const StepConst<T>& c, const FvwScalars& s, const int* it_dev, const HistDesc& h, int* status) {
    int nfres, tiles_x, tiles;
    fault_bc_grid(g, 8, nfres, tiles_x, tiles);
    if (law == 0) {
        if constexpr (sizeof(T) == 4) launch_fault_bc_n<T, 0, FBC_THREADS>(pdl, st, g, f, q, c, s, it_dev, h, status);
        else if (tiles <= nsm) launch_fault_bc_n<T, 0, FBC_THREADS>(pdl, st, g, f, q, c, s, it_dev, h, status);
        else launch_fault_bc_n<T, 0, 256>(pdl, st, g, f, q, c, s, it_dev, h, status);
    } else {
        if (tiles <= nsm) launch_fault_bc_n<T, 1, FBC_THREADS>(pdl, st, g, f, q, c, s, it_dev, h, status);
        else launch_fault_bc_n<T, 1, 256>(pdl, st, g, f, q, c, s, it_dev, h, status);
    }
}

template <class T>
__global__ void k_nucleation(Grid g, Fault<T> q, StepConst<T> c, FvwScalars s, const int* it_dev) {
    pdl_wait();
    pdl_launch_dependents();
    nucleation_body<T>(g, q, c, s, it_dev, blockIdx.x, blockIdx.y, blockIdx.z);
}

}  // namespace fd3d
