// fd3d_common.cuh -- device data layout and launch-wide constants of the B200 path.
//
// Layout in HBM (one model):
//   * 9 wave fields (u,v,w,xx,yy,zz,xy,yz,xz) and 3 media (lam1,mu1,d1), each a
//     separate array of nzt x nyt rows of `px` elements.  Element (i,j,k) of the
//     reference (1-based, x fastest) lives at  off + (i-1) + px*((j-1) + nyt*(k-1)).
//     `off` shifts the row so that i = nabc+1, the first interior column, starts on a
//     128-byte boundary (fp32) and px (a multiple of 32) keeps every row aligned.
//   * fault-plane arrays (i,k) at (i-1) + nxt*(k-1), the reference's own layout.
//   * PML auxiliary (split) components of init_pml (src/fd3d_deriv.f90:1319-1410): one
//     pool indexed by the compact cell index of the strips (4, or 5 under FSPACE), in 32-cell blocks per
//     group of components (PmlAux, fd3d_kernels.cuh).
#pragma once
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

namespace fd3d {

struct Grid {
    int nxt, nyt, nzt, nabc, nfs;
    int fspace;      // FSPACE build: a PML strip above k = ks() instead of the free surface
    int px;          // row pitch (elements)
    int off;         // x offset of i=1 inside a row
    long long plane; // px*nyt
    long long n3;    // plane*nzl + tail pad: the elements of one stored 3-D array
    // z-slab of a model decomposed over several contexts: the context updates planes
    // klo..khi and stores planes kofs+1 .. kofs+nzl (its own and the halo planes of its
    // neighbours).  Field pointers are offset by -kofs planes, so at() takes the global k
    // everywhere.  A whole model: klo = 1, khi = nzt, kofs = 0, nzl = nzt.
    int klo, khi, kofs, nzl;

    __host__ __device__ __forceinline__ long long at(int i, int j, int k) const {
        return (long long)off + (i - 1) + (long long)px * (j - 1) + plane * (k - 1);
    }
    __host__ __device__ __forceinline__ int at2(int i, int k) const { return (i - 1) + nxt * (k - 1); }
    __host__ __device__ __forceinline__ int ks() const { return nzt - nfs; }  // free-surface row (top row of the
                                                                              // interior box under FSPACE)
    __host__ __device__ __forceinline__ bool owns(int k) const { return k >= klo && k <= khi; }
    // the planes of the interior box (and fault rows) this context updates
    __host__ __device__ __forceinline__ int kin_lo() const { return klo > nabc + 1 ? klo : nabc + 1; }
    __host__ __device__ __forceinline__ int kin_hi() const { return khi < ks() ? khi : ks(); }
};

// Split-field PML strip (strip s = 1 x-low, 2 x-high, 3 y-low, 4 z-low, 5 z-high under FSPACE).
struct Strip {
    int nxb, nxe, nyb, nye, nzb, nze;  // reference box (v/xy/yz loops end at nye)
    int ni, nj1, nk;                   // aux dims, nj1 = nye-nyb+2
    int jend_uw;                       // last j of the u/w and normal/xz loops
    long long base;                    // offset of this strip in each aux pool
    long long ncells;                  // ni*nj1*nk
    int ox_off, oxS_off, oy_off, oyS_off, oz_off, ozS_off;  // offsets into the profile table
    float rni, rnj;                    // 1/ni, 1/(jend_uw-nyb+1) for the index split (udiv_small)
    int fastdiv;                       // the strip's u/w range has fewer than 2^24 cells
};

// 24 split components per strip: u(3) v(3) w(3) xx(3) yy(3) zz(3) xy(2) xz(2) yz(2)
enum AuxId {
    AX_U0 = 0, AX_U1, AX_U2, AX_V0, AX_V1, AX_V2, AX_W0, AX_W1, AX_W2,
    AX_XX0, AX_XX1, AX_XX2, AX_YY0, AX_YY1, AX_YY2, AX_ZZ0, AX_ZZ1, AX_ZZ2,
    AX_XY0, AX_XY1, AX_XZ0, AX_XZ1, AX_YZ0, AX_YZ1, AX_N
};

template <class T>
struct Fields {
    T *u, *v, *w, *xx, *yy, *zz, *xy, *yz, *xz;
    const T *lam, *mu, *d;
    // The same medium as a 1-D profile when it varies with k only (the layered medium
    // of readcrustalmodel): lam at lay[k-1], mu at lay[nzt+k-1], d at lay[2*nzt+k-1],
    // dth/d (the IEEE quotient the interior velocity sweep forms per cell) at
    // lay[3*nzt+k-1] and dt/d (the PML velocity sweep's) at lay[4*nzt+k-1]; null
    // otherwise.  The interior and PML sweeps then read values per plane instead of
    // arrays per cell.
    const T* lay;
};
constexpr int LAY_N = 5;  // profile entries per plane

// Fault-plane state.  F = field type, double = accumulators (slip, slip path,
// rupture time, rise, slip time, psi).
//
// avdx, avdz (the damping memory of the trial traction) and distX (the slip path of the
// X nodes) hold two planes each: step it reads plane (it+1)&1 and writes plane it&1, so
// the fault boundary condition, which recomputes the trial and post-friction tractions of
// a tile's neighbouring nodes, never reads a value another CTA is updating.  After n steps
// the current plane is n&1 (pp_rd / pp_wr below).
template <class T>
struct Fault {
    // traction_com
    T *tx, *tz;           // traction after friction (read by next step's fault velocity)
    T *txt, *tzt;         // trial traction (scratch of the separate-launch fault BC only)
    T *RFx, *RFz, *avdx, *avdz, *v1t, *au1, *av1, *aw1;
    // friction_com
    T *uZ, *wX, *tabsX, *tabsZ, *T0X, *T0Z, *T0Xb, *Dc;
    T *peakX, *dynX, *DcX, *peakZ, *dynZ, *DcZ, *coh;
    T *aX, *bX, *vwX, *fwX, *aZ, *bZ, *vwZ, *fwZ;
    double *psiX, *psiZ;
    // source_com
    double *distX, *distZ, *slipX, *slipZ, *ruptime, *rise, *sliptime;
    T *schangeX, *schangeZ;  // last step's shear traction / strength planes
    int n2;                  // nxt*nzt, the size of one plane
};

// plane of a two-plane state array that step `it` reads / writes
template <class U>
__host__ __device__ __forceinline__ U* pp_rd(U* base, int it, int n2) { return base + (size_t)((it + 1) & 1) * n2; }
template <class U>
__host__ __device__ __forceinline__ U* pp_wr(U* base, int it, int n2) { return base + (size_t)(it & 1) * n2; }

struct FvwScalars {
    double Sn, v0, f0, fw, uini, wini;
    int nucleation;
    double hx0, hz0, perturb, RR2, TT2, strinixI;
};

// Scalars of one time step in the field type T, computed on the host exactly as the
// reference computes them in `real` (dth = dt/dh, ...).
template <class T>
struct StepConst {
    T dt, dh, dth, dth2, dht, damp_s, c1, c2;
    T rdh, rdl;              // the pair of dh for div_by
    T ydh;                   // RN(1/dh) for div_steps
    T ds, dsi;               // the scale S of the dividends and 1/S (div_scale)
    int pml_form;            // how the PML sweeps form their quotients (PmlForm)
    double dtA, dhA, dthA;   // FP64 copies for the FP64 parts
};

// x / b rounded to nearest (IEEE) for a divisor b > 0 known before the launch, in one
// multiplication and one multiply-add: RN(x*h + RN(x*l)), with h close to 1/b and l close
// to 1/b - h formed on the host.
//
// Method: N. Brisebarre, J.-M. Muller, S. K. Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", IEEE Trans. Computers
// 53(8), 2004: the sum before its rounding is within a few 2^-48 of x/b (relative), so the
// rounding can only go wrong where x/b lies that close to the midpoint of two consecutive
// floats.  For a given b only a handful of significands of x do; div_pair (fd3d_setup.h)
// enumerates them and takes the first pair (h, l) whose result is right, with a margin, for
// every one.
//
// The bound on the error holds while RN(x*l) does not underflow into it, |x| >= 2^-70 for b
// in the range that div_pair takes.  The wave field's leading edge runs through every magnitude
// down to zero (in the first few hundred steps a third of a small model's PML cells are
// below 2^-70, a tenth below 2^-126), so the sweeps form x scaled by a power of two S (div_scale),
// which commutes with every rounding here, and put the factor back where the quotient is
// used: that takes |x| down to where x/b is still a normal number, for one more
// multiplication a cell.  A zero is exact too
// (with l >= 0 its sign as well; with l < 0 div_by_signed puts the sign back).  Smaller
// dividends are recorded in `key`: the least of 2*bits(x) - 1 over the quotients a thread forms,
// which sends zero to the top of the range, so the test costs two integer operations a quotient
// and one branch a cell.  A cell with key < DIV_KEY is done again with div_small, one with a
// result that is not finite (x*l and x*h can cancel to NaN where x/b is infinite) with
// div_exact.  An exhaustive GPU test over all 2^32 dividends (fd3d_check_division) holds all
// three to the IEEE quotient.
//
// Not every divisor has a pair.  Of 20000 random significands 1218 have none with l >= 0 (nor have
// 11.3, 45.2 or 40000/650) and 38 have none at all (56.3, 112.6, 225.2).  PmlForm is what a model's
// sweeps do about it, one form for the whole model:
//   PML_PAIR    dh has a pair with l >= 0, every 1 + omega a pair: div_by and div_by_signed
//   PML_SIGNED  the pair of dh has l < 0: div_by_signed for both, one operation more a quotient
//   PML_STEPS   some divisor has no pair: div_steps for both
//   PML_EXACT   some divisor is outside [2^-20, 2^20]: div_exact for both
// The last three are kernels of their own (ANY), so that the first keeps its registers.  us a step at
// spacings of the four forms (45.0, 45.2, 56.3, 1.5e6 m): 1.6 M cells 65.3, 66.3, 67.1, 74.0, 68 M cells
// 1547, 1546, 1550, 1853.  (With div_exact for all but the first, formed after div_by's result was
// thrown away: 65.3, 92.6, 92.6, 92.6 and 1547, 2006, 2006, 2006.)
enum PmlForm { PML_PAIR = 0, PML_SIGNED = 1, PML_STEPS = 2, PML_EXACT = 3 };
constexpr unsigned DIV_KEY = 2u * 0x1c800000u - 1u;  // the key of 2^-70
__device__ __forceinline__ float div_by(float x, float h, float l, unsigned& key) {
    key = min(key, 2u * __float_as_uint(x) - 1u);
    return __fmaf_rn(x, h, __fmul_rn(x, l));
}
__device__ __forceinline__ float div_by_signed(float x, float h, float l, unsigned& key) {
    return __uint_as_float(__float_as_uint(div_by(x, h, l, key)) | (__float_as_uint(x) & 0x80000000u));
}
// The same in five operations from y = RN(1/b) alone, for a divisor without a pair.  Markstein's
// theorem (P. W. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34(1), 1990): if y is within half an ulp of 1/b and q within one
// ulp of x/b, the remainder r = x - b*q is exact and RN(q + r*y) = RN(x/b).  RN(x*y) can be 1.5
// ulp off, so one correction brings it within one first; the second is the theorem's.  The remainder
// is exact while it does not underflow, and |x| >= 2^-70 leaves it 2^-117 or more.
__device__ __forceinline__ float div_steps(float x, float b, float y, unsigned& key) {
    key = min(key, 2u * __float_as_uint(x) - 1u);
    float q = __fmul_rn(x, y);
    q = __fmaf_rn(__fmaf_rn(-q, b, x), y, q);
    q = __fmaf_rn(__fmaf_rn(-q, b, x), y, q);
    return __uint_as_float(__float_as_uint(q) | (__float_as_uint(x) & 0x80000000u));
}
// x / b for every finite x: scaled by 2^80 the quotient is div_by's (STEPS: div_steps's, from y = h;
// right for every divisor in range where x / b is finite).  Scaling it back rounds a
// second time if the result is subnormal; where that went to the wrong side of a tie, the
// residual x - q*b (exact here: q is a multiple of 2^-149, and less than a unit off) is more
// than half a unit times b.
template <bool STEPS>
__device__ __forceinline__ float div_small(float x, float b, float h, float l) {
    unsigned key = 0;
    const bool small = fabsf(x) < 0x1p-10f;
    const float xs = x * (small ? 0x1p80f : 1.0f), qs = STEPS ? div_steps(xs, b, h, key) : div_by_signed(xs, h, l, key);
    float q = qs * (small ? 0x1p-80f : 1.0f);
    if (small && fabsf(qs) < 0x1p-46f) {
        const float rest = __fmaf_rn(-(q * 0x1p80f), b, xs), half = b * 0x1p-70f;
        q += rest > half ? 0x1p-149f : rest < -half ? -0x1p-149f : 0.0f;
        q = copysignf(q, x);  // (a negative zero plus zero is positive)
    }
    return q;
}
// The quotient formed in FP64 and rounded to FP32: both operands are exact in FP64, and
// rounding a quotient first to 53 bits and then to 24 (or fewer, for a subnormal result)
// gives the directly rounded one because 53 >= 2*24 + 2 (S. A. Figueroa, "When is double
// rounding innocuous?", SIGNUM Newsletter 30(3), 1995).  Right for every x and b.
__device__ __forceinline__ float div_exact(float x, float b) { return __double2float_rn(__ddiv_rn((double)x, (double)b)); }
// the FP64 build divides directly (parity build, not the fast path)
__device__ __forceinline__ double div_exact(double x, double b) { return x / b; }

// n / d for n < 2^24 and 1 <= d < 2^24 with rd = RN(1/d): the float product is within
// one of the quotient, and one remainder test each way makes it exact (a few integer
// operations instead of a 32-bit division, which the GPU runs as a long sequence).
__host__ __device__ __forceinline__ unsigned udiv_small(unsigned n, unsigned d, float rd, unsigned& rem) {
    unsigned q = (unsigned)((float)n * rd);
    int r = (int)(n - q * d);
    if (r < 0) { --q; r += (int)d; }
    else if (r >= (int)d) { ++q; r -= (int)d; }
    rem = (unsigned)r;
    return q;
}

// Device-side status word bits.
enum { ST_NEWTON = 1, ST_NONFINITE = 2, ST_TIMEOUT = 4 };

#ifndef FD3D_NEWTON_MAXIT
#define FD3D_NEWTON_MAXIT 200
#endif

}  // namespace fd3d
