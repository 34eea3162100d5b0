// Column kernels of the FIM dynamics step: hybgen (regrid_1d, dffusn_lev,
// remap_1d with restp_1d, equilb, inflate, pcwise), hystat, globsum.
//
// hybgen's regrid is serial in k with data-dependent branches, so k_regrid runs
// one thread per column over column arrays (in shared memory while the grid
// fits one round of warps, else local); the 1-ring interface smoothing and
// inflate run in one kernel, 32 columns a block; the remap of the default
// knobs takes whole columns a warp, that of the others a thread a column.
// hystat runs 32 columns a block, its bottom-up Montgomery/geopotential
// recursion with a lane a column over shared memory.
// globsum accumulates per thread (FP64, or float-float compensated sums in the
// FP32 build, whose error is that of an FP64 sum) and reduces per block into a
// deterministic partial buffer.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "fim_internal.h"

namespace fim {

template <typename R> __device__ __forceinline__ R cmax(R a, R b) { return a > b ? a : b; }
template <typename R> __device__ __forceinline__ R cmin(R a, R b) { return a < b ? a : b; }
template <typename R> __device__ __forceinline__ R cabs(R a) { return a < R(0) ? -a : a; }
__device__ __forceinline__ double cabs(double a) { return fabs(a); }

// FP64 comparisons on the integer pipe (fim_internal.h); false for NaNs, as <
__device__ __forceinline__ bool lt(float a, float b) { return a < b; }
__device__ __forceinline__ bool lt(double a, double b) { return f64_lt(a, b); }
__device__ __forceinline__ bool nonzero(float a) { return a != 0.f; }
__device__ __forceinline__ bool nonzero(double a) { return (__double_as_longlong(a) << 1) != 0ll; }
__device__ __forceinline__ double cmax(double a, double b) { return lt(b, a) ? a : b; }
__device__ __forceinline__ double cmin(double a, double b) { return lt(a, b) ? a : b; }
// x / cp, and the pressure that belongs to an Exner function value.  Every kernel
// forms it here, so an interface that has not moved since the initial
// adjustment or the last remap keeps its pressure bit for bit, and the layer
// thicknesses keep summing to the column's mass.
template <typename R>
__device__ __forceinline__ R by_cp(R x) { return divide_by(x, R(kCp), R(1) / R(kCp)); }
template <typename R>
__device__ __forceinline__ R pressure_of(R ex) { return R(kP1000) * pow_cp_rd(by_cp(ex)); }

constexpr int kColBlock = 128;
constexpr int kBlock2 = 256;
inline unsigned nblocks(long long n, int b) { return (unsigned)((n + b - 1) / b); }

// ---------------------------------------------------------------- hybgen --
// What regrid_1d takes from the target column alone, formed once a block: the
// targets, the heat diffusion's factors (dffudt cnv^2 (th(k+1) - th(k-1)) / 2
// and its floor .03 cnv, cnv = g / th(k)) and inflate's minimum layers.
template <typename R, int ML>
struct RegTab {
  R tg[ML], num[ML], fl[ML], d0[ML];
  __device__ __forceinline__ void fill(const R* targt, const R* dpsig, int L) {
    const R grv = R(kGrvity), dffudt = R(.1);
    for (int k = threadIdx.x; k < L; k += blockDim.x) {
      tg[k] = targt[k];
      d0[k] = R(kRd) * dpsig[k] / R(kP1000);
      if (k >= 1 && k <= L - 2) {
        const R cnv = grv / targt[k];
        num[k] = dffudt * cnv * cnv * R(.5) * (targt[k + 1] - targt[k - 1]);
        fl[k] = R(.03) * cnv;
      }
    }
  }
};

// restp_1d (hybgen.F90:792-890).  The running minimum oldth is formed in
// place in thold (the caller's column, not read again), whose layers below
// kmod are one already.  The new theta column is targt except its two end
// layers (hybgen.F90:832-834), so it is not stored: th0 and thL are its ends
// and tn(k) its layer k.
template <typename R, typename C>
__device__ void restp_1d(C oldth, int kmod, C pkold, int kold, C pknew, const R* targt, int knew, int* bad) {
  {
    R up = oldth[kold - 1];
    for (int k = kold - 2; k >= 0; k--) {
      const R x = oldth[k];
      if (k < kmod && !lt(up, x)) break;  // the column below is monotone
      up = cmin(up, x);
      oldth[k] = up;
    }
  }
  const R th0 = cmin(cmin(oldth[0], oldth[kold - 1]), targt[0]);
  const R thL = cmax(cmax(oldth[0], oldth[kold - 1]), targt[knew - 1]);
  auto tn = [&](int k) -> R { return k == 0 ? th0 : k == knew - 1 ? thL : targt[k]; };
  pknew[0] = pkold[0];
  pknew[knew] = pkold[kold];
  R colint = R(0), colscl = R(0), cloutt = R(0);
  {
    R p0 = pkold[0];
#pragma unroll 4
    for (int k = 0; k < kold; k++) {
      const R p1 = pkold[k + 1], w = oldth[k] * (p1 - p0);
      colint = colint + w;
      colscl = colscl + cabs(w);
      p0 = p1;
    }
  }
  int ko = 0;
  R tk = th0, prev = pknew[0], ok = oldth[0], pk = pkold[0];  // layer ko's theta and lower interface
  for (int k = 0; k < knew - 1; k++) {
    const R tk1 = tn(k + 1);
    R pinteg = R(0), tha, thb = tk;
    for (;;) {
      tha = thb;
      thb = cmin(tk1, cmax(tk, ok));
      pinteg = pinteg + pk * (thb - tha);
      if (lt(ok, tk1)) {
        if (ko < kold - 1) {
          ko++;
          ok = oldth[ko];
          pk = pkold[ko];
          continue;
        }
        tha = thb;
        thb = tk1;
        pinteg = pinteg + pkold[kold] * (thb - tha);
      }
      break;
    }
    R pn = prev;
    if (lt(tk, tk1)) pn = divide(pinteg, tk1 - tk);
    pknew[k + 1] = pn;
    cloutt = cloutt + tk * (pn - prev);
    prev = pn;
    tk = tk1;
  }
  cloutt = cloutt + thL * (pknew[knew] - prev);
  if (cabs(cloutt - colint) > cmax(R(1.e-33), col_tol<R>(1.e-6) * colscl)) *bad = 1;
}

// equilb scenario 1 (hybgen.F90:1316-1363); in place on pres, the six
// interfaces of a step kept as the loop moves up
template <typename R, typename C>
__device__ void equilb(const R* thet, C pnew, int kk, R slak) {
  const R thin = R(kRd) / R(kP1000);
  const R top = pnew[0] - thin;
  R p0 = pnew[0], p1 = pnew[1], p2 = pnew[2], p3 = pnew[3], p4 = pnew[4];
  for (int k = 3; k <= kk - 2; k++) {
    const R p5 = pnew[k + 2];
    const R dp1 = p0 - p1, dp2 = p1 - p2, dp4 = p3 - p4, dp5 = p4 - p5;
    if (!lt(top, p0) && lt(dp1, dp2) && lt(dp5, dp4)) {
      const R dp3 = p2 - p3;
      const R goal = R(.5) * (dp3 + cmin(dp2, dp4));
      if (lt(goal, dp2) && lt(goal, dp4)) {
        R dis3 = cmin(dp2 - goal, goal - dp3) * slak;
        R dis4 = cmin(dp4 - goal, goal - dp3) * slak;
        const R th2 = thet[k - 2], th3 = thet[k - 1], th4 = thet[k];
        if (th3 > th2 && th4 > th3) {
          const R ratio = (th4 - th3) / (th3 - th2);
          if (ratio > R(1)) dis4 = dis3 / ratio;
          else dis3 = dis4 * ratio;
        }
        p2 = p2 + dis3;
        p3 = p3 - dis4;
        pnew[k - 1] = p2;
        pnew[k] = p3;
      }
    }
    p0 = p1; p1 = p2; p2 = p3; p3 = p4; p4 = p5;
  }
}

template <typename R>
__device__ __forceinline__ R cushn(R a, R b) {
  const R m = cmin(a, R(2) * b);
  return divide(R(.25) * (m * m), b) + cmax(a, R(2) * b) - b;
}

// inflate (hybgen.F90:893-1007); d0(k) = rd dpsig(k) / p1000
template <typename R, typename D0, typename C>
__device__ void inflate(const Knobs& kn, D0 d0, int L, R psurf, C exner) {
  const R thin = R(kRd) / R(kP1000);
  const R rd = R(kRd), p1000 = R(kP1000), cp = R(kCp);
  R dpsum = R(0);
  const R extop = cp * pow(R(kn.ptop) / p1000, rd / cp);
  const R top = R(.2);
  const R shrink = cmin(R(1), (psurf / p1000 - top) / (R(1) - top));
  const R soft = rd * R(100) / p1000;
  const R ex0 = exner[0];
  R below = ex0;  // exner[k - 1]
  int last = 1;
  for (int k = 1; k <= L - 1; k++) {
    R dp0 = d0(k - 1) * shrink;
    dpsum = dpsum + dp0;
    const R exold = exner[k];
    R now = exold;
    if (k <= kn.kbl) {
      last = k + 1;
      now = below - dp0;
      exner[k] = now;
    } else {
      if (k > last) {
        // / min(10, 1.25 2^(k - last)): 2.5, 5, 10, 10, ... a tenth scaled exactly
        const int n = k - last;
        dp0 = tenth(dp0) * (n == 1 ? R(4) : n == 2 ? R(2) : R(1));
        dp0 = cmax(dp0, soft);
      }
      const R dp1 = cushn(cmax(R(0), below - cmin(exold, ex0 - dpsum)), dp0);
      if (lt(below - dp1, exold - thin)) {
        if (k == last) last = k + 1;
        now = cmax(extop, below - dp1);
        exner[k] = now;
      }
    }
    below = now;
  }
  if (kn.thktop > 0.) {
    const R thk = R(kn.thktop);
    for (int k = L; k >= 2; k--) {
      R q = exner[k - 1] / cp;
      q = q * q * sqrt(q);
      const R dk = R(.25) * R(L - k);
      const R dp0 = rd * thk / p1000 * (R(1) / (R(1) + dk * dk)) / q;
      const R exold = exner[k - 1];
      const R dp1 = cushn(cmax(R(0), exold - exner[k]), dp0);
      if (exner[k] + dp1 > exold + thin) exner[k - 1] = exner[k] + dp1;
      if (exner[k - 1] < exner[k - 2] - dp0) break;
    }
  }
}

// regrid_1d (hybgen.F90:207-512, hybrid-isentropic branch) for one column: a
// serial chain of ~200 instructions a level, bound by its latency (small grids)
// or issue and local memory (large ones).  What the target column decides
// comes in tab, passes keep the neighbours they read in registers: 0.89 -> 0.62
// ms at glvl 8 / nvl 64, 74 -> 41 us at glvl 5 / nvl 38 (with regrid_in_smem), FP64
// glvl 6 0.87 -> 0.47 ms.
// thcol (L) comes as its running minimum from the top and excol (L+1) as its
// running limit from the bottom (columns_in_min, columns_in_limit); both are
// overwritten.  exnew ends as the new Exner function.
template <typename R, int ML, typename C>
__device__ void regrid_1d(const Knobs& kn, const RegTab<R, ML>& tab, int L, int its, C thcol, C excol, C exnew,
                          R prcol0, int* bad) {
  const R thin = R(kRd) / R(kP1000), tolrnce = R(0.001);
  const R eqlb_slak = R(.1) * R(its) / (R(10) + R(its));
  const R* targt = tab.tg;
  C exwrk = excol;
  const R tt = targt[L - 1];
  int kmod = L;  // lowest layer of thcol changed here
  for (int k = L; k >= 2; k--) {
    if (thcol[k - 1] <= tt + tolrnce) break;
    const R wgt1 = cmax(R(0), exwrk[k - 2] - exwrk[k - 1]);
    const R wgt2 = cmax(thin, exwrk[k - 1] - exwrk[k]);
    const R tr = (thcol[k - 2] * wgt1 + thcol[k - 1] * wgt2) / (wgt1 + wgt2);
    if (tr > tt - tolrnce) {
      exwrk[k - 1] = exwrk[L];
      for (int k1 = k - 1; k1 <= L; k1++) thcol[k1 - 1] = tr;
      kmod = k - 2;
    } else {
      exwrk[k - 1] = cmin(exwrk[k - 2], cmax(exwrk[k], (exwrk[k - 1] * (thcol[k - 1] - thcol[k - 2]) +
                                                         exwrk[k] * (tt - thcol[k - 1])) /
                                                            (tt - thcol[k - 2])));
      for (int k1 = k; k1 <= L; k1++) thcol[k1 - 1] = tt;
      kmod = k - 1;
      break;
    }
  }
  restp_1d<R>(thcol, kmod, exwrk, L, exnew, targt, L, bad);
  // heat diffusion (heatfx zero at the end layers and next to the column's
  // ends) from the interfaces before the pass, whose neighbours stay in
  // registers as the pass overwrites them
  const R bot = exnew[0] - R(.01), top = exnew[L] + R(.01);
  for (int iter = 1; iter <= 3; iter++) {
    bool event = false;
    R hprev = R(0);                                        // heatfx(k - 1)
    R lo = exnew[0], at = exnew[1], newlo = lo;            // old k - 1, old k, new k - 1
#pragma unroll 2
    for (int k = 1; k <= L - 1; k++) {
      const R hi = exnew[k + 1];
      R hcur = R(0);
      if (k <= L - 2 && lt(at, bot) && lt(top, hi)) hcur = divide(tab.num[k], cmax(tab.fl[k], at - hi));
      R now = at;
      if (lt(at, bot) && lt(top, at)) {
        now = cmax(hi, cmin(lo, at + divide(hcur - hprev, targt[k] - targt[k - 1])));
        exnew[k] = now;
      }
      event = event || lt(newlo + thin, now);
      hprev = hcur;
      lo = at;
      at = hi;
      newlo = now;
    }
    event = event || lt(newlo + thin, at);
    if (!event) break;
  }
  equilb<R>(targt, exnew, L, eqlb_slak);  // reads layers 1..nvl-2 only
  inflate<R>(kn, [&](int k) { return tab.d0[k]; }, L, prcol0, exnew);
}

// pcwise (hybgen.F90:1010-1279): 1-D PCM/PLM/PPM remap of yold from cell
// boundaries xold to xnew.  Returns true when the column-integral check fails.
template <typename R, int ML>
__device__ bool pcwise(int kk, const R* xold, const R* yold, const R* xnew, R* ynew, int miglim, int remap_optn) {
  R delz[ML + 1], fco[ML], fcn[ML], vertfx[ML + 1], fldnew[ML], a[ML], b[ML], cc[ML];
  const R athird = R(1) / R(3), small = R(1.e-22);
  const bool flip = !(xold[0] < xold[kk]);
  for (int k = 0; k <= kk; k++) delz[k] = flip ? (-xnew[k]) - (-xold[k]) : xnew[k] - xold[k];
  for (int k = 0; k < kk; k++) {
    fco[k] = flip ? cmax(R(0), (-xold[k + 1]) - (-xold[k])) : cmax(R(0), xold[k + 1] - xold[k]);
    fcn[k] = flip ? cmax(R(0), (-xnew[k + 1]) - (-xnew[k])) : cmax(R(0), xnew[k + 1] - xnew[k]);
  }
  R bfore = R(0), colscl = R(0);
  for (int k = 0; k < kk; k++) {
    bfore = bfore + yold[k] * fco[k];
    colscl = colscl + cabs(yold[k] * fco[k]);
  }
  for (int k = 0; k < kk; k++) fldnew[k] = yold[k];
  for (int k = kk - 2; k >= 0; k--) fldnew[k] = (fldnew[k] * fco[k] + fldnew[k + 1] * small) / (fco[k] + small);
  for (int k = 1; k < kk; k++) fldnew[k] = (fldnew[k] * fco[k] + fldnew[k - 1] * small) / (fco[k] + small);
  a[0] = fldnew[0]; b[0] = R(0); cc[0] = R(0);
  a[kk - 1] = fldnew[kk - 1]; b[kk - 1] = R(0); cc[kk - 1] = R(0);
  for (int k = 1; k < kk - 1; k++) {
    if (remap_optn == 1) {
      a[k] = fldnew[k]; b[k] = R(0); cc[k] = R(0);
    } else if (remap_optn == 2) {
      a[k] = fldnew[k];
      b[k] = R(0);
      if (fldnew[k] <= cmin(fldnew[k - 1], fldnew[k + 1]) || fldnew[k] >= cmax(fldnew[k - 1], fldnew[k + 1])) {
        b[k] = R(0);
      } else if ((fldnew[k + 1] - fldnew[k - 1]) * (fldnew[k - 1] + fldnew[k + 1] - R(2) * fldnew[k]) > R(0)) {
        b[k] = fldnew[k] - fldnew[k - 1];
      } else {
        b[k] = fldnew[k + 1] - fldnew[k];
      }
      cc[k] = R(0);
    } else {
      const R yl = (cmax(small, fco[k - 1]) * fldnew[k] + cmax(small, fco[k]) * fldnew[k - 1]) /
                   (cmax(small, fco[k - 1]) + cmax(small, fco[k]));
      const R yr = (cmax(small, fco[k + 1]) * fldnew[k] + cmax(small, fco[k]) * fldnew[k + 1]) /
                   (cmax(small, fco[k + 1]) + cmax(small, fco[k]));
      a[k] = R(1.5) * fldnew[k] - R(.25) * (yl + yr);
      b[k] = yr - yl;
      cc[k] = R(6) * (R(.5) * (yl + yr) - fldnew[k]);
      if (cabs(yr - yl) < R(6) * cabs(R(.5) * (yl + yr) - fldnew[k])) {
        if (cabs(yr - yl) > R(2) * cabs(R(.5) * (yl + yr) - fldnew[k])) {
          if ((yr - yl) * (R(.5) * (yl + yr) - fldnew[k]) > R(0)) {
            a[k] = R(.25) * (R(3) * fldnew[k] + yl);
            cc[k] = R(3) * (fldnew[k] - yl);
            b[k] = cc[k];
          } else {
            a[k] = R(.25) * (R(3) * fldnew[k] + yr);
            cc[k] = R(3) * (fldnew[k] - yr);
            b[k] = -cc[k];
          }
        } else {
          a[k] = fldnew[k]; b[k] = R(0); cc[k] = R(0);
        }
      }
    }
  }
  for (int k = 1; k < kk; k++) {
    R slab = R(0), amount = R(0);
    vertfx[k] = R(0);
    const R dz = delz[k];
    if (miglim == 1) {
      if (dz > R(0)) {
        const int lyr = k;
        if (fco[lyr] > R(0)) {
          const R dslab = cmin(slab + fco[lyr], dz) - cmin(slab, dz);
          const R dx = dslab / fco[lyr];
          const R fcdx = a[lyr] + b[lyr] * R(.5) * (dx - R(1)) + cc[lyr] * (R(.25) - dx * (R(.5) - dx * athird));
          amount = amount + fcdx * dslab;
          slab = slab + dslab;
        }
      } else if (dz < R(0)) {
        const int lyr = k - 1;
        if (fco[lyr] > R(0)) {
          const R dslab = cmin(slab + fco[lyr], -dz) - cmin(slab, -dz);
          const R dx = dslab / fco[lyr];
          const R fcdx = a[lyr] + b[lyr] * R(.5) * (R(1) - dx) + cc[lyr] * (R(.25) - dx * (R(.5) - dx * athird));
          amount = amount + fcdx * dslab;
          slab = slab + dslab;
        }
      }
    } else {
      if (dz > R(0)) {
        int lyr = k - 1;
        for (;;) {
          lyr = lyr + 1;
          if (slab >= dz) break;
          if (fco[lyr] > R(0)) {
            const R dslab = cmin(slab + fco[lyr], dz) - cmin(slab, dz);
            const R dx = dslab / fco[lyr];
            const R fcdx = a[lyr] + b[lyr] * R(.5) * (dx - R(1)) + cc[lyr] * (R(.25) - dx * (R(.5) - dx * athird));
            amount = amount + fcdx * dslab;
            slab = slab + dslab;
          }
          if (!(lyr < kk - 1)) break;
        }
      } else if (dz < R(0)) {
        int lyr = k;
        for (;;) {
          lyr = lyr - 1;
          if (slab >= -dz) break;
          if (fco[lyr] > R(0)) {
            const R dslab = cmin(slab + fco[lyr], -dz) - cmin(slab, -dz);
            const R dx = dslab / fco[lyr];
            const R fcdx = a[lyr] + b[lyr] * R(.5) * (R(1) - dx) + cc[lyr] * (R(.25) - dx * (R(.5) - dx * athird));
            amount = amount + fcdx * dslab;
            slab = slab + dslab;
          }
          if (!(lyr > 0)) break;
        }
      }
    }
    if (slab != R(0)) vertfx[k] = -dz * amount / slab;
  }
  vertfx[0] = R(0);
  vertfx[kk] = R(0);
  R after = R(0);
  for (int k = 0; k < kk; k++) {
    const R amount = fldnew[k] * fco[k] - (vertfx[k + 1] - vertfx[k]);
    ynew[k] = (amount + fldnew[k] * small) / (fcn[k] + small);
    after = after + amount;
  }
  return cabs(bfore - after) > cmax(R(1.e-33), col_tol<R>(1.e-11) * colscl);
}

// A warp's 32 columns (lane = column) move between global memory and the
// lanes' column arrays through a 32 x 33 shared tile, 32 levels at a time, so
// the global accesses run along k (128-byte rows) rather than one column per
// lane.  n values of column i0 + lane start at src + (i0 + lane) * stride.
// take(k, x) receives the levels upward (UP) or downward.
template <bool UP, typename R, typename F>
__device__ __forceinline__ void columns_in(const R* __restrict__ src, size_t stride, int n, int ncol, int i0,
                                           int lane, R (*tile)[33], F take) {
  const int nc = (n + 31) / 32;
  for (int cc = 0; cc < nc; cc++) {
    const int c0 = (UP ? cc : nc - 1 - cc) * 32;
    const int kk = c0 + lane;
#pragma unroll 8
    for (int r = 0; r < 32; r++)
      if (r < ncol && kk < n) tile[r][lane] = src[(size_t)(i0 + r) * stride + kk];
    __syncwarp();
    const int m = n - c0 < 32 ? n - c0 : 32;
    if (lane < ncol) {
#pragma unroll 4
      for (int q = 0; q < m; q++) {
        const int k = UP ? q : m - 1 - q;
        take(c0 + k, tile[lane][k]);
      }
    }
    __syncwarp();
  }
}
template <typename R, typename C>
__device__ __forceinline__ void columns_out(R* __restrict__ dst, size_t stride, int n, int ncol, int i0, int lane,
                                            R (*tile)[33], C col) {
  for (int c0 = 0; c0 < n; c0 += 32) {
    const int m = n - c0 < 32 ? n - c0 : 32;
    if (lane < ncol)
      for (int q = 0; q < m; q++) tile[lane][q] = col[c0 + q];
    __syncwarp();
    const int kk = c0 + lane;
#pragma unroll 8
    for (int r = 0; r < 32; r++)
      if (r < ncol && kk < n) dst[(size_t)(i0 + r) * stride + kk] = tile[r][lane];
    __syncwarp();
  }
}

// a lane's column of a warp's 32 in shared memory
template <typename R>
struct LaneCol {
  R* p;
  __device__ __forceinline__ R& operator[](int k) const { return p[k * 32]; }
};

template <typename R, int ML, bool SM>
__global__ void __launch_bounds__(SM ? 32 : kColBlock) k_regrid(Grid<R> g, Strides s, Knobs kn,
    const StepParams* __restrict__ sp, const R* __restrict__ targt, const R* __restrict__ tr3d,
    const R* __restrict__ ex3d, const R* __restrict__ pr3d, R* __restrict__ exsmo, int* __restrict__ flags,
    int bnd) {
  __shared__ R tiles[SM ? 1 : kColBlock / 32][32][33];
  extern __shared__ __align__(16) unsigned char rgsm[];
  __shared__ RegTab<R, ML> tab;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int i0 = blockIdx.x * blockDim.x + wib * 32;
  const int N = g.N, L = g.L, L1 = L + 1;
  tab.fill(targt, g.dpsig, L);
  __syncthreads();
  if (i0 >= N) return;
  const int ncol = N - i0 < 32 ? N - i0 : 32;
  const int i = i0 + lane;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active || (bnd && sp->its <= 1)) return;
  tr3d += m * s.tr; ex3d += m * s.intf; pr3d += m * s.intf; exsmo += m * s.intf;
  R lth[SM ? 1 : ML], lex[SM ? 1 : ML + 1], lnw[SM ? 1 : ML + 1];
  using C = std::conditional_t<SM, LaneCol<R>, R*>;
  C thcol, excol, exnew;
  if constexpr (SM) {
    R* q = reinterpret_cast<R*>(rgsm) + lane;
    thcol.p = q;
    excol.p = q + 32 * L;
    exnew.p = q + 32 * (L + L1);
  } else {
    thcol = lth;
    excol = lex;
    exnew = lnw;
  }
  const R thin = R(kRd) / R(kP1000);
  // theta's running minimum from the top; no interface above the one below it
  R run = R(0);
  columns_in<false>(tr3d, (size_t)L, L, ncol, i0, lane, tiles[wib], [&](int k, R x) {
    run = k == L - 1 ? x : cmin(x, run);
    thcol[k] = run;
  });
  columns_in<true>(ex3d, (size_t)L1, L1, ncol, i0, lane, tiles[wib], [&](int k, R x) {
    run = k > 0 && lt(run, x - thin) ? run : x;
    excol[k] = run;
  });
  int bad = 0;
  if (lane < ncol)
    regrid_1d<R, ML>(kn, tab, L, sp->its - bnd, thcol, excol, exnew, pr3d[(size_t)i * L1], &bad);
  columns_out(exsmo, (size_t)L1, L1, ncol, i0, lane, tiles[wib], exnew);
  if (bad) atomicOr(flags + m, kFlagColumnIntegral);
}

// dffusn_lev (dffusn.F90:37-58 with dffusn_lev.exe) on interfaces kbl+2..nvl,
// out of place so every cell reads the unsmoothed neighbours.  A thread takes
// kDffK interfaces of one cell, kg + j*ng (ng = ceil((nvl+1)/kDffK)), so each
// load of a warp stays contiguous and the neighbour values of all its
// interfaces are in flight together (all six prox slots hold valid cells; a
// pentagon's slot 5 is left out of the sum).
constexpr int kDffK = 4;
template <typename R>
__global__ void __launch_bounds__(kBlock2) k_dffusn_lev(Grid<R> g, Strides s, const StepParams* __restrict__ sp,
    int bnd, int k1, int k2, const R* __restrict__ fld, R* __restrict__ out) {
  const int N = g.N, L1 = g.L + 1;
  const int ng = (L1 + kDffK - 1) / kDffK;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= N * ng) return;
  const int i = gid / ng, kg = gid - i * ng;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active || (bnd && sp->its <= 1)) return;
  fld += m * s.intf; out += m * s.intf;
  const int np = g.nprox[i];
  const R* col = fld + (size_t)i * L1;
  const R* nb[6];
#pragma unroll
  for (int e = 0; e < 6; e++) nb[e] = fld + (size_t)g.prox[i * 6 + e] * L1;
  R val[kDffK], x[kDffK][6];
#pragma unroll
  for (int j = 0; j < kDffK; j++) {
    const int k = kg + j * ng;
    const bool act = k < L1;
    const int kk = act ? k : 0;
    val[j] = col[kk];
#pragma unroll
    for (int e = 0; e < 6; e++) x[j][e] = nb[e][kk];
  }
  const R rar = g.rarea[i];
#pragma unroll
  for (int j = 0; j < kDffK; j++) {
    const int k = kg + j * ng;
    if (k >= L1) continue;
    R v = val[j];
    if (k >= k1 && k <= k2) {
      R flxdv = R(0);
#pragma unroll
      for (int e = 0; e < 6; e++)
        if (e < np) flxdv = flxdv + (v - x[j][e]) * g.sideln[i * 6 + e];
      const R factor = -g.smoo[k] * rar;
      v = v + flxdv * factor;
    }
    out[(size_t)i * L1 + k] = v;
  }
}

// remap_1d (hybgen.F90:515-789) followed by the hybgen bookkeeping
// (hybgen.F90:189-191): new u, v, tracers, Exner, pressure, thickness, sdot.
template <typename R, int ML>
__global__ void __launch_bounds__(kColBlock) k_remap(Grid<R> g, Strides s, Knobs kn,
    const StepParams* __restrict__ sp, const R* __restrict__ targt, const R* __restrict__ exsmo,
    R* __restrict__ us3d, R* __restrict__ vs3d, R* __restrict__ tr3d, R* __restrict__ sdot,
    R* __restrict__ ex3d, R* __restrict__ dp3d, R* __restrict__ pr3d, int* __restrict__ flags, int bnd) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int N = g.N, L = g.L, L1 = L + 1;
  if (i >= N) return;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active || (bnd && sp->its <= 1)) return;
  const int T = min(g.T, sp->ntr);
  exsmo += m * s.intf; us3d += m * s.cell; vs3d += m * s.cell; tr3d += m * s.tr; sdot += m * s.intf;
  ex3d += m * s.intf; dp3d += m * s.cell; pr3d += m * s.intf;
  const int its = sp->its - bnd;
  const R cp = R(kCp), rd = R(kRd), p1000 = R(kP1000), small = R(1.e-6);
  R exold[ML + 1], exnew[ML + 1], prcol[ML + 1], prnew[ML + 1], pk1col[ML + 1], pk1new[ML + 1];
  R yold[ML], ynew[ML], dpcol[ML];
  for (int k = 0; k <= L; k++) {
    exold[k] = ex3d[(size_t)i * L1 + k];
    prcol[k] = pr3d[(size_t)i * L1 + k];
    exnew[k] = exsmo[(size_t)i * L1 + k];
  }
  for (int k = 0; k <= L; k++) pk1col[k] = exold[k] * prcol[k] / cp;
  const R* dps = g.dpsig;
  if (kn.intfc_smooth > 0.) inflate<R>(kn, [&](int k) { return rd * dps[k] / p1000; }, L, prcol[0], (R*)exnew);
  if (its > 0) {
    const R sl = R(kn.slak);
    for (int k = 0; k <= L; k++) exnew[k] = sl * exnew[k] + (R(1) - sl) * exold[k];
  }
  const int mg = kn.miglim;
  if (mg > 0) {
    for (int k = 1 + mg; k <= L + 1 - mg; k++)
      exnew[k - 1] = cmax(R(.0001) * exold[k - 1] + R(.9999) * exold[k - 1 + mg],
                          cmin(R(.0001) * exold[k - 1] + R(.9999) * exold[k - 1 - mg], exnew[k - 1]));
    for (int k = 2; k <= mg; k++) {
      exnew[k - 1] = cmin(exold[0], exnew[k - 1]);
      exnew[L - k] = cmax(exold[L], exnew[L - k]);
    }
  }
  for (int k = L; k >= 0; k--) prnew[k] = pressure_of(exnew[k]);
  for (int k = 0; k < L; k++) dpcol[k] = prnew[k] - prnew[k + 1];
  for (int k = 0; k <= L; k++) pk1new[k] = exnew[k] * prnew[k] / cp;
  prnew[L] = prcol[L];
  pk1new[L] = pk1col[L];
  prnew[0] = prcol[0];
  pk1new[0] = pk1col[0];
  bool bad = false;
  // u and v
  for (int f = 0; f < 2; f++) {
    R* col = (f == 0 ? us3d : vs3d) + (size_t)i * L;
    for (int k = 0; k < L; k++) yold[k] = col[k];
    bad |= pcwise<R, ML>(L, prcol, yold, prnew, ynew, mg, kn.remap_optn);
    for (int k = 0; k < L; k++) col[k] = ynew[k];
  }
  // tracers 2..ntra in pressure, with the optional massless-layer fill
  for (int t = 1; t < T; t++) {
    R* col = tr3d + ((size_t)t * N + i) * L;
    for (int k = 0; k < L; k++) yold[k] = col[k];
    bad |= pcwise<R, ML>(L, prcol, yold, prnew, ynew, mg, kn.remap_optn);
    if (kn.thktop == 0.) {
      for (int k = 3; k <= L; k++) {
        const R qq = R(1) / (dpcol[k - 1] + small);
        ynew[k - 1] = (ynew[k - 1] * dpcol[k - 1] + ynew[k - 2] * small) * qq;
      }
    }
    for (int k = 0; k < L; k++) col[k] = ynew[k];
  }
  // potential temperature in p^(kappa+1), then the target redistribution
  {
    R* col = tr3d + (size_t)i * L;
    for (int k = 0; k < L; k++) yold[k] = col[k];
    bad |= pcwise<R, ML>(L, pk1col, yold, pk1new, ynew, mg, kn.remap_optn);
    for (int k = L; k >= 3; k--) {
      const R dplo = cmax(pk1new[k - 2] - pk1new[k - 1], pk1new[0] * small);
      const R dpup = cmax(pk1new[k - 1] - pk1new[k], pk1new[0] * small);
      const R tha = ynew[k - 2], thb = ynew[k - 1];
      const R devilo = (tha - targt[k - 2]) * dplo;
      const R deviup = (thb - targt[k - 1]) * dpup;
      if (deviup > R(0) && devilo < R(0)) {
        ynew[k - 2] = tha + cmin(deviup, -devilo) / dplo;
        ynew[k - 1] = thb - cmin(deviup, -devilo) / dpup;
      } else if (deviup < R(0) && devilo > R(0)) {
        ynew[k - 2] = tha - cmin(devilo, -deviup) / dplo;
        ynew[k - 1] = thb + cmin(devilo, -deviup) / dpup;
      }
    }
    {
      R colin = R(0), clout = R(0), colscl = R(0);
      for (int k = 0; k < L; k++) {
        colin = colin + yold[k] * (pk1col[k] - pk1col[k + 1]);
        clout = clout + ynew[k] * (pk1new[k] - pk1new[k + 1]);
        colscl = colscl + cabs(yold[k] * (pk1col[k] - pk1col[k + 1]));
      }
      if (cabs(clout - colin) > cmax(R(1.e-33), col_tol<R>(2.e-6) * colscl)) bad = true;
    }
    for (int k = 0; k < L; k++) col[k] = ynew[k];
  }
  for (int k = 0; k < L; k++)
    if (exnew[k] < exnew[k + 1]) exnew[k + 1] = exnew[k];
  for (int k = 0; k <= L; k++) {
    sdot[(size_t)i * L1 + k] = exnew[k] - exold[k];
    ex3d[(size_t)i * L1 + k] = exnew[k];
    pr3d[(size_t)i * L1 + k] = prnew[k];
  }
  for (int k = 0; k < L; k++) dp3d[(size_t)i * L + k] = dpcol[k];
  if (bad) atomicOr(flags + m, kFlagColumnIntegral);
}

// ------------------------------------------ remap, warp per column, lane = levels --
// remap_1d (hybgen.F90:515-700) for the default knobs: PLM pcwise with
// one-layer migration (remap_optn = 2, miglim = 1).
//  k_smooth_inflate: the interface smoothing and inflate, the one serial
//             recursion of the column set-up, of 32 columns a block;
//  k_remap_v: each warp runs kColsPerWarp consecutive columns.  Lane l holds
//             levels l*VL .. l*VL+VL-1 of the field in hand (u, v, tracers
//             2..ntra in pressure, theta in p^(kappa+1)), so a field's column
//             is one contiguous read and write.  The three interface arrays
//             and the fields of the warp's columns stream through a ring of
//             shared-memory slots filled by cp.async several items ahead,
//             across column boundaries.
// Given the filled values, pcwise's flux form is level-parallel: PLM slopes
// and interface fluxes take the neighbouring levels from the adjacent lanes.
// The massless-layer fills of pcwise and remap_1d's tracer fill are
// first-order linear recurrences x(k) = a(k) x(k-+1) + b(k): each lane
// composes the maps of its levels, a warp scan of the composed maps gives the
// value entering each lane, and the lane runs the recurrence in the
// reference's form over its own levels.  The pairwise theta redistribution
// toward the target (hybgen.F90:648-667) is a nonlinear sweep over the
// column: it runs after the warp's last column with lane = column.
// With one-layer migration the donor layer, slab width and dx of every
// interface depend on the coordinate only, so they are formed once per column
// and held in registers; divisions by the coordinate thicknesses (fco +
// small, fcn + small) become products with reciprocals.  Results differ from
// the serial pcwise by rounding.
constexpr int kWarpsRemapV = 4;
constexpr int kColsPerWarp = 8;  // at most; see remap_columns

// pcwise's massless-layer fill moves y(k) by (y(k+-1) - y(k)) * 1e-22 / fco(k):
// below the rounding of either precision unless fco(k) is under ~1e-4.
template <typename R>
__device__ __forceinline__ R fill_thin() { return R(1.2e-4); }

// PLM slope of a layer from its filled value f and its neighbours' fm, fp
__device__ __forceinline__ float plm_slope(float fm, float f, float fp) {
  const float b = ((fp - fm) * (fm + fp - 2.f * f) > 0.f) ? f - fm : fp - f;
  // (a NaN is dropped from below and kept from above, as cmin and cmax do)
  return (f <= fminf(fm, fp) || f >= fmaxf(fm, fp)) && fp == fp ? 0.f : b;
}

// FP64: monotonicity and the slope's sign by integer comparisons (a zero
// curvature takes the upper difference, as the product test does)
__device__ __forceinline__ double plm_slope(double fm, double f, double fp) {
  const long long km = f64_key(fm), k = f64_key(f), kp = f64_key(fp);
  const bool rise = km < k && k < kp, fall = km > k && k > kp;
  if (!rise && !fall) return 0.;
  const double c = fma(-2., f, fm + fp);
  const bool lower = c != 0. && negative(c) == fall;
  return (lower ? f : fp) - (lower ? fm : f);
}
// the slope as pcwise writes it, for values that are not finite
__device__ __forceinline__ float plain_slope(float fm, float f, float fp) { return plm_slope(fm, f, fp); }
__device__ __forceinline__ double plain_slope(double fm, double f, double fp) {
  const double b = (fp - fm) * (fm + fp - 2. * f) > 0. ? f - fm : fp - f;
  return f <= plain_min(fm, fp) || f >= plain_max(fm, fp) ? 0. : b;
}
// asynchronous global -> shared copy of B = 4, 8 or 16 bytes
template <int B>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sa), "l"(gmem), "n"(B) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// sum over a segment of W lanes (the lanes of one column)
template <typename R, int W = 32>
__device__ __forceinline__ R warp_sum(R v) {
#pragma unroll
  for (int off = W / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off, W);
  return v;
}

// sums of two values over a segment of W lanes: the halves of the segment take
// one value each, so a step is one addition for both; a's sum ends in the
// lower half's lanes and is returned everywhere, b's likewise
template <typename R, int W = 32>
__device__ __forceinline__ void warp_sum2(int lane, R& a, R& b) {
  const bool up = lane >= W / 2;
  const R give = up ? a : b, keep = up ? b : a;
  R t = keep + __shfl_xor_sync(0xffffffffu, give, W / 2, W);
#pragma unroll
  for (int off = W / 4; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off, W);
  a = __shfl_sync(0xffffffffu, t, 0, W);
  b = __shfl_sync(0xffffffffu, t, W / 2, W);
}

// Value entering each lane of a recurrence x <- a x + b whose per-lane
// composed map is (a, b): from the lanes below (up) or above (down); the
// first lane of the sweep receives 0 (its own map is constant there).
// (lane: the lane within its W-lane segment)
template <typename R, int W = 32>
__device__ __forceinline__ R affine_entry_up(int lane, R a, R b) {
#pragma unroll
  for (int off = 1; off < W; off <<= 1) {
    const R ao = __shfl_up_sync(0xffffffffu, a, off, W), bo = __shfl_up_sync(0xffffffffu, b, off, W);
    if (lane >= off) { b = a * bo + b; a = a * ao; }
  }
  const R e = __shfl_up_sync(0xffffffffu, b, 1, W);
  return lane == 0 ? R(0) : e;
}
template <typename R, int W = 32>
__device__ __forceinline__ R affine_entry_down(int lane, R a, R b) {
#pragma unroll
  for (int off = 1; off < W; off <<= 1) {
    const R ao = __shfl_down_sync(0xffffffffu, a, off, W), bo = __shfl_down_sync(0xffffffffu, b, off, W);
    if (lane + off < W) { b = a * bo + b; a = a * ao; }
  }
  const R e = __shfl_down_sync(0xffffffffu, b, 1, W);
  return lane == W - 1 ? R(0) : e;
}

// shared memory of one warp: the copy ring (an item is, for each of the H
// columns in hand, the three interface arrays or three fields), the column
// arrays of those columns, and theta of the warp's columns awaiting the
// redistribution (values, p^(kappa+1) thicknesses, their floor and, FP64
// build, the input column integrals)
template <typename R, int VL, int H>
struct RemapV {
  static constexpr int S = 32 / H * VL + 4;                        // nvl + 1 <= (32/H) VL + 1
  static constexpr int D = H > 1 ? 2 : (sizeof(R) == 4 ? 4 : 3);   // items in flight
  R ring[D][H][3][S];
  R exold[H][S], prcol[H][S], exnew[H][S], prnew[H][S], pk1col[H][S], pk1new[H][S], dpcol[H][S];
  R tg[S];
  R thb[kColsPerWarp][S], dkb[kColsPerWarp][S];
  R dpb[kColsPerWarp][S];  // new thicknesses, for theta x thickness (trdp) after the redistribution
  R flo[kColsPerWarp], colin[kColsPerWarp], colscl[kColsPerWarp];
};
static_assert(sizeof(RemapV<float, 1, 1>) % 16 == 0 && sizeof(RemapV<double, 1, 1>) % 16 == 0 &&
                  sizeof(RemapV<float, 4, 2>) % 16 == 0,
              "ring slots of consecutive warps stay 16-byte aligned");

// Level kb + v of a column of L levels held VL a lane by W lanes: with FULL the
// column fills the lanes (L == W VL), so that the tests cost nothing but for
// the first and last lane's end levels.
template <int VL, int W, bool FULL>
struct Lv {
  int L, lane;
  __device__ __forceinline__ int k(int v) const { return lane * VL + v; }
  __device__ __forceinline__ bool in(int v) const { return FULL || k(v) < L; }
  __device__ __forceinline__ bool first(int v) const { return FULL ? v == 0 && lane == 0 : k(v) == 0; }
  __device__ __forceinline__ bool last(int v) const { return FULL ? v == VL - 1 && lane == W - 1 : k(v) == L - 1; }
};

// pcwise's coordinate quantities for one lane's levels and interfaces
template <typename R, int VL>
struct LaneGeo {
  R fo[VL], rfo[VL], rfn[VL];  // level kb+v: fco, 1/(fco+small), 1/(fcn+small)
  R nd[VL], hh[VL];            // interface kb+v: -delz (0: no flux), (dx-1 | 1-dx)/2
  unsigned up;                 // bit v: interface kb+v takes layer kb+v as donor
  bool thin;                   // (whole warp) some layer is thin enough for the fill to matter
};

// 1 / x and a / b of thicknesses
__device__ __forceinline__ float recip(float x) { return fdiv(1.f, x); }
__device__ __forceinline__ float over(float a, float b) { return fdiv(a, b); }
__device__ __forceinline__ double over(double a, double b) { return divide(a, b); }

template <typename R>
__device__ __forceinline__ R coord_thick(bool flip, const R* x, int k) {
  return flip ? cmax(R(0), (-x[k + 1]) - (-x[k])) : cmax(R(0), x[k + 1] - x[k]);
}

template <typename R, int VL, int W, bool FULL>
__device__ __forceinline__ void lane_geo(int L, int lane, const R* xo, const R* xn, LaneGeo<R, VL>& G) {
  const R small = R(1.e-22);
  const bool flip = !(xo[0] < xo[L]);
  const int kb = lane * VL;
  const Lv<VL, W, FULL> lv{L, lane};
  bool thin = false;
  unsigned up = 0u;
#pragma unroll
  for (int v = 0; v < VL; v++) {
    const int k = kb + v;
    R fo = R(0), fn = R(0);
    if (lv.in(v)) {
      fo = coord_thick(flip, xo, k);
      fn = coord_thick(flip, xn, k);
      thin = thin || lt(fo, fill_thin<R>());
    }
    G.fo[v] = fo;
    if constexpr (sizeof(R) == 4) G.rfo[v] = fdiv(R(1), fo + small);
    G.rfn[v] = recip(fn + small);
    R nd = R(0), hh = R(0);
    if (lv.in(v) && !lv.first(v)) {
      const R d = flip ? (-xn[k]) - (-xo[k]) : xn[k] - xo[k];
      const bool rise = lt(R(0), d);
      if (nonzero(d)) {
        const R fl = coord_thick(flip, xo, rise ? k : k - 1);
        if (lt(R(0), fl)) {
          const R dd = rise ? d : -d;
          const R dsl = cmin(fl, dd);
          const R dx = over(dsl, fl);
          const R hx = rise ? dx - R(1) : R(1) - dx;
          if (nonzero(dsl)) {
            nd = -d;
            hh = R(.5) * hx;
          }
        }
        if (rise) up |= 1u << v;
      }
    }
    G.nd[v] = nd;
    G.hh[v] = hh;
  }
  G.up = up;
  // decided over the whole warp: pcwise's fill branch holds full-warp
  // shuffles, so both columns of a paired warp must take it together (the
  // fill is the reference's own step, exact for columns without thin layers)
  G.thin = __any_sync(0xffffffffu, thin);
  if constexpr (sizeof(R) == 8) {  // read by the fill only
    if (G.thin) {
#pragma unroll
      for (int v = 0; v < VL; v++) G.rfo[v] = R(1) / (G.fo[v] + small);
    }
  }
}

// pcwise (PLM, miglim = 1) of NF fields sharing one coordinate, lane =
// levels kb .. kb+VL-1 of each; the fields' chains are independent and
// interleave.  Returns true when pcwise's column-integral check
// (hybgen.F90:1262) fails.  That check compares two sums of the same
// telescoping fluxes; in FP32 it would only measure the rounding of those
// sums and cost 0.49 ms a step at glvl 8 (a tenth of the remap), so it runs
// in the FP64 build, and the FP32-mixed build keeps the two physical column
// checks (restp_1d's, and remap_1d's theta integral).
template <typename R, int VL, int NF, int W, bool FULL>
__device__ __forceinline__ bool pcwise_v(int L, int lane, R (&y)[NF][VL], const LaneGeo<R, VL>& G) {
  const R small = R(1.e-22);
  const Lv<VL, W, FULL> lv{L, lane};
  R bfore[NF], colscl[NF];
  if (sizeof(R) == 8) {
#pragma unroll
    for (int h = 0; h < NF; h++) {
      bfore[h] = R(0);
      colscl[h] = R(0);
#pragma unroll
      for (int v = 0; v < VL; v++)
        if (lv.in(v)) {
          bfore[h] += y[h][v] * G.fo[v];
          colscl[h] += cabs(y[h][v] * G.fo[v]);
        }
    }
  }
  R yf[NF][VL];
  if (G.thin) {
    // backward fill: nb(nvl) = y(nvl), nb(k) = (y(k) fco(k) + nb(k+1) small) / (fco(k) + small)
    R nb[NF][VL];
#pragma unroll
    for (int h = 0; h < NF; h++) {
      R a = R(1), b = R(0);
#pragma unroll
      for (int v = VL - 1; v >= 0; v--) {
        if (lv.last(v)) {
          a = R(0);
          b = y[h][v];
        } else if (lv.in(v)) {
          const R A = small * G.rfo[v];
          b = A * b + y[h][v] * G.fo[v] * G.rfo[v];
          a = A * a;
        }
      }
      R x = affine_entry_down<R, W>(lane, a, b);
#pragma unroll
      for (int v = VL - 1; v >= 0; v--) {
        if (lv.last(v)) x = y[h][v];
        else if (lv.in(v)) x = (y[h][v] * G.fo[v] + x * small) * G.rfo[v];
        nb[h][v] = x;
      }
    }
    // forward fill: yf(1) = nb(1), yf(k) = (nb(k) fco(k) + yf(k-1) small) / (fco(k) + small)
#pragma unroll
    for (int h = 0; h < NF; h++) {
      R a = R(1), b = R(0);
#pragma unroll
      for (int v = 0; v < VL; v++) {
        if (lv.first(v)) {
          a = R(0);
          b = nb[h][v];
        } else if (lv.in(v)) {
          const R A = small * G.rfo[v];
          b = A * b + nb[h][v] * G.fo[v] * G.rfo[v];
          a = A * a;
        }
      }
      R x = affine_entry_up<R, W>(lane, a, b);
#pragma unroll
      for (int v = 0; v < VL; v++) {
        if (lv.first(v)) x = nb[h][v];
        else if (lv.in(v)) x = (nb[h][v] * G.fo[v] + x * small) * G.rfo[v];
        yf[h][v] = x;
      }
    }
  } else {
#pragma unroll
    for (int h = 0; h < NF; h++)
#pragma unroll
      for (int v = 0; v < VL; v++) yf[h][v] = y[h][v];
  }
  bool bad = false;
#pragma unroll
  for (int h = 0; h < NF; h++) {
    const R ym = __shfl_up_sync(0xffffffffu, yf[h][VL - 1], 1, W);
    const R yp = __shfl_down_sync(0xffffffffu, yf[h][0], 1, W);
    R after;
    // slopes, fluxes and new values; plain: of values that are not finite
    auto advect = [&](bool plain) {
      // PLM slopes (zero in the end layers)
      R bk[VL];
#pragma unroll
      for (int v = 0; v < VL; v++) {
        const R fm = v > 0 ? yf[h][v - 1] : ym;
        const R fp = v < VL - 1 ? yf[h][v + 1] : yp;
        bk[v] = !lv.in(v) || lv.first(v) || lv.last(v) ? R(0)
                : plain ? plain_slope(fm, yf[h][v], fp) : plm_slope(fm, yf[h][v], fp);
      }
      // interface fluxes; one donor layer: vertfx = -dz * (fcdx * slab) / slab = -dz * fcdx
      const R bm = __shfl_up_sync(0xffffffffu, bk[VL - 1], 1, W);
      R fl[VL];
#pragma unroll
      for (int v = 0; v < VL; v++) {
        const bool up = (G.up >> v) & 1u;
        const R a = up ? yf[h][v] : (v > 0 ? yf[h][v - 1] : ym);
        const R b = up ? bk[v] : (v > 0 ? bk[v - 1] : bm);
        // (nothing passes an interface that stays, whatever lies beside it)
        fl[v] = G.nd[v] * (a + b * G.hh[v]);
        if (plain && G.nd[v] == R(0)) fl[v] = R(0);
      }
      const R fnext = __shfl_down_sync(0xffffffffu, fl[0], 1, W);
      after = R(0);
#pragma unroll
      for (int v = 0; v < VL; v++) {
        if (lv.in(v)) {
          const R vn = !lv.last(v) ? (v < VL - 1 ? fl[v + 1] : fnext) : R(0);
          const R amount = yf[h][v] * G.fo[v] - (vn - fl[v]);
          after += amount;
          y[h][v] = (amount + yf[h][v] * small) * G.rfn[v];
        }
      }
    };
    advect(sizeof(R) == 4);
    if constexpr (sizeof(R) == 8) {
      R dif = bfore[h] - after, scl = colscl[h];
      warp_sum2<R, W>(lane, dif, scl);
      bad |= cabs(dif) > floor_at(col_tol<R>(1.e-11) * scl, R(1.e-33));
      // (the same in every lane of the column; the warp's columns go together)
      if (__any_sync(0xffffffffu, f64_odd(dif))) advect(true);
    }
  }
  return bad;
}

// remap_1d's fill of thin layers from above for tracers 2..ntra (thktop = 0):
// y(k) = (y(k) dp(k) + y(k-1) small) / (dp(k) + small), k = 3..nvl
template <typename R, int VL, int NF, int W, bool FULL>
__device__ __forceinline__ void fill_from_above(int L, int lane, R (&y)[NF][VL], const R (&dpv)[VL],
                                                const R (&qqv)[VL]) {
  const R small = R(1.e-6);
  const int kb = lane * VL;
#pragma unroll
  for (int h = 0; h < NF; h++) {
    R a = R(1), b = R(0);
#pragma unroll
    for (int v = 0; v < VL; v++) {
      const int k = kb + v;
      if (k < 2) {
        a = R(0);
        b = y[h][v];
      } else if (k < L) {
        const R A = small * qqv[v];
        b = A * b + y[h][v] * dpv[v] * qqv[v];
        a = A * a;
      }
    }
    R x = affine_entry_up<R, W>(lane, a, b);
#pragma unroll
    for (int v = 0; v < VL; v++) {
      const int k = kb + v;
      if (k < 2) {
        x = y[h][v];
      } else if (k < L) {
        x = (y[h][v] * dpv[v] + x * small) * qqv[v];
        y[h][v] = x;
      }
    }
  }
}

// VL consecutive values at p (VL * sizeof(R) bytes, aligned to min(16, that))
template <typename R, int VL>
__device__ __forceinline__ void st_lane(R* p, const R (&y)[VL]) {
  if constexpr (VL * sizeof(R) <= 16) {
    stv<VL>(p, y);
  } else {
#pragma unroll
    for (int h = 0; h < VL; h += 2) {
      double2 t;
      t.x = y[h];
      t.y = y[h + 1];
      *reinterpret_cast<double2*>(p + h) = t;
    }
  }
}

// one lane's levels of a field column: VL wide when vec, else value by value
template <typename R, int VL>
__device__ __forceinline__ void store_levels(R* dst, int L, int kb, int vec, const R (&y)[VL]) {
  if (vec) {
    if (kb < L) st_lane<R, VL>(dst + kb, y);
  } else {
#pragma unroll
    for (int v = 0; v < VL; v++)
      if (kb + v < L) dst[kb + v] = y[v];
  }
}

// one lane's levels from shared memory (n of the VL lie in the column)
template <typename R, int VL, bool FULL>
__device__ __forceinline__ void ld_levels(const R* p, int n, R (&y)[VL]) {
  if constexpr (FULL && VL * sizeof(R) <= 16) {
    ldv<VL>(p, y);
  } else {
#pragma unroll
    for (int v = 0; v < VL; v++) y[v] = FULL || v < n ? p[v] : R(0);
  }
}

// tracer t (0-based, >= 1) of column i leaving the remap when tracer x
// thickness is formed here: hystat's floor for tracers 2 and 3 (applied to y,
// which the caller then stores), then trdp = y * dp (hystat.F90:90-101)
template <typename R, int VL>
__device__ __forceinline__ void tracer_out(int t, R qvmin, R qwmin, const R (&dp)[VL], R (&y)[VL], R* trdp,
                                           size_t NL, int i, int L, int kb, int vec) {
  if (t == 1 || t == 2) {
    const R floor = t == 1 ? qvmin : qwmin;
#pragma unroll
    for (int v = 0; v < VL; v++) y[v] = cmax(floor, y[v]);
  }
  R z[VL];
#pragma unroll
  for (int v = 0; v < VL; v++) z[v] = y[v] * dp[v];
  store_levels<R, VL>(trdp + (size_t)t * NL + (size_t)i * L, L, kb, vec, z);
}

// dffusn_lev (k_dffusn_lev's arithmetic; none without interface smoothing) and
// inflate (hybgen.F90:893-1007) of 32 columns a block: the smoothed interfaces
// are formed into shared memory with thread = (column, interface), one warp
// runs inflate up its columns, lane = column, and the result leaves as rows.
// Two kernels moved the interfaces through memory in between.  A small grid
// takes wide blocks (256 threads, glvl 5 / nvl 38: 25 -> 16 us, FP64 63 -> 53), one
// of more than four blocks an SM narrow ones, whose serial warps are then more
// of those resident (64 threads, glvl 8 / nvl 64: 0.40 -> 0.36 ms; 256: 0.54).
constexpr int kInfCols = 32;
constexpr int kInfBlock = 256;
template <typename R>
__global__ void __launch_bounds__(kInfBlock) k_smooth_inflate(Grid<R> g, Strides s, Knobs kn,
    const StepParams* __restrict__ sp, int k1, int k2, const R* __restrict__ pr3d, const R* __restrict__ fld,
    R* __restrict__ out, int bnd) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int N = g.N, L = g.L, L1 = L + 1, LS = L1 | 1;  // odd row stride: lane = column is conflict-free
  R* const col = reinterpret_cast<R*>(smraw);           // [32][LS]
  R* const d0 = col + kInfCols * LS;                    // rd dpsig / p1000 [L]
  const int i0 = blockIdx.x * kInfCols;
  const int ncol = N - i0 < kInfCols ? N - i0 : kInfCols;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active || (bnd && sp->its <= 1)) return;
  pr3d += m * s.intf; fld += m * s.intf; out += m * s.intf;
  for (int k = threadIdx.x; k < L; k += blockDim.x) d0[k] = R(kRd) * g.dpsig[k] / R(kP1000);
#pragma unroll 4
  for (int q = threadIdx.x; q < ncol * L1; q += blockDim.x) {
    const int r = q / L1, k = q - r * L1, i = i0 + r;
    R v = fld[(size_t)i0 * L1 + q];
    R x[6];
#pragma unroll
    for (int e = 0; e < 6; e++) x[e] = fld[(size_t)g.prox[i * 6 + e] * L1 + k];
    if (k >= k1 && k <= k2) {
      const int np = g.nprox[i];
      R flxdv = R(0);
#pragma unroll
      for (int e = 0; e < 6; e++)
        if (e < np) flxdv = flxdv + (v - x[e]) * g.sideln[i * 6 + e];
      const R factor = -g.smoo[k] * g.rarea[i];
      v = v + flxdv * factor;
    }
    col[r * LS + k] = v;
  }
  __syncthreads();
  if ((int)threadIdx.x < ncol)
    inflate<R>(kn, [&](int k) { return d0[k]; }, L, pr3d[(size_t)(i0 + threadIdx.x) * L1], col + threadIdx.x * LS);
  __syncthreads();
#pragma unroll 4
  for (int q = threadIdx.x; q < ncol * L1; q += blockDim.x) {
    const int r = q / L1;
    out[(size_t)i0 * L1 + q] = col[r * LS + (q - r * L1)];
  }
}

// vec: every field column starts on a min(16, VL*sizeof(R))-byte boundary
// and nvl is a multiple of VL (the copies and stores are then VL wide)
// WL: lanes per column (32, or 16 with two columns per warp in hand)
template <typename R, int VL, int WL, bool FULL>
__global__ void __launch_bounds__(32 * kWarpsRemapV) k_remap_v(Grid<R> g, Strides s, Knobs kn,
    const StepParams* __restrict__ sp, const R* __restrict__ targt, const R* __restrict__ exsmo,
    R* __restrict__ us3d, R* __restrict__ vs3d, R* __restrict__ tr3d, R* __restrict__ sdot,
    R* __restrict__ ex3d, R* __restrict__ dp3d, R* __restrict__ pr3d, int* __restrict__ flags, int bnd,
    int vec, R* __restrict__ trdp, int cpw) {
  constexpr int H = 32 / WL;  // columns in hand per warp
  using SW = RemapV<R, VL, H>;
  constexpr int D = SW::D;
  constexpr int CB = VL * (int)sizeof(R) < 16 ? VL * (int)sizeof(R) : 16;  // bytes per copy
  constexpr int CE = CB / (int)sizeof(R);                                  // values per copy
  // fields whose pcwise runs interleaved (register budget)
  constexpr int NT = (sizeof(R) == 4 && VL <= 2) ? 3 : 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int N = g.N, L = g.L, L1 = L + 1, T = g.T;
  const int c0 = (blockIdx.x * kWarpsRemapV + wib) * cpw;
  const int ncol = N - c0 < cpw ? max(N - c0, 0) : cpw;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active || (bnd && sp->its <= 1)) return;
  SW& S = reinterpret_cast<SW*>(smraw)[wib];
  exsmo += m * s.intf; us3d += m * s.cell; vs3d += m * s.cell; tr3d += m * s.tr; sdot += m * s.intf;
  ex3d += m * s.intf; dp3d += m * s.cell; pr3d += m * s.intf;
  if (trdp) trdp += m * s.tr;
  const int its = sp->its - bnd;
  const R small = R(1.e-6), sl = R(kn.slak);
  const bool fill = kn.thktop == 0.;  // remap_1d's fill of thin layers
  // hystat's floors of tracers 2 and 3 (hystat.F90:90-93) when trdp is formed here
  const R qvmin = R(kQvmin), qwmin = R(kQwmin);
  const int hw = lane / WL, ls = lane - hw * WL;  // column in hand, lane within it
  const int kb = ls * VL;
  const int ngroups = (ncol + H - 1) / H;            // columns gc*H + hw, gc < ngroups
  // fields in order o: 0 = theta, 1 = u, 2 = v, 3.. = tracers 2..ntra;
  // items per column: the interface arrays (ex3d, pr3d, exsmo), then the
  // fields three by three
  const int F = min(T, sp->ntr) + 2, I = 1 + (F + 2) / 3;
  auto field = [&](int o, int i) -> R* {
    return o == 1 ? us3d + (size_t)i * L : o == 2 ? vs3d + (size_t)i * L
         : tr3d + ((size_t)(o == 0 ? 0 : o - 2) * N + i) * L;
  };
  // copy item j of the columns gc*H + hw into ring slot q (an empty group past the last)
  auto issue = [&](int gc, int j, int q) {
    if (gc < ngroups && gc * H + hw < ncol) {
      const int i = c0 + gc * H + hw;
      if (j == 0) {
#pragma unroll
        for (int h = 0; h < 3; h++) {
          const R* src = (h == 0 ? ex3d : h == 1 ? pr3d : exsmo) + (size_t)i * L1;
          for (int k = ls; k <= L; k += WL) cp_async<sizeof(R)>(&S.ring[q][hw][h][k], src + k);
        }
      } else {
#pragma unroll
        for (int h = 0; h < 3; h++) {
          const int o = 3 * (j - 1) + h;
          if (o < F) {
            const R* src = field(o, i);
            if (vec) {
              if (kb < L) {
#pragma unroll
                for (int e = 0; e < VL; e += CE) cp_async<CB>(&S.ring[q][hw][h][kb + e], src + kb + e);
              }
            } else {
#pragma unroll
              for (int v = 0; v < VL; v++)
                if (kb + v < L) cp_async<sizeof(R)>(&S.ring[q][hw][h][kb + v], src + kb + v);
            }
          }
        }
      }
    }
    cp_async_commit();
  };
  for (int k = lane; k < L; k += 32) S.tg[k] = targt[k];
  int ic = 0, ij = 0;   // next item to copy
  for (int q = 0; q < D; q++) {
    issue(ic, ij, q);
    if (++ij == I) { ij = 0; ++ic; }
  }
  LaneGeo<R, VL> gp;
  R dpv[VL], qqv[VL];
  bool bad = false;
  int gc = 0, j = 0, qs = 0;   // item in hand: column group, item, ring slot
  while (gc < ngroups) {
    cp_async_wait<D - 1>();
    __syncwarp();
    const int cs = gc * H + hw;            // this lane's column (index within the warp)
    const bool valid = cs < ncol;          // the second column of a last odd group is idle
    const int i = c0 + (valid ? cs : 0);
    R y[3][VL];
    if (j == 0) {
      for (int k = ls; k <= L; k += WL) {
        S.exold[hw][k] = S.ring[qs][hw][0][k];
        S.prcol[hw][k] = S.ring[qs][hw][1][k];
        S.exnew[hw][k] = S.ring[qs][hw][2][k];
      }
    } else {
#pragma unroll
      for (int h = 0; h < 3; h++) ld_levels<R, VL, FULL>(&S.ring[qs][hw][h][kb], L - kb, y[h]);
    }
    __syncwarp();
    issue(ic, ij, qs);   // D items ahead, into the slot just read
    if (++ij == I) { ij = 0; ++ic; }
    if (j == 0) {
      // new interfaces (exsmo -> exnew), pressures and p^(kappa+1) of the column
      for (int k = ls; k <= L; k += WL) {
        const R eo = S.exold[hw][k];
        R en = S.exnew[hw][k];
        if (its > 0) {
          en = sl * en + (R(1) - sl) * eo;
        }
        S.exnew[hw][k] = en;
        S.pk1col[hw][k] = by_cp(eo * S.prcol[hw][k]);
      }
      __syncwarp();
      // miglim = 1: exnew(2..nvl) between the neighbouring old interfaces
      for (int k = 2 + ls; k <= L; k += WL)
        S.exnew[hw][k - 1] = cmax(R(.0001) * S.exold[hw][k - 1] + R(.9999) * S.exold[hw][k],
                              cmin(R(.0001) * S.exold[hw][k - 1] + R(.9999) * S.exold[hw][k - 2], S.exnew[hw][k - 1]));
      __syncwarp();
      for (int k = ls; k <= L; k += WL) {
        const R en = S.exnew[hw][k];
        const R pn = pressure_of(en);
        S.prnew[hw][k] = pn;
        S.pk1new[hw][k] = by_cp(en * pn);
      }
      __syncwarp();
      for (int k = ls; k < L; k += WL) S.dpcol[hw][k] = S.prnew[hw][k] - S.prnew[hw][k + 1];
      __syncwarp();
      if (ls == 0) {
        S.prnew[hw][L] = S.prcol[hw][L];
        S.pk1new[hw][L] = S.pk1col[hw][L];
        S.prnew[hw][0] = S.prcol[hw][0];
        S.pk1new[hw][0] = S.pk1col[hw][0];
        S.flo[cs] = S.pk1col[hw][0] * small;
      }
      __syncwarp();
      for (int k = ls; k < L; k += WL) S.dkb[cs][k] = S.pk1new[hw][k] - S.pk1new[hw][k + 1];
      if (trdp)
        for (int k = ls; k < L; k += WL) S.dpb[cs][k] = S.dpcol[hw][k];
      lane_geo<R, VL, WL, FULL>(L, ls, S.prcol[hw], S.prnew[hw], gp);
      ld_levels<R, VL, FULL>(&S.dpcol[hw][kb], L - kb, dpv);
#pragma unroll
      for (int v = 0; v < VL; v++) {
        qqv[v] = sizeof(R) == 4 || fill ? fdiv(R(1), dpv[v] + small) : R(0);
      }
      __syncwarp();
    } else if (j == 1) {
      // theta in p^(kappa+1), held for the redistribution after the last column
      {
        LaneGeo<R, VL> gk;
        lane_geo<R, VL, WL, FULL>(L, ls, S.pk1col[hw], S.pk1new[hw], gk);
        {
          R colin = R(0), colscl = R(0);
#pragma unroll
          for (int v = 0; v < VL; v++)
            if (FULL || kb + v < L) {
              const R w = y[0][v] * (S.pk1col[hw][kb + v] - S.pk1col[hw][kb + v + 1]);
              colin += w;
              colscl += cabs(w);
            }
          colin = warp_sum<R, WL>(colin);
          colscl = warp_sum<R, WL>(colscl);
          if (ls == 0) {
            S.colin[cs] = colin;
            S.colscl[cs] = colscl;
          }
        }
        R t[1][VL];
#pragma unroll
        for (int v = 0; v < VL; v++) t[0][v] = y[0][v];
        const bool bt = pcwise_v<R, VL, 1, WL, FULL>(L, ls, t, gk);
        bad |= valid && bt;
        if constexpr (FULL) {
          st_lane<R, VL>(&S.thb[cs][kb], t[0]);
        } else {
#pragma unroll
          for (int v = 0; v < VL; v++)
            if (kb + v < L) S.thb[cs][kb + v] = t[0][v];
        }
      }
      // u, v in pressure
      if constexpr (NT == 3) {
        R uv[2][VL];
#pragma unroll
        for (int v = 0; v < VL; v++) {
          uv[0][v] = y[1][v];
          uv[1][v] = y[2][v];
        }
        const bool bu = pcwise_v<R, VL, 2, WL, FULL>(L, ls, uv, gp);
        bad |= valid && bu;
        if (valid) {
          store_levels<R, VL>(us3d + (size_t)i * L, L, kb, vec, uv[0]);
          store_levels<R, VL>(vs3d + (size_t)i * L, L, kb, vec, uv[1]);
        }
      } else {
#pragma unroll
        for (int h = 1; h < 3; h++) {
          R t[1][VL];
#pragma unroll
          for (int v = 0; v < VL; v++) t[0][v] = y[h][v];
          const bool bu = pcwise_v<R, VL, 1, WL, FULL>(L, ls, t, gp);
          bad |= valid && bu;
          if (valid) store_levels<R, VL>(field(h, i), L, kb, vec, t[0]);
        }
      }
    } else {
      // tracers 2..ntra in pressure
      const int o0 = 3 * (j - 1);
      if constexpr (NT == 3) {
        const bool bq = pcwise_v<R, VL, 3, WL, FULL>(L, ls, y, gp);
        bad |= valid && bq;
        if (fill) fill_from_above<R, VL, 3, WL, FULL>(L, ls, y, dpv, qqv);
#pragma unroll
        for (int h = 0; h < 3; h++)
          if (valid && o0 + h < F) {
            if (trdp) tracer_out<R, VL>(o0 + h - 2, qvmin, qwmin, dpv, y[h], trdp, (size_t)N * L, i, L, kb, vec);
            store_levels<R, VL>(field(o0 + h, i), L, kb, vec, y[h]);
          }
      } else {
#pragma unroll
        for (int h = 0; h < 3; h++) {
          if (o0 + h < F) {
            R t[1][VL];
#pragma unroll
            for (int v = 0; v < VL; v++) t[0][v] = y[h][v];
            const bool bq = pcwise_v<R, VL, 1, WL, FULL>(L, ls, t, gp);
            bad |= valid && bq;
            if (fill) fill_from_above<R, VL, 1, WL, FULL>(L, ls, t, dpv, qqv);
            if (valid) {
              if (trdp) tracer_out<R, VL>(o0 + h - 2, qvmin, qwmin, dpv, t[0], trdp, (size_t)N * L, i, L, kb, vec);
              store_levels<R, VL>(field(o0 + h, i), L, kb, vec, t[0]);
            }
          }
        }
      }
    }
    if (j == I - 1) {
      // exnew made non-increasing downward: prefix minimum over the
      // interfaces; the column's lane l holds interfaces l*VL .. l*VL+VL-1
      // (running minimum within the lane, one scan of the lane minima over
      // the column's WL lanes), interface nvl (when WL*VL == nvl) takes the
      // minimum over all of them
      const size_t ci = (size_t)i * L1;
      const R top = S.exnew[hw][0];  // fill: no interface lies above the column top
      R pm[VL];
#pragma unroll
      for (int v = 0; v < VL; v++) {
        const int k = kb + v;
        const R x = k <= L ? S.exnew[hw][k] : top;
        pm[v] = v == 0 ? x : cmin(pm[v - 1], x);
      }
      R tot = pm[VL - 1];
#pragma unroll
      for (int off = 1; off < WL; off <<= 1) {
        const R o = __shfl_up_sync(0xffffffffu, tot, off, WL);
        if (ls >= off) tot = cmin(tot, o);
      }
      const R above = __shfl_up_sync(0xffffffffu, tot, 1, WL);
      const R all = __shfl_sync(0xffffffffu, tot, WL - 1, WL);
#pragma unroll
      for (int v = 0; v < VL; v++) {
        const int k = kb + v;
        if (valid && k <= L) {
          const R x = ls > 0 ? cmin(pm[v], above) : pm[v];
          sdot[ci + k] = x - S.exold[hw][k];
          ex3d[ci + k] = x;
          pr3d[ci + k] = S.prnew[hw][k];
          if (k < L) dp3d[(size_t)i * L + k] = S.dpcol[hw][k];
        }
      }
      if (valid && WL * VL == L && ls == 0) {
        const R x = cmin(S.exnew[hw][L], all);
        sdot[ci + L] = x - S.exold[hw][L];
        ex3d[ci + L] = x;
        pr3d[ci + L] = S.prnew[hw][L];
      }
      __syncwarp();
    }
    if (++j == I) { j = 0; ++gc; }
    if (++qs == D) qs = 0;
  }
  cp_async_wait<0>();
  __syncthreads();
  // theta redistribution among neighbouring layers (hybgen.F90:648-667),
  // lane = column over the block's columns: pairs (k-1, k) from the bottom up,
  // each pair seeing the upper layer of the pair below as already adjusted.
  // One warp sweeps for all four: the sweep's instructions cost the same for
  // 8 columns as for 32 (a fifth of the FP64 kernel when each warp swept its
  // own).
  static_assert(kWarpsRemapV * kColsPerWarp <= 32, "one lane a column of the block");
  const int sw = lane / kColsPerWarp, sc = lane - sw * kColsPerWarp;
  if (wib == 0 && L >= 3 && sc < cpw && (blockIdx.x * kWarpsRemapV + sw) * cpw + sc < N) {
    SW& Q = reinterpret_cast<SW*>(smraw)[sw];
    R* th = Q.thb[sc];
    const R* dk = Q.dkb[sc];
    const R fl = Q.flo[sc];
    R thb = th[L - 1], dkup = cmax(dk[L - 1], fl);
    R dev = (thb - S.tg[L - 1]) * dkup;
    for (int k = L; k >= 3; k--) {
      const R tha = th[k - 2];
      const R dplo = cmax(dk[k - 2], fl), dpup = dkup;
      const R devilo = (tha - S.tg[k - 2]) * dplo;
      const R deviup = dev;
      R na = tha, nbv = thb;
      if (lt(R(0), deviup) && lt(devilo, R(0))) {
        const R cc = cmin(deviup, -devilo);
        na = tha + divide(cc, dplo);
        nbv = thb - divide(cc, dpup);
      } else if (lt(deviup, R(0)) && lt(R(0), devilo)) {
        const R cc = cmin(devilo, -deviup);
        na = tha - divide(cc, dplo);
        nbv = thb + divide(cc, dpup);
      }
      th[k - 1] = nbv;
      thb = na;
      dkup = dplo;
      dev = (thb - S.tg[k - 2]) * dkup;
    }
    th[1] = thb;
    {
      R clout = R(0);
      for (int k = 0; k < L; k++) clout = clout + th[k] * dk[k];
      if (cabs(clout - Q.colin[sc]) > cmax(R(1.e-33), col_tol<R>(2.e-6) * Q.colscl[sc])) bad = true;
    }
  }
  __syncthreads();
  for (int cc = hw; cc < ncol; cc += H) {
    R y[VL];
    ld_levels<R, VL, FULL>(&S.thb[cc][kb], L - kb, y);
    store_levels<R, VL>(tr3d + (size_t)(c0 + cc) * L, L, kb, vec, y);
    if (trdp) {
      R z[VL];
#pragma unroll
      for (int v = 0; v < VL; v++) z[v] = kb + v < L ? y[v] * S.dpb[cc][kb + v] : R(0);
      store_levels<R, VL>(trdp + (size_t)(c0 + cc) * L, L, kb, vec, z);
    }
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(flags + m, kFlagColumnIntegral);
}

template <typename R, int VL, int WL>
size_t remap_v_smem() { return sizeof(RemapV<R, VL, 32 / WL>) * kWarpsRemapV; }
template <typename R>
size_t inflate_smem(int L) { return sizeof(R) * (kInfCols * (size_t)((L + 1) | 1) + L); }

// levels per lane of k_remap_v
inline int remap_vl(int L) { return L <= 32 ? 1 : L <= 64 ? 2 : 4; }

// two columns per warp (16 lanes x 4 levels) for FP32 with 32 < nvl <= 64:
// each ring item, scan and shuffle then serves two columns
template <typename R>
inline bool remap_paired(int L) { return sizeof(R) == 4 && L > 32 && L <= 64; }

// Columns a warp of k_remap_v takes in turn.  Many columns a warp amortise its
// start (the first copies, the theta sweep); few leave small grids no nearly
// empty last round of blocks.  FP64 (two blocks an SM by shared memory): the
// rounds of 2 x 152 blocks times (columns + 1/2) follow the measured times at
// glvl 6 / nvl 64 (8 columns 3.07 ms, 6: 2.81, 4: 2.90, 2: 2.98) and glvl 5 / nvl 38
// (6: 0.59, 4: 0.60, 2: 0.55).  FP32: all blocks of a small grid are resident and
// share their SM, blocks an SM times (columns + 3): glvl 5 / nvl 38 8: 62 us,
// 6: 51, 4: 69; glvl 8 / nvl 64 8: 2.95 ms, 6: 3.01, 4: 3.12.  (Two columns a warp
// would be taken by grids of a few hundred columns alone.)
template <typename R>
int remap_columns(int N, int members, bool paired) {
  const int sms = sm_count();
  const long long slots = sizeof(R) == 8 ? 2 * sms : sms;
  long long best = -1;
  int cols = kColsPerWarp;
  for (int c = kColsPerWarp; c >= (paired ? 4 : 3); c -= paired ? 2 : 1) {
    const long long nb = (long long)nblocks(N, kWarpsRemapV * c) * members;
    const long long cost = (nb + slots - 1) / slots * (sizeof(R) == 8 ? 2 * c + 1 : 2 * c + 6);
    if (best < 0 || cost < best) { best = cost; cols = c; }
  }
  return cols;
}

template <typename R, int VL, int WL>
cudaError_t remap_v_attr() {
  const int bytes = (int)remap_v_smem<R, VL, WL>();
  const cudaError_t e =
      cudaFuncSetAttribute(k_remap_v<R, VL, WL, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  return e != cudaSuccess ? e
                          : cudaFuncSetAttribute(k_remap_v<R, VL, WL, false>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

template <typename R>
int prepare_hybgen(int L) {
  cudaError_t e = cudaSuccess;
  const int vl = remap_vl(L);
  if (remap_paired<R>(L)) {
    if constexpr (sizeof(R) == 4) e = remap_v_attr<R, 4, 16>();
  } else if (vl == 1) e = remap_v_attr<R, 1, 32>();
  else if (vl == 2) e = remap_v_attr<R, 2, 32>();
  else e = remap_v_attr<R, 4, 32>();
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_smooth_inflate<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)inflate_smem<R>(kMaxL));
  return e == cudaSuccess ? 0 : (int)e;
}

// ---------------------------------------------------------------- hystat --
// hystat (hystat.F90:53-109), 32 columns a block.  The recursions up the
// columns are the surface pressure sum (warp 0) and the Montgomery potential
// (warp 1), lane = column over shared tiles in the reference's order, in FP64
// (FP64 build) or float-float (FP32-mixed build, which also keeps the (hi, lo)
// Montgomery potential for the pressure gradient).  What each level adds to the
// potential, Exner(k) (theta(k) - theta(k-1)), is formed before and the
// geopotential at each interface after with thread = (column, VK levels).  The
// humidity floors and tracer x thickness are k_hystat_trdp.  One warp doing
// all of it for its 32 columns, 16 levels at a time, kept two warps an SM in
// flight at glvl 5: 25 -> 11 us at glvl 5 / nvl 38, 137 -> 71 us at glvl 7 / nvl
// 64, 0.47 -> 0.35 ms at glvl 8 (FP32), 36 -> 17 us in FP64 at glvl 5.
constexpr int kHyCols = 32;
constexpr int kHyBlock = 256;
template <typename R, int VK>
__global__ void __launch_bounds__(kHyBlock) k_hystat(Grid<R> g, Strides s, const StepParams* __restrict__ sp,
    R* __restrict__ ph3d, const R* __restrict__ ex3d, R* __restrict__ mp3d, const R* __restrict__ dp3d,
    const R* __restrict__ tr3d, R* __restrict__ psrf, R* __restrict__ ptdcy,
    float2* __restrict__ mpf, int bnd) {
  constexpr bool FFB = sizeof(R) == 4;
  extern __shared__ __align__(16) unsigned char hysm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int N = g.N, L = g.L, L1 = L + 1, LV = L / VK;
  const int LS = L | 1;  // odd row stride: lane = column reads are conflict-free
  R* const td = reinterpret_cast<R*>(hysm);  // thickness
  R* const tm = td + kHyCols * LS;           // a level's term, then the potential
  R* const tl = tm + kHyCols * LS;           // their low parts (FP32)
  const int i0 = blockIdx.x * kHyCols;
  const int ncol = N - i0 < kHyCols ? N - i0 : kHyCols;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active || (bnd && sp->its <= 1)) return;
  ph3d += m * s.intf; ex3d += m * s.intf; mp3d += m * s.cell; dp3d += m * s.cell; tr3d += m * s.tr;
  psrf += m * s.col; ptdcy += m * 2 * s.col;
  if (mpf) mpf += m * s.cell;
  const int its = sp->its - bnd;
  for (int it = threadIdx.x; it < ncol * LV; it += kHyBlock) {
    const int r = it / LV, k = (it - r * LV) * VK;
    const size_t c = (size_t)(i0 + r) * L + k, ci = (size_t)(i0 + r) * L1 + k;
    R d[VK], t[VK], e[VK];
    ldv<VK>(dp3d + c, d);
    ldv<VK>(tr3d + c, t);
    R tp = k > 0 ? tr3d[c - 1] : R(0);
    FOR_V e[j] = ex3d[ci + j];
    FOR_V {
      const int o = r * LS + k + j;
      td[o] = d[j];
      if constexpr (FFB) {
        FF2 term;
        if (k + j == 0) {
          term = ff_add(two_prod(e[j], t[j]), FF2{ph3d[ci], 0.f});
        } else {
          const FF2 dd = two_sum(t[j], -tp);
          term = ff_add(two_prod(e[j], dd.hi), FF2{e[j] * dd.lo, 0.f});
        }
        tm[o] = term.hi;
        tl[o] = term.lo;
      } else {
        tm[o] = k + j == 0 ? e[j] * t[j] + ph3d[ci] : e[j] * (t[j] - tp);
      }
      tp = t[j];
    }
  }
  __syncthreads();
  if (lane < ncol) {
    if (wib == 0) {
      const R* q = td + lane * LS;
      R pn;
      if constexpr (FFB) {
        FF2 ps{0.f, 0.f};
#pragma unroll 4
        for (int k = 0; k < L; k++) ps = ff_add(ps, FF2{q[k], 0.f});
        pn = ps.hi;
      } else {
        pn = R(0);
#pragma unroll 4
        for (int k = 0; k < L; k++) pn += q[k];
      }
      const int i = i0 + lane;
      const R work = psrf[i];
      psrf[i] = pn;
      if (its > 0) ptdcy[(size_t)(its % 2) * N + i] = pn - work;
    } else if (wib == 1) {
      R* q = tm + lane * LS;
      if constexpr (FFB) {
        float* ql = (float*)tl + lane * LS;
        FF2 mp{q[0], ql[0]};
#pragma unroll 4
        for (int k = 1; k < L; k++) {
          mp = ff_add(mp, FF2{q[k], ql[k]});
          q[k] = mp.hi;
          ql[k] = mp.lo;
        }
      } else {
        R mp = q[0];
#pragma unroll 4
        for (int k = 1; k < L; k++) {
          mp = mp + q[k];
          q[k] = mp;
        }
      }
    }
  }
  __syncthreads();
  for (int it = threadIdx.x; it < ncol * LV; it += kHyBlock) {
    const int r = it / LV, k = (it - r * LV) * VK;
    const size_t c = (size_t)(i0 + r) * L + k, ci = (size_t)(i0 + r) * L1 + k;
    R t[VK], mo[VK];
    ldv<VK>(tr3d + c, t);
    FOR_V {
      const int o = r * LS + k + j;
      const R e1 = ex3d[ci + j + 1];  // the interface above
      mo[j] = tm[o];
      if constexpr (FFB) {
        if (mpf) mpf[c + j] = make_float2(tm[o], tl[o]);
        ph3d[ci + j + 1] = ff_add(FF2{tm[o], tl[o]}, ff_neg(two_prod(t[j], e1))).hi;
      } else {
        ph3d[ci + j + 1] = tm[o] - t[j] * e1;
      }
    }
    stv<VK>(mp3d + c, mo);
  }
}

// hystat.F90:72-98, the per-level part: humidity floors and tracer x
// thickness, VK levels per thread (a stream over all tracers of a column
// slice; kept apart from the column scans so its loads are not serialised
// behind them)
template <typename R, int VK>
__global__ void __launch_bounds__(kBlock2) k_hystat_trdp(Grid<R> g, Strides s, const StepParams* __restrict__ sp,
    const R* __restrict__ dp3d, R* __restrict__ tr3d, R* __restrict__ trdp, int bnd) {
  int i, k;
  if (!cell_levels<VK>(g.N, g.L, i, k)) return;
  const int N = g.N, L = g.L;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active || (bnd && sp->its <= 1)) return;
  const int T = min(g.T, sp->ntr);
  const size_t NL = (size_t)N * L;
  const size_t c = (size_t)i * L + k;
  dp3d += m * s.cell; tr3d += m * s.tr; trdp += m * s.tr;
  const R qvmin = R(kQvmin), qwmin = R(kQwmin);
  R dp[VK];
  ldv<VK>(dp3d + c, dp);
#pragma unroll 4
  for (int t = 0; t < T; t++) {
    R x[VK], y[VK];
    ldv<VK>(tr3d + (size_t)t * NL + c, x);
    if (t == 1 || t == 2) {
      const R floor = t == 1 ? qvmin : qwmin;
      FOR_V x[j] = cmax(floor, x[j]);
      stv<VK>(tr3d + (size_t)t * NL + c, x);
    }
    FOR_V y[j] = x[j] * dp[j];
    stv<VK>(trdp + (size_t)t * NL + c, y);
  }
}

// --------------------------------------------------------------- globsum --
// float-float compensated accumulator (Knuth two-sum), ~48-bit significand
struct FF {
  float hi, lo;
  __device__ void add(float x) {
    const float s = hi + x;
    const float bp = s - hi;
    const float err = (hi - (s - bp)) + (x - bp);
    hi = s;
    lo += err;
  }
  __device__ double value() const { return (double)hi + (double)lo; }
};
template <typename R> struct Acc;
template <> struct Acc<double> {
  double v = 0.0;
  __device__ void add(double x) { v += x; }
  __device__ double value() const { return v; }
};
template <> struct Acc<float> {
  FF f{0.f, 0.f};
  __device__ void add(float x) { f.add(x); }
  __device__ double value() const { return f.value(); }
};

constexpr int kMaxT = 32;

// Slots of one block's partial sums: 0 = sum(area*dp), 1+t = sum(area*dp*tr_t)
// (level sums), kMaxT+1.. = the column sums of globsum.F90:81-85
// (rain, convective rain, non-convective rain, latent energy).
constexpr int kGsCol = kMaxT + 1;
constexpr int kGsSlots = kMaxT + 5;

// Level sums: a block takes one chunk of 256 VK iters cell-levels and a
// group of kGsGroup consecutive slots q (0: area x dp, 1..ntr: area x dp x
// tracer q-1): it reads the chunk's thicknesses and cell areas once for the
// group and one tracer array per slot.  The group holding slot 0 also forms
// the column sums of the cells whose first level lies in the chunk.  Every
// slot is summed per thread in level order and per block in a fixed order,
// and the partials are per (chunk, slot): the sums are deterministic and do
// not depend on the grouping.
constexpr int kGsGroup = 7;
// Iterations of a block: 16 where that leaves 1.5 blocks an SM, fewer for
// small grids.  (A block's reduction takes ~60 FP64 operations a warp, so many
// short blocks cost more than an idle SM: glvl 5 / nvl 38, one level a thread:
// 760 blocks of two iterations 33 us, 380 of four 21 us.)
// A function of the grid alone, the blocks a constant (1.5 of 152 SMs): the
// order of the sums depends on neither the tracers or members beside them nor
// the device.
inline int gs_iters(long long NL, int vk) {
  int it = 16;
  while (it > 1 && NL / ((long long)kBlock2 * vk * it) < 228) it /= 2;
  return it;
}
inline int gs_chunks(long long NL, int vk) {
  const long long per = (long long)kBlock2 * vk * gs_iters(NL, vk);
  return (int)((NL + per - 1) / per);
}

template <typename R, int VK> struct GsVec;
template <typename R> struct GsVec<R, 1> {
  static __device__ __forceinline__ void ld(const R* p, R (&r)[1]) { r[0] = *p; }
};
template <> struct GsVec<float, 4> {
  static __device__ __forceinline__ void ld(const float* p, float (&r)[4]) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    r[0] = t.x; r[1] = t.y; r[2] = t.z; r[3] = t.w;
  }
};
template <> struct GsVec<double, 2> {
  static __device__ __forceinline__ void ld(const double* p, double (&r)[2]) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    r[0] = t.x; r[1] = t.y;
  }
};

// One step of a warp's sums of 2 n values: the lanes with bit `off` set keep
// the upper n values' sums of their pair, the others the lower.
template <int n>
__device__ __forceinline__ void tree_step(int lane, int off, double* v) {
  const bool up = lane & off;
#pragma unroll
  for (int i = 0; i < n; i++) {
    const double give = up ? v[i] : v[n + i], keep = up ? v[n + i] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
  }
}
// sums of eight values over a warp: v[0] of a lane ends as the sum of value
// warp_tree8's result (the same in each four lanes)
__device__ __forceinline__ int warp_tree8(int lane, double (&v)[8]) {
  tree_step<4>(lane, 16, v);
  tree_step<2>(lane, 8, v);
  tree_step<1>(lane, 4, v);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return (lane & 16 ? 4 : 0) + (lane & 8 ? 2 : 0) + (lane & 4 ? 1 : 0);
}
__device__ __forceinline__ int warp_tree4(int lane, double (&v)[4]) {
  tree_step<2>(lane, 16, v);
  tree_step<1>(lane, 8, v);
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
  return (lane & 16 ? 2 : 0) + (lane & 8 ? 1 : 0);
}

template <typename R, int VK>
__global__ void __launch_bounds__(kBlock2) k_globsum_levels(Grid<R> g, Strides s, const StepParams* __restrict__ sp,
    int T, const R* __restrict__ dp3d, const R* __restrict__ tr, const R* __restrict__ rn2d, const R* __restrict__ rc2d,
    const R* __restrict__ pr3d, const R* __restrict__ ex3d, const R* __restrict__ qf2d,
    double* __restrict__ partial, int nchunk, int iters) {
  const int N = g.N, L = g.L, L1 = L + 1;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active) return;
  const int ngrp = (T + kGsGroup) / kGsGroup;  // groups of the T + 1 slots
  const int chunk = blockIdx.x / ngrp, q0 = (blockIdx.x - chunk * ngrp) * kGsGroup;
  const int nq = (T + 1 - q0 < kGsGroup) ? T + 1 - q0 : kGsGroup;
  dp3d += m * s.cell; tr += m * s.tr; pr3d += m * s.intf; ex3d += m * s.intf;
  // N * L < 2^31 (checked on the host): 32-bit cell-level indices
  const unsigned NL = (unsigned)N * (unsigned)L;
  const unsigned CH = kBlock2 * VK * (unsigned)iters;
  const unsigned e0 = (unsigned)chunk * CH;
  Acc<R> acc[kGsGroup];
  // the group's arrays: slot 0 reads the thicknesses again (an L1 hit) and
  // adds area x dp; slots past the last repeat slot T and add nothing, so
  // every load of an iteration is issued before the first sum
  const R* xp[kGsGroup];
  // tracers past the member's own count add nothing (and are not read)
  const int ntm = min(T, sp->ntr);
#pragma unroll
  for (int u = 0; u < kGsGroup; u++) {
    const int q = q0 + u <= T ? q0 + u : T;
    xp[u] = (q == 0 || q > ntm) ? dp3d : tr + (size_t)(q - 1) * NL;
  }
  auto sum_at = [&](unsigned idx) {
    const R ar = g.area[idx / (unsigned)L];
    R dp[VK], ad[VK], x[kGsGroup][VK];
    GsVec<R, VK>::ld(dp3d + idx, dp);
#pragma unroll
    for (int u = 0; u < kGsGroup; u++) GsVec<R, VK>::ld(xp[u] + idx, x[u]);
#pragma unroll
    for (int j = 0; j < VK; j++) ad[j] = ar * dp[j];
#pragma unroll
    for (int u = 0; u < kGsGroup; u++)
      if (u < nq && q0 + u <= ntm) {
#pragma unroll
        for (int j = 0; j < VK; j++) acc[u].add(u == 0 && q0 == 0 ? ad[j] : ad[j] * x[u][j]);
      }
  };
  if (e0 + CH <= NL) {
    for (int it = 0; it < iters; it++) sum_at(e0 + ((unsigned)it * kBlock2 + threadIdx.x) * VK);
  } else {
    for (int it = 0; it < iters; it++) {
      const unsigned idx = e0 + ((unsigned)it * kBlock2 + threadIdx.x) * VK;
      if (idx < NL) sum_at(idx);
    }
  }
  double col[4] = {0., 0., 0., 0.};
  if (q0 == 0) {
    const double dt = sp->dt, rdcp = kRd / kCp;
    const size_t i0 = ((size_t)e0 + L - 1) / L;
    size_t i1 = ((size_t)e0 + CH + L - 1) / L;
    if (i1 > (size_t)N) i1 = N;
    for (size_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
      const double a = g.area_d[i];
      const double rn = rn2d ? (double)rn2d[m * s.col + i] : 0.0;
      const double rc = rc2d ? (double)rc2d[m * s.col + i] : 0.0;
      const double qf = qf2d ? (double)qf2d[m * s.col + i] : 0.0;
      col[0] += a * rn;
      col[1] += a * rc;
      col[2] += a * (rn - rc);
      const double den = (double)pr3d[i * L1] / (rdcp * (double)ex3d[i * L1] * (double)tr[i * L]);
      col[3] += a * den * qf * dt / (1.25 * 2.5e6);
    }
  }
  // block sums: each warp's tree over its lanes (pairs 16, 8, 4, 2, 1 apart,
  // the slots of a group in different lanes from the first pair on, so a step
  // adds for all of them), then over the warps in order
  __shared__ double red[kBlock2 / 32][kGsGroup + 5];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  {
    double v[8];
#pragma unroll
    for (int u = 0; u < kGsGroup; u++) v[u] = acc[u].value();
    v[7] = 0.;
    const int u = warp_tree8(lane, v);
    if ((lane & 3) == 0 && u < kGsGroup) red[wib][u] = v[0];
  }
  if (q0 == 0) {
    const int w = warp_tree4(lane, col);
    if ((lane & 7) == 0) red[wib][kGsGroup + w] = col[0];
  }
  __syncthreads();
  double* out = partial + (m * nchunk + chunk) * kGsSlots;
  const int u = threadIdx.x;
  if (u < nq || (q0 == 0 && u >= kGsGroup && u < kGsGroup + 4)) {
    double t = 0.0;
    for (int w = 0; w < kBlock2 / 32; w++) t += red[w][u];
    out[u < nq ? q0 + u : kGsCol + (u - kGsGroup)] = t;
  }
}

// Final reduction of the block partials; one warp per output slot, a block per
// member and eight slots.
template <typename R>
__global__ void __launch_bounds__(kBlock2) k_globsum_final(const StepParams* __restrict__ sp, int T, const double* __restrict__ partial,
                                int nblk, double* __restrict__ sums) {
  const size_t m = blockIdx.x;
  sp += m;
  if (!sp->active) return;
  const int lane = threadIdx.x & 31;
  double* out = sums + m * (8 + T);
  const int j = blockIdx.y * (kBlock2 / 32) + (threadIdx.x >> 5);
  if (j < T + 5) {
    const int q = j <= T ? j : kGsCol + (j - T - 1);
    double t = 0.;
#pragma unroll 8
    for (int b = lane; b < nblk; b += 32) t += partial[(m * nblk + b) * kGsSlots + q];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
    if (lane != 0) return;
    if (q == 0) {
      out[0] = t / kGrvity;
    } else if (q <= T) {
      out[8 + (q - 1)] = t;
      if (q == 2) out[1] = t / kGrvity;
      if (q == 3) out[2] = t / kGrvity;
      if (q == 4) out[3] = t / kGrvity;
    } else {
      // qmstr (sumr), qmstrc (sumrc), qmstrn (sumrn), qmste (sume)
      const int c = q - kGsCol;
      out[c == 0 ? 5 : c == 1 ? 7 : c == 2 ? 6 : 4] = t;
    }
  }
}

// pressure and thickness from Exner (dyn_init.F90:895-906)
template <typename R>
__global__ void __launch_bounds__(kBlock2) k_prdp_from_ex(Grid<R> g, Strides s, const R* __restrict__ ex3d,
    R* __restrict__ pr3d, R* __restrict__ dp3d) {
  const int N = g.N, L = g.L, L1 = L + 1;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= N * L1) return;
  const int i = gid / L1, k = gid - i * L1;
  const size_t m = blockIdx.y;
  ex3d += m * s.intf; pr3d += m * s.intf; dp3d += m * s.cell;
  const R p = pressure_of(ex3d[(size_t)i * L1 + k]);
  pr3d[(size_t)i * L1 + k] = p;
  if (k < L) {
    const R pu = pressure_of(ex3d[(size_t)i * L1 + k + 1]);
    dp3d[(size_t)i * L + k] = p - pu;
  }
}


// k_regrid's column arrays in shared memory, a warp a block, while every warp
// of the launch fits the chip at once: the columns' serial chains then see
// shared-memory latency (glvl 5 / nvl 38: 41 against 59 us, FP64 125 against 144).
// Larger launches hide the latency of local memory behind more warps than
// shared memory holds (glvl 6 / nvl 64 x 4 members: 181 against 298 us; glvl 8
// 0.62 against 1.16 ms).
template <typename R>
bool regrid_in_smem(int N, int L, int members) {
  const size_t block = 32 * (size_t)(3 * L + 2) * sizeof(R) + (32 * 33 + 4 * (L <= 64 ? 64 : kMaxL)) * sizeof(R) + 1024;
  return (long long)nblocks(N, 32) * members <= (long long)sm_count() * (long long)(227 * 1024 / block);
}

template <typename R>
bool launch_hybgen(const Launch& l, const Grid<R>& g, const Strides& s, const Knobs& kn, const HybgenScratch<R>& w,
                   const R* targt, R* us3d, R* vs3d, R* tr3d, R* sdot, R* ex3d, R* dp3d, R* pr3d, R* trdp) {
  bool trdp_done = false;
  dim3 gc(nblocks(g.N, kColBlock), l.members);
  FIM_KBEGIN(l, "k_regrid");
  const bool rsm = regrid_in_smem<R>(g.N, g.L, l.members);
  const size_t rs = rsm ? (size_t)32 * (3 * g.L + 2) * sizeof(R) : 0;
  const dim3 gr(nblocks(g.N, rsm ? 32 : kColBlock), l.members);
#define FIM_REGRID(ML, SM)                                                                                    \
  do {                                                                                                        \
    if (rs > (size_t)24 * 1024)                                                                               \
      cudaFuncSetAttribute(k_regrid<R, ML, SM>, cudaFuncAttributeMaxDynamicSharedMemorySize,                  \
                           (int)(32 * (3 * ML + 2) * sizeof(R)));                                             \
    k_regrid<R, ML, SM><<<gr, SM ? 32 : kColBlock, rs, l.stream>>>(g, s, kn, l.sp, targt, tr3d, ex3d, pr3d,   \
                                                                   w.exsmo, l.flags, l.boundary);             \
  } while (0)
  if (g.L <= 64) {
    if (rsm) FIM_REGRID(64, true);
    else FIM_REGRID(64, false);
  } else if (rsm) FIM_REGRID(kMaxL, true);
  else FIM_REGRID(kMaxL, false);
#undef FIM_REGRID
  FIM_KEND(l);
  const R* ex_in = w.exsmo;
  // Fortran levels kbl+2..nvl -> 0-based interfaces kbl+1..nvl-1
  const int k1 = kn.kbl + 1, k2 = g.L - 1;
  const bool plm1 = kn.remap_optn == 2 && kn.miglim == 1;
  if (kn.intfc_smooth > 0. && plm1) {
    FIM_KBEGIN(l, "k_smooth_inflate");
    const unsigned nb = nblocks(g.N, kInfCols);
    const int tb = (long long)nb * l.members <= 4ll * sm_count() ? kInfBlock : kInfBlock / 4;
    k_smooth_inflate<R><<<dim3(nb, l.members), tb, inflate_smem<R>(g.L), l.stream>>>(
        g, s, kn, l.sp, k1, k2, pr3d, w.exsmo, w.exsmo2, l.boundary);
    FIM_KEND(l);
    ex_in = w.exsmo2;
  } else if (kn.intfc_smooth > 0.) {
    // the remap of the other knobs inflates its columns itself
    dim3 gs(nblocks((long long)g.N * ((g.L + kDffK) / kDffK), kBlock2), l.members);
    FIM_KBEGIN(l, "k_dffusn_lev");
    k_dffusn_lev<R><<<gs, kBlock2, 0, l.stream>>>(g, s, l.sp, l.boundary, k1, k2, w.exsmo, w.exsmo2);
    FIM_KEND(l);
    ex_in = w.exsmo2;
  }
  if (plm1) {
    const int cpw = remap_columns<R>(g.N, l.members, remap_paired<R>(g.L));
    dim3 gw(nblocks(g.N, kWarpsRemapV * cpw), l.members);
    const bool paired = remap_paired<R>(g.L);
    const int vl = paired ? 4 : remap_vl(g.L);
    const int cb = (int)(vl * sizeof(R) < 16 ? vl * sizeof(R) : 16);
    int vec = g.L % vl == 0;
    for (const void* p : {(const void*)us3d, (const void*)vs3d, (const void*)tr3d})
      if ((uintptr_t)p % cb != 0) vec = 0;
    FIM_KBEGIN(l, "k_remap");
    // a column that fills its lanes, copied 16 bytes at a time, needs no level tests
#define FIM_REMAP_V(VL, WL)                                                                                  \
  if (vec && g.L == VL * WL) FIM_REMAP_VF(VL, WL, true);                                                     \
  else FIM_REMAP_VF(VL, WL, false)
#define FIM_REMAP_VF(VL, WL, FULL)                                                                           \
  k_remap_v<R, VL, WL, FULL><<<gw, 32 * kWarpsRemapV, remap_v_smem<R, VL, WL>(), l.stream>>>(                 \
      g, s, kn, l.sp, targt, ex_in, us3d, vs3d, tr3d, sdot, ex3d, dp3d, pr3d, l.flags, l.boundary, vec, trdp, cpw)
    if (paired) {
      if constexpr (sizeof(R) == 4) { FIM_REMAP_V(4, 16); }
    } else if (vl == 1) { FIM_REMAP_V(1, 32); }
    else if (vl == 2) { FIM_REMAP_V(2, 32); }
    else { FIM_REMAP_V(4, 32); }
#undef FIM_REMAP_V
#undef FIM_REMAP_VF
    trdp_done = trdp != nullptr;
  } else if (g.L <= 64) {
    FIM_KBEGIN(l, "k_remap");
    k_remap<R, 64><<<gc, kColBlock, 0, l.stream>>>(g, s, kn, l.sp, targt, ex_in, us3d, vs3d, tr3d, sdot, ex3d,
                                                    dp3d, pr3d, l.flags, l.boundary);
  } else {
    FIM_KBEGIN(l, "k_remap");
    k_remap<R, kMaxL><<<gc, kColBlock, 0, l.stream>>>(g, s, kn, l.sp, targt, ex_in, us3d, vs3d, tr3d, sdot, ex3d,
                                                       dp3d, pr3d, l.flags, l.boundary);
  }
  FIM_KEND(l);
  return trdp_done;
}

template <typename R>
void launch_hystat(const Launch& l, const Grid<R>& g, const Strides& s, R* ph3d, const R* ex3d, R* mp3d,
                   const R* dp3d, R* tr3d, R* trdp, R* psrf, R* ptdcy, float2* mpf, bool trdp_done) {
  {
    const int vk = pick_vk<R>(g.L, {dp3d, tr3d, mp3d}, sizeof(R) == 8 ? 1 : 0);
    const size_t smem = (size_t)(sizeof(R) == 4 ? 3 : 2) * kHyCols * (g.L | 1) * sizeof(R);
    const dim3 grid(nblocks(g.N, kHyCols), l.members);
    FIM_KBEGIN(l, "k_hystat");
    FIM_VK_DISPATCH(R, vk, ({
      if (smem > (size_t)48 * 1024)  // columns of more than 95 (FP64) or 127 levels
        cudaFuncSetAttribute(k_hystat<R, VK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)((sizeof(R) == 4 ? 3 : 2) * kHyCols * (kMaxL | 1) * sizeof(R)));
      k_hystat<R, VK><<<grid, kHyBlock, smem, l.stream>>>(g, s, l.sp, ph3d, ex3d, mp3d, dp3d, tr3d, psrf, ptdcy, mpf,
                                                          l.boundary);
    }));
    FIM_KEND(l);
  }
  if (trdp_done) return;  // the remap formed the floors and tracer x thickness
  const int vk = pick_vk<R>(g.L, {dp3d, tr3d, trdp});
  FIM_KBEGIN(l, "k_hystat_trdp");
  FIM_VK_DISPATCH(R, vk, (k_hystat_trdp<R, VK><<<dim3(nblocks((long long)g.N * (g.L / VK), kBlock2), l.members),
                                                 kBlock2, 0, l.stream>>>(g, s, l.sp, dp3d, tr3d, trdp,
                                                                         l.boundary)));
  FIM_KEND(l);
}

// partial buffer: the most chunks any layout uses
size_t globsum_partials(int N, int L, int T, int members) {
  (void)T;
  int n = 0;
  for (int vk : {1, 2, 4}) n = std::max(n, gs_chunks((long long)N * L, vk));
  return (size_t)members * (size_t)n * kGsSlots;
}

template <typename R>
void launch_globsum(const Launch& l, const Grid<R>& g, const Strides& s, int ntr, const R* dp3d, const R* tr,
                    const R* rn2d, const R* rc2d, const R* pr3d, const R* ex3d, const R* qf2d,
                    double* partial, double* sums) {
  FIM_KBEGIN(l, "k_globsum_levels");
  constexpr int VK = sizeof(R) == 4 ? 4 : 2;
  const bool vec = g.L % VK == 0 && (uintptr_t)dp3d % (VK * sizeof(R)) == 0 && (uintptr_t)tr % (VK * sizeof(R)) == 0;
  const long long NL = (long long)g.N * g.L;
  const unsigned ngrp = (unsigned)(ntr + kGsGroup) / kGsGroup;
  const int vk = vec ? VK : 1, nchunk = gs_chunks(NL, vk), iters = gs_iters(NL, vk);
  if (vec) {
    k_globsum_levels<R, VK><<<dim3((unsigned)nchunk * ngrp, l.members), kBlock2, 0, l.stream>>>(
        g, s, l.sp, ntr, dp3d, tr, rn2d, rc2d, pr3d, ex3d, qf2d, partial, nchunk, iters);
  } else {
    k_globsum_levels<R, 1><<<dim3((unsigned)nchunk * ngrp, l.members), kBlock2, 0, l.stream>>>(
        g, s, l.sp, ntr, dp3d, tr, rn2d, rc2d, pr3d, ex3d, qf2d, partial, nchunk, iters);
  }
  FIM_KEND(l);
  FIM_KBEGIN(l, "k_globsum_final");
  k_globsum_final<R><<<dim3(l.members, (unsigned)((ntr + 5 + kBlock2 / 32 - 1) / (kBlock2 / 32))), kBlock2, 0,
                       l.stream>>>(l.sp, ntr, partial, nchunk, sums);
  FIM_KEND(l);
}

template <typename R>
void launch_prdp_from_ex(const Launch& l, const Grid<R>& g, const Strides& s, const R* ex3d, R* pr3d, R* dp3d) {
  dim3 gs(nblocks((long long)g.N * (g.L + 1), kBlock2), l.members);
  FIM_KBEGIN(l, "k_prdp_from_ex");
  k_prdp_from_ex<R><<<gs, kBlock2, 0, l.stream>>>(g, s, ex3d, pr3d, dp3d);
  FIM_KEND(l);
}

#define INSTANTIATE(R)                                                                                       \
  template int prepare_hybgen<R>(int);                                                                       \
  template bool launch_hybgen<R>(const Launch&, const Grid<R>&, const Strides&, const Knobs&,               \
                                 const HybgenScratch<R>&, const R*, R*, R*, R*, R*, R*, R*, R*, R*);            \
  template void launch_hystat<R>(const Launch&, const Grid<R>&, const Strides&, R*, const R*, R*, const R*, \
                                 R*, R*, R*, R*, float2*, bool);                                                  \
  template void launch_globsum<R>(const Launch&, const Grid<R>&, const Strides&, int, const R*, const R*,        \
                                  const R*, const R*, const R*, const R*, const R*, double*, double*);      \
  template void launch_prdp_from_ex<R>(const Launch&, const Grid<R>&, const Strides&, const R*, R*, R*);
INSTANTIATE(float)
INSTANTIATE(double)

}  // namespace fim
