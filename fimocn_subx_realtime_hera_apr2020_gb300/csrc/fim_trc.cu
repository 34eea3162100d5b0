// Tracer transport of the fused step: edgvar3's tracer reconstruction and
// trcadv1..3 (trcadv_compute.F90:19-315) for all tracers, on cell patches
// staged in shared memory.
//
// A patch is a parallelogram of up to 8 x 8 cells of one rhombus (each pole
// is a patch of its own); its frame adds every cell within two neighbour
// steps of the patch.  A block takes one patch, one tile of LK levels and one
// ensemble member, and runs the tracers of a chunk in turn, staging the next
// tracer's operands by cp.async while it works on the current one.
//
//   k_trf_lo  edgvalEval (edgvar3.F90:66-94): the own-side edge values of the
//             patch cells and the ring-1 neighbours' values on the patch's
//             boundary edges, in shared memory only; trcadv1 (:19-141):
//             high- and low-order fluxes, low-order AB3 update, trcr_lo; the
//             antidiffusive fluxes and the Zalesak sums S+/S- of trcadv2
//             (:143-241); a copy of the old tracer.
//   k_trf_hi  trcadv2: R+/R- of the patch cells and of their first ring, the
//             bounds taken over the 1-ring of the old tracer and of trcr_lo;
//             trcadv3 (:243-315): the antidiffusive fluxes clipped with the
//             limiters of their two cells, AB3 update of tracer x thickness,
//             new tracer.
//
// The per-routine trcadv runs the same two kernels with the caller's edge
// values (EV): 38 words a cell-level and tracer at 16-byte accesses where one
// thread a cell-level took about 60 at 4 (glvl 7, nvl 64, 11 tracers, FP32:
// 8.04 -> 2.95 ms; FP64, glvl 5, nvl 37, 5 tracers: 0.82 -> 0.43 ms).
//
// The edge values (six per cell-level and tracer) and R+/R- never reach HBM:
// per cell-level and tracer the pair reads and writes 32 words (10 of them
// the step's own state traffic), where edge values written and read back and
// R+/R- stored cost 46.  The old tracer is copied because k_trf_hi overwrites
// the tracer in place while the blocks of neighbouring patches still read it.
//
// Every value is formed from the same operands in the same order as in the
// per-routine entries (k_edgvar3_patch, or in FP64 k_edgvar3_own/_avg, then
// these kernels with EV), so the fused step is bit-identical to the routine
// sequence.  nprox is 5 or 6 (checked when the context is created), so only
// slot 5 of a cell can be missing: the tests "e < nprox" are written
// (e < 5 || e < np) and cost nothing for slots 0..4.
#include "fim_internal.h"

#include <algorithm>
#include <cmath>

namespace fim {

namespace {

template <typename R> __device__ __forceinline__ R tmax(R a, R b) { return a > b ? a : b; }
template <typename R> __device__ __forceinline__ R tmin(R a, R b) { return a < b ? a : b; }

// asynchronous global -> shared copy of B = 4, 8 or 16 bytes (16: through L2 only)
template <int B>
__device__ __forceinline__ void stage_copy(void* smem, const void* gmem) {
  const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  if constexpr (B == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sa), "l"(gmem), "n"(B) : "memory");
}
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }
// all but the last group
__device__ __forceinline__ void stage_wait1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// Row of slot e of patch cell x in the edge-indexed shared arrays (edge
// values, mass fluxes, antidiffusive fluxes): the slots of odd cells are
// swapped in pairs, so the same slot of two consecutive cells falls in
// different halves of the shared-memory banks (rows of 64 bytes).  The
// patch tables' mirror rows use the same mapping.
__host__ __device__ __forceinline__ int erow(int x, int e) { return x * 6 + (e ^ (x & 1)); }

// frame-local index of prox slot e (one byte each, slots 0..3 in x, 4..5 in y)
__device__ __forceinline__ int nb_at(uint2 nb, int e) {
  return e < 4 ? (int)((nb.x >> (8 * e)) & 255u) : (int)((nb.y >> (8 * (e - 4))) & 255u);
}

// Shared-memory layout of the two kernels (offsets in elements of R, then the
// patch tables after a 16-byte boundary).
//   lo: tracer frame x 2 buffers [S2][LK]; edge values [SE][LK]; mass
//       fluxes [SE][LK] in the rows of the edge values (the patch cells' six
//       slots, then the ring edges' neighbour sides); the patch cells'
//       low-order AB3 slots of and vof and tracer x thickness, x 2 buffers
//       [3][SC][LK]; least-squares coefficients, 36 per patch cell (row
//       stride 36), then 6 per ring edge.  With the caller's edge values
//       (EV) neither edge values nor coefficients are held.
//   hi: old-tracer and trcr_lo frames [S2][LK]; the ring-1 frame's AB3 slots
//       of and vof, S+ and S- [4][S1][LK]; R+, R- [S1][LK]; the patch cells'
//       antidiffusive fluxes [SC][6][LK], low-order tendency and tracer x
//       thickness [SC][LK]; the ring-1 frame's thickness [S1][LK] and cell
//       areas [S1].
struct PatchLayout {
  size_t trs, E, mf, ops, hf;                          // lo
  size_t TO, TL, opq, Rp, Rm, af, tlt, tdb, dpf, arf;  // hi
  size_t r_elems, tab, bytes;
  template <typename R>
  __host__ __device__ static PatchLayout make(const FrameTab& f, int LK, bool hi, bool ev = false) {
    PatchLayout p{};
    const size_t S2 = f.S2, S1 = f.S1, SC = f.SC, SE = f.SE;
    size_t o = 0;
    if (!hi) {
      p.trs = o; o += 2 * S2 * LK;
      p.E = o; o += ev ? 0 : SE * LK;
      p.mf = o; o += SE * LK;
      p.ops = o; o += 2 * 3 * SC * LK;
      p.hf = o; o += ev ? 0 : (size_t)f.cstride;
    } else {
      p.TO = o; o += S2 * LK;
      p.TL = o; o += S2 * LK;
      p.opq = o; o += 4 * S1 * LK;
      p.Rp = o; o += S1 * LK;
      p.Rm = o; o += S1 * LK;
      p.af = o; o += 6 * SC * LK;
      p.tlt = o; o += SC * LK;
      p.tdb = o; o += SC * LK;
      p.dpf = o; o += S1 * LK;
      p.arf = o; o += S1;
    }
    return p.tables<R>(hi ? f.head : f.bytes, o);
  }
  // edges: field frame x 2 buffers [S2][LK]; edge values [SE][LK];
  // least-squares coefficients as in lo
  template <typename R>
  __host__ __device__ static PatchLayout edges(const FrameTab& f, int LK) {
    PatchLayout p{};
    size_t o = 0;
    p.trs = o; o += (size_t)2 * f.S2 * LK;
    p.E = o; o += (size_t)f.SE * LK;
    p.hf = o; o += (size_t)f.cstride;
    return p.tables<R>(f.bytes, o);
  }
  // the patch tables after o elements of R
  template <typename R>
  __host__ __device__ PatchLayout tables(int nbytes, size_t o) const {
    PatchLayout p = *this;
    p.r_elems = o;
    size_t b = (o * sizeof(R) + 15) & ~(size_t)15;
    p.tab = b;
    b += (size_t)nbytes;
    p.bytes = (b + 15) & ~(size_t)15;
    return p;
  }
};

struct FrameSm {
  const int* cells;
  const uint2* nbr;
  const unsigned char* np;  // nprox of the interior and ring-1 cells
  const unsigned short* mir;
  const unsigned short* red;
  const int* mfr;
};

// asynchronous copy of n bytes (a multiple of 16, both ends on 16 bytes)
__device__ __forceinline__ void stage_bytes(void* dst, const void* src, int n) {
  for (int q = threadIdx.x * 16; q < n; q += blockDim.x * 16)
    stage_copy<16>(static_cast<unsigned char*>(dst) + q, static_cast<const unsigned char*>(src) + q);
}

// the patch's tables (the first n bytes of them) on their way into shared
// memory; callers commit, wait and synchronise before use
__device__ __forceinline__ FrameSm stage_tables(const FrameTab& ft, unsigned char* base, size_t tab, int tile, int n) {
  unsigned char* q = base + tab;
  stage_bytes(q, ft.tab + (size_t)tile * ft.bytes, n);
  return {reinterpret_cast<const int*>(q), reinterpret_cast<const uint2*>(q + ft.nbr), q + ft.np,
          reinterpret_cast<const unsigned short*>(q + ft.mir), reinterpret_cast<const unsigned short*>(q + ft.red),
          reinterpret_cast<const int*>(q + ft.mfr)};
}

// halved least-squares coefficients of the patch cells (36 each) and of the
// ring edges (the row of the edge's slot) on their way into hf.  The edge
// values are kept halved (exactly), so that the average of an edge's two sides
// is one addition.
template <typename R>
__device__ __forceinline__ void stage_coefs(const FrameTab& ft, R* hf, int tile, int C, int nre) {
  stage_bytes(hf, static_cast<const R*>(ft.coef) + (size_t)tile * ft.cstride,
              ((C * 36 + nre * 6) * (int)sizeof(R) + 15) & ~15);
}

template <typename R>
__global__ void k_patch_coefs(Grid<R> g, FrameTab ft, R* __restrict__ coef) {
  const int tile = blockIdx.x;
  const unsigned char* q = ft.tab + (size_t)tile * ft.bytes;
  const int* cells = reinterpret_cast<const int*>(q);
  const unsigned short* red = reinterpret_cast<const unsigned short*>(q + ft.red);
  const int4 cn = ft.cnt[tile];
  R* out = coef + (size_t)tile * ft.cstride;
  for (int a = threadIdx.x; a < ft.cstride; a += blockDim.x) {
    R h = R(0);
    if (a < cn.x * 36) {
      const int x = a / 36;
      h = g.hfcoef[(size_t)cells[x] * 36 + (a - x * 36)];
    } else if (a < cn.x * 36 + cn.w * 6) {
      const int b = a - cn.x * 36, r = b / 6, code = red[r];
      h = g.hfcoef[(size_t)cells[code >> 3] * 36 + (code & 7) * 6 + (b - r * 6)];
    }
    out[a] = R(0.5) * h;
  }
}

// rows of lk levels (from src, already offset to the tile's first level) of
// the n cells cells[0..n) into dst[x * LK + level]
template <typename R, int VK, int GC>
__device__ __forceinline__ void stage_rows(R* dst, const R* src, const int* cells, int n, int lk, int L) {
  constexpr int LK = VK * GC;
  for (int it = threadIdx.x; it < n * GC; it += blockDim.x) {
    const int x = it / GC, v = (it - x * GC) * VK;
    if (v < lk) stage_copy<VK * (int)sizeof(R)>(dst + x * LK + v, src + cells[x] * L + v);
  }
}

// The frame rows a thread copies.  The block has SC * GC threads and GC
// threads take one row, so thread (x0, v) takes rows x0, x0 + SC, x0 + 2 SC
// of every frame field (the frame lists interior, ring-1 and ring-2 cells in
// that order, so a field over its first n rows takes the rows below n).  The
// element offsets of those rows' level tiles are formed once per block; a
// copy is then an add and one cp.async.  Frames of more than 3 SC cells (the
// small patches of coarse grids) take the general loop.
template <typename R, int VK, int GC>
struct RowPlan {
  int x0, v, off[3];
  bool fast;
  __device__ __forceinline__ void init(const FrameSm& fs, int SC, int n2, int lk, int L) {
    x0 = threadIdx.x / GC;
    v = (threadIdx.x - x0 * GC) * VK;
    fast = n2 <= 3 * SC;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int x = x0 + j * SC;
      off[j] = (x < n2 && v < lk) ? fs.cells[x] * L + v : -1;
    }
  }
  // rows [0, n) of the field at src (offset to the tile's first level) into
  // dst[x * LK + level]
  __device__ __forceinline__ void copy(R* dst, const R* src, const FrameSm& fs, int SC, int n, int lk,
                                       int L) const {
    constexpr int LK = VK * GC;
    if (fast) {
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const int x = x0 + j * SC;
        if (x < n && off[j] >= 0) stage_copy<VK * (int)sizeof(R)>(dst + x * LK + v, src + off[j]);
      }
    } else {
      stage_rows<R, VK, GC>(dst, src, fs.cells, n, lk, L);
    }
  }
};

// six coefficients hf[0..6) as three pairs (8- or 16-byte shared loads)
template <typename R>
__device__ __forceinline__ void coef6(const R* hf, R (&h)[6]) {
  using P2 = typename VecOf<R, 2>::T;
  const P2* q = reinterpret_cast<const P2*>(hf);
#pragma unroll
  for (int u = 0; u < 3; u++) {
    const P2 w = q[u];
    h[2 * u] = w.x;
    h[2 * u + 1] = w.y;
  }
}

// the twelve coefficients of two slots of a patch cell (a 16-byte boundary:
// 16-byte shared loads)
__device__ __forceinline__ void coef12(const float* hf, float (&h)[12]) {
#pragma unroll
  for (int u = 0; u < 3; u++) {
    const float4 w = reinterpret_cast<const float4*>(hf)[u];
    h[4 * u] = w.x; h[4 * u + 1] = w.y; h[4 * u + 2] = w.z; h[4 * u + 3] = w.w;
  }
}
__device__ __forceinline__ void coef12(const double* hf, double (&h)[12]) {
#pragma unroll
  for (int u = 0; u < 6; u++) {
    const double2 w = reinterpret_cast<const double2*>(hf)[u];
    h[2 * u] = w.x; h[2 * u + 1] = w.y;
  }
}

// half the own-side least-squares edge value of every slot ie of a patch cell
// (k_edgvar3_own's arithmetic, halved): val = bc + sum_e hfcoef(e, ie) (tr_e -
// bc), d[e] = tr_e - bc (0 past nprox); hf = the cell's 36 halved coefficients
template <typename R, int VK, int LK>
__device__ __forceinline__ void own_values(const R* hf, int x, int v, const R (&bc)[VK], const R (&d)[6][VK],
                                           int np, R* E) {
#pragma unroll
  for (int i2 = 0; i2 < 6; i2 += 2) {
    R h[12];
    coef12(hf + i2 * 6, h);
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int ie = i2 + q;
      R val[VK];
      FOR_V val[j] = mul_rn(R(0.5), bc[j]);
#pragma unroll
      for (int e = 0; e < 6; e++) {
        FOR_V val[j] = (e < 5 || e < np) ? fma_rn(d[e][j], h[q * 6 + e], val[j]) : val[j];
      }
      FOR_V val[j] = (ie < 5 || ie < np) ? val[j] : R(0);
      stv<VK>(E + erow(x, ie) * LK + v, val);
    }
  }
}

// half the value on slot p of ring-1 cell y (its side of the edge it shares with a
// patch cell), into edge-value row 6C + r; hf = that slot's 6 coefficients
template <typename R, int VK, int LK>
__device__ __forceinline__ void ring_value(const R* T, const FrameSm& fs, const R* hf, int code, int row, int v,
                                           R* E) {
  const int y = code >> 3;
  const int np = fs.np[y];
  const uint2 nb = fs.nbr[y];
  R bc[VK], val[VK], h[6];
  coef6<R>(hf, h);
  ldv<VK>(T + y * LK + v, bc);
  FOR_V val[j] = mul_rn(R(0.5), bc[j]);
#pragma unroll
  for (int e = 0; e < 6; e++) {
    R d[VK];
    ldv<VK>(T + nb_at(nb, e) * LK + v, d);
    FOR_V d[j] = (e < 5 || e < np) ? d[j] - bc[j] : R(0);
    FOR_V val[j] = (e < 5 || e < np) ? fma_rn(d[j], h[e], val[j]) : val[j];
  }
  stv<VK>(E + row * LK + v, val);
}

// The thread's patch cell and levels (one per thread: the block has SC * GC
// threads), with the layer thickness (at least the threshold) and its
// reciprocal, which it keeps in registers for the whole tracer loop.
template <typename R, int VK>
struct CellItem {
  bool on;
  int i, x, v, k, c, np;
  R rar;
  R dp[VK], rdp[VK];
  template <int GC>
  __device__ __forceinline__ void load(const Grid<R>& g, const Strides& s, const FrameSm& fs, size_t m,
                                       const R* delp, int C, int k0, int lk) {
    x = threadIdx.x / GC;
    v = (threadIdx.x - x * GC) * VK;
    on = x < C && v < lk;
    if (!on) return;
    const int L = g.L;
    i = fs.cells[x];
    k = k0 + v;
    c = i * L + k;
    np = fs.np[x];
    rar = g.rarea[i];
    ldv<VK>(delp + m * s.cell + c, dp);
    FOR_V {
      dp[j] = tmax(R(1.e-11), dp[j]);
      rdp[j] = fdiv(R(1), dp[j]);
    }
  }
};

// The AB3 weights of the slot a launch writes (nf) and of those it reads (of,
// vof).  Where a caller's slots are the same one (fim_set_ab takes any), the
// weights of the slots that are nf's go to the new tendency, as trcadv1 and 3
// read it after they set it, and trcadv2's limiters see no old one (trcadv1
// clears it): a block never reads a slot that another is writing.
template <typename R>
struct Ab3 {
  R now, old, very_old;
  __device__ __forceinline__ explicit Ab3(const StepParams& p)
      : now(p.w1<R>()), old(p.w2<R>()), very_old(p.w3<R>()) {
    if (p.of == p.nf) {
      now = now + old;
      old = R(0);
    }
    if (p.vof == p.nf) {
      now = now + very_old;
      very_old = R(0);
    }
  }
};
template <typename R>
__device__ __forceinline__ void zero_rows(R* p, int n) {
  for (int q = threadIdx.x; q < n; q += blockDim.x) p[q] = R(0);
}

// One level of a cell as the routines write it, for items that hold a value
// that is not finite (or, in FP64, a mass flux positive on both sides).
// trcadv1's bounds of frame cell x: T the tracer's frame at that level.
template <typename R> struct UpDown { R up, down; };
template <typename R, int LK>
__device__ __forceinline__ UpDown<R> plain_bounds(const R* T, uint2 nb, int x) {
  UpDown<R> b{T[x * LK], T[x * LK]};
#pragma unroll 1
  for (int e = 0; e < 6; e++) {
    const R a = T[nb_at(nb, e) * LK];
    b = {plain_max(b.up, a), plain_min(b.down, a)};
  }
  return {plain_max(R(0), b.up), plain_max(R(0), b.down)};
}

// fluxes, sums and bounds of patch cell x in trcadv1 and trcadv2; te: its six
// edge values in memory (stride L), or null where they are E's; mir: its six
// entries; anti: its antidiffusive fluxes (stride L)
template <typename R> struct LoItem { R sum, sp, sm, hx, hn; };
template <typename R, int LK>
__device__ __forceinline__ LoItem<R> plain_lo(const R* T, const R* MF, const R* E, const R* te,
                                              const unsigned short* mir, uint2 nb, int x, int np, int L, R* anti) {
  const UpDown<R> b = plain_bounds<R, LK>(T, nb, x);
  LoItem<R> w{R(0), R(0), R(0), b.up, b.down};
  const R tri = T[x * LK];
#pragma unroll 1
  for (int e = 0; e < np; e++) {
    const R mf = MF[erow(x, e) * LK], mfx = MF[mir[e] * LK], trx = T[nb_at(nb, e) * LK];
    const R tev = te ? te[e * L] : E[erow(x, e) * LK] + E[mir[e] * LK];
    const R lo = plain_donor(mf, mfx, tri, trx);
    const R a = fma_rn(mf, tev, -lo);
    w.sum = w.sum + lo;
    w.sp = w.sp - plain_min(R(0), a);
    w.sm = w.sm + plain_max(R(0), a);
    anti[e * L] = a;
  }
  return w;
}
// the same as a call: at 16 bytes of levels a thread k_trf_lo is 1% faster with it,
// at 8 it is 6% slower (glvl 5 / nvl 38 / 5 tracers 59.7 against 63.6 us)
template <typename R, int LK>
__device__ __noinline__ LoItem<R> plain_lo_call(const R* T, const R* MF, const R* E, const R* te,
                                                const unsigned short* mir, uint2 nb, int x, int np, int L, R* anti) {
  return plain_lo<R, LK>(T, MF, E, te, mir, nb, x, np, L, anti);
}

// bounds and limiters of frame cell x in trcadv2 (ar: the cell's area, in FP64
// over ab1).  routine: the bounds as trcadv1 and 2 form them one after the other;
// else as the fused step does, old tracer and trcr_lo of a neighbour at a time
// (in FP32 by the three-input instructions, which drop a NaN).
template <typename R> struct LimItem { R hx, hn, rp, rm; };
__device__ __forceinline__ float pair_max(float m, float a, float b) { return fmaxf(m, fmaxf(a, b)); }
__device__ __forceinline__ float pair_min(float m, float a, float b) { return fminf(m, fminf(a, b)); }
__device__ __forceinline__ double pair_max(double m, double a, double b) { return plain_max(m, plain_max(a, b)); }
__device__ __forceinline__ double pair_min(double m, double a, double b) { return plain_min(m, plain_min(a, b)); }
template <typename R, int LK>
__device__ __noinline__ LimItem<R> plain_limits(const R* TO, const R* TL, uint2 nb, int x, R dp, R tof, R tvf, R spl,
                                                R smn, R ab2, R ab3, R rab1, R ar, bool routine) {
  const R lc = TL[x * LK], tc = TO[x * LK];
  UpDown<R> b = {tc, tc};
  if (routine) b = plain_bounds<R, LK>(TO, nb, x);
  b = {plain_max(b.up, lc), plain_min(b.down, lc)};
#pragma unroll 1
  for (int e = 0; e < 6; e++) {
    const R a = TL[nb_at(nb, e) * LK], o = TO[nb_at(nb, e) * LK];
    if (routine) b = {plain_max(b.up, a), plain_min(b.down, a)};
    else b = {pair_max(b.up, o, a), pair_min(b.down, o, a)};
  }
  b = {plain_max(R(0), b.up), plain_max(R(0), b.down)};
  const R qp = per_ab1((b.up - lc) * dp - (ab2 * plain_min(R(0), tof) + ab3 * plain_max(R(0), tvf)), rab1, ar);
  const R qm = per_ab1((lc - b.down) * dp + (ab2 * plain_max(R(0), tof) + ab3 * plain_min(R(0), tvf)), rab1, ar);
  return {b.up, b.down, plain_ratio01(qp, spl), plain_ratio01(qm, smn)};
}

// trcadv1 + the S+/S- sums of trcadv2 + copy of the old tracer, per patch.
// EV: the edge values of every tracer are the caller's (trc_edg of the
// per-routine trcadv, or edgvar1's without hi_order_flux_comp); a thread
// loads its cell's six rows before it waits for the staged operands, and the
// member's own tracer count does not apply.  EV = false forms them on chip
// (theta's are edgvar1's).
//
// Two blocks an SM at GC 4, the shared memory's limit with 16-byte rows a
// thread.  FP64 at one level a thread takes the three that fit then (80
// registers: glvl 5 / nvl 37 / 5 tracers 273 -> 257 us when chosen, 184 us with
// the present flux arithmetic); FP32 at two levels a
// thread is slower there (59 -> 62 us).
template <typename R, int VK, int GC, bool EV>
__global__ void __launch_bounds__(64 * GC, sizeof(R) == 8 && VK == 1 ? 12 / GC : 8 / GC) k_trf_lo(Grid<R> g, Strides s, FrameTab ft,
    const StepParams* __restrict__ sp, int t0, int nt, const R* __restrict__ massfx, const R* __restrict__ trc_edg,
    const R* __restrict__ tracr, const R* __restrict__ trcdp, R* __restrict__ trl_tdcy, const R* __restrict__ delp,
    R* __restrict__ trcr_lo, R* __restrict__ s_plus, R* __restrict__ s_mnus, R* __restrict__ trold,
    R* __restrict__ antifx, size_t sc) {
  constexpr int LK = VK * GC;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active) return;
  // the member's tracers in this chunk (fim_member_set_tracers); the
  // scratch keeps the chunk's layout
  const int ntm = EV ? nt : min(nt, sp->ntr - t0);
  if (ntm <= 0) return;
  const int L = g.L, N = g.N;
  const int nlc = (L + LK - 1) / LK;
  const int tile = blockIdx.x / nlc;
  const int k0 = (blockIdx.x - tile * nlc) * LK;
  const int lk = min(LK, L - k0);
  const int4 cn = ft.cnt[tile];
  const int C = cn.x, n1 = cn.y, n2 = cn.z, nre = cn.w;
  extern __shared__ __align__(16) unsigned char fsm[];
  const PatchLayout lay = PatchLayout::make<R>(ft, LK, false, EV);
  R* const sr = reinterpret_cast<R*>(fsm);
  R* const trs = sr + lay.trs;
  R* const E = sr + lay.E;
  R* const MF = sr + lay.mf;
  R* const ops = sr + lay.ops;
  R* const hf = sr + lay.hf;
  // the tables, then (arriving with the first operands) the coefficients
  const FrameSm fs = stage_tables(ft, fsm, lay.tab, tile, ft.bytes);
  stage_commit();
  if (!EV) stage_coefs<R>(ft, hf, tile, C, nre);
  stage_commit();
  stage_wait1();
  __syncthreads();
  const size_t NL = (size_t)N * L;
  const int nf = sp->nf, of = sp->of, vof = sp->vof;
  const Ab3<R> ab(*sp);
  const R* mfn = massfx + m * s.mf + (size_t)nf * 6 * NL;
  const R* te0 = trc_edg + m * s.tredg;  // EV: tracer t's at t * 6 NL; else theta's (edgvar1)
  // this step's tracer t: its frame, and the patch cells' AB3 slots of/vof
  // and tracer x thickness
  RowPlan<R, VK, GC> rp;
  rp.init(fs, ft.SC, n2, lk, L);
  auto stage = [&](int t, int b) {
    rp.copy(trs + b * ft.S2 * LK, tracr + m * s.tr + (size_t)t * NL + k0, fs, ft.SC, n2, lk, L);
    const R* tl = trl_tdcy + m * s.trab + (size_t)t * 3 * NL + k0;
    R* o = ops + b * 3 * ft.SC * LK;
    if (of != nf) rp.copy(o, tl + (size_t)of * NL, fs, ft.SC, C, lk, L);
    if (vof != nf) rp.copy(o + ft.SC * LK, tl + (size_t)vof * NL, fs, ft.SC, C, lk, L);
    rp.copy(o + 2 * ft.SC * LK, trcdp + m * s.tr + (size_t)t * NL + k0, fs, ft.SC, C, lk, L);
    stage_commit();
  };
  // the mass fluxes of the patch cells' edges and of the ring edges'
  // neighbour sides (tracer independent), with the first tracer's operands
  for (int it = threadIdx.x; it < (6 * C + nre) * GC; it += blockDim.x) {
    const int r = it / GC, v = (it - r * GC) * VK;
    if (v < lk) stage_copy<VK * (int)sizeof(R)>(MF + r * LK + v, mfn + fs.mfr[r] * L + k0 + v);
  }
  for (int b = 0; b < 2; b++) {  // rows that no copy fills
    if (of == nf) zero_rows(ops + b * 3 * ft.SC * LK, ft.SC * LK);
    if (vof == nf) zero_rows(ops + (b * 3 + 1) * ft.SC * LK, ft.SC * LK);
  }
  stage(t0, 0);
  CellItem<R, VK> ci;
  ci.template load<GC>(g, s, fs, m, delp, C, k0, lk);
  bool mf_rare = false;
  for (int tz = 0; tz < ntm; tz++) {
    const int t = t0 + tz, b = tz & 1;
    R ter[6][VK];  // EV: the edge values of the thread's cell, in flight over the wait
    if constexpr (EV) {
      if (ci.on) {
        const R* te = te0 + (size_t)t * 6 * NL;
#pragma unroll
        for (int e = 0; e < 6; e++) ldv<VK>(te + (ci.i * 6 + e) * L + ci.k, ter[e]);
      }
    }
    stage_wait();
    __syncthreads();
    if (tz + 1 < ntm) stage(t + 1, b ^ 1);
    const R* T = trs + b * ft.S2 * LK;
    if (!EV && t != 0) {
      // edge values: the six of the thread's patch cell, then the ring cells'
      // sides of the patch's boundary edges
      if (ci.on) {
        const uint2 nb = fs.nbr[ci.x];
        R bc[VK], d[6][VK];
        ldv<VK>(T + ci.x * LK + ci.v, bc);
#pragma unroll
        for (int e = 0; e < 6; e++) {
          ldv<VK>(T + nb_at(nb, e) * LK + ci.v, d[e]);
          FOR_V d[e][j] = (e < 5 || e < ci.np) ? d[e][j] - bc[j] : R(0);
        }
        own_values<R, VK, LK>(hf + ci.x * 36, ci.x, ci.v, bc, d, ci.np, E);
      }
      for (int it = threadIdx.x; it < nre * GC; it += blockDim.x) {
        const int r = it / GC, ve = (it - r * GC) * VK;
        if (ve < lk) ring_value<R, VK, LK>(T, fs, hf + C * 36 + r * 6, fs.red[r], 6 * C + r, ve, E);
      }
      __syncthreads();
    }
    if (!ci.on) continue;
    const int x = ci.x, v = ci.v, i = ci.i, c = ci.c;
    const uint2 nb = fs.nbr[x];
    // a mass flux of the cell needs plain_donor: FP64 looks once, FP32 keeps the
    // largest magnitude as the fluxes pass (one instruction each)
    float top = 0.f;
    if (sizeof(R) == 8 && tz == 0) {
#pragma unroll
      for (int e = 0; e < 6; e++) {
        R a[VK], b[VK];
        ldv<VK>(MF + erow(x, e) * LK + v, a);
        ldv<VK>(MF + fs.mir[x * 6 + e] * LK + v, b);
        FOR_V mf_rare |= (e < 5 || e < ci.np) & donor_rare(a[j], b[j]);
      }
    }
    R tri[VK], sumlo[VK], sp_[VK], sm_[VK];
    Bound<R> mx[VK], mn[VK];
    ldv<VK>(T + x * LK + v, tri);
    FOR_V { sumlo[j] = R(0); sp_[j] = R(0); sm_[j] = R(0); mx[j] = mn[j] = Bound<R>::of(tri[j]); }
#pragma unroll
    for (int e = 0; e < 6; e++) {
      R trx[VK];
      ldv<VK>(T + nb_at(nb, e) * LK + v, trx);
      FOR_V {
        const Bound<R> bx = Bound<R>::of(trx[j]);
        mx[j].up(bx);
        mn[j].down(bx);
      }
      if (e < 5 || e < ci.np) {
        R tev[VK];
        if constexpr (EV) {
          FOR_V tev[j] = ter[e][j];
        } else if (t != 0) {
          R tem[VK];
          ldv<VK>(E + erow(x, e) * LK + v, tev);
          ldv<VK>(E + fs.mir[x * 6 + e] * LK + v, tem);
          FOR_V tev[j] = tev[j] + tem[j];
        } else {
          ldv<VK>(te0 + (i * 6 + e) * L + ci.k, tev);
        }
        R anti[VK];
        R mfo[VK], mfm[VK];
        ldv<VK>(MF + erow(x, e) * LK + v, mfo);
        ldv<VK>(MF + fs.mir[x * 6 + e] * LK + v, mfm);
        FOR_V {
          if constexpr (sizeof(R) == 4) top = max_nan(top, fabsf(mfo[j]), fabsf(mfm[j]));
          const R lo = donor(mfo[j], mfm[j], tri[j], trx[j]);
          anti[j] = fma_rn(mfo[j], tev[j], -lo);
          sumlo[j] = sumlo[j] + lo;
          split_sum(anti[j], sp_[j], sm_[j]);
        }
        stv<VK>(antifx + (m * nt + tz) * 6 * sc + (size_t)(i * 6 + e) * L + ci.k, anti);
      }
    }
    const size_t q = (m * nt + tz) * sc + c;
    R* const af = antifx + (m * nt + tz) * 6 * sc + (size_t)i * 6 * L + ci.k;
    R hx[VK], hn[VK];
    bool rare = mf_rare | !(top < __int_as_float(0x7f800000));
    FOR_V {
      hx[j] = mx[j].at_least_zero();
      hn[j] = mn[j].at_least_zero();
      rare |= bounds_rare(mx[j], mn[j]) | sums_rare(sp_[j], sm_[j]);
    }
    if (rare) {
      const R* te = EV || t == 0 ? te0 + (EV ? (size_t)t * 6 * NL : (size_t)0) + (size_t)i * 6 * L + ci.k : nullptr;
      FOR_V {
        constexpr auto plain = VK * sizeof(R) == 16 ? plain_lo_call<R, LK> : plain_lo<R, LK>;
        const LoItem<R> w = plain(T + v + j, MF + v + j, E + v + j, te ? te + j : te, fs.mir + x * 6, nb, x, ci.np, L,
                                  af + j);
        sumlo[j] = w.sum;
        sp_[j] = w.sp;
        sm_[j] = w.sm;
        hx[j] = w.hx;
        hn[j] = w.hn;
      }
    }
    const R* o = ops + b * 3 * ft.SC * LK + x * LK + v;
    R tn[VK], tlo[VK], tlv[VK], td[VK], out[VK];
    FOR_V tn[j] = -sumlo[j] * ci.rar;
    stv<VK>(trl_tdcy + m * s.trab + (size_t)t * 3 * NL + (size_t)nf * NL + c, tn);
    ldv<VK>(o, tlo);
    ldv<VK>(o + ft.SC * LK, tlv);
    ldv<VK>(o + 2 * ft.SC * LK, td);
    FOR_V {
      const R lo = td[j] + ab.now * tn[j] + ab.old * tlo[j] + ab.very_old * tlv[j];
      out[j] = tmax(hn[j], tmin(hx[j], quot(lo, ci.dp[j], ci.rdp[j])));
    }
    stv<VK>(trcr_lo + q, out);
    stv<VK>(s_plus + q, sp_);
    stv<VK>(s_mnus + q, sm_);
    stv<VK>(trold + q, tri);
  }
}

// Where k_trf_hi writes tracer x thickness and the new tracer: the state
// (member stride s.tr, tracer t at t * NL), or, for the shape probe, chunk
// scratch (member stride nt * NL, tracer t at (t - t0) * NL).
template <typename R>
struct TrOut {
  R* trdp;
  R* tr;
  size_t mstride;
  int tbase;
};

// R+/R- of trcadv2 for frame cell xe at levels ve, from the staged old tracer
// and trcr_lo, AB3 slots, S+/S- and thickness (arf: the cell areas, in FP64
// over ab1); the bounds
// (clamped at zero) and the slots of/vof are returned for trcadv3
template <typename R, int VK, int LK>
__device__ __forceinline__ void limiters(const FrameSm& fs, const R* TO, const R* TL, const R* opq, const R* dpf,
                                         const R* arf, int S1, int xe, int ve, R ab2, R ab3, R rab1, bool routine,
                                         R* Rp, R* Rm, R (&hx)[VK], R (&hn)[VK], R (&tof)[VK], R (&tvf)[VK]) {
  const R thshld = R(1.e-11);
  const uint2 nb = fs.nbr[xe];
  const int o = xe * LK + ve;
  R lc[VK], tc0[VK];
  Bound<R> mx[VK], mn[VK];
  ldv<VK>(TL + o, lc);
  ldv<VK>(TO + o, tc0);
  FOR_V {
    mx[j] = mn[j] = Bound<R>::of(lc[j]);
    const Bound<R> b = Bound<R>::of(tc0[j]);
    mx[j].up(b);
    mn[j].down(b);
  }
#pragma unroll
  for (int e = 0; e < 6; e++) {
    R aa[VK], bb[VK];
    ldv<VK>(TO + nb_at(nb, e) * LK + ve, aa);
    ldv<VK>(TL + nb_at(nb, e) * LK + ve, bb);
    FOR_V {
      const Bound<R> a = Bound<R>::of(aa[j]), b = Bound<R>::of(bb[j]);
      mx[j].up(a, b);
      mn[j].down(a, b);
    }
  }
  R dp[VK], spl[VK], smn[VK], rp[VK], rm[VK];
  ldv<VK>(opq + o, tof);
  ldv<VK>(opq + S1 * LK + o, tvf);
  ldv<VK>(opq + 2 * S1 * LK + o, spl);
  ldv<VK>(opq + 3 * S1 * LK + o, smn);
  ldv<VK>(dpf + o, dp);
  const R ar = arf[xe];
  bool rare = false;
  FOR_V {
    hx[j] = mx[j].at_least_zero();
    hn[j] = mn[j].at_least_zero();
    const R q_plus = per_ab1((hx[j] - lc[j]) * dp[j] - (ab2 * neg(tof[j]) + ab3 * pos(tvf[j])), rab1, ar);
    const R q_mnus = per_ab1((lc[j] - hn[j]) * dp[j] + (ab2 * pos(tof[j]) + ab3 * neg(tvf[j])), rab1, ar);
    rp[j] = ratio01(q_plus, floor_at(spl[j], thshld));
    rm[j] = ratio01(q_mnus, floor_at(smn[j], thshld));
    rare |= bounds_rare(mx[j], mn[j]) | ratio_rare(q_plus, q_mnus);
  }
  if (rare) {
    FOR_V {
      const LimItem<R> w = plain_limits<R, LK>(TO + ve + j, TL + ve + j, nb, xe, dp[j], tof[j], tvf[j], spl[j],
                                               smn[j], ab2, ab3, rab1, ar, routine);
      hx[j] = w.hx;
      hn[j] = w.hn;
      rp[j] = w.rp;
      rm[j] = w.rm;
    }
  }
  stv<VK>(Rp + o, rp);
  stv<VK>(Rm + o, rm);
}

// trcadv2's limiters over the patch and its first ring, then trcadv3: the
// antidiffusive fluxes k_trf_lo stored are clipped with the limiters of
// their two cells and summed; the low-order tendency k_trf_lo stored
// (-sum of the low-order fluxes x rarea, rounded) is added; AB3 update of
// tracer x thickness; new tracer.
//
// Copies: the limiters' operands of tracer t (frames, slots, S+/S-) are
// staged while the block clips tracer t-1; the clip's operands of tracer t
// (fluxes, tendency, tracer x thickness) while it forms tracer t's limiters.
//
// Registers: the blocks an SM that the shared memory lets in at GC 4, two of
// 98 KB with 16-byte rows a thread, more below (three at up to 80 registers
// are as fast as four at 64).  Left to itself the compiler takes 80 and 64
// and serialises the neighbour loads (FP32 glvl 7 / nvl 64 / 11 tracers 1.43
// -> 1.41 ms, glvl 5 / nvl 38 / 5 tracers 66 -> 61 us, FP64 glvl 6 / nvl 64 /
// 11 tracers 2.84 -> 2.78 ms; FP64 one level a thread at two blocks 252 us
// against 239 at three; measured when chosen, the FP64 kernel has since come to
// 2.48 ms and 212 us).
template <typename R, int VK, int GC>
__global__ void __launch_bounds__(64 * GC, VK * (int)sizeof(R) == 16 ? 8 / GC : 12 / GC) k_trf_hi(Grid<R> g, Strides s, FrameTab ft,
    const StepParams* __restrict__ sp, int t0, int nt, const R* __restrict__ trl_tdcy, const R* trcdp,
    R* __restrict__ trc_tdcy, const R* __restrict__ delp, const R* __restrict__ trold,
    const R* __restrict__ trcr_lo, const R* __restrict__ s_plus, const R* __restrict__ s_mnus,
    const R* __restrict__ antifx, TrOut<R> out, size_t sc, int all) {
  // all: every tracer of the chunk, whatever the member's own count
  // trcdp (read) and out.trdp (written) are the same array in the step
  constexpr int LK = VK * GC;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active) return;
  // the member's tracers in this chunk (fim_member_set_tracers); the
  // scratch keeps the chunk's layout
  const int ntm = all ? nt : min(nt, sp->ntr - t0);
  if (ntm <= 0) return;
  const int L = g.L, N = g.N;
  const int nlc = (L + LK - 1) / LK;
  const int tile = blockIdx.x / nlc;
  const int k0 = (blockIdx.x - tile * nlc) * LK;
  const int lk = min(LK, L - k0);
  const int4 cn = ft.cnt[tile];
  const int C = cn.x, n1 = cn.y, n2 = cn.z, nre = cn.w;
  extern __shared__ __align__(16) unsigned char fsm[];
  const PatchLayout lay = PatchLayout::make<R>(ft, LK, true);
  R* const sr = reinterpret_cast<R*>(fsm);
  R* const TO = sr + lay.TO;
  R* const TL = sr + lay.TL;
  R* const opq = sr + lay.opq;
  R* const Rp = sr + lay.Rp;
  R* const Rm = sr + lay.Rm;
  R* const af = sr + lay.af;
  R* const tlt = sr + lay.tlt;
  R* const tdb = sr + lay.tdb;
  R* const dpf = sr + lay.dpf;
  R* const arf = sr + lay.arf;
  const FrameSm fs = stage_tables(ft, fsm, lay.tab, tile, ft.head);
  stage_commit();
  stage_wait();
  __syncthreads();
  const size_t NL = (size_t)N * L;
  const int nf = sp->nf, of = sp->of, vof = sp->vof;
  const Ab3<R> ab(*sp);
  const R rab1 = R(1) / sp->template w1<R>();  // Q+/Q- divide by ab1: one reciprocal
  for (int x = threadIdx.x; x < n1; x += blockDim.x) arf[x] = g.area[fs.cells[x]] * (sizeof(R) == 8 ? rab1 : R(1));
  // the limiters' operands of tracer t0 + tz
  RowPlan<R, VK, GC> rp;
  rp.init(fs, ft.SC, n2, lk, L);
  auto stage_lim = [&](int tz) {
    const size_t so = (m * nt + tz) * sc + k0;
    rp.copy(TO, trold + so, fs, ft.SC, n2, lk, L);
    rp.copy(TL, trcr_lo + so, fs, ft.SC, n2, lk, L);
    const R* tc = trc_tdcy + m * s.trab + (size_t)(t0 + tz) * 3 * NL + k0;
    if (of != nf) rp.copy(opq, tc + (size_t)of * NL, fs, ft.SC, n1, lk, L);
    if (vof != nf) rp.copy(opq + ft.S1 * LK, tc + (size_t)vof * NL, fs, ft.SC, n1, lk, L);
    rp.copy(opq + 2 * ft.S1 * LK, s_plus + so, fs, ft.SC, n1, lk, L);
    rp.copy(opq + 3 * ft.S1 * LK, s_mnus + so, fs, ft.SC, n1, lk, L);
    stage_commit();
  };
  // the clip's operands: the patch cells' six fluxes, low-order tendency
  // (slot nf) and tracer x thickness
  // (each thread copies the six flux rows of its own cell)
  const int afo = (rp.x0 < C && rp.v < lk) ? fs.cells[rp.x0] * 6 * L + rp.v : -1;
  auto stage_clip = [&](int tz) {
    const R* a = antifx + (m * nt + tz) * 6 * sc + k0;
    if (afo >= 0) {
#pragma unroll
      for (int e = 0; e < 6; e++)
        stage_copy<VK * (int)sizeof(R)>(af + erow(rp.x0, e) * LK + rp.v, a + afo + e * L);
    }
    const size_t tt = (size_t)(t0 + tz);
    rp.copy(tlt, trl_tdcy + m * s.trab + tt * 3 * NL + (size_t)nf * NL + k0, fs, ft.SC, C, lk, L);
    rp.copy(tdb, trcdp + m * s.tr + tt * NL + k0, fs, ft.SC, C, lk, L);
    stage_commit();
  };
  stage_rows<R, VK, GC>(dpf, delp + m * s.cell + k0, fs.cells, n1, lk, L);
  if (of == nf) zero_rows(opq, ft.S1 * LK);  // rows that no copy fills
  if (vof == nf) zero_rows(opq + ft.S1 * LK, ft.S1 * LK);
  stage_lim(0);
  const int x = threadIdx.x / GC, v = (threadIdx.x - x * GC) * VK;
  const bool on = x < C && v < lk;
  // FP64: the thickness (at least the threshold) and its reciprocal, once a
  // block (FP32 has no registers left and divides in three instructions)
  R dpk[VK], rdp[VK];
  if constexpr (sizeof(R) == 8) {
    if (on) {
      ldv<VK>(delp + m * s.cell + (size_t)fs.cells[x] * L + k0 + v, dpk);
      FOR_V {
        dpk[j] = tmax(R(1.e-11), dpk[j]);
        rdp[j] = R(1) / dpk[j];
      }
    }
  }
  for (int tz = 0; tz < ntm; tz++) {
    const int t = t0 + tz;
    stage_wait();
    __syncthreads();
    stage_clip(tz);
    // R+/R- of the thread's patch cell (its bounds and slots kept for
    // trcadv3), then of the ring-1 cells
    R hx[VK], hn[VK], tof[VK], tvf[VK];
    if (on) limiters<R, VK, LK>(fs, TO, TL, opq, dpf, arf, ft.S1, x, v, ab.old, ab.very_old, rab1, all, Rp, Rm, hx, hn, tof,
                                   tvf);
    for (int it = threadIdx.x; it < (n1 - C) * GC; it += blockDim.x) {
      const int xe = C + it / GC, ve = (it % GC) * VK;
      if (ve >= lk) continue;
      R mx2[VK], mn2[VK], tof2[VK], tvf2[VK];
      limiters<R, VK, LK>(fs, TO, TL, opq, dpf, arf, ft.S1, xe, ve, ab.old, ab.very_old, rab1, all, Rp, Rm, mx2, mn2,
                           tof2, tvf2);
    }
    stage_wait();
    __syncthreads();
    if (tz + 1 < ntm) stage_lim(tz + 1);
    if (!on) continue;
    const int i = fs.cells[x];
    const int c = i * L + k0 + v;
    const int np = fs.np[x];
    const uint2 nb = fs.nbr[x];
    R rpc[VK], rmc[VK], at[VK];
    ldv<VK>(Rp + x * LK + v, rpc);
    ldv<VK>(Rm + x * LK + v, rmc);
    FOR_V {
      rpc[j] = own_limit(rpc[j]);
      rmc[j] = own_limit(rmc[j]);
      at[j] = R(0);
    }
#pragma unroll
    for (int e = 0; e < 6; e++) {
      if (e < 5 || e < np) {
        const int y = nb_at(nb, e);
        R a[VK], rpx[VK], rmx[VK];
        ldv<VK>(af + erow(x, e) * LK + v, a);
        ldv<VK>(Rp + y * LK + v, rpx);
        ldv<VK>(Rm + y * LK + v, rmx);
        FOR_V {
          const bool in = below0(a[j]);
          at[j] = fma_rn(a[j], min0(in ? rpc[j] : rmc[j], in ? rmx[j] : rpx[j]), at[j]);
        }
      }
    }
    const R rar = g.rarea[i];
    R tl[VK], tdv[VK], dp[VK], tn[VK], res[VK];
    ldv<VK>(tlt + x * LK + v, tl);
    ldv<VK>(tdb + x * LK + v, tdv);
    ldv<VK>(dpf + x * LK + v, dp);
    // the low-order tendency plus the clipped fluxes' divergence
    FOR_V tn[j] = tl[j] + (-at[j] * rar);
    stv<VK>(trc_tdcy + m * s.trab + (size_t)t * 3 * NL + (size_t)nf * NL + c, tn);
    const size_t ob = m * out.mstride + (size_t)(t - out.tbase) * NL + c;
    FOR_V {
      tdv[j] = tdv[j] + ab.now * tn[j] + ab.old * tof[j] + ab.very_old * tvf[j];
      const R q = sizeof(R) == 8 ? quot(tdv[j], dpk[j], rdp[j]) : fdiv(tdv[j], tmax(R(1.e-11), dp[j]));
      res[j] = tmax(hn[j], tmin(hx[j], q));
    }
    stv<VK>(out.trdp + ob, tdv);
    stv<VK>(out.tr + ob, res);
  }
}

// edgvar3 (edgvar3.F90:66-133) of several fields per patch: the own-side
// values of the patch cells and the ring cells' sides of its boundary edges in
// shared memory, then the two-sided average 0.5 own + 0.5 other side of every
// slot of the patch cells (0 in a pentagon's sixth).  Field 0 is the layer
// thickness, field f tracer f.  One read and six writes a value, where storing
// the own-side values and averaging them in a second pass (k_edgvar3_own,
// k_edgvar3_avg) moves 19.  Held by the shared-memory pipe (77% busy: 1,400
// wavefronts a patch, 16 levels and field), three blocks an SM (80 registers;
// two 0.98 ms, four 0.91 ms, against 0.89): at glvl 7 / nvl 64, dp and 10
// tracers, 0.84 ms (0.89 before the tables were packed) against 0.65 + 0.90 ms
// for the two passes.  blockIdx.z takes every
// gridDim.z-th field, so small grids fill the chip.
template <typename R, int VK, int GC>
__global__ void __launch_bounds__(64 * GC, 3) k_edgvar3_patch(Grid<R> g, Strides s, FrameTab ft, int nfields,
    const R* __restrict__ delp, const R* __restrict__ tracr, R* __restrict__ dp_edg, R* __restrict__ trc_edg) {
  constexpr int LK = VK * GC;
  const size_t m = blockIdx.y;
  const int L = g.L, N = g.N;
  const int nlc = (L + LK - 1) / LK;
  const int tile = blockIdx.x / nlc;
  const int k0 = (blockIdx.x - tile * nlc) * LK;
  const int lk = min(LK, L - k0);
  const int4 cn = ft.cnt[tile];
  const int C = cn.x, n1 = cn.y, n2 = cn.z, nre = cn.w;
  extern __shared__ __align__(16) unsigned char fsm[];
  const PatchLayout lay = PatchLayout::edges<R>(ft, LK);
  R* const sr = reinterpret_cast<R*>(fsm);
  R* const trs = sr + lay.trs;
  R* const E = sr + lay.E;
  R* const hf = sr + lay.hf;
  const FrameSm fs = stage_tables(ft, fsm, lay.tab, tile, ft.bytes);
  stage_commit();
  stage_coefs<R>(ft, hf, tile, C, nre);
  stage_commit();
  stage_wait1();
  __syncthreads();
  const size_t NL = (size_t)N * L;
  RowPlan<R, VK, GC> rp;
  rp.init(fs, ft.SC, n2, lk, L);
  auto stage = [&](int f, int b) {
    const R* src = f == 0 ? delp + m * s.cell : tracr + m * s.tr + (size_t)f * NL;
    rp.copy(trs + b * ft.S2 * LK, src + k0, fs, ft.SC, n2, lk, L);
    stage_commit();
  };
  int f = blockIdx.z;
  stage(f, 0);
  const int x = threadIdx.x / GC, v = (threadIdx.x - x * GC) * VK;
  const bool on = x < C && v < lk;
  const int i = on ? fs.cells[x] : 0, np = on ? fs.np[x] : 0;
  for (int b = 0; f < nfields; f += gridDim.z, b ^= 1) {
    stage_wait();
    __syncthreads();
    if (f + (int)gridDim.z < nfields) stage(f + gridDim.z, b ^ 1);
    const R* T = trs + b * ft.S2 * LK;
    if (on) {
      const uint2 nb = fs.nbr[x];
      R bc[VK], d[6][VK];
      ldv<VK>(T + x * LK + v, bc);
#pragma unroll
      for (int e = 0; e < 6; e++) {
        ldv<VK>(T + nb_at(nb, e) * LK + v, d[e]);
        FOR_V d[e][j] = (e < 5 || e < np) ? d[e][j] - bc[j] : R(0);
      }
      own_values<R, VK, LK>(hf + x * 36, x, v, bc, d, np, E);
    }
    for (int it = threadIdx.x; it < nre * GC; it += blockDim.x) {
      const int r = it / GC, ve = (it - r * GC) * VK;
      if (ve < lk) ring_value<R, VK, LK>(T, fs, hf + C * 36 + r * 6, fs.red[r], 6 * C + r, ve, E);
    }
    __syncthreads();
    if (!on) continue;
    R* dst = (f == 0 ? dp_edg + m * s.edge : trc_edg + m * s.tredg + (size_t)f * 6 * NL) + (size_t)i * 6 * L + k0 + v;
#pragma unroll
    for (int e = 0; e < 6; e++) {
      R a[VK], o[VK];
      ldv<VK>(E + erow(x, e) * LK + v, a);
      ldv<VK>(E + fs.mir[x * 6 + e] * LK + v, o);
      FOR_V a[j] = a[j] + o[j];
      stv<VK>(dst + e * L, a);
    }
  }
}

template <typename R, int VK>
void edges_launch(const Launch& l, const Grid<R>& g, const Strides& s, const FrameTab& ft, int nfields,
                  const R* delp, const R* tracr, R* dp_edg, R* trc_edg) {
  constexpr int GC = 4, LK = VK * GC;
  const unsigned nb = (unsigned)(ft.ntile * ((g.L + LK - 1) / LK));
  // enough blocks for two waves of three an SM, at most one field a block
  const unsigned want = 6u * (unsigned)sm_count() / (nb * l.members) + 1u;
  const unsigned nz = want < (unsigned)nfields ? want : (unsigned)nfields;
  k_edgvar3_patch<R, VK, GC><<<dim3(nb, l.members, nz), ft.SC * GC, PatchLayout::edges<R>(ft, LK).bytes, l.stream>>>(
      g, s, ft, nfields, delp, tracr, dp_edg, trc_edg);
}

template <typename R, int VK, int GC, bool EV>
void trf_chunks(const Launch& l, const Grid<R>& g, const Strides& s, const TrcFusedScratch<R>& w, R* trc_edg,
                R* tracr, R* trcdp, R* trc_tdcy, R* trl_tdcy, const R* massfx, const R* delp, bool probe,
                const ChunkHook* hook) {
  constexpr int LK = VK * GC;
  const FrameTab& ft = w.ft;
  const size_t sc = (size_t)g.N * g.L;
  const int nlc = (g.L + LK - 1) / LK;
  const size_t sm_lo = PatchLayout::make<R>(ft, LK, false, EV).bytes,
               sm_hi = PatchLayout::make<R>(ft, LK, true).bytes;
  dim3 grid((unsigned)(ft.ntile * nlc), l.members);
  const int tb = ft.SC * GC;
  for (int t0 = 0; t0 < g.T; t0 += w.tchunk) {
    const int nt = (g.T - t0 < w.tchunk) ? g.T - t0 : w.tchunk;
    if (hook && hook->fn) hook->fn(hook->arg, 0, t0, nt);
    FIM_KBEGIN(l, "k_trf_lo");
    k_trf_lo<R, VK, GC, EV><<<grid, tb, sm_lo, l.stream>>>(g, s, ft, l.sp, t0, nt, massfx, trc_edg, tracr, trcdp,
                                                            trl_tdcy, delp, w.trcr_lo, w.s_plus, w.s_mnus, w.trold,
                                                            w.antifx, sc);
    FIM_KEND(l);
    // the probe sends the new tracer and tracer x thickness to scratch
    const TrOut<R> out = probe ? TrOut<R>{w.r_plus, w.r_mnus, (size_t)nt * sc, t0} : TrOut<R>{trcdp, tracr, s.tr, 0};
    FIM_KBEGIN(l, "k_trf_hi");
    k_trf_hi<R, VK, GC><<<grid, tb, sm_hi, l.stream>>>(g, s, ft, l.sp, t0, nt, trl_tdcy, trcdp, trc_tdcy, delp,
                                                        w.trold, w.trcr_lo, w.s_plus, w.s_mnus, w.antifx, out, sc,
                                                        EV ? 1 : 0);
    FIM_KEND(l);
    if (probe) return;  // the first chunk only
    if (hook && hook->fn) hook->fn(hook->arg, 1, t0, nt);
  }
}

// Levels per thread: 16-byte accesses where nvl allows; every array offset
// is then a multiple of VK elements, and every base is a cudaMalloc'd field
// (256-byte aligned), checked here.
template <typename R>
int tracer_vk(const Grid<R>& g, std::initializer_list<const void*> ptrs, int want) {
  return pick_vk<R>(g.L, ptrs, want);
}

template <typename R>
void fused_dispatch(const Launch& l, const Grid<R>& g, const Strides& s, const TrcFusedScratch<R>& w, R* trc_edg,
                    R* tracr, R* trcdp, R* trc_tdcy, R* trl_tdcy, const R* massfx, const R* delp, bool probe,
                    const ChunkHook* hook) {
  const int vk = tracer_vk(g, {trc_edg, tracr, trcdp, trc_tdcy, trl_tdcy, massfx, delp, w.trcr_lo, w.s_plus,
                               w.s_mnus, w.trold, w.r_plus, w.r_mnus, w.antifx}, w.vk);
  const bool g4 = w.gc >= 4;
#define FIM_TRF(VKV)                                                                                            \
  do {                                                                                                          \
    if (w.edges)                                                                                                \
      trf_chunks<R, VKV, 4, true>(l, g, s, w, trc_edg, tracr, trcdp, trc_tdcy, trl_tdcy, massfx, delp, probe, hook);  \
    else if (g4)                                                                                                \
      trf_chunks<R, VKV, 4, false>(l, g, s, w, trc_edg, tracr, trcdp, trc_tdcy, trl_tdcy, massfx, delp, probe, hook); \
    else                                                                                                        \
      trf_chunks<R, VKV, 2, false>(l, g, s, w, trc_edg, tracr, trcdp, trc_tdcy, trl_tdcy, massfx, delp, probe, hook); \
  } while (0)
  if (vk == 4) FIM_TRF((sizeof(R) == 4 ? 4 : 2));
  else if (vk == 2) FIM_TRF(2);
  else FIM_TRF(1);
#undef FIM_TRF
}

// The attribute belongs to the kernel, not to a context: it is raised to the
// architecture's limit, so that contexts of different grids do not lower it
// for each other.
template <typename K>
cudaError_t allow_smem(K kernel, size_t bytes) {
  constexpr int kLimit = 227 * 1024;
  if (bytes > (size_t)kLimit) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLimit);
}

template <typename R, int VK, int GC>
int prepare_one(const FrameTab& ft) {
  constexpr int LK = VK * GC;
  cudaError_t e = allow_smem(k_trf_lo<R, VK, GC, false>, PatchLayout::make<R>(ft, LK, false).bytes);
  if constexpr (GC == 4)
    if (e == cudaSuccess)
      e = allow_smem(k_trf_lo<R, VK, GC, true>, PatchLayout::make<R>(ft, LK, false, true).bytes);
  if (e == cudaSuccess) e = allow_smem(k_trf_hi<R, VK, GC>, PatchLayout::make<R>(ft, LK, true).bytes);
  return (int)e;
}

}  // namespace

int prepare_edges(const FrameTab& ft) {
  cudaError_t e = allow_smem(k_edgvar3_patch<float, 1, 4>, PatchLayout::edges<float>(ft, 4).bytes);
  if (e == cudaSuccess) e = allow_smem(k_edgvar3_patch<float, 2, 4>, PatchLayout::edges<float>(ft, 8).bytes);
  if (e == cudaSuccess) e = allow_smem(k_edgvar3_patch<float, 4, 4>, PatchLayout::edges<float>(ft, 16).bytes);
  return (int)e;
}

void launch_edges_patch(const Launch& l, const Grid<float>& g, const Strides& s, const FrameTab& ft, int nfields,
                        const float* delp, const float* tracr, float* dp_edg, float* trc_edg) {
  const int vk = pick_vk<float>(g.L, {delp, tracr, dp_edg, trc_edg});
  FIM_KBEGIN(l, "k_edgvar3_patch");
  FIM_VK_DISPATCH(float, vk, (edges_launch<float, VK>(l, g, s, ft, nfields, delp, tracr, dp_edg, trc_edg)));
  FIM_KEND(l);
}

// ---- cell patches ---------------------------------------------------------

int build_frames(int N, const int* prox, const int* proxs, const int* nprox, int side, FrameHost* F, bool sixth) {
  if (side < 1 || side > 8) return 1;
  std::vector<std::vector<int>> tiles;
  // the reference's IJ numbering: north pole, 10 rhombi of sl x sl cells in
  // rows of sl, south pole; a cell strictly inside a rhombus then has the
  // cells +-1 and +-sl among its neighbours
  const long long sl = std::llround(std::sqrt((N - 2) / 10.0));
  bool ij = sl >= 1 && 10 * sl * sl + 2 == N;
  auto has = [&](int c, int n) {
    for (int e = 0; e < nprox[c]; e++)
      if (prox[c * 6 + e] == n) return true;
    return false;
  };
  for (long long r = 0; ij && r < 10; r++)
    for (long long a = 1; ij && a + 1 < sl; a++)
      for (long long b = 1; ij && b + 1 < sl; b++) {
        const int c = (int)(1 + r * sl * sl + a * sl + b);
        if (!has(c, c - 1) || !has(c, c + 1) || !has(c, c - (int)sl) || !has(c, c + (int)sl)) ij = false;
      }
  if (ij) {
    tiles.push_back({0});
    for (long long r = 0; r < 10; r++)
      for (long long ta = 0; ta < sl; ta += side)
        for (long long tb = 0; tb < sl; tb += side) {
          std::vector<int> t;
          for (long long a = ta; a < std::min(ta + side, sl); a++)
            for (long long b = tb; b < std::min(tb + side, sl); b++) t.push_back((int)(1 + r * sl * sl + a * sl + b));
          tiles.push_back(t);
        }
    tiles.push_back({N - 1});
  } else {
    // any other numbering: grow each patch breadth-first from the lowest
    // unassigned cell
    std::vector<char> used(N, 0);
    const size_t cap = (size_t)side * side;
    for (int c0 = 0; c0 < N; c0++) {
      if (used[c0]) continue;
      std::vector<int> t{c0};
      used[c0] = 1;
      for (size_t q = 0; q < t.size() && t.size() < cap; q++)
        for (int e = 0; e < nprox[t[q]] && t.size() < cap; e++) {
          const int n = prox[t[q] * 6 + e];
          if (!used[n]) { used[n] = 1; t.push_back(n); }
        }
      std::sort(t.begin(), t.end());
      tiles.push_back(t);
    }
  }
  // frames
  const int nt = (int)tiles.size();
  std::vector<int> loc(N, -1);
  struct Fr { std::vector<int> cells; int C, n1, n2; std::vector<uint32_t> nbr; std::vector<uint16_t> mir, red; };
  std::vector<Fr> fr(nt);
  int S2 = 0, S1 = 0, SC = 0, SR = 0;
  for (int ti = 0; ti < nt; ti++) {
    Fr& f = fr[ti];
    f.cells = tiles[ti];
    f.C = (int)f.cells.size();
    for (int x = 0; x < f.C; x++) loc[f.cells[x]] = x;
    for (int ring = 0; ring < 2; ring++) {
      const int lo = ring == 0 ? 0 : f.C, hi = (int)f.cells.size();
      std::vector<int> add;
      for (int x = lo; x < hi; x++) {
        const int c = f.cells[x];
        for (int e = 0; e < (sixth ? 6 : nprox[c]); e++) {
          const int n = prox[c * 6 + e];
          if (loc[n] == -1) { loc[n] = -2; add.push_back(n); }
        }
      }
      std::sort(add.begin(), add.end());
      for (int n : add) { loc[n] = (int)f.cells.size(); f.cells.push_back(n); }
      if (ring == 0) f.n1 = (int)f.cells.size();
    }
    f.n2 = (int)f.cells.size();
    if (f.n2 > 255) {
      for (int c : f.cells) loc[c] = -1;
      return 2;
    }
    f.nbr.assign((size_t)f.n1 * 2, 0u);
    for (int x = 0; x < f.n1; x++)
      for (int e = 0; e < 6; e++) {
        const int l6 = loc[prox[f.cells[x] * 6 + e]];
        if (l6 < 0) { for (int c : f.cells) loc[c] = -1; return 3; }
        f.nbr[(size_t)x * 2 + e / 4] |= (uint32_t)l6 << (8 * (e % 4));
      }
    f.mir.assign((size_t)f.C * 6, 0);
    for (int x = 0; x < f.C; x++) {
      const int c = f.cells[x];
      for (int e = 0; e < 6; e++) {
        if (e >= nprox[c]) { f.mir[(size_t)x * 6 + e] = (uint16_t)erow(x, e); continue; }
        const int y = loc[prox[c * 6 + e]], p = proxs[c * 6 + e];
        if (y < f.C) {
          f.mir[(size_t)x * 6 + e] = (uint16_t)erow(y, p);
        } else {
          f.mir[(size_t)x * 6 + e] = (uint16_t)(6 * f.C + f.red.size());
          f.red.push_back((uint16_t)((y << 3) | p));
        }
      }
    }
    for (int c : f.cells) loc[c] = -1;
    S2 = std::max(S2, f.n2);
    S1 = std::max(S1, f.n1);
    SC = std::max(SC, f.C);
    SR = std::max(SR, (int)f.red.size());
  }
  S2 = (S2 + 3) & ~3;  // keeps the tables after the cell list 16-byte aligned
  S1 = (S1 + 1) & ~1;
  SR = std::max(2, (SR + 1) & ~1);
  F->ntile = nt; F->S2 = S2; F->S1 = S1; F->SC = SC; F->SR = SR; F->SE = 6 * SC + SR;
  F->cells.assign((size_t)nt * S2, 0);
  F->nbr.assign((size_t)nt * S1 * 2, 0u);
  F->cnt.assign((size_t)nt * 4, 0);
  F->mir.assign((size_t)nt * SC * 6, 0);
  F->red.assign((size_t)nt * SR, 0);
  for (int ti = 0; ti < nt; ti++) {
    const Fr& f = fr[ti];
    std::copy(f.cells.begin(), f.cells.end(), F->cells.begin() + (size_t)ti * S2);
    std::copy(f.nbr.begin(), f.nbr.end(), F->nbr.begin() + (size_t)ti * S1 * 2);
    std::copy(f.mir.begin(), f.mir.end(), F->mir.begin() + (size_t)ti * SC * 6);
    std::copy(f.red.begin(), f.red.end(), F->red.begin() + (size_t)ti * SR);
    F->cnt[(size_t)ti * 4 + 0] = f.C;
    F->cnt[(size_t)ti * 4 + 1] = f.n1;
    F->cnt[(size_t)ti * 4 + 2] = f.n2;
    F->cnt[(size_t)ti * 4 + 3] = (int)f.red.size();
  }
  return 0;
}

void pack_frames(const FrameHost& f, const int* nprox, FrameTab* tab, std::vector<unsigned char>* out) {
  FrameTab& t = *tab;
  t.ntile = f.ntile; t.S2 = f.S2; t.S1 = f.S1; t.SC = f.SC; t.SE = f.SE; t.SR = f.SR;
  auto up = [](int n) { return (n + 15) & ~15; };
  t.nbr = up(4 * f.S2);
  t.np = t.nbr + up(8 * f.S1);
  t.head = t.np + up(f.S1);
  t.mir = t.head;
  t.red = t.mir + up(12 * f.SC);
  t.mfr = t.red + up(2 * f.SR);
  t.bytes = t.mfr + up(4 * f.SE);
  t.cstride = (f.SC * 36 + f.SR * 6 + 3) & ~3;
  out->assign((size_t)f.ntile * t.bytes, 0);
  for (int i = 0; i < f.ntile; i++) {
    unsigned char* q = out->data() + (size_t)i * t.bytes;
    const int* cells = &f.cells[(size_t)i * f.S2];
    const int C = f.cnt[(size_t)i * 4], n1 = f.cnt[(size_t)i * 4 + 1], nre = f.cnt[(size_t)i * 4 + 3];
    std::copy(cells, cells + f.S2, reinterpret_cast<int*>(q));
    std::copy(&f.nbr[(size_t)i * f.S1 * 2], &f.nbr[(size_t)i * f.S1 * 2] + (size_t)f.S1 * 2,
              reinterpret_cast<uint32_t*>(q + t.nbr));
    for (int x = 0; x < n1; x++) q[t.np + x] = (unsigned char)nprox[cells[x]];
    std::copy(&f.mir[(size_t)i * f.SC * 6], &f.mir[(size_t)i * f.SC * 6] + (size_t)f.SC * 6,
              reinterpret_cast<uint16_t*>(q + t.mir));
    const uint16_t* red = &f.red[(size_t)i * f.SR];
    std::copy(red, red + f.SR, reinterpret_cast<uint16_t*>(q + t.red));
    int* mfr = reinterpret_cast<int*>(q + t.mfr);
    for (int x = 0; x < C; x++)
      for (int e = 0; e < 6; e++) mfr[erow(x, e)] = cells[x] * 6 + e;
    for (int r = 0; r < nre; r++) mfr[6 * C + r] = cells[red[r] >> 3] * 6 + (red[r] & 7);
  }
}

template <typename R>
void launch_patch_coefs(cudaStream_t stream, const Grid<R>& g, const FrameTab& ft, R* coef) {
  k_patch_coefs<R><<<(unsigned)ft.ntile, 256, 0, stream>>>(g, ft, coef);
}

int check_frames(int N, const int* prox, const int* proxs, const int* nprox, const FrameHost& F) {
  std::vector<int> seen(N, 0);
  for (int t = 0; t < F.ntile; t++) {
    const int C = F.cnt[(size_t)t * 4], n1 = F.cnt[(size_t)t * 4 + 1], n2 = F.cnt[(size_t)t * 4 + 2],
              nre = F.cnt[(size_t)t * 4 + 3];
    if (C < 1 || C > F.SC || n1 > F.S1 || n2 > F.S2 || nre > F.SR || 6 * C + nre > F.SE) return 1;
    const int* cells = &F.cells[(size_t)t * F.S2];
    for (int x = 0; x < n2; x++)
      if (cells[x] < 0 || cells[x] >= N) return 2;
    for (int x = 0; x < C; x++) seen[cells[x]]++;
    for (int x = 0; x < n1; x++)
      for (int e = 0; e < 6; e++) {
        const int y = (F.nbr[((size_t)t * F.S1 + x) * 2 + e / 4] >> (8 * (e % 4))) & 255;
        if (y >= n2 || cells[y] != prox[cells[x] * 6 + e]) return 3;
      }
    for (int x = 0; x < C; x++) {
      const int c = cells[x];
      for (int e = 0; e < nprox[c]; e++) {
        const int row = F.mir[((size_t)t * F.SC + x) * 6 + e];
        int y, p;
        if (row < 6 * C) {
          y = row / 6;
          p = (row % 6) ^ (y & 1);
        } else {
          const int r = row - 6 * C;
          if (r >= nre) return 4;
          const int code = F.red[(size_t)t * F.SR + r];
          y = code >> 3;
          p = code & 7;
          if (y < C || y >= n1) return 5;
        }
        if (cells[y] != prox[c * 6 + e] || p != proxs[c * 6 + e]) return 6;
      }
    }
  }
  for (int i = 0; i < N; i++)
    if (seen[i] != 1) return 7;
  return 0;
}

template <typename R>
int prepare_tracers(const FrameTab& ft) {
  int e;
  if ((e = prepare_one<R, 1, 2>(ft)) || (e = prepare_one<R, 1, 4>(ft))) return e;
  if ((e = prepare_one<R, 2, 2>(ft)) || (e = prepare_one<R, 2, 4>(ft))) return e;
  if (sizeof(R) == 4) {
    if ((e = prepare_one<R, (sizeof(R) == 4 ? 4 : 2), 2>(ft)) || (e = prepare_one<R, (sizeof(R) == 4 ? 4 : 2), 4>(ft)))
      return e;
  }
  return 0;
}

template <typename R>
void launch_tracers_fused(const Launch& l, const Grid<R>& g, const Strides& s, const TrcFusedScratch<R>& w,
                          R* trc_edg, R* tracr, R* trcdp, R* trc_tdcy, R* trl_tdcy, const R* massfx,
                          const R* delp, const ChunkHook* hook) {
  fused_dispatch<R>(l, g, s, w, trc_edg, tracr, trcdp, trc_tdcy, trl_tdcy, massfx, delp, false, hook);
}

// Autotuner: time k_trf_lo + k_trf_hi (first tracer chunk, results of
// k_trf_hi sent to scratch) for every (levels per thread, level tile) that
// the layout admits and keep the fastest.  The caller provides step
// parameters whose nf slot the next step overwrites, so the probe leaves no
// state behind.
template <typename R>
int tune_tracers(const Launch& l, const Grid<R>& g, const Strides& s, const TrcFusedScratch<R>& w, R* trc_edg,
                 R* tracr, R* trcdp, R* trc_tdcy, R* trl_tdcy, const R* massfx, const R* delp, int* best_vk,
                 int* best_gc, float* best_ms) {
  cudaEvent_t a, b;
  if (cudaEventCreate(&a) != cudaSuccess) return (int)cudaGetLastError();
  if (cudaEventCreate(&b) != cudaSuccess) { cudaEventDestroy(a); return (int)cudaGetLastError(); }
  Launch lq = l;
  lq.prof = nullptr;
  lq.counter = nullptr;
  float best = 1e30f;
  int rc = 0;
  const int vmax = (int)(16 / sizeof(R));
  for (int gc : {2, 4}) {
    for (int vk = vmax; vk >= 1 && vk >= vmax / 2; vk /= 2) {
      TrcFusedScratch<R> wv = w;
      wv.vk = vk;
      wv.gc = gc;
      if (tracer_vk(g, {trc_edg, tracr, trcdp, trc_tdcy, trl_tdcy, massfx, delp, w.trcr_lo}, vk) != vk) continue;
      float ms = 0.f;
      for (int rep = 0; rep < 3; rep++) {  // the first repetition warms up
        cudaEventRecord(a, lq.stream);
        fused_dispatch<R>(lq, g, s, wv, trc_edg, tracr, trcdp, trc_tdcy, trl_tdcy, massfx, delp, true, nullptr);
        cudaEventRecord(b, lq.stream);
        if (cudaEventSynchronize(b) != cudaSuccess) { rc = (int)cudaGetLastError(); break; }
        float t = 0.f;
        cudaEventElapsedTime(&t, a, b);
        if (rep > 0) ms += t;
      }
      if (rc) break;
      if (ms < best) { best = ms; *best_vk = vk; *best_gc = gc; }
    }
    if (rc) break;
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (!rc) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) rc = (int)e;
  }
  if (best_ms) *best_ms = best / 2;
  return rc;
}

#define INSTANTIATE(R)                                                                                        \
  template void launch_tracers_fused<R>(const Launch&, const Grid<R>&, const Strides&,                       \
                                        const TrcFusedScratch<R>&, R*, R*, R*, R*, R*, const R*, const R*,   \
                                        const ChunkHook*);                                                    \
  template void launch_patch_coefs<R>(cudaStream_t, const Grid<R>&, const FrameTab&, R*);                     \
  template int prepare_tracers<R>(const FrameTab&);                                                           \
  template int tune_tracers<R>(const Launch&, const Grid<R>&, const Strides&, const TrcFusedScratch<R>&, R*, \
                               R*, R*, R*, R*, const R*, const R*, int*, int*, float*);
INSTANTIATE(float)
INSTANTIATE(double)

}  // namespace fim
