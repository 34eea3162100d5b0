// Horizontal stencil kernels of the FIM dynamics step: edgvar1, edgvar3,
// cnuity1..5, del4prep/dissip/momtum1 (trcadv1..3: fim_trc.cu).
//
// Layout is the reference's (level index fastest), so one thread per
// (level group, cell) gives fully coalesced loads along k for own and
// neighbour columns alike; a warp covers consecutive levels of a cell and the
// grid tables of that cell are broadcast loads.  Where levels of one column
// are coupled, cnuity5 (pressure and omega sums) takes 32 columns a block and
// sums with a lane a column over shared memory, and momtum1 (Rayleigh
// damping) a warp a column.
// Ensemble members map to gridDim.y; all members share the grid tables.
//
// Every kernel restates the arithmetic of the reference routine it names,
// in the same order, with the reference's 'real' mapped to the template type R.
#include "fim_internal.h"

namespace fim {

template <typename R> __device__ __forceinline__ R rmax(R a, R b) { return a > b ? a : b; }
template <typename R> __device__ __forceinline__ R rmin(R a, R b) { return a < b ? a : b; }
template <typename R> __device__ __forceinline__ R rabs(R a) { return a < R(0) ? -a : a; }

constexpr int kBlock = 256;

__device__ __forceinline__ bool cell_level(int N, int L, int& i, int& k) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= N * L) return false;
  i = gid / L;
  k = gid - i * L;
  return true;
}

inline unsigned blocks_for(long long n, int b = kBlock) { return (unsigned)((n + b - 1) / b); }

// |(a, b)|: IEEE sqrt in FP64; x * rsqrt(x) in FP32, a few ulp from the
// rounded root and about a third of its instructions
__device__ __forceinline__ double vmag(double a, double b) { return sqrt(a * a + b * b); }
__device__ __forceinline__ float vmag(float a, float b) {
  const float x = a * a + b * b;
  return x > 0.f ? x * rsqrtf(x) : 0.f;
}

// four table entries of an edge (cs or sn): 16-byte loads
__device__ __forceinline__ void ld4(const float* p, float (&r)[4]) { ldv<4>(p, r); }
__device__ __forceinline__ void ld4(const double* p, double (&r)[4]) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  r[0] = a.x; r[1] = a.y; r[2] = b.x; r[3] = b.y;
}

// --------------------------------------------------------------------------
// edgvar1 (edgvar1.F90:156-511, eqwgt=.true., janjic=0): rotate u,v of the
// cell, the cell across the edge and the cells across the two adjacent edges
// into the edge frame, equal-weight interpolate with magnitude correction;
// mid-layer pressure, Montgomery potential, kinetic energy and tracer 1 (all
// tracers and dp when hi_order == 0) on the cell's own edges.
//
// A thread loads each of its cell's six neighbours once and keeps what the
// three edges that see it share: the wind, the float-float difference of the
// Montgomery potential, theta; in FP64, where operations bound the kernel,
// also the wind's speed.  The magnitude is that of the rotated components, and
// the matrix (cs sn; -sn cs) scales every vector by sqrt(cs^2 + sn^2), so the
// speeds enter with that factor (g.vw): tables in real*4, as a grid file holds
// them, are off a rotation by 6e-8.  (The FP32 build forms it from the rotated
// components, because the thickness tendencies, differences of large fluxes,
// show the last bit of the edge winds.)  FP64 folds the edge wind's common
// factors: with U, V six times the interpolated components and M the
// interpolated magnitude, u m_2 / max(eps, m_1) = U M / sqrt(U^2 + V^2).
// The winds and the scalars are formed one after the other, so their operands
// share registers: 64 a thread, four blocks an SM (three: 1.53 ms, five,
// spilling: 1.88 ms).  At glvl 8 / nvl 64 in FP32 1.41 ms, 4,880 GB/s of its
// 41 words, where loading each neighbour for each of its edges took 1.98 ms;
// glvl 6 in FP64 3.08 -> 1.70 ms.
#define FIM_TRAIL(x) (e == 0 ? (five ? x[4][j] : x[5][j]) : x[e == 0 ? 0 : e - 1][j])
#define FIM_LEAD(x) (e == 5 ? x[0][j] : e == 4 ? (five ? x[0][j] : x[5][j]) : x[e == 5 ? 0 : e + 1][j])
// (2 (a + b) + c + d) / 6 on the live edges of a cell: x0 the cell's value, x
// its neighbours'; written to rows of o
template <typename R, int VK>
__device__ __forceinline__ void edge_means(bool five, int L, const R (&x0)[VK], const R (&x)[6][VK], R* o) {
  const R divby6 = R(1) / R(6), two = R(2);
#pragma unroll
  for (int e = 0; e < 6; e++) {
    if (e == 5 && five) continue;
    R out[VK];
    FOR_V out[j] = (two * (x0[j] + x[e][j]) + FIM_TRAIL(x) + FIM_LEAD(x)) * divby6;
    stv<VK>(o + (size_t)e * L, out);
  }
}
// a cell field's values at the cell and its six prox slots (all valid cells)
template <typename R, int VK>
__device__ __forceinline__ void around(const R* f, int L, int i, int k, const int (&nb)[6], R (&x0)[VK],
                                       R (&x)[6][VK]) {
  ldv<VK>(f + (size_t)i * L + k, x0);
#pragma unroll
  for (int e = 0; e < 6; e++) ldv<VK>(f + (size_t)nb[e] * L + k, x[e]);
}

template <typename R, int VK>
__global__ void __launch_bounds__(kBlock, 4) k_edgvar1(Grid<R> g, Strides s, int hi_order,
    const R* __restrict__ u, const R* __restrict__ v, const R* __restrict__ delp,
    const R* __restrict__ pres, const R* __restrict__ montg, const R* __restrict__ tracr,
    R* __restrict__ u_edg, R* __restrict__ v_edg, R* __restrict__ dp_edg, R* __restrict__ lp_edg,
    R* __restrict__ mont_edg, R* __restrict__ uvsq_edg, R* __restrict__ trc_edg, const float2* __restrict__ mpf,
    R* __restrict__ thold) {
  int i, k;
  if (!cell_levels<VK>(g.N, g.L, i, k)) return;
  const int L = g.L, N = g.N, L1 = L + 1;
  const size_t m = blockIdx.y;
  const size_t c = (size_t)i * L + k;
  const bool five = g.nprox[i] < 6;
  int nb[6];
#pragma unroll
  for (int e = 0; e < 6; e++) nb[e] = g.prox[i * 6 + e];
  const size_t oe = (size_t)i * 6 * L + k;
  // the wind
  {
    R u0[VK], v0[VK], ux[6][VK], vx[6][VK];
    around<R, VK>(u + m * s.cell, L, i, k, nb, u0, ux);
    around<R, VK>(v + m * s.cell, L, i, k, nb, v0, vx);
    R m0[VK], mx[6][VK];
    if constexpr (sizeof(R) == 8) {
      FOR_V {
        m0[j] = vmag(u0[j], v0[j]);
#pragma unroll
        for (int e = 0; e < 6; e++) mx[e][j] = vmag(ux[e][j], vx[e][j]);
      }
    }
    const R divby6 = R(1) / R(6), eps = R(0.001), two = R(2), half = R(0.5);
    R* pu = u_edg + m * s.edge + oe;
    R* pv = v_edg + m * s.edge + oe;
    R* pq = uvsq_edg + m * s.edge + oe;
#pragma unroll
    for (int e = 0; e < 6; e++) {
      if (e == 5 && five) continue;
      R cs[4], sn[4];
      ld4(g.cs + (i * 6 + e) * 4, cs);
      ld4(g.sn + (i * 6 + e) * 4, sn);
      R ue[VK], ve[VK], uv[VK];
      FOR_V {
        const R ut = FIM_TRAIL(ux), vt = FIM_TRAIL(vx), ul = FIM_LEAD(ux), vl = FIM_LEAD(vx);
        if constexpr (sizeof(R) == 8) {
          R w[4];
          ld4(g.vw + (i * 6 + e) * 4, w);
          R un = cs[0] * u0[j] + sn[0] * v0[j] + cs[1] * ux[e][j] + sn[1] * vx[e][j];
          R vn = cs[0] * v0[j] - sn[0] * u0[j] + cs[1] * vx[e][j] - sn[1] * ux[e][j];
          un = two * un + cs[2] * ut + sn[2] * vt + cs[3] * ul + sn[3] * vl;
          vn = two * vn + cs[2] * vt - sn[2] * ut + cs[3] * vl - sn[3] * ul;
          const R sq = un * un + vn * vn;
          const R ms = w[0] * m0[j] + w[1] * mx[e][j] + w[2] * FIM_TRAIL(mx) + w[3] * FIM_LEAD(mx);
          const R q = ms * (f64_lt(sq, R(36) * eps * eps) ? R(1) / (R(6) * eps) : f64_rsqrt(sq));
          ue[j] = un * q;
          ve[j] = vn * q;
        } else {
          const R u3trl = cs[2] * ut + sn[2] * vt, v3trl = -sn[2] * ut + cs[2] * vt;
          const R u1ldg = cs[0] * u0[j] + sn[0] * v0[j], v1ldg = -sn[0] * u0[j] + cs[0] * v0[j];
          const R u2ldg = cs[1] * ux[e][j] + sn[1] * vx[e][j], v2ldg = -sn[1] * ux[e][j] + cs[1] * vx[e][j];
          const R u3ldg = cs[3] * ul + sn[3] * vl, v3ldg = -sn[3] * ul + cs[3] * vl;
          const R uu = (two * (u1ldg + u2ldg) + u3trl + u3ldg) * divby6;
          const R vv = (two * (v1ldg + v2ldg) + v3trl + v3ldg) * divby6;
          const R m_1 = vmag(uu, vv);
          const R m_2 = (two * (vmag(u1ldg, v1ldg) + vmag(u2ldg, v2ldg)) + vmag(u3trl, v3trl) + vmag(u3ldg, v3ldg)) *
                        divby6;
          const R q = fdiv(m_2, rmax(eps, m_1));  // one division for both components
          ue[j] = uu * q;
          ve[j] = vv * q;
        }
        uv[j] = half * (ue[j] * ue[j] + ve[j] * ve[j]);
      }
      stv<VK>(pu + (size_t)e * L, ue);
      stv<VK>(pv + (size_t)e * L, ve);
      stv<VK>(pq + (size_t)e * L, uv);
    }
  }
  // mid-layer pressure
  {
    const R divby6 = R(1) / R(6), half = R(0.5);
    const R* pm = pres + m * s.intf;
    R p0[VK], pa[6][VK], pb[6][VK];  // FP64: pa the layer's sum
    FOR_V p0[j] = pm[(size_t)i * L1 + k + j] + pm[(size_t)i * L1 + k + j + 1];
#pragma unroll
    for (int e = 0; e < 6; e++) {
      const R* pe = pm + (size_t)nb[e] * L1 + k;
      R a = pe[0];
      FOR_V {
        const R b = pe[j + 1];
        pa[e][j] = sizeof(R) == 8 ? a + b : a;
        pb[e][j] = b;
        a = b;
      }
    }
    R* o = lp_edg + m * s.edge + oe;
#pragma unroll
    for (int e = 0; e < 6; e++) {
      if (e == 5 && five) continue;
      R lp[VK];
      if constexpr (sizeof(R) == 8)
        FOR_V lp[j] = (p0[j] + pa[e][j] + half * (FIM_TRAIL(pa) + FIM_LEAD(pa))) * divby6;
      else
        FOR_V lp[j] = (p0[j] + pa[e][j] + pb[e][j] + half * (FIM_TRAIL(pa) + FIM_TRAIL(pb) + FIM_LEAD(pa) + FIM_LEAD(pb))) *
                    divby6;
      stv<VK>(o + (size_t)e * L, lp);
    }
  }
  // Montgomery potential
  {
    R x0[VK], x[6][VK];
    if (mpf) {
      // edge minus cell value from float-float differences (no cancellation)
      const float2* mp = mpf + m * s.cell;
      float2 mc[VK];
      FOR_V {
        mc[j] = mp[c + j];
        x0[j] = R(0);
      }
#pragma unroll
      for (int e = 0; e < 6; e++) FOR_V x[e][j] = R(ff_diff(mp[(size_t)nb[e] * L + k + j], mc[j]));
    } else {
      around<R, VK>(montg + m * s.cell, L, i, k, nb, x0, x);
    }
    edge_means<R, VK>(five, L, x0, x, mont_edg + m * s.edge + oe);
  }
  if (!hi_order) {
    R x0[VK], x[6][VK];
    around<R, VK>(delp + m * s.cell, L, i, k, nb, x0, x);
    edge_means<R, VK>(five, L, x0, x, dp_edg + m * s.edge + oe);
  }
  const int ntr = hi_order ? 1 : g.T;
  for (int t = 0; t < ntr; t++) {
    R x0[VK], x[6][VK];
    around<R, VK>(tracr + m * s.tr + (size_t)t * N * L, L, i, k, nb, x0, x);
    // the potential temperature of this step's edge values, for momtum1
    if (t == 0 && thold) stv<VK>(thold + m * s.cell + c, x0);
    R* te = trc_edg + m * s.tredg + (size_t)t * N * 6 * L + oe;
    edge_means<R, VK>(five, L, x0, x, te);
    if (five) {
      R z[VK];
      FOR_V z[j] = R(0);
      stv<VK>(te + (size_t)5 * L, z);
    }
  }
}
#undef FIM_TRAIL
#undef FIM_LEAD

// g.vw; the first square's rounding is kept, so exact rotations give 1 / 3 and
// 1 / 6 to the last bit
__global__ void __launch_bounds__(kBlock) k_speed_weights(int n, const double* __restrict__ cs,
                                                          const double* __restrict__ sn, double* __restrict__ vw) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const double a = cs[q], b = sn[q], aa = a * a;
  vw[q] = sqrt((fma(b, b, aa) + fma(a, a, -aa)) / ((q & 3) < 2 ? 9. : 36.));
}
void launch_speed_weights(cudaStream_t stream, int N, const double* cs, const double* sn, double* vw) {
  k_speed_weights<<<blocks_for((long long)N * 24), kBlock, 0, stream>>>(N * 24, cs, sn, vw);
}

// --------------------------------------------------------------------------
// edgvar2 (edgvar2.F90:24-319, hiOrderUVComp; the MORE_VARS block is compiled
// out in the reference): the edge wind is rescaled to the mean of the speeds
// at the edge's two corners seen from the three cells around each corner,
// each a cell's speed plus its speed-gradient projected on the corner.
//  k_edgvar2_grad: per cell-level the speed |u| and the gradient of the edge
//                  speeds (gradient(), edgvar2.F90:231-258) -> w[0..2]
//  k_edgvar2:      per cell-level and edge, the corner speeds of the cell, the
//                  neighbour across the edge and the neighbours across the
//                  adjacent edges, the ratio to |u_edg| (1 below 1e-5), and
//                  uvsq_edg of the rescaled wind.
template <typename R>
__global__ void __launch_bounds__(kBlock) k_edgvar2_grad(Grid<R> g, Strides s, const R* __restrict__ u,
    const R* __restrict__ v, const R* __restrict__ u_edg, const R* __restrict__ v_edg, R* __restrict__ w) {
  int i, k;
  if (!cell_levels<1>(g.N, g.L, i, k)) return;
  const int L = g.L;
  const size_t m = blockIdx.y, NL = (size_t)g.N * L;
  u += m * s.cell; v += m * s.cell; u_edg += m * s.edge; v_edg += m * s.edge; w += m * 3 * NL;
  const size_t c = (size_t)i * L + k;
  const int np = g.nprox[i];
  R g1 = R(0), g2 = R(0);
  for (int e = 0; e < np; e++) {
    const size_t o = ((size_t)i * 6 + e) * L + k;
    const R sp = sqrt(u_edg[o] * u_edg[o] + v_edg[o] * v_edg[o]);
    g1 = g1 + sp * g.svc[(i * 6 + e) * 2 + 1];
    g2 = g2 - sp * g.svc[(i * 6 + e) * 2 + 0];
  }
  const R rar = g.rarea[i];
  w[c] = sqrt(u[c] * u[c] + v[c] * v[c]);
  w[NL + c] = g1 * rar;
  w[2 * NL + c] = g2 * rar;
}

template <typename R>
__global__ void __launch_bounds__(kBlock) k_edgvar2(Grid<R> g, Strides s, const R* __restrict__ w,
    R* __restrict__ u_edg, R* __restrict__ v_edg, R* __restrict__ uvsq_edg) {
  int i, k;
  if (!cell_levels<1>(g.N, g.L, i, k)) return;
  const int L = g.L;
  const size_t m = blockIdx.y, NL = (size_t)g.N * L;
  u_edg += m * s.edge; v_edg += m * s.edge; uvsq_edg += m * s.edge; w += m * 3 * NL;
  const R divby6 = R(1) / R(6), eps = R(0.00001);
  const int np = g.nprox[i];
  // corner q of cell x: its speed plus 0.5 * (grad . corner_xy(q))
  auto corner = [&](int x, int q) -> R {
    const size_t cx = (size_t)x * L + k;
    const R gc = R(0.5) * (w[NL + cx] * g.cxy[(x * 2 + 0) * 6 + q] + w[2 * NL + cx] * g.cxy[(x * 2 + 1) * 6 + q]);
    return w[cx] + gc;
  };
  for (int e = 0; e < np; e++) {
    const int nba = g.prox[i * 6 + e], nbaedg = g.proxs[i * 6 + e];
    const int em1 = (e - 1 + np) % np, ep1 = (e + 1) % np;
    const int nbm1 = g.prox[i * 6 + em1], nbp1 = g.prox[i * 6 + ep1];
    const R uv1conr1 = corner(i, e);
    const R uv2conr1 = corner(nba, (nbaedg + 1) % g.nprox[nba]);
    const R uv3conr1 = corner(nbm1, g.proxs[i * 6 + em1]);
    const R uv1conr2 = corner(i, ep1);
    const R uv2conr2 = corner(nba, nbaedg);
    const R uv3conr2 = corner(nbp1, (g.proxs[i * 6 + ep1] + 1) % g.nprox[nbp1]);
    const size_t o = ((size_t)i * 6 + e) * L + k;
    R ue = u_edg[o], ve = v_edg[o];
    const R uvm1 = sqrt(ue * ue + ve * ve);
    const R uvm2 = (uv1conr1 + uv2conr1 + uv3conr1 + uv1conr2 + uv2conr2 + uv3conr2) * divby6;
    const R r_m = uvm1 < eps ? R(1) : uvm2 / uvm1;
    ue = ue * r_m;
    ve = ve * r_m;
    u_edg[o] = ue;
    v_edg[o] = ve;
    uvsq_edg[o] = R(.5) * (ue * ue + ve * ve);
  }
}

template <typename R>
void launch_edgvar2(const Launch& l, const Grid<R>& g, const Strides& s, const R* u, const R* v, R* u_edg,
                    R* v_edg, R* uvsq_edg, R* w) {
  dim3 grid(blocks_for((long long)g.N * g.L), l.members);
  FIM_KBEGIN(l, "k_edgvar2_grad");
  k_edgvar2_grad<R><<<grid, kBlock, 0, l.stream>>>(g, s, u, v, u_edg, v_edg, w);
  FIM_KEND(l);
  FIM_KBEGIN(l, "k_edgvar2");
  k_edgvar2<R><<<grid, kBlock, 0, l.stream>>>(g, s, w, u_edg, v_edg, uvsq_edg);
  FIM_KEND(l);
}

// --------------------------------------------------------------------------
// edgvar3 loop 1 with edgvalEval (edgvar3.F90:66-94,136-163): least-squares
// (hfcoef) reconstruction of dp (field 0) and tracers 2..ntra (field t) on the
// cell's own edges; pentagons store 0 in the sixth slot.
template <typename R, int VK>
__global__ void __launch_bounds__(kBlock) k_edgvar3_own(Grid<R> g, Strides s,
    const R* __restrict__ delp, const R* __restrict__ tracr, R* __restrict__ dp_edg, R* __restrict__ trc_edg) {
  int i, k;
  if (!cell_levels<VK>(g.N, g.L, i, k)) return;
  const int L = g.L, N = g.N;
  const size_t m = blockIdx.y;
  const int f = blockIdx.z;
  const R* src = (f == 0) ? delp + m * s.cell : tracr + m * s.tr + (size_t)f * N * L;
  R* dst = (f == 0) ? dp_edg + m * s.edge : trc_edg + m * s.tredg + (size_t)f * N * 6 * L;
  const int np = g.nprox[i];
  const int* pr = g.prox + i * 6;
  R bc[VK];
  ldv<VK>(src + (size_t)i * L + k, bc);
  // branch-free gathers over the six prox slots (all valid cells); a
  // pentagon's slot 5 is dropped by selects
  R d[6][VK];
#pragma unroll
  for (int e = 0; e < 6; e++) {
    ldv<VK>(src + (size_t)pr[e] * L + k, d[e]);
    FOR_V d[e][j] = e < np ? d[e][j] - bc[j] : R(0);
  }
  const R* hf = g.hfcoef + (size_t)i * 36;
#pragma unroll
  for (int ie = 0; ie < 6; ie++) {
    R val[VK];
    FOR_V val[j] = bc[j];
#pragma unroll
    for (int e = 0; e < 6; e++) {
      const R h = hf[ie * 6 + e];
      FOR_V val[j] = e < np ? val[j] + d[e][j] * h : val[j];
    }
    FOR_V val[j] = ie < np ? val[j] : R(0);
    stv<VK>(dst + ((size_t)i * 6 + ie) * L + k, val);
  }
}

// edgvar3 loop 2 (edgvar3.F90:110-132): the lower-numbered cell of each pair
// stores the two-sided average in both slots, as the reference does; each slot
// has exactly one writer, which is also its only reader.
template <typename R, int VK>
__global__ void __launch_bounds__(kBlock) k_edgvar3_avg(Grid<R> g, Strides s, R* __restrict__ dp_edg,
                                                       R* __restrict__ trc_edg) {
  int i, k;
  if (!cell_levels<VK>(g.N, g.L, i, k)) return;
  const int L = g.L, N = g.N;
  const size_t m = blockIdx.y;
  const int f = blockIdx.z;
  R* x = (f == 0) ? dp_edg + m * s.edge : trc_edg + m * s.tredg + (size_t)f * N * 6 * L;
  const int np = g.nprox[i];
  for (int e = 0; e < np; e++) {
    const int nb = g.prox[i * 6 + e];
    if (i < nb) {
      const int os = g.proxs[i * 6 + e];
      const size_t a = ((size_t)i * 6 + e) * L + k, b = ((size_t)nb * 6 + os) * L + k;
      R xa[VK], xb[VK], w[VK];
      ldv<VK>(x + a, xa);
      ldv<VK>(x + b, xb);
      FOR_V w[j] = R(0.5) * (xa[j] + xb[j]);
      stv<VK>(x + a, w);
      stv<VK>(x + b, w);
    }
  }
}

// --------------------------------------------------------------------------
// cnuity1 + cnuity2 (cnuity_compute.F90:41-146): normal velocity on the cell's
// edge and on the neighbour's copy of it, donor-cell mass flux, antidiffusive
// flux, low-order tendency and low-order thickness; also the Zalesak sums
// P+/P- of cnuity3 (cnuity_compute.F90:186-194), which only need own edges.
// The bodies of cnuity12/3/4 take the (virtual) block index, so the persistent
// variant below runs the same code; their pointers carry no __restrict__ (the
// persistent variant reads in one stage what another block wrote in the
// stage before, which read-only loads must not do).
template <typename R, int VK>
__device__ __forceinline__ void cnuity12_body(int bx, int by, const Grid<R>& g, const Strides& s,
    const StepParams* sp, const R* u_edg, const R* v_edg, const R* dp_edg, const R* delp, R* massfx,
    R* dplo_tndcy, R* antifx, R* delp_lo, R* p_plus, R* p_mnus) {
  int i, k;
  if (!cell_levels_at<VK>(g.N, g.L, bx, i, k)) return;
  const int L = g.L, N = g.N;
  const size_t m = by;
  sp += m;
  if (!sp->active) return;
  u_edg += m * s.edge; v_edg += m * s.edge; dp_edg += m * s.edge; delp += m * s.cell;
  massfx += m * s.mf; dplo_tndcy += m * s.ab; antifx += m * s.edge; delp_lo += m * s.cell;
  p_plus += m * s.cell; p_mnus += m * s.cell;
  const int nf = sp->nf, of = sp->of, vof = sp->vof;
  const R ab1 = sp->template w1<R>(), ab2 = sp->template w2<R>(), ab3 = sp->template w3<R>();
  R* mfn = massfx + (size_t)nf * N * 6 * L;
  const int np = g.nprox[i];
  const R half = R(0.5);
  R dpi[VK], sum[VK], pp[VK], pm[VK];
  ldv<VK>(delp + (size_t)i * L + k, dpi);
  bool rare = false;  // FP64: a flux needs plain_donor
  FOR_V { sum[j] = R(0); pp[j] = R(0); pm[j] = R(0); }
  if (np < 6) {
    R z[VK];
    FOR_V z[j] = R(0);
    stv<VK>(mfn + ((size_t)i * 6 + 5) * L + k, z);
    stv<VK>(antifx + ((size_t)i * 6 + 5) * L + k, z);
  }
  // branch-free over the six slots: a pentagon's slot 5 reads valid rows
  // (mirror edge 0) and is neither accumulated nor stored
#pragma unroll
  for (int e = 0; e < 6; e++) {
    const bool live = e < np;
    const int ipx = g.prox[i * 6 + e], edx = live ? g.proxs[i * 6 + e] : 0;
    const R* sv = g.sve + (i * 6 + e) * 2;
    const R* sx = g.sve + (ipx * 6 + edx) * 2;
    const size_t o = ((size_t)i * 6 + e) * L + k, ox = ((size_t)ipx * 6 + edx) * L + k;
    R ue[VK], ve[VK], ux[VK], vx_[VK], de[VK], dx[VK], mf[VK], an[VK];
    ldv<VK>(u_edg + o, ue);
    ldv<VK>(v_edg + o, ve);
    ldv<VK>(u_edg + ox, ux);
    ldv<VK>(v_edg + ox, vx_);
    // edgvar3's two-sided average 0.5*(own + neighbour's own), formed here
    // (exact also when dp_edg already holds it: 0.5*(w + w) == w)
    R dm[VK];
    ldv<VK>(dp_edg + o, de);
    ldv<VK>(dp_edg + ox, dm);
    if constexpr (sizeof(R) == 4) FOR_V de[j] = half * (de[j] + dm[j]);
    ldv<VK>(delp + (size_t)ipx * L + k, dx);
    FOR_V {
      const R vn = sv[1] * ue[j] - sv[0] * ve[j];
      const R vx = sx[1] * ux[j] - sx[0] * vx_[j];
      if constexpr (sizeof(R) == 8) {  // the same, with half the FP64 operations
        mf[j] = donor(vn, vx, dpi[j], dx[j]);
        an[j] = fma(half * vn, de[j] + dm[j], -mf[j]);
        if (live) {
          sum[j] = sum[j] + mf[j];
          split_sum(an[j], pp[j], pm[j]);
          rare |= donor_rare(vn, vx) | f64_odd(dx[j]);
        }
        continue;
      }
      const R flxhi = vn * de[j];
      mf[j] = half * ((vn + rabs(vn)) * dpi[j] - (vx + rabs(vx)) * dx[j]);
      const R a = flxhi - mf[j];
      an[j] = a;
      sum[j] = live ? sum[j] + mf[j] : sum[j];
      if (live && a <= R(0)) pp[j] = pp[j] - a;
      else if (live) pm[j] = pm[j] + a;
    }
    if (live) {
      stv<VK>(mfn + o, mf);
      stv<VK>(antifx + o, an);
    }
  }
  if constexpr (sizeof(R) == 8) {
    FOR_V rare |= f64_odd(dpi[j]) | sums_rare(pp[j], pm[j]);
    if (rare) {
      FOR_V { sum[j] = R(0); pp[j] = R(0); pm[j] = R(0); }
#pragma unroll 1
      for (int e = 0; e < np; e++) {
        const int ipx = g.prox[i * 6 + e], edx = g.proxs[i * 6 + e];
        const R* sv = g.sve + (i * 6 + e) * 2;
        const R* sx = g.sve + (ipx * 6 + edx) * 2;
        const size_t o = ((size_t)i * 6 + e) * L + k, ox = ((size_t)ipx * 6 + edx) * L + k;
        FOR_V {
          const R vn = sv[1] * u_edg[o + j] - sv[0] * v_edg[o + j];
          const R vx = sx[1] * u_edg[ox + j] - sx[0] * v_edg[ox + j];
          const R mf = plain_donor(vn, vx, dpi[j], delp[(size_t)ipx * L + k + j]);
          const R a = fma(half * vn, dp_edg[o + j] + dp_edg[ox + j], -mf);
          sum[j] = sum[j] + mf;
          if (a <= R(0)) pp[j] = pp[j] - a;
          else pm[j] = pm[j] + a;
          mfn[o + j] = mf;
          antifx[o + j] = a;
        }
      }
    }
  }
  const size_t c = (size_t)i * L + k;
  const R rar = g.rarea[i];
  R tn[VK], to[VK], tv[VK], lo[VK];
  FOR_V tn[j] = -sum[j] * rar;
  stv<VK>(dplo_tndcy + (size_t)nf * N * L + c, tn);
  ldv<VK>(dplo_tndcy + (size_t)of * N * L + c, to);
  ldv<VK>(dplo_tndcy + (size_t)vof * N * L + c, tv);
  FOR_V lo[j] = dpi[j] + ab1 * tn[j] + ab2 * to[j] + ab3 * tv[j];
  stv<VK>(delp_lo + c, lo);
  stv<VK>(p_plus + c, pp);
  stv<VK>(p_mnus + c, pm);
}
// FP32 at four levels a thread: the three blocks an SM that 80 registers let
// in (the compiler's own 72 also give three, with its loads serialised: glvl 7
// / nvl 64 283 -> 255 us; two 294, four 322).  Narrower accesses keep the
// compiler's choice (0): at two levels more registers make the kernel 3 us
// faster alone and the step 4 us slower, its companion stream's blocks wait.
template <typename R, int VK>
__global__ void __launch_bounds__(kBlock, VK == 4 ? 3 : 0) k_cnuity12(Grid<R> g, Strides s, const StepParams* __restrict__ sp,
    const R* __restrict__ u_edg, const R* __restrict__ v_edg, const R* __restrict__ dp_edg,
    const R* __restrict__ delp, R* __restrict__ massfx, R* __restrict__ dplo_tndcy, R* __restrict__ antifx,
    R* __restrict__ delp_lo, R* __restrict__ p_plus, R* __restrict__ p_mnus) {
  cnuity12_body<R, VK>(blockIdx.x, blockIdx.y, g, s, sp, u_edg, v_edg, dp_edg, delp, massfx, dplo_tndcy, antifx,
                       delp_lo, p_plus, p_mnus);
}

// cnuity3 (cnuity_compute.F90:206-252): 1-ring max/min of old and low-order
// thickness, Zalesak Q+/Q- and the limiters R+/R-.
template <typename R, int VK>
__device__ __forceinline__ void cnuity3_body(int bx, int by, const Grid<R>& g, const Strides& s,
    const StepParams* sp, const R* delp_lo, const R* delp, const R* dp_tndcy, const R* p_plus, const R* p_mnus,
    R* r_plus, R* r_mnus) {
  int i, k;
  if (!cell_levels_at<VK>(g.N, g.L, bx, i, k)) return;
  const int L = g.L, N = g.N;
  const size_t m = by;
  sp += m;
  if (!sp->active) return;
  delp_lo += m * s.cell; delp += m * s.cell; dp_tndcy += m * s.ab;
  p_plus += m * s.cell; p_mnus += m * s.cell; r_plus += m * s.cell; r_mnus += m * s.cell;
  const int of = sp->of, vof = sp->vof;
  const R ab1 = sp->template w1<R>(), ab2 = sp->template w2<R>(), ab3 = sp->template w3<R>();
  const R rab1 = R(1) / ab1;  // Q+/Q- divide by ab1: one reciprocal
  const R thshld = R(1.e-11);
  const size_t c = (size_t)i * L + k;
  const int* pr = g.prox + i * 6;
  R dlo[VK], dc[VK];
  ldv<VK>(delp_lo + c, dlo);
  ldv<VK>(delp + c, dc);
  Bound<R> mx[VK], mn[VK];
  FOR_V {
    mx[j] = mn[j] = Bound<R>::of(dlo[j]);
    const Bound<R> b = Bound<R>::of(dc[j]);
    mx[j].up(b);
    mn[j].down(b);
  }
#pragma unroll
  for (int e = 0; e < 6; e++) {
    R a[VK], b[VK];
    ldv<VK>(delp_lo + (size_t)pr[e] * L + k, a);
    ldv<VK>(delp + (size_t)pr[e] * L + k, b);
    FOR_V {
      const Bound<R> ba = Bound<R>::of(a[j]), bb = Bound<R>::of(b[j]);
      mx[j].up(ba, bb);
      mn[j].down(ba, bb);
    }
  }
  R to[VK], tv[VK], pp[VK], pm[VK], rp[VK], rm[VK];
  ldv<VK>(dp_tndcy + (size_t)of * N * L + c, to);
  ldv<VK>(dp_tndcy + (size_t)vof * N * L + c, tv);
  ldv<VK>(p_plus + c, pp);
  ldv<VK>(p_mnus + c, pm);
  const R ar = sizeof(R) == 8 ? g.area[i] * rab1 : g.area[i];
  bool rare = false;
  FOR_V {
    const R dpmax = mx[j].at_least_zero(), dpmin = mn[j].at_least_zero();
    const R q_plus = per_ab1(dpmax - dlo[j] - (ab2 * neg(to[j]) + ab3 * pos(tv[j])), rab1, ar);
    const R q_mnus = per_ab1(dlo[j] - dpmin + (ab2 * pos(to[j]) + ab3 * neg(tv[j])), rab1, ar);
    rp[j] = ratio01(q_plus, floor_at(pp[j], thshld));
    rm[j] = ratio01(q_mnus, floor_at(pm[j], thshld));
    rare |= bounds_rare(mx[j], mn[j]) | ratio_rare(q_plus, q_mnus);
  }
  if (rare) {  // as the routine writes it
    FOR_V {
      R hi = rmax(dlo[j], dc[j]), lo = rmin(dlo[j], dc[j]);
#pragma unroll 1
      for (int e = 0; e < 6; e++) {
        const R a = delp_lo[(size_t)pr[e] * L + k + j], b = delp[(size_t)pr[e] * L + k + j];
        hi = rmax(hi, rmax(a, b));
        lo = rmin(lo, rmin(a, b));
      }
      hi = rmax(R(0), hi);
      lo = rmax(R(0), lo);
      rp[j] = plain_ratio01(per_ab1(hi - dlo[j] - (ab2 * rmin(R(0), to[j]) + ab3 * rmax(R(0), tv[j])), rab1, ar), pp[j]);
      rm[j] = plain_ratio01(per_ab1(dlo[j] - lo + (ab2 * rmax(R(0), to[j]) + ab3 * rmin(R(0), tv[j])), rab1, ar), pm[j]);
    }
  }
  stv<VK>(r_plus + c, rp);
  stv<VK>(r_mnus + c, rm);
}
template <typename R, int VK>
__global__ void __launch_bounds__(kBlock) k_cnuity3(Grid<R> g, Strides s, const StepParams* __restrict__ sp,
    const R* __restrict__ delp_lo, const R* __restrict__ delp, const R* __restrict__ dp_tndcy,
    const R* __restrict__ p_plus, const R* __restrict__ p_mnus, R* __restrict__ r_plus, R* __restrict__ r_mnus) {
  cnuity3_body<R, VK>(blockIdx.x, blockIdx.y, g, s, sp, delp_lo, delp, dp_tndcy, p_plus, p_mnus, r_plus, r_mnus);
}

// cnuity4 (cnuity_compute.F90:291-369): clip the antidiffusive flux with the
// own and neighbour limiters, total mass flux, AB3 thickness update.
template <typename R, int VK>
__device__ __forceinline__ void cnuity4_body(int bx, int by, const Grid<R>& g, const Strides& s,
    const StepParams* sp, const R* antifx, const R* r_plus, const R* r_mnus, R* massfx, const R* dplo_tndcy,
    R* dp_tndcy, R* delp, int* flags) {
  int i, k;
  if (!cell_levels_at<VK>(g.N, g.L, bx, i, k)) return;
  const int L = g.L, N = g.N;
  const size_t m = by;
  sp += m;
  if (!sp->active) return;
  antifx += m * s.edge; r_plus += m * s.cell; r_mnus += m * s.cell; massfx += m * s.mf;
  dplo_tndcy += m * s.ab; dp_tndcy += m * s.ab; delp += m * s.cell;
  const int nf = sp->nf, of = sp->of, vof = sp->vof;
  const R ab1 = sp->template w1<R>(), ab2 = sp->template w2<R>(), ab3 = sp->template w3<R>();
  R* mfn = massfx + (size_t)nf * N * 6 * L;
  const size_t c = (size_t)i * L + k;
  R rp[VK], rm[VK], at[VK];
  ldv<VK>(r_plus + c, rp);
  ldv<VK>(r_mnus + c, rm);
  FOR_V {
    if (sizeof(R) == 8) {
      rp[j] = own_limit(rp[j]);
      rm[j] = own_limit(rm[j]);
    }
    at[j] = R(0);
  }
  const int np = g.nprox[i];
  for (int e = 0; e < np; e++) {
    const int px = g.prox[i * 6 + e];
    const size_t o = ((size_t)i * 6 + e) * L + k;
    R a[VK], mf[VK], rpx[VK], rmx[VK];
    ldv<VK>(antifx + o, a);
    ldv<VK>(mfn + o, mf);
    ldv<VK>(r_plus + (size_t)px * L + k, rpx);
    ldv<VK>(r_mnus + (size_t)px * L + k, rmx);
    FOR_V {
      const bool in = below0(a[j]);
      const R own = in ? rp[j] : rm[j], other = in ? rmx[j] : rpx[j];
      const R clip = sizeof(R) == 8 ? min0(own, other) : rmin(own, other);
      const R ac = a[j] * clip;
      mf[j] = mf[j] + ac;
      at[j] = at[j] + ac;
    }
    stv<VK>(mfn + o, mf);
  }
  const R rar = g.rarea[i];
  R tl[VK], tn[VK], to[VK], tv[VK], dn[VK];
  ldv<VK>(dplo_tndcy + (size_t)nf * N * L + c, tl);
  FOR_V tn[j] = tl[j] + (-at[j] * rar);
  stv<VK>(dp_tndcy + (size_t)nf * N * L + c, tn);
  ldv<VK>(dp_tndcy + (size_t)of * N * L + c, to);
  ldv<VK>(dp_tndcy + (size_t)vof * N * L + c, tv);
  ldv<VK>(delp + c, dn);
  bool bad = false;
  FOR_V {
    dn[j] = dn[j] + ab1 * tn[j] + ab2 * to[j] + ab3 * tv[j];
    bad = bad || !(dn[j] > R(0));
  }
  stv<VK>(delp + c, dn);
  if (bad) atomicOr(flags + m, kFlagBadDp);
}
template <typename R, int VK>
__global__ void __launch_bounds__(kBlock) k_cnuity4(Grid<R> g, Strides s, const StepParams* __restrict__ sp,
    const R* __restrict__ antifx, const R* __restrict__ r_plus, const R* __restrict__ r_mnus,
    R* __restrict__ massfx, const R* __restrict__ dplo_tndcy, R* __restrict__ dp_tndcy, R* __restrict__ delp,
    int* __restrict__ flags) {
  cnuity4_body<R, VK>(blockIdx.x, blockIdx.y, g, s, sp, antifx, r_plus, r_mnus, massfx, dplo_tndcy, dp_tndcy, delp,
                      flags);
}

// ---- persistent variant of cnuity1..4 ---------------------------------------
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid-wide barrier of a cooperative launch.  Every block adds one to *ctr
// and waits until it reaches target; the wait gives up after limit_ns (and
// after 2^22 polls whatever the timer says), sets kFlagTimeout in *flags and
// returns false, so the kernel ends and the host reads FIM_ETIMEDOUT.
__device__ bool coop_barrier(unsigned* ctr, unsigned target, unsigned long long limit_ns, int* flags) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(ctr, 1u);
    int good = 1;
    const unsigned long long t0 = global_ns();
    for (unsigned it = 0;; it++) {
      if (*(volatile unsigned*)ctr >= target) break;
      if (it >= (1u << 22) || global_ns() - t0 > limit_ns) {
        good = 0;
        break;
      }
      __nanosleep(64);
    }
    if (!good) atomicOr(flags, kFlagTimeout);
    __threadfence();
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// cnuity1..4 of every member in one cooperative launch: the blocks resident
// on the GPU walk the virtual blocks of each stage, with a grid barrier
// between the stages in place of kernel boundaries.  extra arrivals are added
// to each barrier's target (a barrier that can never complete: the test of
// the time limit).
template <typename R, int VK>
__global__ void __launch_bounds__(kBlock) k_cnuity_coop(Grid<R> g, Strides s, const StepParams* sp, int members,
    const R* u_edg, const R* v_edg, const R* dp_edg, R* delp, R* massfx, R* dplo_tndcy, R* dp_tndcy, R* antifx,
    R* delp_lo, R* p_plus, R* p_mnus, R* r_plus, R* r_mnus, int* flags, unsigned* bar, unsigned extra,
    unsigned long long limit_ns) {
  const int nvb = (int)(((long long)g.N * (g.L / VK) + kBlock - 1) / kBlock);
  const int total = nvb * members;
  for (int w = blockIdx.x; w < total; w += gridDim.x)
    cnuity12_body<R, VK>(w % nvb, w / nvb, g, s, sp, u_edg, v_edg, dp_edg, delp, massfx, dplo_tndcy, antifx,
                         delp_lo, p_plus, p_mnus);
  if (!coop_barrier(bar, gridDim.x + extra, limit_ns, flags)) return;
  for (int w = blockIdx.x; w < total; w += gridDim.x)
    cnuity3_body<R, VK>(w % nvb, w / nvb, g, s, sp, delp_lo, delp, dp_tndcy, p_plus, p_mnus, r_plus, r_mnus);
  if (!coop_barrier(bar, 2 * gridDim.x + extra, limit_ns, flags)) return;
  for (int w = blockIdx.x; w < total; w += gridDim.x)
    cnuity4_body<R, VK>(w % nvb, w / nvb, g, s, sp, antifx, r_plus, r_mnus, massfx, dplo_tndcy, dp_tndcy, delp,
                        flags);
}

// cnuity5 (cnuity_compute.F90:408-445), 32 columns a block.  The layer
// thickness and pressure tendency of every level are formed with thread =
// (column, VK levels) into shared tiles; the top-down pressure sum (warp 0) and
// the omega flux-convergence integral (warp 1) run with lane = column up the
// tiles in the reference's order (FP64, or float-float in the FP32-mixed
// build); the Exner function and the v.grad(p) term are formed with thread =
// (column, VK levels) again.  The sums are a serial chain of ~nvl steps, so the
// block's other warps and its neighbours on the SM cover it: one warp doing
// all three parts of its 32 columns, 32 levels at a time, left two to four warps
// an SM in flight on small grids.  FP32, nvl 64: glvl 8 0.84 -> 0.44 ms (5,340
// GB/s of its 14 words), glvl 5 / nvl 38 78 -> 14 us (4 levels a thread; one:
// 0.65 ms and 18 us).  FP64, glvl 6: 0.70 -> 0.35 ms, with the power of
// fim_internal.h; one level a thread, bound by the FP64 pipe.
constexpr int kC5Cols = 32;
constexpr int kC5Block = 256;
template <typename R, int VK>
__global__ void __launch_bounds__(kC5Block, 4) k_cnuity5(Grid<R> g, Strides s,
    const StepParams* __restrict__ sp, R* __restrict__ pres, R* __restrict__ delp, R* __restrict__ exner,
    const R* __restrict__ dp_tndcy, R* __restrict__ omega, const R* __restrict__ lp_edg, const R* __restrict__ u,
    const R* __restrict__ v, int ab3_delp) {
  extern __shared__ __align__(16) unsigned char c5sm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int N = g.N, L = g.L, L1 = L + 1, LV = L / VK;
  const int LS = L | 1;  // odd row stride: lane = column reads are conflict-free
  R* const tp = reinterpret_cast<R*>(c5sm);  // thickness in, pressure out
  R* const tw = tp + kC5Cols * LS;           // layer pressure tendency in, omega's first terms out
  const int i0 = blockIdx.x * kC5Cols;
  const int ncol = N - i0 < kC5Cols ? N - i0 : kC5Cols;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active) return;
  pres += m * s.intf; delp += m * s.cell; exner += m * s.intf; dp_tndcy += m * s.ab;
  omega += m * s.cell; lp_edg += m * s.edge; u += m * s.cell; v += m * s.cell;
  const int nf = sp->nf, of = sp->of, vof = sp->vof;
  const R ab1 = sp->template w1<R>(), ab2 = sp->template w2<R>(), ab3 = sp->template w3<R>(), dt = sp->template step<R>();
  const R cp = R(kCp), p1000 = R(kP1000), rdt = R(1) / dt;
  const size_t NL = (size_t)N * L;
#pragma unroll 2
  for (int it = threadIdx.x; it < ncol * LV; it += kC5Block) {
    const int r = it / LV, k = (it - r * LV) * VK;
    const size_t c = (size_t)(i0 + r) * L + k;
    R tnf[VK], tof[VK], tvf[VK], d[VK];
    ldv<VK>(dp_tndcy + (size_t)nf * NL + c, tnf);
    ldv<VK>(dp_tndcy + (size_t)of * NL + c, tof);
    ldv<VK>(dp_tndcy + (size_t)vof * NL + c, tvf);
    ldv<VK>(delp + c, d);
    if (ab3_delp) {
      // massflux_newdepth's AB3 thickness update (massadv_compute.F90:85-91)
      FOR_V {
        const R dn = d[j] + ab1 * tnf[j] + ab2 * tof[j] + ab3 * tvf[j];
        d[j] = dn > R(0) ? dn : R(0);
      }
      stv<VK>(delp + c, d);
    }
    FOR_V {
      tp[r * LS + k + j] = d[j];
      tw[r * LS + k + j] = divide_by(ab1 * tnf[j] + ab2 * tof[j] + ab3 * tvf[j], dt, rdt);
    }
  }
  __syncthreads();
  if (lane < ncol) {
    if (wib == 0) {
      R* t = tp + lane * LS;
      const R ptop = pres[(size_t)(i0 + lane) * L1 + L];
      if constexpr (sizeof(R) == 4) {
        FF2 pf{(float)ptop, 0.f};
#pragma unroll 4
        for (int k = L - 1; k >= 0; k--) {
          pf = ff_add(pf, FF2{t[k], 0.f});
          t[k] = pf.hi;
        }
      } else {
        double pd = (double)ptop;
#pragma unroll 4
        for (int k = L - 1; k >= 0; k--) {
          pd = pd + (double)t[k];
          t[k] = R(pd);
        }
      }
    } else if (wib == 1) {
      // omega = (integral of the layers above) + half of this layer
      R* t = tw + lane * LS;
      if constexpr (sizeof(R) == 4) {
        FF2 cf{0.f, 0.f};
#pragma unroll 4
        for (int k = L - 1; k >= 0; k--) {
          const R lyr = t[k];
          t[k] = R(cf.hi + cf.lo) + R(0.5) * lyr;
          cf = ff_add(cf, FF2{lyr, 0.f});
        }
      } else {
        double cd = 0.0;
#pragma unroll 4
        for (int k = L - 1; k >= 0; k--) {
          const double lyr = (double)t[k];
          t[k] = R(cd + 0.5 * lyr);
          cd = cd + lyr;
        }
      }
    }
  }
  __syncthreads();
  for (int it = threadIdx.x; it < ncol * LV; it += kC5Block) {
    const int r = it / LV, k = (it - r * LV) * VK;
    const int i = i0 + r;
    const size_t c = (size_t)i * L + k;
    // pressure gradient over the cell's edges (all six slots hold valid
    // rows; a pentagon's slot 5 is left out)
    const int np = g.nprox[i];
    R lp[6][VK], uu[VK], vv[VK], om[VK];
#pragma unroll
    for (int e = 0; e < 6; e++) ldv<VK>(lp_edg + ((size_t)i * 6 + e) * L + k, lp[e]);
    ldv<VK>(u + c, uu);
    ldv<VK>(v + c, vv);
    R dpdx[VK], dpdy[VK];
    FOR_V {
      const R pr = tp[r * LS + k + j];
      pres[(size_t)i * L1 + k + j] = pr;
      exner[(size_t)i * L1 + k + j] = cp * pow_rd_cp(divide_by(pr, p1000, R(1) / R(kP1000)));
      dpdx[j] = R(0);
      dpdy[j] = R(0);
    }
#pragma unroll
    for (int e = 0; e < 6; e++)
      if (e < np) {
        const R* sv = g.svc + (i * 6 + e) * 2;
        FOR_V {
          dpdx[j] = dpdx[j] + lp[e][j] * sv[1];
          dpdy[j] = dpdy[j] - lp[e][j] * sv[0];
        }
      }
    const R rar = g.rarea[i];
    FOR_V om[j] = tw[r * LS + k + j] + (uu[j] * dpdx[j] + vv[j] * dpdy[j]) * rar;
    stv<VK>(omega + c, om);
  }
}

template <typename R>
void launch_cnuity5(const Launch& l, const Grid<R>& g, const Strides& s, R* pres, R* delp, R* exner,
                    const R* dp_tndcy, R* omega, const R* lp_edg, const R* u, const R* v, int ab3_delp) {
  const int vk = pick_vk<R>(g.L, {delp, dp_tndcy, omega, lp_edg, u, v}, sizeof(R) == 8 ? 1 : 0);
  const size_t smem = (size_t)2 * kC5Cols * (g.L | 1) * sizeof(R);
  const dim3 grid((unsigned)((g.N + kC5Cols - 1) / kC5Cols), l.members);
  FIM_KBEGIN(l, "k_cnuity5");
  FIM_VK_DISPATCH(R, vk, ({
    if (smem > (size_t)48 * 1024)  // FP64 columns of more than 95 levels
      cudaFuncSetAttribute(k_cnuity5<R, VK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(2 * kC5Cols * (kMaxL | 1) * sizeof(R)));
    k_cnuity5<R, VK><<<grid, kC5Block, smem, l.stream>>>(g, s, l.sp, pres, delp, exner, dp_tndcy, omega, lp_edg, u, v,
                                                         ab3_delp);
  }));
  FIM_KEND(l);
}

// --------------------------------------------------------------------------
// mass_adv (flux_conserv_schm = 2, the reference default): flux_limiter.F90
// edgeNormVel + limiter (M1 branch).  k_massadv_lim: bounded edge thickness
// q* per edge and the outflow bounds q_min_out/q_max_out per cell
// (flux_limiter.F90:149-233).  k_massadv_flux: limited edge thickness with
// the upwind cell's bounds, mass flux, dp tendency (flux_limiter.F90:247-259,
// massadv_compute.F90:45-83); the AB3 thickness update runs in k_cnuity5.
template <typename R>
__device__ __forceinline__ void ma_edge(const Grid<R>& g, int i, int k, int e, int np, const R* u_edg,
                                        const R* v_edg, const R* dp_edg, const R* delp, R& vn, R& qs, int& ipx) {
  const int L = g.L;
  const int* pr = g.prox + i * 6;
  ipx = pr[e];
  const int nbm1 = pr[e == 0 ? np - 1 : e - 1], nbp1 = pr[e == np - 1 ? 0 : e + 1];
  const R* sv = g.sve + (i * 6 + e) * 2;
  const size_t o = ((size_t)i * 6 + e) * L + k;
  vn = sv[1] * u_edg[o] - sv[0] * v_edg[o];
  const R a = delp[(size_t)i * L + k], b = delp[(size_t)ipx * L + k], c = delp[(size_t)nbm1 * L + k],
          d = delp[(size_t)nbp1 * L + k];
  const R qmn = rmin(rmin(rmin(a, b), c), d), qmx = rmax(rmax(rmax(a, b), c), d);
  qs = rmax(qmn, rmin(qmx, dp_edg[o]));
}

template <typename R>
__global__ void __launch_bounds__(kBlock) k_massadv_lim(Grid<R> g, Strides s, const StepParams* __restrict__ sp,
    const R* __restrict__ u_edg, const R* __restrict__ v_edg, const R* __restrict__ dp_edg,
    const R* __restrict__ delp, const R* __restrict__ dp_tndcy, R* __restrict__ qmin_out, R* __restrict__ qmax_out) {
  int i, k;
  if (!cell_level(g.N, g.L, i, k)) return;
  const int L = g.L, N = g.N;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active) return;
  u_edg += m * s.edge; v_edg += m * s.edge; dp_edg += m * s.edge; delp += m * s.cell; dp_tndcy += m * s.ab;
  qmin_out += m * s.cell; qmax_out += m * s.cell;
  const int of = sp->of, vof = sp->vof;
  const R ab1 = sp->template w1<R>(), ab2 = sp->template w2<R>(), ab3 = sp->template w3<R>(), dt = sp->template step<R>();
  const size_t c = (size_t)i * L + k;
  const R gv = delp[c], rar = g.rarea[i];
  const int np = g.nprox[i];
  R qminin = sizeof(R) == 8 ? R(1.79769313486231571e308) : R(3.40282347e38f), qmaxin = R(0);
  R cqmin = R(0), cqmax = R(0), cin = R(0), cout = R(0);
  for (int e = 0; e < np; e++) {
    R vn, qs;
    int ipx;
    ma_edge(g, i, k, e, np, u_edg, v_edg, dp_edg, delp, vn, qs, ipx);
    const R cn = rabs(vn) * dt * rar;
    if (vn > R(0)) {
      cout = cout + cn;
    } else {
      const R gx = delp[(size_t)ipx * L + k];
      const R qmn = rmin(qs, gx), qmx = rmax(qs, gx);
      cin = cin + cn;
      qminin = rmin(qminin, qmn);
      qmaxin = rmax(qmaxin, qmx);
      cqmin = cqmin + cn * qmn;
      cqmax = cqmax + cn * qmx;
    }
  }
  const R qmin_next = rmin(gv, qminin), qmax_next = rmax(gv, qmaxin);
  if (cout != R(0)) {
    const R to = dp_tndcy[(size_t)of * N * L + c], tv = dp_tndcy[(size_t)vof * N * L + c];
    qmin_out[c] = (gv + ab1 / dt * cqmax - qmax_next * (R(1) + cin - cout) + ab2 * to + ab3 * tv) / cout / ab1 * dt;
    qmax_out[c] = (gv + ab1 / dt * cqmin - qmin_next * (R(1) + cin - cout) + ab2 * to + ab3 * tv) / cout / ab1 * dt;
  } else {
    qmin_out[c] = R(-100000.0);
    qmax_out[c] = R(100000.0);
  }
}

template <typename R>
__global__ void __launch_bounds__(kBlock) k_massadv_flux(Grid<R> g, Strides s, const StepParams* __restrict__ sp,
    const R* __restrict__ u_edg, const R* __restrict__ v_edg, R* __restrict__ dp_edg, const R* __restrict__ delp,
    const R* __restrict__ qmin_out, const R* __restrict__ qmax_out, R* __restrict__ massfx, R* __restrict__ dp_tndcy) {
  int i, k;
  if (!cell_level(g.N, g.L, i, k)) return;
  const int L = g.L, N = g.N;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active) return;
  u_edg += m * s.edge; v_edg += m * s.edge; dp_edg += m * s.edge; delp += m * s.cell; dp_tndcy += m * s.ab;
  qmin_out += m * s.cell; qmax_out += m * s.cell; massfx += m * s.mf;
  const int nf = sp->nf;
  R* mfn = massfx + (size_t)nf * N * 6 * L;
  const int np = g.nprox[i];
  R vnv[6], dpe[6];
#pragma unroll
  for (int e = 0; e < 6; e++) {
    if (e < np) {
      R vn, qs;
      int ipx;
      ma_edge(g, i, k, e, np, u_edg, v_edg, dp_edg, delp, vn, qs, ipx);
      const size_t cs = (size_t)(vn > R(0) ? i : ipx) * L + k;
      vnv[e] = vn;
      dpe[e] = rmax(qmin_out[cs], rmin(qmax_out[cs], qs));
    }
  }
  R t = R(0);
#pragma unroll
  for (int e = 0; e < 6; e++) {
    if (e < np) {
      const size_t o = ((size_t)i * 6 + e) * L + k;
      dp_edg[o] = dpe[e];
      const R mf = vnv[e] * dpe[e];
      mfn[o] = mf;
      t = t + mf;
    }
  }
  dp_tndcy[(size_t)nf * N * L + (size_t)i * L + k] = -t * g.rarea[i];
}

template <typename R>
void launch_massadv(const Launch& l, const Grid<R>& g, const Strides& s, const CnuityScratch<R>& w, const R* u,
                    const R* v, const R* u_edg, const R* v_edg, R* dp_edg, const R* lp_edg, R* delp, R* pres,
                    R* exner, R* dp_tndcy, R* massfx, R* omega) {
  dim3 grid(blocks_for((long long)g.N * g.L), l.members);
  FIM_KBEGIN(l, "k_massadv_lim");
  k_massadv_lim<R><<<grid, kBlock, 0, l.stream>>>(g, s, l.sp, u_edg, v_edg, dp_edg, delp, dp_tndcy, w.r_plus,
                                                   w.r_mnus);
  FIM_KEND(l);
  FIM_KBEGIN(l, "k_massadv_flux");
  k_massadv_flux<R><<<grid, kBlock, 0, l.stream>>>(g, s, l.sp, u_edg, v_edg, dp_edg, delp, w.r_plus, w.r_mnus,
                                                    massfx, dp_tndcy);
  FIM_KEND(l);
  launch_cnuity5<R>(l, g, s, pres, delp, exner, dp_tndcy, omega, lp_edg, u, v, 1);
}

// --------------------------------------------------------------------------
// del4prep (momtum_compute.F90:16-95) on u+grndspd, v; writes prepared fields.
template <typename R>
__global__ void __launch_bounds__(kBlock) k_del4prep(Grid<R> g, Strides s, const R* __restrict__ u,
    const R* __restrict__ v, R* __restrict__ wu, R* __restrict__ wv) {
  int i, k;
  if (!cell_level(g.N, g.L, i, k)) return;
  const int L = g.L;
  const size_t m = blockIdx.y;
  u += m * s.cell; v += m * s.cell; wu += m * s.cell; wv += m * s.cell;
  const int np = g.nprox[i];
  R au = R(0), av = R(0);
  for (int e = 0; e < np; e++) {
    const int ipx = g.prox[i * 6 + e];
    const R* cs = g.cs + (i * 6 + e) * 4;
    const R* sn = g.sn + (i * 6 + e) * 4;
    const R ux = u[(size_t)ipx * L + k] + g.grndspd[ipx], vx = v[(size_t)ipx * L + k];
    const R uxy2 = cs[1] * ux + sn[1] * vx;
    const R vxy2 = -sn[1] * ux + cs[1] * vx;
    au = au + cs[0] * uxy2 - sn[0] * vxy2;
    av = av + sn[0] * uxy2 + cs[0] * vxy2;
  }
  const R factor = g.biharw[k] / R(np);
  const size_t c = (size_t)i * L + k;
  wu[c] = (u[c] + g.grndspd[i]) - au * factor;
  wv[c] = v[c] - av * factor;
}

// dissip (momtum_compute.F90:149-208): thickness-weighted harmonic momentum
// fluxes across the edges, rotated back; increments du, dv. The work fields are
// u+grndspd, v (momtum.F90:99-106) or the del4prep output when wu != nullptr.
template <typename R, int VK>
__global__ void __launch_bounds__(kBlock) k_dissip(Grid<R> g, Strides s, const R* __restrict__ u,
    const R* __restrict__ v, const R* __restrict__ wu, const R* __restrict__ wv, const R* __restrict__ delp,
    R* __restrict__ du, R* __restrict__ dv) {
  int i, k;
  if (!cell_levels<VK>(g.N, g.L, i, k)) return;
  const int L = g.L;
  const size_t m = blockIdx.y;
  u += m * s.cell; v += m * s.cell; delp += m * s.cell; du += m * s.cell; dv += m * s.cell;
  const bool prep = wu != nullptr;
  if (prep) { wu += m * s.cell; wv += m * s.cell; }
  const R thshld = R(1.e-11), two = R(2);
  const size_t c = (size_t)i * L + k;
  R ui[VK], vi[VK], dpi[VK], factor[VK], dfl[VK], dfl2[VK], su[VK], sv[VK];
  if (prep) {
    ldv<VK>(wu + c, ui);
    ldv<VK>(wv + c, vi);
  } else {
    ldv<VK>(u + c, ui);
    ldv<VK>(v + c, vi);
    const R gs = g.grndspd[i];
    FOR_V ui[j] = ui[j] + gs;
  }
  ldv<VK>(delp + c, dpi);
  const R rar = g.rarea[i];
  FOR_V {
    dpi[j] = rmax(dpi[j], thshld);
    factor[j] = fdiv(rar, dpi[j]);
    dfl[j] = g.dfflen[k + j];
    dfl2[j] = two * dfl[j];
    su[j] = R(0);
    sv[j] = R(0);
  }
  const int np = g.nprox[i];
  // all six prox slots hold valid cells (a pentagon's slot 5 repeats a
  // neighbour), so the gathers carry no branch; slot 5 of a pentagon is
  // dropped by the selects
#pragma unroll
  for (int e = 0; e < 6; e++) {
    const bool live = e < np;
    const int ipx = g.prox[i * 6 + e];
    const R* cs = g.cs + (i * 6 + e) * 4;
    const R* sn = g.sn + (i * 6 + e) * 4;
    const size_t cx = (size_t)ipx * L + k;
    R ux[VK], vx[VK], bx[VK];
    if (prep) {
      ldv<VK>(wu + cx, ux);
      ldv<VK>(wv + cx, vx);
    } else {
      ldv<VK>(u + cx, ux);
      ldv<VK>(v + cx, vx);
      const R gx = g.grndspd[ipx];
      FOR_V ux[j] = ux[j] + gx;
    }
    ldv<VK>(delp + cx, bx);
    const R sl = g.sideln[i * 6 + e];
    if constexpr (sizeof(R) == 8) {
      // the same with the factors gathered and the jumps formed in one chain
      if (live) FOR_V {
        const R b = floor_at(bx[j], thshld);
        const R w = (dfl2[j] * sl) * f64_quot(dpi[j] * b, dpi[j] + b, f64_recip(dpi[j] + b)) * factor[j];
        const R ju = cs[1] * ux[j] + sn[1] * vx[j] - cs[0] * ui[j] - sn[0] * vi[j];
        const R jv = cs[1] * vx[j] - sn[1] * ux[j] - cs[0] * vi[j] + sn[0] * ui[j];
        su[j] = su[j] + (cs[0] * ju - sn[0] * jv) * w;
        sv[j] = sv[j] + (sn[0] * ju + cs[0] * jv) * w;
      }
      continue;
    }
    FOR_V {
      const R uxy1 = cs[0] * ui[j] + sn[0] * vi[j], vxy1 = -sn[0] * ui[j] + cs[0] * vi[j];
      const R uxy2 = cs[1] * ux[j] + sn[1] * vx[j], vxy2 = -sn[1] * ux[j] + cs[1] * vx[j];
      const R b = rmax(bx[j], thshld);
      const R hf = fdiv(dpi[j] * b, dpi[j] + b);
      const R ufx = (uxy2 - uxy1) * dfl[j] * sl * two * hf;
      const R vfx = (vxy2 - vxy1) * dfl[j] * sl * two * hf;
      const R uflux = cs[0] * ufx - sn[0] * vfx;
      const R vflux = sn[0] * ufx + cs[0] * vfx;
      su[j] = live ? su[j] + uflux * factor[j] : su[j];
      sv[j] = live ? sv[j] + vflux * factor[j] : sv[j];
    }
  }
  stv<VK>(du + c, su);
  stv<VK>(dv + c, sv);
}

// momtum1 (momtum_compute.F90:278-423, janjic=0) after adding the dissipation
// increments (momtum.F90:130-139); one warp per column so the Rayleigh damping
// of the top layers can read the updated top three levels.  A lane takes VK
// consecutive levels (one chunk of 32 VK levels covers nvl 64 with two), so the
// cell's tables and row addresses are formed once for both.  SPLIT: the
// FP32-mixed step's form (mpf, tr0).  Bound by HBM: at glvl 8 / nvl 64 the step's
// form takes 1.11 ms, 6,630 GB/s of its 44 words (one level a lane 1.57 ms; two
// blocks an SM 1.32, four 1.34); the plain form at glvl 7 0.30 ms at four blocks
// an SM (three 0.34; one level a lane 0.43).  FP64, one level a lane, is bound
// by its operations: glvl 6 0.44 -> 0.32 ms with M + K - exm th formed once.
template <typename R, int NC, int VK, bool SPLIT>
__global__ void __launch_bounds__(kBlock, SPLIT ? 3 : 4) k_momtum1(Grid<R> g, Strides s, R rlthresh, R rleigh,
    R rltaper, const StepParams* __restrict__ sp,
    R* __restrict__ u, R* __restrict__ v, const R* __restrict__ du, const R* __restrict__ dv,
    const R* __restrict__ exner, R* __restrict__ relvor, const R* __restrict__ u_edg, const R* __restrict__ v_edg,
    const R* __restrict__ trc_edg, const R* __restrict__ mont_edg, const R* __restrict__ uvsq_edg,
    R* __restrict__ u_tndcy, R* __restrict__ v_tndcy, const float2* __restrict__ mpf, const R* __restrict__ tr0) {
  __shared__ R top[kBlock / 32][3][2];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int N = g.N, L = g.L, L1 = L + 1;
  if (warp >= N) return;
  const int i = warp;
  const size_t m = blockIdx.y;
  sp += m;
  if (!sp->active) return;
  u += m * s.cell; v += m * s.cell; exner += m * s.intf; relvor += m * s.cell;
  u_edg += m * s.edge; v_edg += m * s.edge; trc_edg += m * s.tredg; mont_edg += m * s.edge;
  uvsq_edg += m * s.edge; u_tndcy += m * s.ab; v_tndcy += m * s.ab;
  const bool have_d = du != nullptr;
  if (have_d) { du += m * s.cell; dv += m * s.cell; }
  if constexpr (SPLIT) { mpf += m * s.cell; tr0 += m * s.cell; }
  const int nf = sp->nf, of = sp->of, vof = sp->vof;
  const R ab1 = sp->template w1<R>(), ab2 = sp->template w2<R>(), ab3 = sp->template w3<R>();
  const size_t NL = (size_t)N * L;
  const int np = g.nprox[i];
  const int* pr = g.prox + i * 6;
  const R rar = g.rarea[i], cor = g.corio[i];
  // Loads use clamped levels and the six edge slots of every cell (a
  // pentagon's slot 5 and its prox entry are valid memory), so they carry no
  // branch and can be issued together; results and stores are masked.
  R un[NC][VK], vn[NC][VK];
#pragma unroll
  for (int ch = 0; ch < NC; ch++) {
    const int k = (ch * 32 + lane) * VK;
    const int kk = k < L ? k : L - VK;
    const size_t c = (size_t)i * L + kk;
    R uu[VK], vv[VK], exm[VK];
    ldv<VK>(u + c, uu);
    ldv<VK>(v + c, vv);
    if (have_d) {
      R a[VK], b[VK];
      ldv<VK>(du + c, a);
      ldv<VK>(dv + c, b);
      FOR_V { uu[j] = uu[j] + a[j]; vv[j] = vv[j] + b[j]; }
    }
    {
      const R* e = exner + (size_t)i * L1 + kk;
      R lo = e[0];
      FOR_V {
        const R hi = e[j + 1];
        exm[j] = R(0.5) * (lo + hi);
        lo = hi;
      }
    }
    R pgfx[VK], pgfy[VK], rv[VK];
    FOR_V { pgfx[j] = R(0); pgfy[j] = R(0); rv[j] = R(0); }
    if constexpr (!SPLIT) {
#pragma unroll
      for (int e = 0; e < 6; e++) {
        const bool live = e < np;
        const R* svc = g.svc + (i * 6 + e) * 2;
        const R* sve = g.sve + (i * 6 + e) * 2;
        const size_t o = ((size_t)i * 6 + e) * L + kk;
        R mo[VK], kv[VK], th[VK], ue[VK], ve[VK];
        ldv<VK>(mont_edg + o, mo);
        ldv<VK>(uvsq_edg + o, kv);
        ldv<VK>(trc_edg + o, th);
        ldv<VK>(u_edg + o, ue);
        ldv<VK>(v_edg + o, ve);
        if (live) {
          FOR_V {
            if constexpr (sizeof(R) == 8) {  // the fewest operations: (M + K - exm th) s
              const R w = (mo[j] + kv[j]) - exm[j] * th[j];
              pgfx[j] = pgfx[j] - w * svc[1];
              pgfy[j] = pgfy[j] + w * svc[0];
            } else {
              const R mu = mo[j] + kv[j];
              pgfx[j] = pgfx[j] - mu * svc[1] + exm[j] * th[j] * svc[1];
              pgfy[j] = pgfy[j] + mu * svc[0] - exm[j] * th[j] * svc[0];
            }
            rv[j] = rv[j] + (sve[0] * ue[j] + sve[1] * ve[j]);
          }
        }
      }
    } else {
      // FP32-mixed: the same line integrals with the cell values split off,
      // sum_e (M_e + K_e - exm th_e) s_e
      //   = sum_e (dM_e + K_e - exm dth_e) s_e + (M_c - exm th_c) sum_e s_e,
      // dM_e, dth_e the edge-minus-cell values (edgvar1's weights applied to
      // neighbour differences); the large cell term is formed in FP64.
      R thc[VK], dth[6][VK];
      ldv<VK>(tr0 + c, thc);
#pragma unroll
      for (int q = 0; q < 6; q++) {
        ldv<VK>(tr0 + (size_t)pr[q] * L + kk, dth[q]);
        FOR_V dth[q][j] = (q < np) ? dth[q][j] - thc[j] : R(0);
      }
      const R divby6 = R(1) / R(6);
#pragma unroll
      for (int e = 0; e < 6; e++) {
        const bool live = e < np;
        const R* svc = g.svc + (i * 6 + e) * 2;
        const R* sve = g.sve + (i * 6 + e) * 2;
        const size_t o = ((size_t)i * 6 + e) * L + kk;
        const int et = e == 0 ? np - 1 : e - 1, el = e == np - 1 ? 0 : e + 1;
        R mo[VK], kv[VK], ue[VK], ve[VK];
        ldv<VK>(mont_edg + o, mo);
        ldv<VK>(uvsq_edg + o, kv);
        ldv<VK>(u_edg + o, ue);
        ldv<VK>(v_edg + o, ve);
        FOR_V {
          R dte = R(0);
#pragma unroll
          for (int q = 0; q < 6; q++) {
            if (q == e) dte = dte + R(2) * dth[q][j];
            if (q == et || q == el) dte = dte + dth[q][j];
          }
          dte = dte * divby6;
          if (live) {
            const R w = mo[j] + kv[j] - exm[j] * dte;
            pgfx[j] = pgfx[j] - w * svc[1];
            pgfy[j] = pgfy[j] + w * svc[0];
            rv[j] = rv[j] + (sve[0] * ue[j] + sve[1] * ve[j]);
          }
        }
      }
      // Montgomery potential minus exner x theta, cancellation-free
      FOR_V {
        const float2 mp = mpf[c + j];
        const FF2 cf = ff_add(FF2{mp.x, mp.y}, ff_neg(two_prod(float(exm[j]), float(thc[j]))));
        const R cell = R(cf.hi + cf.lo);
        pgfx[j] = pgfx[j] - cell * g.svsum[i * 2 + 1];
        pgfy[j] = pgfy[j] + cell * g.svsum[i * 2 + 0];
      }
    }
    R ut[VK], vt[VK], uo[VK], uv[VK], vo[VK], vw[VK];
    ldv<VK>(u_tndcy + (size_t)of * NL + c, uo);
    ldv<VK>(u_tndcy + (size_t)vof * NL + c, uv);
    ldv<VK>(v_tndcy + (size_t)of * NL + c, vo);
    ldv<VK>(v_tndcy + (size_t)vof * NL + c, vw);
    FOR_V {
      pgfx[j] = pgfx[j] * rar;
      pgfy[j] = pgfy[j] * rar;
      rv[j] = rv[j] * rar;
      const R uzeta = (cor + rv[j]) * uu[j], vzeta = (cor + rv[j]) * vv[j];
      ut[j] = pgfx[j] + vzeta;
      vt[j] = pgfy[j] - uzeta;
      uu[j] = uu[j] + ab1 * ut[j] + ab2 * uo[j] + ab3 * uv[j];
      vv[j] = vv[j] + ab1 * vt[j] + ab2 * vo[j] + ab3 * vw[j];
      un[ch][j] = uu[j];
      vn[ch][j] = vv[j];
    }
    if (k < L) {
      stv<VK>(relvor + c, rv);
      stv<VK>(u_tndcy + (size_t)nf * NL + c, ut);
      stv<VK>(v_tndcy + (size_t)nf * NL + c, vt);
      FOR_V
        if (k + j >= L - 3) { top[wib][L - 1 - k - j][0] = uu[j]; top[wib][L - 1 - k - j][1] = vv[j]; }
    }
  }
  __syncwarp();
  const R q1 = top[wib][0][0] * top[wib][0][0] + top[wib][0][1] * top[wib][0][1];
  const R q2 = top[wib][1][0] * top[wib][1][0] + top[wib][1][1] * top[wib][1][1];
  const R q3 = top[wib][2][0] * top[wib][2][0] + top[wib][2][1] * top[wib][2][1];
  R qq = rmax(rmax(q1, q2), q3) / (rlthresh * rlthresh);
  const int ndamp = L / 4;
  const bool damp = qq > R(1);
  if (damp) {
    qq = sqrt((qq - R(1)) * qq);
    const R dtf = sp->template step<R>() / R(86400.);
#pragma unroll
    for (int ch = 0; ch < NC; ch++) {
      FOR_V {
        const int k = (ch * 32 + lane) * VK + j;
        if (k >= L - 1 - ndamp) {
          const R factor = R(1) - dtf * rleigh * qq * pow(R(2), rltaper * R(k + 1 - L));
          un[ch][j] = un[ch][j] * factor;
          vn[ch][j] = vn[ch][j] * factor;
        }
      }
    }
  }
#pragma unroll
  for (int ch = 0; ch < NC; ch++) {
    const int k = (ch * 32 + lane) * VK;
    if (k < L) {
      stv<VK>(u + (size_t)i * L + k, un[ch]);
      stv<VK>(v + (size_t)i * L + k, vn[ch]);
    }
  }
}

// abstart (abstart.F90:33-65) advanced on the device so a captured step graph
// can be replayed: its += 1, rotate the AB3 slots, set the weights.
__global__ void k_step_begin(StepParams* sp, int members) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= members || !sp[m].active) return;
  sp += m;
  StepParams p = *sp;
  p.its += 1;
  p.nf = (p.nf + 1) % 3;
  p.of = (p.of + 1) % 3;
  p.vof = (p.vof + 1) % 3;
  if (p.its == 1) { p.ab1 = p.dt; p.ab2 = 0.; p.ab3 = 0.; }
  if (p.its == 2) { p.ab1 = p.dt * 1.5; p.ab2 = -p.dt * .5; p.ab3 = 0.; }
  if (p.its == 3) { p.ab1 = p.dt * 23. / 12.; p.ab2 = -p.dt * 16. / 12.; p.ab3 = p.dt * 5. / 12.; }
  p.narrow();
  *sp = p;
}

// ---------------------------- launchers -----------------------------------

template <typename R>
void launch_edgvar1(const Launch& l, const Grid<R>& g, const Strides& s, int hi_order, const R* u,
                    const R* v, const R* delp, const R* pres, const R* montg, const R* tracr,
                    R* u_edg, R* v_edg, R* dp_edg, R* lp_edg, R* mont_edg, R* uvsq_edg, R* trc_edg,
                    const float2* mpf, R* thold) {
  // FP32: 8-byte accesses; at 4 levels a thread the neighbours' values take
  // twice the registers and half the occupancy (glvl 8: 1.47 against 1.41 ms),
  // at one level a thread half the bytes a load (1.87 ms)
  const int vk = pick_vk<R>(g.L, {u, v, delp, montg, tracr, u_edg, v_edg, dp_edg, lp_edg, mont_edg, uvsq_edg,
                                  trc_edg, thold}, sizeof(R) == 8 ? 1 : 2);
  FIM_KBEGIN(l, "k_edgvar1");
  FIM_VK_DISPATCH(R, vk, (k_edgvar1<R, VK><<<dim3(blocks_for((long long)g.N * (g.L / VK)), l.members), kBlock, 0,
                                             l.stream>>>(g, s, hi_order, u, v, delp, pres, montg, tracr, u_edg,
                                                         v_edg, dp_edg, lp_edg, mont_edg, uvsq_edg, trc_edg, mpf,
                                                         thold)));
  FIM_KEND(l);
}

template <typename R>
void launch_edgvar3(const Launch& l, const Grid<R>& g, const Strides& s, const R* delp, const R* tracr,
                    R* dp_edg, R* trc_edg, int nfields, const FrameTab& ft, bool average) {
  if constexpr (sizeof(R) == 4) {
    if (average) return launch_edges_patch(l, g, s, ft, nfields, delp, tracr, dp_edg, trc_edg);
  }
  const int vk = pick_vk<R>(g.L, {delp, tracr, dp_edg, trc_edg});
  FIM_KBEGIN(l, "k_edgvar3_own");
  FIM_VK_DISPATCH(R, vk, (k_edgvar3_own<R, VK><<<dim3(blocks_for((long long)g.N * (g.L / VK)), l.members, nfields),
                                                 kBlock, 0, l.stream>>>(g, s, delp, tracr, dp_edg, trc_edg)));
  FIM_KEND(l);
  if constexpr (sizeof(R) == 8) {
    if (!average) return;
    FIM_KBEGIN(l, "k_edgvar3_avg");
    FIM_VK_DISPATCH(R, vk, (k_edgvar3_avg<R, VK><<<dim3(blocks_for((long long)g.N * (g.L / VK)), l.members, nfields),
                                                   kBlock, 0, l.stream>>>(g, s, dp_edg, trc_edg)));
    FIM_KEND(l);
  }
}

template <typename R>
void launch_cnuity(const Launch& l, const Grid<R>& g, const Strides& s, const CnuityScratch<R>& w, const R* u,
                   const R* v, const R* u_edg, const R* v_edg, const R* dp_edg, const R* lp_edg,
                   R* delp, R* pres, R* exner, R* dp_tndcy, R* dplo_tndcy, R* massfx, R* omega, bool columns) {
  const int vk = pick_vk<R>(g.L, {u_edg, v_edg, dp_edg, delp, massfx, dplo_tndcy, dp_tndcy, w.antifx, w.delp_lo,
                                  w.p_plus, w.p_mnus, w.r_plus, w.r_mnus});
  if (l.coop) {
    // one cooperative launch of as many blocks as the GPU holds at once
    FIM_KBEGIN(l, "k_cnuity_coop");
    cudaMemsetAsync(l.coop->barrier, 0, sizeof(unsigned), l.stream);
    FIM_VK_DISPATCH(R, vk, ({
      int dev = 0, sms = 0, per = 0;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cnuity_coop<R, VK>, kBlock, 0);
      const long long need = (long long)blocks_for((long long)g.N * (g.L / VK)) * l.members;
      const unsigned nb = (unsigned)(need < (long long)sms * per ? need : (long long)sms * per);
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(nb > 0 ? nb : 1);
      cfg.blockDim = dim3(kBlock);
      cfg.stream = l.stream;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeCooperative;
      attr[0].val.cooperative = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      cudaLaunchKernelEx(&cfg, k_cnuity_coop<R, VK>, g, s, l.sp, l.members, u_edg, v_edg, dp_edg, delp, massfx,
                         dplo_tndcy, dp_tndcy, w.antifx, w.delp_lo, w.p_plus, w.p_mnus, w.r_plus, w.r_mnus,
                         l.flags, l.coop->barrier, l.coop->extra, l.coop->limit_ns);
    }));
    FIM_KEND(l);
  } else {
  FIM_KBEGIN(l, "k_cnuity12");
  FIM_VK_DISPATCH(R, vk, (k_cnuity12<R, VK><<<dim3(blocks_for((long long)g.N * (g.L / VK)), l.members), kBlock, 0,
                                              l.stream>>>(g, s, l.sp, u_edg, v_edg, dp_edg, delp, massfx,
                                                          dplo_tndcy, w.antifx, w.delp_lo, w.p_plus, w.p_mnus)));
  FIM_KEND(l);
  FIM_KBEGIN(l, "k_cnuity3");
  FIM_VK_DISPATCH(R, vk, (k_cnuity3<R, VK><<<dim3(blocks_for((long long)g.N * (g.L / VK)), l.members), kBlock, 0,
                                             l.stream>>>(g, s, l.sp, w.delp_lo, delp, dp_tndcy, w.p_plus, w.p_mnus,
                                                         w.r_plus, w.r_mnus)));
  FIM_KEND(l);
  FIM_KBEGIN(l, "k_cnuity4");
  FIM_VK_DISPATCH(R, vk, (k_cnuity4<R, VK><<<dim3(blocks_for((long long)g.N * (g.L / VK)), l.members), kBlock, 0,
                                             l.stream>>>(g, s, l.sp, w.antifx, w.r_plus, w.r_mnus, massfx,
                                                         dplo_tndcy, dp_tndcy, delp, l.flags)));
  FIM_KEND(l);
  }
  if (columns) launch_cnuity5<R>(l, g, s, pres, delp, exner, dp_tndcy, omega, lp_edg, u, v, 0);
}

template <typename R>
void launch_momtum(const Launch& l, const Grid<R>& g, const Strides& s, const Knobs& kn, const MomtumScratch<R>& w,
                   R* u, R* v, const R* exner, R* relvor, const R* u_edg, const R* v_edg,
                   const R* trc_edg, const R* mont_edg, const R* uvsq_edg, R* u_tndcy, R* v_tndcy,
                   const R* dp3d, const float2* mpf, const R* tr0) {
  dim3 grid(blocks_for((long long)g.N * g.L), l.members);
  const R* du = nullptr;
  const R* dv = nullptr;
  if (kn.dfflen_max > 0.) {
    const R* wu = nullptr;
    const R* wv = nullptr;
    if (kn.biharm) {
      FIM_KBEGIN(l, "k_del4prep");
      k_del4prep<R><<<grid, kBlock, 0, l.stream>>>(g, s, u, v, w.wu, w.wv);
      FIM_KEND(l);
      wu = w.wu;
      wv = w.wv;
    }
    const int vk = pick_vk<R>(g.L, {u, v, wu, wv, dp3d, w.du, w.dv});
    FIM_KBEGIN(l, "k_dissip");
    FIM_VK_DISPATCH(R, vk, (k_dissip<R, VK><<<dim3(blocks_for((long long)g.N * (g.L / VK)), l.members), kBlock, 0,
                                              l.stream>>>(g, s, u, v, wu, wv, dp3d, w.du, w.dv)));
    FIM_KEND(l);
    du = w.du;
    dv = w.dv;
  }
  dim3 gw(blocks_for((long long)g.N * 32), l.members);
  FIM_KBEGIN(l, "k_momtum1");
  const int vm = pick_vk<R>(g.L, {u, v, du, dv, relvor, u_edg, v_edg, trc_edg, mont_edg, uvsq_edg, u_tndcy, v_tndcy,
                                  tr0}, sizeof(R) == 8 ? 1 : 2);
  const int nc = (g.L + 32 * vm - 1) / (32 * vm);
#define FIM_MOMTUM1S(NC, VK, SPLIT)                                                                            \
  k_momtum1<R, NC, VK, SPLIT><<<gw, kBlock, 0, l.stream>>>(g, s, R(kn.rlthresh), R(kn.rleigh), R(kn.rltaper), l.sp, u, \
                                                            v, du, dv, exner, relvor, u_edg, v_edg, trc_edg, mont_edg, \
                                                            uvsq_edg, u_tndcy, v_tndcy, mpf, tr0)
#define FIM_MOMTUM1(NC, VK)                                                                                    \
  do {                                                                                                         \
    if constexpr (sizeof(R) == 4) {                                                                            \
      if (mpf) FIM_MOMTUM1S(NC, VK, true);                                                                     \
      else FIM_MOMTUM1S(NC, VK, false);                                                                        \
    } else {                                                                                                   \
      FIM_MOMTUM1S(NC, VK, false);                                                                             \
    }                                                                                                          \
  } while (0)
  if (vm == 2) {
    if constexpr (sizeof(R) == 4) {
      if (nc == 1) FIM_MOMTUM1(1, 2);
      else FIM_MOMTUM1(2, 2);
    }
  } else if (nc == 1) FIM_MOMTUM1(1, 1);
  else if (nc == 2) FIM_MOMTUM1(2, 1);
  else if (nc == 3) FIM_MOMTUM1(3, 1);
  else FIM_MOMTUM1(4, 1);
#undef FIM_MOMTUM1S
#undef FIM_MOMTUM1
  FIM_KEND(l);
}

void launch_step_begin(const Launch& l, StepParams* sp) {
  FIM_KBEGIN(l, "k_step_begin");
  k_step_begin<<<(l.members + 31) / 32, 32, 0, l.stream>>>(sp, l.members);
  FIM_KEND(l);
}

#define INSTANTIATE(R)                                                                                          \
  template void launch_edgvar1<R>(const Launch&, const Grid<R>&, const Strides&, int, const R*, const R*,      \
                                  const R*, const R*, const R*, const R*, R*, R*, R*, R*, R*, R*, R*,          \
                                  const float2*, R*);                                                         \
  template void launch_edgvar2<R>(const Launch&, const Grid<R>&, const Strides&, const R*, const R*, R*, R*,  \
                                  R*, R*);                                                                    \
  template void launch_edgvar3<R>(const Launch&, const Grid<R>&, const Strides&, const R*, const R*, R*, R*,  \
                                  int, const FrameTab&, bool);                                                                \
  template void launch_cnuity<R>(const Launch&, const Grid<R>&, const Strides&, const CnuityScratch<R>&,      \
                                 const R*, const R*, const R*, const R*, const R*, const R*, R*, R*, R*, R*,  \
                                 R*, R*, R*, bool);                                                                 \
  template void launch_cnuity5<R>(const Launch&, const Grid<R>&, const Strides&, R*, R*, R*, const R*, R*,    \
                                  const R*, const R*, const R*, int);                                         \
  template void launch_massadv<R>(const Launch&, const Grid<R>&, const Strides&, const CnuityScratch<R>&,     \
                                  const R*, const R*, const R*, const R*, R*, const R*, R*, R*, R*, R*, R*,   \
                                  R*);                                                                       \
  template void launch_momtum<R>(const Launch&, const Grid<R>&, const Strides&, const Knobs&,                 \
                                 const MomtumScratch<R>&, R*, R*, const R*, R*, const R*, const R*, const R*, \
                                 const R*, const R*, R*, R*, const R*, const float2*, const R*);
INSTANTIATE(float)
INSTANTIATE(double)

}  // namespace fim
