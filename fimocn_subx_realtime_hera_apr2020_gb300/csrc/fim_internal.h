// Internal declarations shared by the kernels and the C-ABI layer.
#pragma once

#include <cuda_runtime.h>

#include <chrono>
#include <cstddef>
#include <cstdint>
#include <initializer_list>
#include <map>
#include <string>
#include <vector>

namespace fim {

// Physical constants of FIMsrc/cntl/module_constants.F90:14-27.
constexpr double kPi = 3.14159265;
constexpr double kEarthRad = 6371220.;
constexpr double kOmegx2 = 1.4584e-4;
constexpr double kGrvity = 9.80665;
constexpr double kP1000 = 100000.;
constexpr double kCp = 1004.6855;
constexpr double kRd = 287.0586;
constexpr double kQvmin = 1.e-10;
constexpr double kQwmin = 1.e-10;

// Largest layer count the column kernels accept.
constexpr int kMaxL = 128;

// Step-dependent scalars that the reference keeps in module_variables
// (nf, of, vof, adbash1..3) plus the step number used by hybgen and hystat.
// They live in device memory so a captured step graph can be replayed.
// One block per ensemble member (indexed by the member, blockIdx.y in the
// kernels), so members of one batch can be at different steps.
struct StepParams {
  int its;
  int nf, of, vof;      // 0-based AB3 slots
  double ab1, ab2, ab3; // AB3 weights (s)
  double dt;
  int active;           // 0: the member's slot is idle, kernels skip it
  // tracers the member transports (fim_member_set_tracers): the tracer
  // transport, the remap and the budget sums leave slots ntr.. as they are
  int ntr = 0x7fffffff;
  // the weights and dt in FP32 (narrow(), wherever the doubles are set for the
  // device): a conversion a thread costs the FP32 kernels 16 clocks of the FP64
  // pipe a warp
  float f1 = 0.f, f2 = 0.f, f3 = 0.f, fdt = 0.f;
  __host__ __device__ void narrow() {
    f1 = (float)ab1;
    f2 = (float)ab2;
    f3 = (float)ab3;
    fdt = (float)dt;
  }
  template <typename R> __device__ __forceinline__ R w1() const { if constexpr (sizeof(R) == 4) return f1; else return ab1; }
  template <typename R> __device__ __forceinline__ R w2() const { if constexpr (sizeof(R) == 4) return f2; else return ab2; }
  template <typename R> __device__ __forceinline__ R w3() const { if constexpr (sizeof(R) == 4) return f3; else return ab3; }
  template <typename R> __device__ __forceinline__ R step() const { if constexpr (sizeof(R) == 4) return fdt; else return dt; }
};

// device status bits
enum : int {
  kFlagBadDp = 1,       // non-positive or NaN layer thickness after cnuity
  kFlagColumnIntegral = 2,  // hybgen column-integral conservation check failed
  kFlagNaN = 4,
  kFlagTimeout = 8,     // a grid barrier of a persistent launch gave up waiting
};

// Relative tolerance of hybgen's column-integral checks: the reference's own
// in FP64 (acurcy of restp_1d 1e-6, hybgen.F90:873; of remap_1d 2e-6, :694;
// of the real*8 pcwise 1e-11, :1262); in the FP32-mixed build one bound for
// the checks it runs, ~500 float epsilons, well above the rounding of a
// column sum of nvl <= 128 FP32 terms and well below a lost or doubled layer.
template <typename R>
__host__ __device__ constexpr R col_tol(double ref) {
  return R(sizeof(R) == 8 ? ref : 3.e-5);
}

// Grid tables on the device, metric tables in the compute type R.
template <typename R>
struct Grid {
  int N, L, T;
  const int* __restrict__ prox;   // [N*6] 0-based
  const int* __restrict__ proxs;  // [N*6] 0-based (pentagon slot 5 = -1)
  const int* __restrict__ nprox;  // [N]
  const R* __restrict__ cs;       // [N*6*4]
  const R* __restrict__ sn;
  // [N*6*4] sqrt(cs^2 + sn^2) x (2, 2, 1, 1) / 6, what edgvar1's magnitude
  // takes of the four cells' speeds (FP64 contexts; else null)
  const R* __restrict__ vw;
  const R* __restrict__ svc;      // sidevec_c [N*6*2]
  const R* __restrict__ sve;      // sidevec_e [N*6*2]
  const R* __restrict__ sideln;   // [N*6]
  const R* __restrict__ area;     // [N]
  const R* __restrict__ rarea;
  const R* __restrict__ corio;
  const R* __restrict__ grndspd;
  const R* __restrict__ hfcoef;   // [N*6*6]: hfcoef[(i*6+edge)*6+j]
  const R* __restrict__ cxy;      // [N*2*6]: corner_xy(6,2,nip), cxy[(i*2+xy)*6+corner]; null if not given
  const double* __restrict__ area_d;  // [N] double areas for budgets
  const R* __restrict__ svsum;        // [N*2] sum over edges of sidevec_c(1:2), summed in FP64
  // per-level tables
  const R* __restrict__ dfflen;   // [L]
  const R* __restrict__ biharw;   // [L]
  const R* __restrict__ smoo;     // [L+1]
  const R* __restrict__ thetac;   // [L]
  const R* __restrict__ dpsig;    // [L]
};

struct Knobs {
  int kbl, miglim, remap_optn, hi_order;
  double intfc_smooth, slak, ptop, thktop, rleigh, rlthresh, rltaper;
  double dfflen_max;
  int biharm;  // any biharw > 0
};

// Per-member element strides of the state arrays.
struct Strides {
  size_t cell;   // L*N
  size_t intf;   // (L+1)*N
  size_t edge;   // 6*L*N
  size_t ab;     // 3*L*N
  size_t tr;     // (T+TB)*L*N: tr3d and trdp
  size_t trab;   // 3*T*L*N
  size_t tredg;  // 6*T*L*N
  size_t mf;     // 3*6*L*N
  size_t col;    // N
};

// T class-A tracers (edges, tendencies); tr3d/trdp also hold TB class-B ones
inline Strides make_strides(int N, int L, int T, int TB = 0) {
  Strides s;
  s.cell = (size_t)L * N;
  s.intf = (size_t)(L + 1) * N;
  s.edge = (size_t)6 * L * N;
  s.ab = (size_t)3 * L * N;
  s.tr = (size_t)(T + TB) * L * N;
  s.trab = (size_t)3 * T * L * N;
  s.tredg = (size_t)6 * T * L * N;
  s.mf = (size_t)18 * L * N;
  s.col = (size_t)N;
  return s;
}

// Per-kernel timing with CUDA events on the launching stream (bench only).
struct Prof {
  bool on = false;
  struct Rec { const char* name; cudaEvent_t a, b; };
  std::vector<Rec> pending;
  std::vector<cudaEvent_t> pool;
  std::map<std::string, std::pair<long long, double>> agg;  // name -> (launches, ms)
  cudaEvent_t get() {
    if (!pool.empty()) { cudaEvent_t e = pool.back(); pool.pop_back(); return e; }
    cudaEvent_t e;
    cudaEventCreate(&e);
    return e;
  }
  void begin(const char* name, cudaStream_t s) {
    Rec r{name, get(), get()};
    cudaEventRecord(r.a, s);
    pending.push_back(r);
  }
  void end(cudaStream_t s) { cudaEventRecord(pending.back().b, s); }
  void collect() {
    for (auto& r : pending) {
      cudaEventSynchronize(r.b);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, r.a, r.b);
      auto& a = agg[r.name];
      a.first += 1;
      a.second += ms;
      pool.push_back(r.a);
      pool.push_back(r.b);
    }
    pending.clear();
  }
  // fim_step_io's timeline: host time stamps taken by callbacks queued on
  // the compute and copy streams, kept as offsets from the step's first
  // mark; each name accumulates (steps, ms) in agg as "io:<name>"
  struct Mark { std::string name; double ms = 0.0; };
  std::vector<Mark*> marks;
  static void CUDART_CB stamp(void* p) {
    static_cast<Mark*>(p)->ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
  }
  void mark(const std::string& name, cudaStream_t s) {
    Mark* m = new Mark{name};
    if (cudaLaunchHostFunc(s, stamp, m) != cudaSuccess) {
      cudaGetLastError();
      delete m;
      return;
    }
    marks.push_back(m);
  }
  // once the streams holding the marks are idle
  void collect_marks() {
    for (Mark* m : marks) {
      auto& a = agg["io:" + m->name];
      a.first += 1;
      a.second += m->ms - marks[0]->ms;
    }
    for (Mark* m : marks) delete m;
    marks.clear();
  }
  ~Prof() {
    for (auto& r : pending) { cudaEventDestroy(r.a); cudaEventDestroy(r.b); }
    for (auto e : pool) cudaEventDestroy(e);
    for (Mark* m : marks) delete m;
  }
};

// Launch context handed to every launcher.
struct CoopCfg;
struct Launch {
  cudaStream_t stream;
  int members;         // gridDim.y
  const StepParams* sp;  // device
  int* flags;          // device status word per member [members]
  long long* counter;  // host launch counter
  Prof* prof = nullptr;  // per-kernel event timing when enabled
  // 1 for the column adjustment that opens a step (dyn_run's hybgen/hystat
  // of step its-1): the column kernels then act for its-1 and skip a member
  // at its first step, where dyn_init's adjustment stands in
  int boundary = 0;
  // non-null: cnuity1..4 run as one cooperative persistent launch
  const CoopCfg* coop = nullptr;
};

// The persistent cnuity1..4 launch: its grid barrier's counter (device),
// arrivals added to each barrier's target (0; a test sets 1 so that the first
// barrier never completes) and the barrier's time limit.
struct CoopCfg {
  unsigned* barrier;
  unsigned extra;
  unsigned long long limit_ns;
};

#define FIM_KBEGIN(l, name) do { if ((l).prof && (l).prof->on) (l).prof->begin(name, (l).stream); } while (0)
#define FIM_KEND(l)                                                      \
  do {                                                                   \
    if ((l).prof && (l).prof->on) (l).prof->end((l).stream);             \
    if ((l).counter) ++*(l).counter;                                     \
  } while (0)


// ---- level vectors: VK consecutive levels per thread ----------------------
// Cell and edge fields are level-fastest, so VK consecutive levels of one
// column are one 4/8/16-byte access.  pick_vk chooses the widest VK (at most
// 16 bytes) that nvl and the alignment of every pointer admit.
template <typename R, int VK> struct VecOf;
template <typename R> struct VecOf<R, 1> { using T = R; };
template <> struct VecOf<float, 2> { using T = float2; };
template <> struct VecOf<float, 4> { using T = float4; };
template <> struct VecOf<double, 2> { using T = double2; };

template <int VK, typename R>
__device__ __forceinline__ void ldv(const R* p, R (&r)[VK]) {
  if constexpr (VK == 1) {
    r[0] = *p;
  } else if constexpr (VK == 2) {
    const typename VecOf<R, 2>::T t = *reinterpret_cast<const typename VecOf<R, 2>::T*>(p);
    r[0] = t.x; r[1] = t.y;
  } else {
    const float4 t = *reinterpret_cast<const float4*>(p);
    r[0] = t.x; r[1] = t.y; r[2] = t.z; r[3] = t.w;
  }
}

template <int VK, typename R>
__device__ __forceinline__ void stv(R* p, const R (&r)[VK]) {
  if constexpr (VK == 1) {
    *p = r[0];
  } else if constexpr (VK == 2) {
    typename VecOf<R, 2>::T t; t.x = r[0]; t.y = r[1];
    *reinterpret_cast<typename VecOf<R, 2>::T*>(p) = t;
  } else {
    float4 t; t.x = r[0]; t.y = r[1]; t.z = r[2]; t.w = r[3];
    *reinterpret_cast<float4*>(p) = t;
  }
}

#define FOR_V _Pragma("unroll") for (int j = 0; j < VK; j++)

// a / b for the clamped quotients of the FCT limiters: IEEE division in FP64;
// __fdividef in the FP32-mixed build (within 2 ulp while |b| < 2^126; the
// denominators are clamped to >= 1e-11 and are far below that bound).  The
// fused and the per-routine tracer kernels use it alike, so they stay
// bit-identical.
template <typename R>
__device__ __forceinline__ R fdiv(R a, R b) { return a / b; }
template <>
__device__ __forceinline__ float fdiv<float>(float a, float b) { return __fdividef(a, b); }

// (cell, first level) of thread threadIdx.x of (virtual) block bx over
// nip x (nvl/VK)
template <int VK>
__device__ __forceinline__ bool cell_levels_at(int N, int L, int bx, int& i, int& k) {
  const int LV = L / VK;
  const int gid = bx * blockDim.x + threadIdx.x;
  if (gid >= N * LV) return false;
  i = gid / LV;
  k = (gid - i * LV) * VK;
  return true;
}

// (cell, first level) of thread gid over nip x (nvl/VK)
template <int VK>
__device__ __forceinline__ bool cell_levels(int N, int L, int& i, int& k) {
  const int LV = L / VK;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= N * LV) return false;
  i = gid / LV;
  k = (gid - i * LV) * VK;
  return true;
}

template <typename R>
inline int pick_vk(int L, std::initializer_list<const void*> ptrs, int want = 0) {
  int vk = want > 0 ? want : (int)(16 / sizeof(R));
  if ((int)sizeof(R) * vk > 16) vk = (int)(16 / sizeof(R));
  while (vk > 1 && L % vk != 0) vk /= 2;
  for (const void* p : ptrs)
    while (vk > 1 && p && ((uintptr_t)p % (vk * sizeof(R))) != 0) vk /= 2;
  return vk;
}

// streaming multiprocessors of the current device
inline int sm_count() {
  int dev = 0, sms = 152;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// run CALL with the compile-time constant VK equal to vk (4 only for float)
#define FIM_VK_DISPATCH(R, vk, CALL)                          \
  do {                                                        \
    if ((vk) >= 4 && sizeof(R) == 4) {                        \
      constexpr int VK = sizeof(R) == 4 ? 4 : 2;              \
      CALL;                                                   \
    } else if ((vk) >= 2) {                                   \
      constexpr int VK = 2;                                   \
      CALL;                                                   \
    } else {                                                  \
      constexpr int VK = 1;                                   \
      CALL;                                                   \
    }                                                         \
  } while (0)

// ---- FP64 with few FP64 operations ------------------------------------------
// GB300 issues 2 FP64 lanes a clock and SM (against 128 FP32 and 64 integer
// ones), so the FP64 build is bound by its FP64 operations.  Comparisons run
// on the integer pipe (a double's bits, the magnitude of negative values
// complemented, order as int64), reciprocals and powers by few steps from the
// hardware's approximations (good to 2^-19).  Error bounds are relative and in
// units of 2^-53, half a last place at most; tests/test_f64_arithmetic_gpu.py
// holds each against 113-bit arithmetic.
__device__ __forceinline__ long long f64_key(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
// by the upper word: a NaN (quiet, as all arithmetic makes them); an infinity
// or a NaN; negative and no NaN
__device__ __forceinline__ bool f64_nan(double x) { return (__double2hiint(x) & 0x7fffffff) > 0x7ff00000; }
__device__ __forceinline__ bool f64_odd(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }
__device__ __forceinline__ bool f64_below0(double x) {
  return ((unsigned)__double2hiint(x) ^ 0x80000000u) <= 0x7ff00000u;
}
// a < b, false where either is a NaN (zeros are ordered by their signs)
__device__ __forceinline__ bool f64_lt(double a, double b) {
  const long long x = f64_key(a), y = f64_key(b);
  return x < y && (int)(y >> 32) <= 0x7ff00000 && (int)(x >> 32) >= (int)0x800fffff;
}
// 1 / b, 2^-1000 < |b| < 2^1000: the approximation r and its residual e = 1 - b r
// in the geometric series of 1 / (1 - e) to e^2 (the hyperpower iteration of
// order three); the last rounding and e^3, 1.1 units
__device__ __forceinline__ double f64_recip(double b) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
  const double e = fma(-b, r, 1.);
  return fma(r, fma(e, e, e), r);
}
// a / b with rb = 1 / b: the product and one residual correction (Markstein),
// the division's result but for quotients next to half-way between two doubles
__device__ __forceinline__ double f64_quot(double a, double b, double rb) {
  const double q = a * rb;
  return fma(fma(-b, q, a), rb, q);
}
// 1 / b and a / b of any operands: where b is zero or infinite, or a is, the
// steps make NaNs of the approximation or the product, which are the result
// then (selected on the integer pipe; a division as written in a branch cost
// k_dissip 28% and k_regrid 45%).  FP32: as written.
__device__ __forceinline__ double recip(double b) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
  const double e = fma(-b, r, 1.), s = fma(r, fma(e, e, e), r);
  return f64_odd(e) ? r : s;
}
__device__ __forceinline__ double divide_by(double a, double b, double rb) {
  const double q = a * rb, e = fma(-b, q, a), s = fma(e, rb, q);
  return f64_odd(e) ? q : s;
}
__device__ __forceinline__ float divide_by(float a, float b, float) { return a / b; }
__device__ __forceinline__ double divide(double a, double b) { return divide_by(a, b, recip(b)); }
__device__ __forceinline__ float divide(float a, float b) { return a / b; }
// x / 10, rounded as the division (Markstein's correction from the rounded
// reciprocal)
__device__ __forceinline__ float tenth(float x) {
  const float q = x * .1f;
  return fmaf(fmaf(-10.f, q, x), .1f, q);
}
__device__ __forceinline__ double tenth(double x) { return divide_by(x, 10., .1); }
// the limiters' quotient: FP32 by the reciprocal
__device__ __forceinline__ float quot(float a, float, float rb) { return a * rb; }
__device__ __forceinline__ double quot(double a, double b, double rb) { return divide_by(a, b, rb); }
// 1 / sqrt(x), x normal: the approximation r and e = 1 - x r^2 in the binomial
// series of (1 - e)^(-1/2) to e^2 (an iteration of order three); 1.6 units,
// where a root and a division have 2
__device__ __forceinline__ double f64_rsqrt(double x) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-(x * r), r, 1.);
  return fma(r, e * fma(.375, e, .5), r);
}
// ln(x) to ~1e-13 absolute, 2^-20 < x < 2^20: x = 2^n m, m in [0.71, 1.42),
// ln m = 2 (s + s^3/3 + s^5/5 + ...), s = (m - 1) / (m + 1), |s| < 0.172
__device__ __forceinline__ double f64_ln13(double x) {
  const int hi = __double2hiint(x);
  const int n = (hi - 0x3fe6a09e) >> 20;
  const double m = __hiloint2double(hi - (n << 20), __double2loint(x));
  const double s = (m - 1.) * f64_recip(m + 1.), z = s * s;
  double p = 2. / 15.;
  p = fma(p, z, 2. / 13.);
  p = fma(p, z, 2. / 11.);
  p = fma(p, z, 2. / 9.);
  p = fma(p, z, 2. / 7.);
  p = fma(p, z, 2. / 5.);
  p = fma(p, z, 2. / 3.);
  p = fma(p, z, 2.);
  return fma(s, p, (double)n * 0.69314718055994530942);
}
// x^(cp/rd) and x^(rd/cp), the Exner function's powers.  cp/rd = 3.5 + d and
// rd/cp = 2/7 + d' with |d| < 1e-4, |d'| < 1e-5, so the root is taken by
// Newton-type steps with its rounding kept in a second term, and x^d =
// exp(d ln x) needs ln x to 1e-12 only.  About 40 FP64 operations, 1.2 and 2.6
// units (pow: 2 last places), where pow takes several times as many.
__device__ __forceinline__ double f64_expm1_small(double y) {  // |y| < 2e-3
  return fma(y * y, fma(y, fma(y, 1. / 24., 1. / 6.), .5), y);
}
__device__ __forceinline__ bool f64_pow_range(double x) {
  return __double2hiint(x) >= 0x3eb00000 && __double2hiint(x) < 0x41300000;  // 2^-20 <= x < 2^20
}
__device__ __forceinline__ double pow_cp_rd(double x) {
  constexpr double a = kCp / kRd, d = a - 3.5;
  if (!f64_pow_range(x)) return pow(x, a);
  // sqrt(x) = sh + sl
  const double r = f64_rsqrt(x), sh = x * r, sl = fma(-sh, sh, x) * (.5 * r);
  // x^3 = qh + ql, their product bh + bl
  const double ph = x * x, pl = fma(x, x, -ph);
  const double qh = ph * x, ql = fma(ph, x, -qh) + pl * x;
  const double bh = qh * sh, bl = fma(qh, sh, -bh) + (qh * sl + ql * sh);
  return bh + fma(bh, f64_expm1_small(d * f64_ln13(x)), bl);
}
__device__ __forceinline__ double pow_rd_cp(double x) {
  // 2/7 = hi + lo
  constexpr double b = kRd / kCp, h27 = 2. / 7., l27 = 1. / 63050394783186944.;  // 2/7 - h27 = 2^-54 2/7
  constexpr double d = (b - h27) - l27;
  if (!f64_pow_range(x)) return pow(x, b);
  // v = x^(2/7) to FP32 accuracy, exact in FP64; v (1 - e)^(-1/7), e = 1 - v^7 / x^2
  const double v = (double)exp2f(0.2857142857f * log2f((float)x));
  const double rx = f64_recip(x), v2 = v * v;
  const double e = fma(-((v2 * v2) * (v2 * v)) * rx, rx, 1.);
  const double c = fma(e * e, 4. / 49., e * (1. / 7.));
  const double g = f64_expm1_small(d * f64_ln13(x));
  return fma(v, fma(c, g, c + g), v);
}
__device__ __forceinline__ float pow_cp_rd(float x) { return pow(x, float(kCp) / float(kRd)); }
__device__ __forceinline__ float pow_rd_cp(float x) { return pow(x, float(kRd) / float(kCp)); }

// ---- flux limiters: bounds, signs and quotients ------------------------------
// FP32 takes the min/max instructions; FP64 compares on the integer pipe and
// divides with the fewest FP64 operations (above).  At glvl 6 / nvl 64 / 11
// tracers this took the FP64 k_trf_lo from 9.56 to 5.0 ms and k_trf_hi from
// 8.15 to 2.48 ms a step (FP32: 2% of k_trf_hi).
//
// These forms hold for numbers.  What is not finite has to go where the
// routines, written with a > b ? a : b, send it (a NaN in a tracer, a thickness
// or a flux reaches the cells around it through fluxes and limiters), so every
// item asks the _rare tests at its end and, if one says so, is formed again
// as the routine writes it (plain_*).  One branch an item: the tests a level
// cost 0-1 FP32 or ~6 integer instructions, where tests in every helper cost
// the FP64 k_trf_lo 18%, k_trf_hi 19%, and the FP32 trcadv 5%.

// max / min that keep a NaN of any value
__device__ __forceinline__ float max_nan(float a, float b) { float r; asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float min_nan(float a, float b) { float r; asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float max_nan(float a, float b, float c) { float r; asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ float min_nan(float a, float b, float c) { float r; asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
template <typename R> struct Bound;
template <> struct Bound<float> {
  float v;
  __device__ __forceinline__ static Bound of(float x) { return {x}; }
  __device__ __forceinline__ void up(Bound a) { v = max_nan(v, a.v); }
  __device__ __forceinline__ void down(Bound a) { v = min_nan(v, a.v); }
  // with two values at once (three-input instructions)
  __device__ __forceinline__ void up(Bound a, Bound b) { v = max_nan(v, a.v, b.v); }
  __device__ __forceinline__ void down(Bound a, Bound b) { v = min_nan(v, a.v, b.v); }
  __device__ __forceinline__ float at_least_zero() const { return max_nan(v, 0.f); }
};
template <> struct Bound<double> {
  long long v;
  __device__ __forceinline__ static Bound of(double x) { return {f64_key(x)}; }
  __device__ __forceinline__ void up(Bound a) { v = a.v > v ? a.v : v; }
  __device__ __forceinline__ void down(Bound a) { v = a.v < v ? a.v : v; }
  __device__ __forceinline__ void up(Bound a, Bound b) { up(a); up(b); }
  __device__ __forceinline__ void down(Bound a, Bound b) { down(a); down(b); }
  __device__ __forceinline__ double at_least_zero() const { return __longlong_as_double(v > 0 ? v : 0); }
};
// upper and lower bound of a ring: some value is a NaN, or (FP64, whose one-
// product fluxes leave it out) infinite
__device__ __forceinline__ bool bounds_rare(Bound<float> up, Bound<float>) { return up.v != up.v; }
__device__ __forceinline__ bool bounds_rare(Bound<double> up, Bound<double> down) {
  return ((int)(up.v >> 32) >= 0x7ff00000) | ((int)(down.v >> 32) <= (int)0x800fffff);
}
template <typename R> __device__ __forceinline__ R plain_max(R a, R b) { return a > b ? a : b; }
template <typename R> __device__ __forceinline__ R plain_min(R a, R b) { return a < b ? a : b; }

// the positive / negative part of x; a NaN in both
__device__ __forceinline__ float pos(float x) { return max_nan(x, 0.f); }
__device__ __forceinline__ float neg(float x) { return min_nan(x, 0.f); }
__device__ __forceinline__ double pos(double x) { return f64_below0(x) ? 0. : x; }
__device__ __forceinline__ double neg(double x) { return (unsigned)__double2hiint(x) > 0x7ff00000u ? x : 0.; }
// own < other ? own : other of two cells' limiters (0 .. 1; a NaN comes sign
// set from plain_ratio01), the cell's own through own_limit first
__device__ __forceinline__ float own_limit(float r) { return r != r ? 2.f : r; }
__device__ __forceinline__ double own_limit(double r) { return __double2hiint(r) < 0 ? 2. : r; }
__device__ __forceinline__ float min0(float own, float other) { return min_nan(own, other); }
__device__ __forceinline__ double min0(double own, double other) {
  const long long x = __double_as_longlong(own), y = __double_as_longlong(other);
  return __longlong_as_double(x < y ? x : y);
}
// a > b ? a : b, b > 0
__device__ __forceinline__ float floor_at(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double floor_at(double a, double b) {
  const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  return x > y && (int)(x >> 32) <= 0x7ff00000 ? a : b;
}
__device__ __forceinline__ bool negative(float x) { return x < 0.f; }
__device__ __forceinline__ bool negative(double x) { return __double2hiint(x) < 0; }
// a < 0 of a number: a zero of either sign is not
__device__ __forceinline__ bool below0(float a) { return a < 0.f; }
__device__ __forceinline__ bool below0(double a) { return (int)((0ull - (unsigned long long)__double_as_longlong(a)) >> 32) > 0; }

// products and sums whose contraction is pinned: the same value must come out
// of every instantiation (the per-routine and the fused kernels, every shape)
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// low-order flux ((mf + |mf|) tri - (mfx + |mfx|) trx) / 2 of the two sides'
// mass fluxes (plain_donor).  They are the same with opposite signs, up to
// rounding, so one of the products is zero but for fluxes of a rounding error's
// size: FP64 forms the other one only.  donor_rare: FP64 mass fluxes that are
// not finite or are positive on both sides (FP32: not finite, asked by the
// largest magnitude).
template <typename R>
__device__ __forceinline__ R plain_donor(R mf, R mfx, R tri, R trx) {
  return mul_rn(R(0.5), fma_rn(mf + fabs(mf), tri, -mul_rn(mfx + fabs(mfx), trx)));
}
__device__ __forceinline__ float donor(float mf, float mfx, float tri, float trx) {
  return fma_rn(fmaxf(mf, 0.f), tri, -mul_rn(fmaxf(mfx, 0.f), trx));
}
__device__ __forceinline__ double donor(double mf, double mfx, double tri, double trx) {
  const bool out = __double2hiint(mf) >= 0;
  const double b = negative(mfx) ? 0. : mfx;
  return mul_rn(out ? mf : -b, out ? tri : trx);
}
__device__ __forceinline__ bool donor_rare(double mf, double mfx) {
  const int a = __double2hiint(mf), b = __double2hiint(mfx);
  return (max(a & 0x7fffffff, b & 0x7fffffff) >= 0x7ff00000) | ((a >= 0) & (__double_as_longlong(mfx) > 0ll));
}

// S+ -= min(0, a), S- += max(0, a); FP64: one addition, to the sum a's sign
// names (sums_rare: one of them ended as a NaN)
__device__ __forceinline__ void split_sum(float a, float& sp, float& sm) {
  sp = sp - neg(a);
  sm = sm + pos(a);
}
__device__ __forceinline__ void split_sum(double a, double& sp, double& sm) {
  const bool n = negative(a);
  const double t = (n ? sp : sm) + fabs(a);
  sp = n ? t : sp;
  sm = n ? sm : t;
}
__device__ __forceinline__ bool sums_rare(float, float) { return false; }
__device__ __forceinline__ bool sums_rare(double sp, double sm) { return f64_nan(sp) | f64_nan(sm); }

// max(0, min(1, a / b)), b > 0; ratio_rare: a NaN or an infinity among the
// numerators of R+ and R-
__device__ __forceinline__ float ratio01(float a, float b) { return __saturatef(__fdividef(a, b)); }
__device__ __forceinline__ double ratio01(double a, double b) {
  const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  if (x <= 0) return 0.;
  if (x >= y) return 1.;
  if (y >= 0x7e00000000000000ll) return a / b;
  return f64_quot(a, b, f64_recip(b));  // 0 < a < b
}
__device__ __forceinline__ bool ratio_rare(float a, float b) { return !(fabsf(a + b) < __int_as_float(0x7f800000)); }
__device__ __forceinline__ bool ratio_rare(double a, double b) { return f64_odd(a) | f64_odd(b); }
__device__ __forceinline__ float plain_ratio01(float a, float b) {
  const float q = plain_max(0.f, plain_min(1.f, fdiv(a, plain_max(b, 1.e-11f))));
  return q != q ? __int_as_float(0xffc00000) : q;
}
__device__ __forceinline__ double plain_ratio01(double a, double b) {
  const double q = plain_max(0., plain_min(1., a / plain_max(b, 1.e-11)));
  return q != q ? __longlong_as_double((long long)0xfff8000000000000ull) : q;
}

// q / ab1 x area: FP64 holds the factor once a cell; FP32 keeps two products
// (theta's last bits decide branches of hybgen in the next step)
__device__ __forceinline__ float per_ab1(float q, float rab1, float area) { return q * rab1 * area; }
__device__ __forceinline__ double per_ab1(double q, double, double f) { return q * f; }

// ---- float-float arithmetic (FP32-mixed build) ----------------------------
// A value hi + lo with |lo| <= ulp(hi)/2 carries ~48 significant bits on the
// FP32 pipes, which GB300 runs at 64x its FP64 rate.  two_sum and two_prod are
// exact (Knuth; Dekker with a fused multiply-add); ff_add is the usual
// double-float sum with one renormalisation.
struct FF2 {
  float hi, lo;
};
__device__ __forceinline__ FF2 two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ FF2 two_prod(float a, float b) {
  const float p = a * b;
  return {p, fmaf(a, b, -p)};
}
__device__ __forceinline__ FF2 ff_add(FF2 a, FF2 b) {
  const FF2 s = two_sum(a.hi, b.hi);
  const float e = s.lo + (a.lo + b.lo);
  const float hi = s.hi + e;
  return {hi, e - (hi - s.hi)};
}
__device__ __forceinline__ FF2 ff_neg(FF2 a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ FF2 ff_shfl_up(FF2 a, int off) {
  return {__shfl_up_sync(0xffffffffu, a.hi, off), __shfl_up_sync(0xffffffffu, a.lo, off)};
}
__device__ __forceinline__ FF2 ff_shfl(FF2 a, int src) {
  return {__shfl_sync(0xffffffffu, a.hi, src), __shfl_sync(0xffffffffu, a.lo, src)};
}
__device__ __forceinline__ FF2 ff_shfl_xor(FF2 a, int m) {
  return {__shfl_xor_sync(0xffffffffu, a.hi, m), __shfl_xor_sync(0xffffffffu, a.lo, m)};
}
// (x.hi + x.lo) - (y.hi + y.lo) rounded once to float
__device__ __forceinline__ float ff_diff(float2 x, float2 y) {
  const FF2 d = two_sum(x.x, -y.x);
  return d.hi + (d.lo + (x.y - y.y));
}

// ---- launchers (instantiated for float and double) ----------------------
// mpf (FP32-mixed step only, may be null): float-float copy (hi, lo) of the
// Montgomery potential; mont_edg then holds the edge value minus the cell value.
// fills Grid::vw on the device (N cells)
void launch_speed_weights(cudaStream_t stream, int N, const double* cs, const double* sn, double* vw);
template <typename R>
void launch_edgvar1(const Launch&, const Grid<R>&, const Strides&, int hi_order, const R* u,
                    const R* v, const R* delp, const R* pres, const R* montg, const R* tracr,
                    R* u_edg, R* v_edg, R* dp_edg, R* lp_edg, R* mont_edg, R* uvsq_edg, R* trc_edg,
                    const float2* mpf = nullptr, R* thold = nullptr);
template <typename R>
struct CnuityScratch { R *antifx, *delp_lo, *p_plus, *p_mnus, *r_plus, *r_mnus; };
template <typename R>
void launch_cnuity(const Launch&, const Grid<R>&, const Strides&, const CnuityScratch<R>&, const R* u,
                   const R* v, const R* u_edg, const R* v_edg, const R* dp_edg, const R* lp_edg,
                   R* delp, R* pres, R* exner, R* dp_tndcy, R* dplo_tndcy, R* massfx, R* omega,
                   bool columns = true);
// cnuity5 (launch_cnuity runs it too when columns is set)
template <typename R>
void launch_cnuity5(const Launch&, const Grid<R>&, const Strides&, R* pres, R* delp, R* exner, const R* dp_tndcy,
                    R* omega, const R* lp_edg, const R* u, const R* v, int ab3_delp);
// flux_conserv_schm = 2 (the bounds use the r_plus/r_mnus scratch slots)
template <typename R>
void launch_massadv(const Launch&, const Grid<R>&, const Strides&, const CnuityScratch<R>&, const R* u,
                    const R* v, const R* u_edg, const R* v_edg, R* dp_edg, const R* lp_edg, R* delp, R* pres,
                    R* exner, R* dp_tndcy, R* massfx, R* omega);
// Cell patches of the fused tracer kernels (fim_trc.cu).  A patch is a set
// of interior cells; its frame lists them first, then every other cell one
// neighbour step away (ring 1), then two steps away (ring 2), so a block can
// stage the frame in shared memory and find every neighbour it needs there.
struct FrameTab {
  int ntile = 0;
  // capacities: frame cells, interior + ring-1 cells, interior cells,
  // edge-value rows (6 per interior cell + ring edges), ring edges
  int S2 = 0, S1 = 0, SC = 0, SE = 0, SR = 0;
  const int4* cnt = nullptr;             // [ntile] interior cells, + ring 1, + ring 2, ring edges
  // A patch's tables, as its block holds them in shared memory (copied 16
  // bytes at a time): `bytes` of them a patch, the first `head` what
  // k_trf_hi needs.  Laid out and resolved once, so that a block's set-up is
  // a straight copy: gathering the tables, the coefficients and the flux rows
  // through each other cost k_trf_lo the time of 1.5 tracers (FP32 at 655,362
  // cells x 64 levels x 11 tracers, k_trf_lo 6.77 -> 6.28 ms and k_trf_hi
  // 5.96 -> 5.85 ms; a step of 10,242 x 38 x 5 286 -> 260 us).  Byte offsets:
  //   0    [S2] int            cell index, frame order
  //   nbr  [S1] uint2          frame-local index of prox slots 0..5, a byte each
  //   np   [S1] u8             nprox of the interior and ring-1 cells
  //   mir  [SC][6] u16         edge-value row of the other side of each edge
  //   red  [SR] u16            ring edges: (frame-local cell << 3) | slot
  //   mfr  [SE] int            cell x 6 + slot of each edge-value row
  const unsigned char* tab = nullptr;
  int bytes = 0, head = 0, nbr = 0, np = 0, mir = 0, red = 0, mfr = 0;
  // halved least-squares coefficients (of the context's precision): cstride
  // values a patch, 36 per interior cell, then 6 per ring edge
  const void* coef = nullptr;
  int cstride = 0;
};
struct FrameHost {
  int ntile = 0, S2 = 0, S1 = 0, SC = 0, SE = 0, SR = 0;
  std::vector<int> cells, cnt;
  std::vector<uint32_t> nbr;
  std::vector<uint16_t> mir, red;
};
// patches of side x side cells of each rhombus (the reference's IJ
// numbering), else grown breadth-first; 0 on success
int build_frames(int N, const int* prox, const int* proxs, const int* nprox, int side, FrameHost* out,
                 bool sixth = false);
// 0 if every cell is in exactly one patch and every frame neighbour and edge
// mirror of the tables resolves to prox/proxs
int check_frames(int N, const int* prox, const int* proxs, const int* nprox, const FrameHost& f);
// fused tracer path of the step (fim_trc.cu)
template <typename R>
struct TrcFusedScratch {
  R *trcr_lo, *s_plus, *s_mnus, *trold;
  R *r_plus, *r_mnus;  // scratch for the shape probe's outputs
  R* antifx;           // antidiffusive fluxes (6 per cell-level) of the chunk
  int tchunk;
  int vk;  // levels per thread (0: widest the layout admits)
  int gc;  // threads per cell and level tile: the tile is vk * gc levels
  FrameTab ft;
  bool edges = false;  // trc_edg holds every tracer's edge values (the per-routine trcadv); 4 threads a cell
};
// nfields: 1 = dp only, T = dp and tracers 2..ntra (edgvar3's full output);
// average = false leaves the own-side values (k_cnuity12 averages the layer
// thickness's itself); ft: the context's cell patches
template <typename R>
void launch_edgvar3(const Launch&, const Grid<R>&, const Strides&, const R* delp, const R* tracr,
                    R* dp_edg, R* trc_edg, int nfields, const FrameTab& ft, bool average = true);
// edgvar3 with the two-sided average on cell patches (fim_trc.cu; FP32: the
// FP64 build is bound by its FP64 operations, which recomputing the ring
// cells' sides would add to); prepare_edges: its one-time launch attributes
int prepare_edges(const FrameTab& ft);
void launch_edges_patch(const Launch&, const Grid<float>&, const Strides&, const FrameTab&, int nfields,
                        const float* delp, const float* tracr, float* dp_edg, float* trc_edg);
// packs the patches' tables as FrameTab describes and sets its sizes and
// offsets (not its pointers); edge-value rows of cells and slots follow proxs
void pack_frames(const FrameHost& f, const int* nprox, FrameTab* tab, std::vector<unsigned char>* out);
// fills coef (ntile x cstride values) from the grid's least-squares coefficients
template <typename R>
void launch_patch_coefs(cudaStream_t stream, const Grid<R>& g, const FrameTab& ft, R* coef);
// one-time launch attributes (shared-memory size) of the tracer kernels for
// these patches; returns a cudaError_t value
template <typename R>
int prepare_tracers(const FrameTab& ft);
// times the tracer kernel shapes on the given state (see fim_trc.cu); returns a cudaError_t value
template <typename R>
int tune_tracers(const Launch&, const Grid<R>&, const Strides&, const TrcFusedScratch<R>&, R* trc_edg, R* tracr,
                 R* trcdp, R* trc_tdcy, R* trl_tdcy, const R* massfx, const R* delp, int* best_vk, int* best_gc,
                 float* best_ms);
// Called by launch_tracers_fused before (phase 0) and after (phase 1) the
// kernels of each tracer chunk [t0, t0 + nt): the step with host transfers
// (fim_step_io) orders the chunk's AB3 slot uploads and its downloads there.
struct ChunkHook {
  void (*fn)(void* arg, int phase, int t0, int nt) = nullptr;
  void* arg = nullptr;
};
template <typename R>
void launch_tracers_fused(const Launch&, const Grid<R>&, const Strides&, const TrcFusedScratch<R>&,
                          R* trc_edg, R* tracr, R* trcdp, R* trc_tdcy, R* trl_tdcy, const R* massfx,
                          const R* delp, const ChunkHook* hook = nullptr);
template <typename R>
struct MomtumScratch { R *du, *dv, *wu, *wv; };
// With mpf != null (FP32-mixed step) the pressure-gradient line integrals use
// the cell values split off (see k_momtum1): tr0 = the potential temperature
// edgvar1 saw (thold), svsum = per-cell sums of sidevec_c.
template <typename R>
void launch_momtum(const Launch&, const Grid<R>&, const Strides&, const Knobs&, const MomtumScratch<R>&,
                   R* u, R* v, const R* exner, R* relvor, const R* u_edg, const R* v_edg,
                   const R* trc_edg, const R* mont_edg, const R* uvsq_edg, R* u_tndcy, R* v_tndcy,
                   const R* dp3d, const float2* mpf = nullptr, const R* tr0 = nullptr);
template <typename R>
struct HybgenScratch { R *exsmo, *exsmo2; };
// one-time launch attributes of the hybgen kernels (shared-memory size);
// returns a cudaError_t value
template <typename R>
int prepare_hybgen(int L);
// trdp != null: the default-knob remap also applies hystat's humidity floors
// and writes tracer x thickness of the new state (returns true; hystat can
// then skip that stream)
template <typename R>
bool launch_hybgen(const Launch&, const Grid<R>&, const Strides&, const Knobs&, const HybgenScratch<R>&,
                   const R* targt, R* us3d, R* vs3d, R* tr3d, R* sdot, R* ex3d, R* dp3d, R* pr3d,
                   R* trdp = nullptr);
template <typename R>
void launch_hystat(const Launch&, const Grid<R>&, const Strides&, R* ph3d, const R* ex3d, R* mp3d,
                   const R* dp3d, R* tr3d, R* trdp, R* psrf, R* ptdcy, float2* mpf = nullptr,
                   bool trdp_done = false);
// class-B transport (fim_trb.cu); scratch per member: w (nvl x nip), the
// other fields (nvl x nip x ntrb)
template <typename R>
struct ClassBScratch { R *w, *F, *V, *fmx, *fmn, *flo, *flp, *fln; };
template <typename R>
void launch_transp1(const Launch&, const Grid<R>&, const Strides&, R* cumufx, const R* massfx);
// every > 0: only members at a step its with its % every == 0
template <typename R>
void launch_transp0(const Launch&, const Grid<R>&, const Strides&, int every, R* cumufx, const R* dp3d,
                    R* dpinit);
template <typename R>
void launch_transp2(const Launch&, const Grid<R>&, const Strides&, const ClassBScratch<R>&, int every, int ntrb,
                    R* tracr, const R* cumufx, const R* dpinit, const R* dpfinl);
template <typename R>
int prepare_classb(int L);
// sums per member: [member][8 + T] doubles; partial buffer sized by globsum_partials()
// ntr: tracers summed (class A and B); sums per member: [member][8 + ntr]
template <typename R>
void launch_globsum(const Launch&, const Grid<R>&, const Strides&, int ntr, const R* dp3d, const R* tr,
                    const R* rn2d, const R* rc2d, const R* pr3d, const R* ex3d, const R* qf2d,
                    double* partial, double* sums);
size_t globsum_partials(int N, int L, int T, int members);
// edgvar2 (fim_dyn.cu): w = 3 N L values of scratch
template <typename R>
void launch_edgvar2(const Launch&, const Grid<R>&, const Strides&, const R* u, const R* v, R* u_edg, R* v_edg,
                    R* uvsq_edg, R* w);
// physics coupling (fim_cpl.cu); GFS arrays (nip, nvl), cell fastest, FP64
// gfs = ps, dp, p, u, v, dpdt, q, oz, cld, t; old6 = u, v, t, q, oz, cld
template <typename R>
void launch_cpl_dyn_to_phy(const Launch&, const Grid<R>&, const R* pr3d, const R* us3d, const R* vs3d,
                           const R* ws3d, const R* tr3d, double* const gfs[10], double* old6);
// gfs7 = p, u, v, q, cld, oz, t; col3 = geshem, rainc, evap; tend: 12 N L
// doubles of scratch with addtend (6 N L without smoothtend)
template <typename R>
void launch_cpl_phy_to_dyn(const Launch&, const Grid<R>&, double dt, double dtp, bool addtend, bool smoothtend,
                           const double* const gfs7[7], const double* old6, const double* const col3[3],
                           const R* dp3d, R* us3d, R* vs3d, R* tr3d, R* rn2d, R* rc2d, R* qf2d, double* tend);
template <typename R>
void launch_prdp_from_ex(const Launch&, const Grid<R>&, const Strides&, const R* ex3d, R* pr3d, R* dp3d);
void launch_step_begin(const Launch&, StepParams* sp);  // advances every active member

// fim_synth.cu: the seeded balanced state of one member slot
template <typename R>
int launch_synthetic(cudaStream_t stream, int N, int L, int nslot, int ntra, const double* lat,
                     const double* dps, unsigned long long seed, double sigma_ps, double noise, double ptop,
                     R* us3d, R* vs3d, R* dp3d, R* pr3d, R* ex3d, R* ph3d, R* mp3d, R* tr3d);

}  // namespace fim
