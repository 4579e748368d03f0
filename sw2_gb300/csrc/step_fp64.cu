// Reference-exact FP64 step, in core.c's order (core.c:134-338) wherever the
// order reaches a value. What reads old fields only (CFL maxima, TVD bodies,
// first Laplacian levels) runs in one launch; the first two steps after an
// upload then run one kernel per reference routine; from the third (AB3) the
// tails of the tendencies are fused, the Laplacians write their own halo
// images and wall fixes, and the range checks are made by the kernels that
// write the state. Compiled with -fmad=false so that no a*b+c is fused: every
// expression keeps the association of the reference expression it restates,
// which makes the results bit-identical to the reference's own single-rank
// run. GB300 executes FP64 at 2 lanes per SM per clock, so quotients, most
// products, scalings by powers of two, zero numerators and comparisons are
// answered on the integer pipe (sigmath.cuh: the same IEEE results), and the
// FP64 unit keeps the additions.
#include <cuda_runtime.h>

#include <atomic>

#include "sigmath.cuh"
#include "sw2g_internal.h"

namespace sw2g {
namespace {

constexpr int TX = 128;

__device__ __forceinline__ int IX(int W, int i, int j) { return (i + 1) + (j + 1) * W; }
__device__ __forceinline__ double RW(const DevState& s, int t, int j) { return s.rows[t * s.H + j + 1]; }
// A field of a polar cap at padded index q.
__device__ __forceinline__ double PF(const DevState& s, int t, int q) { return s.pf[(size_t)t * s.W * s.H + q]; }

// Brings the line of a value that a later row reads into L1, without a
// register to hold it: a load whose result nothing uses.
__device__ __forceinline__ void touch(const double* p) {
  [[maybe_unused]] double x;
  asm volatile("ld.global.ca.f64 %0, [%1];" : "=d"(x) : "l"(p));
}

// The bit pattern of a double, through an opaque move: tests written on the
// integer image (sign, exponent, zero) then stay integer operations; given
// the plain reinterpretation, the compiler may turn them back into FP64
// comparisons, which issue on GB300's narrow FP64 unit.
__device__ __forceinline__ long long dbits(double x) {
  long long r;
  asm("mov.b64 %0, %1;" : "=l"(r) : "d"(x));
  return r;
}

__device__ __forceinline__ int dexp(double x) {
  return (int)(((unsigned long long)dbits(x) >> 52) & 0x7ffULL);
}

// a / b with a zero numerator answered from the bits: IEEE division gives
// +-0 / b the zero whose sign is the exclusive or of the operands' signs for
// every b other than a zero or a NaN; there the hardware sequence would take
// its special-case path (about 15 FP64 instructions). Other operands divide.
// The literal cells use it: in a state at rest their velocities, Courant
// numbers and differences are zeros.
__device__ __forceinline__ double zdiv(double a, double b) {
  const long long A = dbits(a), B = dbits(b);
  const long long mb = B & 0x7fffffffffffffffLL;
  if ((A & 0x7fffffffffffffffLL) == 0 && mb != 0 && mb <= 0x7ff0000000000000LL)
    return __longlong_as_double((A ^ B) & (long long)0x8000000000000000ULL);
  return a / b;
}

// The literal cells' division: on the integer pipe where both operands and
// the quotient are normal numbers (sigmath.cuh), else as zdiv. Out of line: a
// cell has up to eighteen of them.
__device__ __noinline__ double ldiv(double a, double b) {
  const unsigned ea = (unsigned)(((unsigned long long)dbits(a) >> 52) & 0x7ff);
  const unsigned eb = (unsigned)(((unsigned long long)dbits(b) >> 52) & 0x7ff);
  if (ea - 1 < 2046u && eb - 1 < 2046u && ea - eb + 1021u < 2043u) {
    const unsigned long long m = 0x7fffffffffffffffULL, A = (unsigned long long)dbits(a), B = (unsigned long long)dbits(b);
    return __longlong_as_double((long long)(sig_div(A & m, B & m) | ((A ^ B) & ~m)));
  }
  return zdiv(a, b);
}

// x * 2^k for k in -2..1 (p = 2^k), the same value as the FP64 product: when
// x and the product are normal numbers, the product only changes the exponent
// field, done here on the integer pipe; zeros are their own product; other
// cases (subnormal operand or result, inf, NaN) multiply, out of line.
__device__ __noinline__ double mul_pow2_fp64(double x, double p) { return x * p; }
__device__ __forceinline__ double mul_pow2(double x, int k, double p) {
  const long long b = dbits(x);
  if ((b & 0x7fffffffffffffffLL) == 0) return x;
  const int e = (int)((b >> 52) & 0x7ff);
  if (e >= 1 && e <= 2046 && e + k >= 1 && e + k <= 2046) return __longlong_as_double(b + ((long long)k << 52));
  return mul_pow2_fp64(x, p);
}
#define HALF(x) mul_pow2((x), -1, 0.5)
#define QUARTER(x) mul_pow2((x), -2, 0.25)
#define TWICE(x) mul_pow2((x), 1, 2.0)

// Correctly rounded a/b given y = RN(1/b), b a positive normal number, with
// one multiplication and two fused multiply-adds (Markstein's method:
// P. Markstein, IBM J. Res. Dev. 34(1), 1990; J.-M. Muller et al., Handbook
// of Floating-Point Arithmetic, ch. "division with an FMA"): q0 = RN(a*y),
// r0 = a - b*q0 (exact), RN(q0 + r0*y) = RN(a/b). Markstein's theorem covers
// q0 within one ulp of a/b; RN(a*y) can be up to 1.5 ulps off, and the one
// correction still rounds correctly there by the case analysis of a/b in
// [1/2, 1) scaled (a wrong rounding would need a and b both within a few
// ulps of a power of two, a set the self-check walks exhaustively, with
// random and near-midpoint numerators on top: fp64_check_division).
// A zero numerator gives itself (+-0 / b = +-0 for b > 0); other numerators
// outside [2^-900, 2^776] (subnormals: remainders could underflow; inf, NaN)
// use the IEEE division. The row tables hold y = 1.0/b computed by IEEE
// division on the host. fp64_check_division compares this with the IEEE
// quotient on random and near-halfway numerators.
__device__ __forceinline__ double div_rcp(double a, double b, double y) {
  if ((dbits(a) & 0x7fffffffffffffffLL) == 0) return a;
  if ((unsigned)(dexp(a) - 123) > 1799u - 123u) return a / b;
  const double q0 = __dmul_rn(a, y);
  const double r0 = __fma_rn(-b, q0, a);
  return __fma_rn(r0, y, q0);
}

// a + b rounded to nearest, ties to even, computed on the integer pipe (the
// textbook IEEE 754 adder: order the operands by magnitude, align the
// smaller significand with ten guard bits and a sticky bit, add or subtract,
// renormalise, round) when both operands and the sum are normal numbers. A
// zero operand gives the other operand (two zeros give -0 only if both are
// -0), and exact cancellation gives +0, as the FP64 unit's round-to-nearest
// does. Everything else (subnormals, inf, NaN, a sum that overflows or falls
// below the normal range) adds on the FP64 unit, out of line. fp64_check_add
// compares sadd and ssub with the FP64 unit on random and edge-case operands.
// An integer-pipe addition takes about a hundred instructions where the FP64
// unit takes one: it pays only in a kernel whose FP64 work leaves most issue
// slots idle, as the Coriolis updates of the first two steps do (0.139 ->
// 0.105 ms each at 2048x1024). Where products and quotients already take the
// integer pipe (all other kernels) additions stay on the FP64 unit.
__device__ __noinline__ double add_fp64(double a, double b) { return a + b; }
__device__ __forceinline__ double sadd(double a, double b) {
  constexpr unsigned long long MAG = 0x7fffffffffffffffULL, FRAC = 0x000fffffffffffffULL, ONE = 1ULL << 52;
  unsigned long long A = (unsigned long long)dbits(a), B = (unsigned long long)dbits(b);
  if ((A & MAG) < (B & MAG)) {  // |A| >= |B| from here on
    const unsigned long long t = A;
    A = B;
    B = t;
  }
  const int ea = (int)((A >> 52) & 0x7ff), eb = (int)((B >> 52) & 0x7ff);
  if ((B & MAG) == 0)  // the smaller is a zero: the larger (a NaN stays a NaN);
    // two zeros: -0 if both are, else +0
    return __longlong_as_double((long long)(((A & MAG) == 0) ? (A & B) : A));
  if (ea == 0x7ff || eb == 0) return add_fp64(a, b);  // inf, NaN or a subnormal operand
  const int d = ea - eb;
  const unsigned long long ma = ((A & FRAC) | ONE) << 10;  // significand at bits 62..10
  unsigned long long mb = ((B & FRAC) | ONE) << 10;
  if (d >= 63) {
    mb = 1;  // only the sticky bit is left
  } else if (d > 0) {
    mb = (mb >> d) | ((mb << (64 - d)) != 0 ? 1ULL : 0ULL);
  }
  int e = ea;
  unsigned long long m;
  if (((A ^ B) >> 63) == 0) {
    m = ma + mb;
    if (m >> 63) {  // carry: one bit right, keeping the sticky bit
      m = (m >> 1) | (m & 1ULL);
      e += 1;
    }
  } else {
    m = ma - mb;
    if (m == 0) return 0.0;
    const int lz = __clzll((long long)m) - 1;  // back to bit 62 (at most one place when bits were lost)
    m <<= lz;
    e -= lz;
  }
  unsigned long long r = m >> 10;
  const unsigned long long rem = m & 0x3ffULL;
  if (rem > 0x200ULL || (rem == 0x200ULL && (r & 1ULL))) r += 1;
  if (r >> 53) {
    r >>= 1;
    e += 1;
  }
  if (e <= 0 || e >= 0x7ff) return add_fp64(a, b);
  return __longlong_as_double((long long)((A & ~MAG) | ((unsigned long long)e << 52) | (r & FRAC)));
}
// a - b = a + (-b), exactly and for every operand (a NaN operand gives a
// NaN either way; NaN bit patterns are not compared anywhere). The step's kernels
// add only; the self-check takes the adder's other signs through it.
__device__ __forceinline__ double ssub(double a, double b) {
  return sadd(a, __longlong_as_double(dbits(b) ^ (long long)0x8000000000000000ULL));
}

// calc.c:54-63 with sw.h:104-105 MIN/MAX as ternaries (NaN order as written).
template <int SCH>
__device__ __forceinline__ double limiter(double r) {
#define MN(a, b) (((a) < (b)) ? (a) : (b))
#define MX(a, b) (((a) > (b)) ? (a) : (b))
  if constexpr (SCH == 0) return MX(0.0, MN(MN((1 + r) / 2.0, 2.0 * r), 2.0));
  else if constexpr (SCH == 1) return MX(MX(0.0, MN(2.0 * r, 1.0)), MX(0.0, MN(r, 2.0)));
  else if constexpr (SCH == 2) return MN(r, 1.0);
  else if constexpr (SCH == 3) return zdiv(r + fabs(r), 1.0 + r);
  else if constexpr (SCH == 4) return MX(0.0, MN(2.0 * r, MN((1 + 2.0 * r) / 3.0, 2.0)));
  else if constexpr (SCH == 5) return zdiv(1.5 * (r * r + r), r * r + r + 1.0);
  else if constexpr (SCH == 6) return zdiv(r * r + r, r * r + 1.0);
  else if constexpr (SCH == 7) return MX(0.0, MN(MN(2.0, 2.0 * r), MN(0.25 + 0.75 * r, 0.75 + 0.25 * r)));
  else if constexpr (SCH == 8) return 0.0;
  else if constexpr (SCH == 9) return 1.0;
  else return (r == -1.0) ? 0.0 : zdiv(r + fabs(r), 1.0 + r);
#undef MN
#undef MX
}

// One face q0|q1 with outer neighbours qm, q2 (calc.c:41-49).
template <int SCH>
__device__ __forceinline__ void tvd_face(double qm, double q0, double q1, double q2, double cP, double cM,
                                         double& BP, double& BM) {
  const double d = q1 - q0;
  const double rP = (d != 0) ? ldiv(q0 - qm, d) : 0.0;
  const double rM = (d != 0) ? ldiv(q2 - q1, d) : 0.0;
  BP = q0 + limiter<SCH>(rP) * 0.5 * (1 - cP) * d;
  BM = q1 - limiter<SCH>(rM) * 0.5 * (1 + cM) * d;
}

// Sum C*B over the four faces in the reference's order (calc.c:100).
template <int SCH>
__device__ __forceinline__ double tvd_sum(const double* qx, const double* qy, double cwP, double cwM, double ceP,
                                          double ceM, double csP, double csM, double cnP, double cnM) {
  double wP, wM, eP, eM, sP, sM, nP, nM;
  tvd_face<SCH>(qx[0], qx[1], qx[2], qx[3], cwP, cwM, wP, wM);
  tvd_face<SCH>(qx[1], qx[2], qx[3], qx[4], ceP, ceM, eP, eM);
  tvd_face<SCH>(qy[0], qy[1], qy[2], qy[3], csP, csM, sP, sM);
  tvd_face<SCH>(qy[1], qy[2], qy[3], qy[4], cnP, cnM, nP, nM);
  return cwP * wP + cwM * wM - ceP * eP - ceM * eM + csP * sP + csM * sM - cnP * nP - cnM * nM;
}

__device__ __forceinline__ double cpos(double a, double dt, double dx) { return ldiv(0.5 * (a + fabs(a)) * dt, dx); }
__device__ __forceinline__ double cneg(double a, double dt, double dx) { return ldiv(0.5 * (a - fabs(a)) * dt, dx); }
__device__ __forceinline__ double cpos2(double a, double b, double dt, double dx) {
  return ldiv(0.5 * (0.5 * (a + fabs(a)) + 0.5 * (b + fabs(b))) * dt, dx);
}
__device__ __forceinline__ double cneg2(double a, double b, double dt, double dx) {
  return ldiv(0.5 * (0.5 * (a - fabs(a)) + 0.5 * (b - fabs(b))) * dt, dx);
}

struct F7 {
  const double *eta, *u, *v, *tr, *wx, *wy, *hb;
};

#define UW(i, j) (f.u[IX(W, i, j)] + f.wx[IX(W, i, j)])                   /* sw.h:216 */
#define VW(i, j) (f.v[IX(W, i, j)] + f.wy[IX(W, i, j)])                   /* sw.h:217 */
#define HH(i, j) (f.eta[IX(W, i, j)] + s.depth - f.hb[IX(W, i, j)])       /* sw.h:213 */

#define INTERIOR_IJ                                   \
  const int W = s.W;                                  \
  const int i = blockIdx.x * TX + threadIdx.x + 1;    \
  const int j = blockIdx.y + 1;                       \
  if (i > s.nx) return;

// BODYH + damping (calc.c:70-113), one cell
template <int SCH>
__device__ __forceinline__ double mass_cell(const DevState& s, const F7& f, int i, int j) {
  const int W = s.W;
  const double Dt = s.Dt, dxe = RW(s, R_DXE, j), dyn = RW(s, R_DYN, j);
  double qx[5], qy[5];
#pragma unroll
  for (int o = -2; o <= 2; o++) { qx[o + 2] = HH(i + o, j); qy[o + 2] = HH(i, j + o); }
  const double a = UW(i - 1, j), b = UW(i, j), c = VW(i, j - 1), d = VW(i, j);
  double acc = tvd_sum<SCH>(qx, qy, cpos(a, Dt, dxe), cneg(a, Dt, dxe), cpos(b, Dt, dxe), cneg(b, Dt, dxe),
                            cpos(c, Dt, dyn), cneg(c, Dt, dyn), cpos(d, Dt, dyn), cneg(d, Dt, dyn));
  const double sigma = s.polar ? PF(s, P_SH, IX(W, i, j)) : s.sigma;  // the sponge, calc.c:102-111
  acc -= 2.0 * Dt * (sigma) * f.eta[IX(W, i, j)];
  return acc;
}

// Programmatic dependent launch of the step's kernels: each kernel starts by
// waiting for the previous kernel of the stream to complete (a no-op for a
// kernel launched without the attribute), so its launch overlaps the kernel
// before it, and no kernel reads or writes memory before its predecessor has
// finished. None lets its dependents in before it ends
// (griddepcontrol.launch_dependents): blocks that wait where the predecessor's
// last blocks still run cost more than they save (a step at 256x128 98 us with
// it, 88 without; at 1201x607 660 and 631; at 2048x1024 0.2 % less with it).
#define SW2G_PDL_ENTRY() asm volatile("griddepcontrol.wait;" ::: "memory")

template <typename... KArgs, typename... Args>
void pdl_launch(void (*k)(KArgs...), dim3 g, dim3 b, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = g;
  cfg.blockDim = b;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(args)...);
}

template <int SCH>
__global__ void k_mass(DevState s, F7 f, double* out) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  out[IX(W, i, j)] = mass_cell<SCH>(s, f, i, j);
}

// BODYTRACER (calc.c:117-163), one cell
template <int SCH>
__device__ __forceinline__ double tracer_cell(const DevState& s, const F7& f, int i, int j) {
  const int W = s.W;
  const double Dt = s.Dt, dxe = RW(s, R_DXE, j), dyn = RW(s, R_DYN, j);
  double qx[5], qy[5];
#pragma unroll
  for (int o = -2; o <= 2; o++) { qx[o + 2] = f.tr[IX(W, i + o, j)]; qy[o + 2] = f.tr[IX(W, i, j + o)]; }
  const double a = UW(i - 1, j), b = UW(i, j), c = VW(i, j - 1), d = VW(i, j);
  const double pv1 = tvd_sum<SCH>(qx, qy, cpos(a, Dt, dxe), cneg(a, Dt, dxe), cpos(b, Dt, dxe), cneg(b, Dt, dxe),
                                  cpos(c, Dt, dyn), cneg(c, Dt, dyn), cpos(d, Dt, dyn), cneg(d, Dt, dyn));
  const double t = qx[2];
  double pv2 = ldiv(Dt * t * (b - a), dxe);
  pv2 += ldiv(Dt * t * (d - c), dyn);
  double acc = pv1 + pv2;
  const double sigma = s.polar ? PF(s, P_STR, IX(W, i, j)) : s.sigma_tr;  // calc.c:152-161
  acc -= 2.0 * Dt * (sigma) * t;
  return acc;
}

template <int SCH>
__global__ void k_tracer(DevState s, F7 f, double* out) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  out[IX(W, i, j)] = tracer_cell<SCH>(s, f, i, j);
}

// BODYU (calc.c:168-200), one cell
template <int SCH>
__device__ __forceinline__ double advu_cell(const DevState& s, const F7& f, int i, int j) {
  const int W = s.W;
  const double Dt = s.Dt, dxc = RW(s, R_DXC, j), dyv = RW(s, R_DYV, j);
  double qx[5], qy[5];
#pragma unroll
  for (int o = -2; o <= 2; o++) { qx[o + 2] = UW(i + o, j); qy[o + 2] = UW(i, j + o); }
  const double uwm = qx[1], u0 = qx[2], uep = qx[3];
  const double vs0 = VW(i, j - 1), vs1 = VW(i + 1, j - 1), vn0 = VW(i, j), vn1 = VW(i + 1, j);
  const double p1 = tvd_sum<SCH>(qx, qy, cpos2(uwm, u0, Dt, dxc), cneg2(uwm, u0, Dt, dxc), cpos2(u0, uep, Dt, dxc),
                                 cneg2(u0, uep, Dt, dxc), cpos2(vs0, vs1, Dt, dyv), cneg2(vs0, vs1, Dt, dyv),
                                 cpos2(vn0, vn1, Dt, dyv), cneg2(vn0, vn1, Dt, dyv));
  const double p2 = Dt * (ldiv(u0 * (uep - uwm), RW(s, R_DXE2, j)) + ldiv(u0 * ((vn0 + vn1) / 2. - (vs0 + vs1) / 2.), dyv));
  return p1 + p2;
}

template <int SCH>
__global__ void k_adv_u(DevState s, F7 f, double* out) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  out[IX(W, i, j)] = advu_cell<SCH>(s, f, i, j);
}

// BODYV (calc.c:205-237), one cell
template <int SCH>
__device__ __forceinline__ double advv_cell(const DevState& s, const F7& f, int i, int j) {
  const int W = s.W;
  const double Dt = s.Dt, dxv = RW(s, R_DXV, j), dyc = RW(s, R_DYC, j);
  double qx[5], qy[5];
#pragma unroll
  for (int o = -2; o <= 2; o++) { qx[o + 2] = VW(i + o, j); qy[o + 2] = VW(i, j + o); }
  const double vsm = qy[1], v0 = qy[2], vnp = qy[3];
  const double uw1 = UW(i - 1, j + 1), uw0 = UW(i - 1, j), ue1 = UW(i, j + 1), ue0 = UW(i, j);
  const double p1 = tvd_sum<SCH>(qx, qy, cpos2(uw1, uw0, Dt, dxv), cneg2(uw1, uw0, Dt, dxv), cpos2(ue1, ue0, Dt, dxv),
                                 cneg2(ue1, ue0, Dt, dxv), cpos2(vsm, v0, Dt, dyc), cneg2(vsm, v0, Dt, dyc),
                                 cpos2(v0, vnp, Dt, dyc), cneg2(v0, vnp, Dt, dyc));
  const double p2 = Dt * (ldiv(v0 * ((ue0 + ue1) / 2. - (uw0 + uw1) / 2.), dxv) + ldiv(v0 * (vnp - vsm), RW(s, R_DYNS, j)));
  return p1 + p2;
}

template <int SCH>
__global__ void k_adv_v(DevState s, F7 f, double* out) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  out[IX(W, i, j)] = advv_cell<SCH>(s, f, i, j);
}

// Literal cells for the fast kernels' fallback, kept out of line.
template <int SCH>
__device__ __noinline__ double mass_cell_ool(const DevState& s, const F7& f, int i, int j) {
  return mass_cell<SCH>(s, f, i, j);
}
template <int SCH>
__device__ __noinline__ double tracer_cell_ool(const DevState& s, const F7& f, int i, int j) {
  return tracer_cell<SCH>(s, f, i, j);
}
template <int SCH>
__device__ __noinline__ double advu_cell_ool(const DevState& s, const F7& f, int i, int j) {
  return advu_cell<SCH>(s, f, i, j);
}
template <int SCH>
__device__ __noinline__ double advv_cell_ool(const DevState& s, const F7& f, int i, int j) {
  return advv_cell<SCH>(s, f, i, j);
}

// ------------------------------------------------------------ fast TVD bodies
// The same values as k_mass, k_tracer, k_adv_u and k_adv_v, bit for bit, with
// about a tenth of their FP64 instructions. Four properties of the reference
// formulas (calc.c:41-49, 70-237) and of the unit make that possible:
//  (1) x faces. The metric factors DXE, DXC, DXV depend on j only, so the
//      Courant numbers, limiter ratios and limited values of the
//      face between columns i-1 and i are the same operations on the same
//      operands for cell i (its west face) and cell i-1 (its east face). Each
//      lane of a warp computes the face west of its column; a warp covers 31
//      cells with 32 faces and takes the east face from the next lane.
//  (2) y faces. The ratios and limiter values of the face between rows j and
//      j+1 are shared by both cells; only the Courant numbers differ, since
//      each cell divides by its own DYN, DYV or DYC. A warp marches up its
//      rows and carries the face's shared part from one row to the next, and
//      the differences q(j+1)-q(j), which serve three faces.
//  (3) Upwind split. C+ = 0.5(U+|U|)*Dt/DX is +0 when U <= 0, and C- is a
//      zero when U >= 0 (for the two-velocity averages, when both are), so
//      the term C*B of an unused side is a zero whenever B is finite, and
//      0.5(U+|U|) = U exactly when U > 0 (0.5(U-|U|) = U when U < 0). Leaving
//      zero terms out of a sum of otherwise identical terms, in the same
//      order, can change only the sign of a zero result (see below). When
//      both velocities of an average have one sign, the sum of their used
//      halves is the sum of the velocities, which the second term of the
//      body needs as well.
//  (4) The integer pipe. The quotients (limiter ratios, Courant numbers, the
//      second term's divisions) and the products that enter them are taken
//      from the operands' bits (sigmath.cuh: IEEE results); the FP64 unit
//      keeps the additions and the products around them.
// Ranges. Each value that a warp reads is zero or of magnitude 2^-850 ..
// 2^100 (in_range); otherwise the warp's cells are recomputed literally for
// the rest of its strip. Differences and sums of such values are zero or at
// least 2^-902 (they are multiples of the smallest unit among them), so slope
// ratios and Courant numbers are normal; products of several factors are
// tested (slope_term, two_products). The
// skipped side is finite if its slope ratio is below 2^498 (then every
// limiter, squares included, is), which a difference of at least 2^-397
// ensures; below that the ratio's exponent is looked at (make_face).
// Zero sums. A sum that is zero because nonzero terms cancel is +0, as the
// reference's is (x - x = +0, and +0 plus or minus a zero is +0). When every
// term is zero the reference's sum is +0 if its first term is +0: the + side
// at the west face, whose Courant number is never negative, with a face value
// that is not negative (first_term_plus_zero). So it is in a flow at rest and
// for a tracer that is zero. Otherwise the cell is recomputed literally.
// The Van Leer limiter in its reference form (0/0 at r = -1) keeps the
// literal kernels, and so do cases whose Dt or metric divisors lie outside
// 2^-20 .. 2^60 (DevState::sig_ok).
constexpr int FW = 31;      // cells per strip along x (32 faces)
constexpr int FWARPS = 4;   // warps per block; each warp takes strips from the launch's queue
// Resident blocks per SM the register allocation must allow: 7 blocks (28
// warps) at 72 registers hide the FP64 unit's latency best. k_adv_u at
// 2048x1024 with 4, 5, 6, 7, 8 and 10 blocks: 0.138, 0.133, 0.128, 0.122,
// 0.124 and 0.125 ms. In one launch with the other kinds, whole steps with 6, 7
// and 8: four at 2048x1024 3.229, 3.212, 3.197 ms; four of a 500x500 cap 0.763,
// 0.759, 0.771; two forced ones from rest at 1024x512 2.147, 2.000, 2.051. At 72
// registers the launch's frame, which seven kinds of strips share, spills 120 to 124
// bytes a thread for limiter 2, 152 to 236 for the others (limiter 8); k_lapv alone
// takes 56 registers and spills none.
#define FAST_MIN_BLOCKS 7
constexpr unsigned FULL = 0xffffffffu;

// Comparisons on the integer pipe (GB300 issues FP64 compares on its narrow
// FP64 unit). For finite values they agree with the IEEE comparisons except
// that -0 orders below +0; on the fast path that can only change the sign of
// a zero, which cannot reach a nonzero sum (see above), and non-finite inputs
// are recomputed literally.
__device__ __forceinline__ long long key(double x) {  // order-preserving integer image
  const long long b = dbits(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ bool nz(double x) { return (dbits(x) & 0x7fffffffffffffffLL) != 0; }
__device__ __forceinline__ double mn(double a, double b) { return key(a) < key(b) ? a : b; }  // sw.h MIN
__device__ __forceinline__ double mx(double a, double b) { return key(a) > key(b) ? a : b; }  // sw.h MAX

// The limiters of calc.c:54-63 that compare, with the comparisons above, but
// for those whose formula half_psi writes out (2, 4, 5, 6 and the safe Van Leer).
template <int SCH>
__device__ __forceinline__ double limiter_fast(double r) {
  if constexpr (SCH == 0) return mx(0.0, mn(mn(HALF(1 + r), TWICE(r)), 2.0));
  else if constexpr (SCH == 1) return mx(mx(0.0, mn(TWICE(r), 1.0)), mx(0.0, mn(r, 2.0)));
  else if constexpr (SCH == 7) return mx(0.0, mn(mn(2.0, TWICE(r)), mn(0.25 + 0.75 * r, 0.75 + QUARTER(r))));
  else return limiter<SCH>(r);
}

// Operands of the integer-pipe quotients and products.
constexpr unsigned long long kSign = 0x8000000000000000ULL;
__device__ __forceinline__ unsigned long long mag(double x) {
  return (unsigned long long)dbits(x) & 0x7fffffffffffffffULL;
}
__device__ __forceinline__ unsigned hi_word(double x) { return (unsigned)((unsigned long long)dbits(x) >> 32); }
__device__ __forceinline__ bool usable(double x) { return in_window(hi_word(x)); }
// the upper word of |x|, and of 2^k
__device__ __forceinline__ unsigned hi_mag(double x) { return hi_word(x) & 0x7fffffffu; }
#define HI_POW2(k) ((unsigned)(1023 + (k)) << 20)
// zero, or 2^-850 <= |x| < 2^100
__device__ __forceinline__ bool in_range(double x) {
  return hi_mag(x) - HI_POW2(-850) < (950u << 20) || !nz(x);
}
__device__ __forceinline__ double from_bits(unsigned long long b) { return __longlong_as_double((long long)b); }
// p ? a : b, opaque: one operation on the selected value stays one FP64
// instruction (the compiler would evaluate it for both and select after).
__device__ __forceinline__ double pick(bool p, double a, double b) {
  long long r;
  asm("mov.b64 %0, %1;" : "=l"(r) : "l"(p ? __double_as_longlong(a) : __double_as_longlong(b)));
  return __longlong_as_double(r);
}
// x with its sign bit changed by `neg` (0 or the sign bit), on the integer
// pipe: the compiler's negation of a double is an FP64 addition.
__device__ __forceinline__ double flip(double x, unsigned long long neg) {
  return __longlong_as_double(dbits(x) ^ (long long)neg);
}
__device__ __forceinline__ unsigned long long sign_of(double x) {
  return (unsigned long long)dbits(x) & kSign;
}

// A row metric as a divisor: its bits and its reciprocal (sig_recip).
struct Metric {
  unsigned long long b, y;
};
__device__ __forceinline__ Metric metric(const DevState& s, int t, int ty, int j) {
  return Metric{(unsigned long long)dbits(RW(s, t, j)), (unsigned long long)dbits(RW(s, ty, j))};
}
#define METRIC(NAME, j) metric(s, R_##NAME, R_Y##NAME, j)

// Products and quotients of any operands, on the integer pipe when the
// operands are of magnitude 2^-255 .. 2^257 (the result is then normal), on
// the FP64 unit, out of line, otherwise. A zero times a factor is a zero: the
// factors are finite (DevState::finite; without it k_hyper_add and k_pres_sum
// take plain FP64 in every step: asking here costs flows from rest 1.5 %).
__device__ __forceinline__ bool mid(double x) { return ((hi_word(x) - 0x30000000u) & 0x60000000u) == 0; }
// 2^-700 (2^-850) <= |x| < 2^257: times a factor of 2^-255 (2^-130) or more
// still normal, and over a metric factor
__device__ __forceinline__ bool wide(double x) { return hi_mag(x) - HI_POW2(-700) < (957u << 20); }
__device__ __forceinline__ bool wider(double x) { return hi_mag(x) - HI_POW2(-850) < (1107u << 20); }
__device__ __noinline__ double mul_fp64(double a, double b) { return a * b; }
__device__ __forceinline__ double smul(double a, double b) {
  if (mid(a) && mid(b)) return from_bits(sig_mul(mag(a), mag(b)) | ((unsigned long long)(dbits(a) ^ dbits(b)) & kSign));
  return mul_fp64(a, b);
}
// k: a factor of which `ok` (DevState::lap_ok, nu_ok) says that it is of
// magnitude 2^-130 .. 2^250.
__device__ __forceinline__ double rmul(bool ok, double k, double a) {
  const unsigned long long sg = (unsigned long long)(dbits(a) ^ dbits(k)) & kSign;
  if (wider(a) && ok) return from_bits(sig_mul(mag(a), mag(k)) | sg);
  if (!nz(a)) return from_bits(sg);
  return mul_fp64(k, a);
}
__device__ __forceinline__ double cmul(double c, double a) {
  const unsigned long long sg = (unsigned long long)(dbits(a) ^ dbits(c)) & kSign;
  if (wide(a) && mid(c)) return from_bits(sig_mul(mag(a), mag(c)) | sg);
  if (!nz(a)) return from_bits(sg);
  return mul_fp64(c, a);
}
__device__ __noinline__ double div_fp64(double a, double b) { return a / b; }
// a / x.b (x.b > 0): a zero gives itself.
__device__ __forceinline__ double mdiv(const DevState& s, double a, const Metric& x) {
  if (wider(a) && s.sig_ok) return from_bits(sig_div_known(mag(a), x.b, x.y) | sign_of(a));
  if (!nz(a)) return a;
  return div_fp64(a, from_bits(x.b));
}

// (a*(b*2^kx))/X + (a*(c*2^ky))/Y of zero or in-range a, b, c (kx20 = kx << 20,
// kx 0 or -1, and ky alike: the scalings are exact). Where a product could be
// subnormal, on the FP64 unit, out of line.
__device__ __forceinline__ double scaled(double b, unsigned k20) {
  return nz(b) ? from_bits((unsigned long long)dbits(b) + ((unsigned long long)k20 << 32)) : b;
}
__device__ __noinline__ double two_products_fp64(double a, double b, double x, double c, double y) {
  return zdiv(a * b, x) + zdiv(a * c, y);
}
__device__ __forceinline__ double product_over(double a, double b, unsigned k20, const Metric& x) {
  const unsigned long long q = sig_div_known(sig_mul(mag(a), mag(b), k20), x.b, x.y);
  return (nz(a) && nz(b)) ? from_bits(q | (sign_of(a) ^ sign_of(b))) : 0.0;
}
__device__ __forceinline__ double two_products(double a, double b, unsigned kx20, const Metric& X, double c,
                                               unsigned ky20, const Metric& Y) {
  if (min(hi_mag(a) - 1, min(hi_mag(b) - 1, hi_mag(c) - 1)) < HI_POW2(-450) - 1) {  // zeros wrap
    // both products below 2^-1076: zeros, whose signs do not matter
    if ((hi_mag(a) >> 20) + (max(hi_mag(b), hi_mag(c)) >> 20) < 969u) return 0.0;
    return two_products_fp64(a, scaled(b, kx20), from_bits(X.b), scaled(c, ky20), from_bits(Y.b));
  }
  return product_over(a, b, kx20, X) + product_over(a, c, ky20, Y);
}

// a/b on the integer pipe where both are usable (the quotient is then normal),
// a zero numerator from the bits; otherwise on the FP64 unit, out of line.
__device__ __noinline__ double quotient_fp64(double a, double b) { return zdiv(a, b); }
__device__ __forceinline__ double quotient(double a, double b) {
  if (usable(a) && usable(b)) return from_bits(sig_div(mag(a), mag(b)) | (sign_of(a) ^ sign_of(b)));
  return quotient_fp64(a, b);
}

// Half the limited slope factor: 0.5*limiter(n/d), n/d read as 0 for d = 0
// (calc.c:42-47), of zero or in-range differences. The limiters whose formula
// divides take that quotient on the integer pipe too.
template <int SCH>
__device__ __forceinline__ double half_psi(double n, double d) {
  const bool zero = !nz(d) || !nz(n);
  const unsigned long long q = sig_div(mag(n), mag(d)) | (sign_of(n) ^ sign_of(d));
  if constexpr (SCH == 2) {  // min(r, 1): a negative r has a negative image
    const long long m = (long long)q < dbits(1.0) ? (long long)q : dbits(1.0);
    return zero ? 0.0 : __longlong_as_double(m - (1LL << 52));
  }
  const double r = zero ? 0.0 : from_bits(q);
  if constexpr (SCH == 4) {
    const double r2 = TWICE(r);
    return HALF(mx(0.0, mn(r2, mn(quotient(1 + r2, 3.0), 2.0))));
  } else if constexpr (SCH == 5) {
    return HALF(quotient(1.5 * (r * r + r), r * r + r + 1.0));
  } else if constexpr (SCH == 6) {
    return HALF(quotient(r * r + r, r * r + 1.0));
  } else if constexpr (SCH == kVanLeerSafe) {
    return (dbits(r) == dbits(-1.0)) ? 0.0 : HALF(quotient(r + fabs(r), 1.0 + r));
  } else {
    return HALF(limiter_fast<SCH>(r));
  }
}

// The velocity of a face: one (calc.c:72-79) or the sum of two to be averaged
// (calc.c:170-177), w; the side in use is + (pos) or -, none when !act; `both`
// if the two have opposite signs, each then using one side.
struct Vel {
  double w, a, b;
  bool pos, act, both;
};
__device__ __forceinline__ Vel vel_one(double a) { return Vel{a, 0.0, 0.0, dbits(a) >= 0 || !nz(a), nz(a), false}; }
__device__ __forceinline__ Vel vel_pair(double a, double b, double sum) {
  Vel v;
  v.w = sum;
  v.a = a;
  v.b = b;
  v.both = (dbits(a) ^ dbits(b)) < 0 && nz(a) && nz(b);
  v.act = nz(sum) || v.both;
  v.pos = v.both || dbits(sum) >= 0 || !nz(sum);
  return v;
}
// Shared part of a face q0|q1. p: magnitude bits of the used side's numerator
// 0.5(...+-|...|)*Dt; hp: half its limited slope factor; p2, hp2: those of
// the - side when both are in use.
struct Face {
  double d, q0, q1, hp, hp2;
  unsigned long long p, p2;
  bool pos, act, both;
};
// PAIR: w is a sum of two velocities, to be halved. n1: q0 - qm when v.pos,
// q2 - q1 otherwise; n2(): the other of the two. bad is set where a skipped
// side might not be finite (both are skipped without a velocity).
template <int SCH, bool PAIR, typename N2>
__device__ __forceinline__ Face make_face(const Vel& v, double d, double n1, N2 n2, double q0, double q1,
                                          unsigned long long dt, bool& bad) {
  constexpr unsigned K = PAIR ? 0xfff00000u : 0u;  // exponent of the halving
  Face F;
  F.d = d;
  F.q0 = q0;
  F.q1 = q1;
  F.pos = v.pos;
  F.act = v.act;
  F.both = v.both;
  F.hp = half_psi<SCH>(n1, d);
  if (hi_mag(d) < HI_POW2(-397) && nz(d)) {
    bad = bad || hi_mag(n2()) >= hi_mag(d) + (490u << 20);
    if constexpr (SCH == 5 || SCH == 6) bad = bad || (!v.act && hi_mag(n1) >= hi_mag(d) + (490u << 20));
  }
  F.p = sig_mul(mag(v.w), dt, K);
  F.hp2 = 0.0;
  F.p2 = 0;
  if constexpr (PAIR) {
    if (__any_sync(FULL, v.both)) {
      if (v.both) {
        const bool apos = dbits(v.a) > 0;
        F.p = sig_mul(mag(apos ? v.a : v.b), dt, K);
        F.p2 = sig_mul(mag(apos ? v.b : v.a), dt, K);
        F.hp2 = half_psi<SCH>(n2(), d);
      }
    }
  }
  return F;
}

// (hp*g)*d, rounded twice as written. On the
// integer pipe: k_adv_u at 2048x1024 0.146 ms with both products on the FP64
// unit, 0.136 with one of them, 0.133 with none (the mass body 0.118, 0.109,
// 0.101); c*B, whose B may be anything, stays there.
// bad is set where a factor or a product is not a normal number, g = 1 - c = 0
// (a Courant number of exactly 1) among them. d is in range, and |hp*d| at
// most the larger of |d| and half the ratio's numerator, at most 2^101.
__device__ __forceinline__ double slope_term(double hp, double g, double d, bool& bad) {
  const unsigned long long sg = (unsigned long long)(dbits(hp) ^ dbits(g) ^ dbits(d)) & kSign;
  const bool zero = !nz(hp) || !nz(d);
  bad = bad || (!zero && sig_mul3_far(hi_mag(hp), hi_mag(g), hi_mag(d)));
  return zero ? 0.0 : from_bits(sig_mul3(mag(hp), mag(g), mag(d)) | sg);
}
// C*B of one side with c = |C|: B2BP (pos) = q0 + psi*0.5*(1-c)*(q1-q0), or
// B2BM = q1 - psi*0.5*(1-c)*(q1-q0) (C- = -c; q1 - X = q1 + (-X) exactly).
__device__ __forceinline__ double side_term(bool pos, unsigned long long p, const Metric& dx, double hp, double q0,
                                            double q1, double d, bool& bad) {
  const double c = from_bits(sig_div_known(p, dx.b, dx.y));
  const double X = slope_term(hp, 1.0 - c, d, bad);
  const unsigned long long neg = pos ? 0 : kSign;
  return flip(c * (pick(pos, q0, q1) + flip(X, neg)), neg);
}

// A face's terms as seen by one cell: that of the side in use (0 when none
// is), and the - side's when both are.
struct Side {
  double t, m;
  bool pos, both;
};
template <bool PAIR>
__device__ __forceinline__ Side side_of(const Face& F, const Metric& dx, bool& bad) {
  Side r;
  bool far = false;  // says nothing of a face that is not in use
  const double t = side_term(F.pos, F.p, dx, F.hp, F.q0, F.q1, F.d, far);
  r.t = F.act ? t : 0.0;
  bad = bad || (F.act && far);
  r.m = 0.0;
  r.pos = F.pos;
  r.both = F.both;
  if constexpr (PAIR) {
    if (__any_sync(FULL, F.both)) {
      if (F.both) r.m = side_term(false, F.p2, dx, F.hp2, F.q0, F.q1, F.d, bad);
    }
  }
  return r;
}

// calc.c:100 over the four faces: +wP +wM -eP -eM +sP +sM -nP -nM. Unless a
// face of the warp's cells uses both sides, each face has one term and the sum
// takes three additions; otherwise all eight are summed, out of line so that
// the common case does not carry the extra FP64 operations.
__device__ __noinline__ double sum_faces8(double wP, double wM, double eP, double eM, double sP, double sM,
                                          double nP, double nM) {
  double S = wP + wM;
  S = S - eP;
  S = S - eM;
  S = S + sP;
  S = S + sM;
  S = S - nP;
  S = S - nM;
  return S;
}
// Whether the reference's first term, C+*B of the west face qm | q0 | q1, is
// +0 when it is a zero: C+ is +0 or positive, so its sign is that of the face
// value B = q0 + X. If the + side is in use, t is that term. Otherwise C+ is
// +0, X is a zero where q1 = q0, and |X| <= |q1-q0| + |q0-qm| for every limiter
// (|psi(r)| <= 2 + |r|).
__device__ __forceinline__ bool first_term_plus_zero(bool act, bool pos, double t, double qm, double q0, double q1) {
  if (dbits(q0) == (long long)kSign) return false;  // -0 + X: the sign of X's zero matters
  if (act && pos) return dbits(t) >= 0;
  if (dbits(q0) < 0) return false;
  const double d = q1 - q0, n = q0 - qm;
  if (!nz(d)) return true;
  return max(hi_mag(d), hi_mag(n)) + (3u << 20) <= hi_word(q0);
}

// The sum for the lane's cell: w its west face (whose east neighbour's is taken
// from the next lane), so and n its south and north faces; slow: a zero sum
// whose sign only the literal expression tells. act, qm, q0, q1: the west
// face's, for that question.
template <bool PAIR>
__device__ __forceinline__ double sum_faces(const Side& w, const Side& so, const Side& n, int lane, bool act,
                                            double qm, double q0, double q1, bool& slow) {
  const double te = __shfl_sync(FULL, w.t, (lane + 1) & 31);
  if constexpr (PAIR) {
    if (__any_sync(FULL, w.both || so.both || n.both)) {
      const double me = __shfl_sync(FULL, w.m, (lane + 1) & 31);
      const bool epos = __shfl_sync(FULL, (int)w.pos, (lane + 1) & 31) != 0;
      const double S = sum_faces8(w.pos ? w.t : 0.0, w.pos ? w.m : w.t, epos ? te : 0.0, epos ? me : te,
                                  so.pos ? so.t : 0.0, so.pos ? so.m : so.t, n.pos ? n.t : 0.0, n.pos ? n.m : n.t);
      slow = !nz(S);
      return S;
    }
  }
  const double S = ((w.t - te) + so.t) - n.t;
  slow = false;
  if (!nz(S)) {
    slow = !nz(w.t) && !nz(te) && !nz(so.t) && !nz(n.t) && !first_term_plus_zero(act, w.pos, w.t, qm, q0, q1);
    return 0.0;  // -0 where the terms are -0, +0, -0 and +0; the literal sum starts at +0 and stays there
  }
  return S;
}

// Values of the lane's x neighbours at one row: own value v of column i,
// aux = the value of column base-2 (lane 0), base-1 (lane 1) or base+32 (lane 31).
struct XN {
  double m2, m1, p1;
};
__device__ __forceinline__ XN x_neighbours(double v, double aux, int lane) {
  XN n;
  n.m2 = __shfl_sync(FULL, v, (lane + 30) & 31);
  n.m1 = __shfl_sync(FULL, v, (lane + 31) & 31);
  n.p1 = __shfl_sync(FULL, v, (lane + 1) & 31);
  const double a1 = __shfl_sync(FULL, aux, 1);
  if (lane < 2) n.m2 = aux;
  if (lane == 0) n.m1 = a1;
  if (lane == 31) n.p1 = aux;
  return n;
}
// The face west of the lane's column from its x neighbours: q0 = m1, q1 = v.
template <int SCH, bool PAIR>
__device__ __forceinline__ Face x_face(const Vel& vel, const XN& n, double v, unsigned long long dt, bool& bad) {
  const double n1 = pick(vel.pos, n.m1, n.p1) - pick(vel.pos, n.m2, v);
  auto n2 = [&]() { return pick(vel.pos, n.p1, n.m1) - pick(vel.pos, v, n.m2); };
  return make_face<SCH, PAIR>(vel, v - n.m1, n1, n2, n.m1, v, dt, bad);
}
// The face between rows with differences dm, d, d1 (below, across, above): q0 | q1.
template <int SCH, bool PAIR>
__device__ __forceinline__ Face y_face(const Vel& vel, double dm, double d, double d1, double q0, double q1,
                                       unsigned long long dt, bool& bad) {
  auto n2 = [&]() { return vel.pos ? d1 : dm; };
  return make_face<SCH, PAIR>(vel, d, vel.pos ? dm : d1, n2, q0, q1, dt, bad);
}

// A strip is 31 columns x s.fk rows (chosen per launch, see fast_launch).
// The warps of the grid (the resident warps) take strips from a queue, the
// next strip index being an atomic counter: a warp that finishes early takes
// more, so the SMs finish together. The last warp of the launch to find the
// queue empty sets both counters back to zero for the next launch (every
// other warp has made its last fetch by then). No warp ever waits.
__device__ __forceinline__ int next_strip(unsigned* q, int lane) {
  unsigned v = 0;
  if (lane == 0) v = atomicAdd(q, 1u);
  return (int)__shfl_sync(FULL, v, 0);
}
__device__ __forceinline__ void strips_done(unsigned* q, int lane) {
  if (lane == 0 && atomicAdd(q + 1, 1u) == gridDim.x * (blockDim.x >> 5) - 1) {
    atomicExch(q, 0u);
    atomicExch(q + 1, 0u);
  }
}
#define STRIP_SETUP                                                                         \
  const int W = s.W, nx = s.nx, ny = s.ny;                                                  \
  const int FK = s.fk;                                                                      \
  const int nsx = (nx + FW - 1) / FW;                                                       \
  const double Dt = s.Dt;                                                                   \
  const unsigned long long dt = (unsigned long long)dbits(Dt);                              \
  const int j0 = (strip / nsx) * FK + 1;                                                    \
  const int jn = min(j0 + FK - 1, ny);                                                      \
  const int base = (strip % nsx) * FW + 1;                                                  \
  const int i = base + lane;                                                                \
  const int ic = min(i, nx + 2);                                                            \
  const int ia = (lane == 0) ? base - 2 : (lane == 1) ? base - 1 : min(base + 32, nx + 2);  \
  const bool own = (lane < FW) && (i <= nx);
// Field values of the fast bodies. PL (plain form): windx, windy and hB are
// +0.0 everywhere, so x - hB = x exactly, and u + windx = u except that -0
// becomes +0, which the fast path cannot tell apart (see (3) above).
#define UF(i, j) (PL ? f.u[IX(W, i, j)] : UW(i, j))
#define VF(i, j) (PL ? f.v[IX(W, i, j)] : VW(i, j))
#define HF(i, j) (PL ? (f.eta[IX(W, i, j)] + s.depth) : HH(i, j))

// BODYH + damping, fast form.
template <int SCH, bool PL, bool UD>
__device__ __forceinline__ void mass_strip(const DevState& s, const F7& f, double* out, int strip, int lane) {
  STRIP_SETUP
  const int iu = min(i - 1, nx + 2);
  const double damp = 2.0 * Dt * (s.sigma);  // calc.c:112: (2.0*Dt*sigma)*ETA
  // H at this lane's column, rows j and j+1, the differences of rows j-1 .. j+1,
  // and the face south of j0
  double h2 = HF(ic, j0), h3 = HF(ic, j0 + 1), dm, d0;
  bool bad = !in_range(h2) || !in_range(h3);  // any value of the strip so far out of range
  // UD (no damping: sigma = 0, a band): the product damp*eta is a zero (eta is
  // finite on the fast path), and a nonzero S minus a zero is S
  Side ts;
  {
    const double h0 = HF(ic, j0 - 2), h1 = HF(ic, j0 - 1);
    bad = bad || !in_range(h0) || !in_range(h1);
    const double vs = VF(ic, j0 - 1);
    bad = bad || !in_range(vs);
    const Vel b = vel_one(vs);
    dm = h2 - h1;
    d0 = h3 - h2;
    const Face F = y_face<SCH, false>(b, h1 - h0, dm, d0, h1, h2, dt, bad);
    ts = side_of<false>(F, METRIC(DYN, j0), bad);
  }
  for (int j = j0; j <= jn; j++) {
    const double h4 = HF(ic, j + 2), ha = HF(ia, j);
    const double d1 = h4 - h3;
    bad = bad || !in_range(h4) || !in_range(ha);
    // x face west of column i, row j
    const double a = UF(iu, j);
    const XN xn = x_neighbours(h2, ha, lane);
    const Face FX = x_face<SCH, false>(vel_one(a), xn, h2, dt, bad);
    const Side tw = side_of<false>(FX, METRIC(DXE, j), bad);
    // y face north of row j: shared by this cell and the cell above
    const double vn = VF(ic, j);
    bad = bad || !in_range(a) || !in_range(vn);
    const Vel b = vel_one(vn);
    const Face FY = y_face<SCH, false>(b, dm, d0, d1, h2, h3, dt, bad);
    const Side tn = side_of<false>(FY, METRIC(DYN, j), bad);
    const Side ns = side_of<false>(FY, METRIC(DYN, j + 1), bad);
    bool slow;
    const double S = sum_faces<false>(tw, ts, tn, lane, FX.act, xn.m2, xn.m1, h2, slow);  // calc.c:100 in its order: +w -e +s -n
    slow = __any_sync(FULL, bad) || slow;
    if (own) {
      double r;
      if (slow) r = mass_cell_ool<SCH>(s, f, i, j);
      else if (UD) r = S;
      else r = S - (s.polar ? 2.0 * Dt * PF(s, P_SH, IX(W, i, j)) : damp) * f.eta[IX(W, i, j)];
      out[IX(W, i, j)] = r;
    }
    ts = ns;
    h2 = h3;
    h3 = h4;
    dm = d0;
    d0 = d1;
  }
}

// BODYTRACER, fast form (calc.c:117-163).
template <int SCH, bool PL>
__device__ __forceinline__ void tracer_strip(const DevState& s, const F7& f, double* out, int strip, int lane) {
  STRIP_SETUP
  const int iu = min(i - 1, nx + 2);
  const double damp = 2.0 * Dt * (s.sigma_tr);  // calc.c:161
  double h2 = f.tr[IX(W, ic, j0)], h3 = f.tr[IX(W, ic, j0 + 1)], dm, d0;
  bool bad = !in_range(h2) || !in_range(h3);
  double vs = VF(ic, j0 - 1);
  Side ts;
  {
    const double h0 = f.tr[IX(W, ic, j0 - 2)], h1 = f.tr[IX(W, ic, j0 - 1)];
    bad = bad || !in_range(h0) || !in_range(h1) || !in_range(vs);
    const Vel b = vel_one(vs);
    dm = h2 - h1;
    d0 = h3 - h2;
    const Face F = y_face<SCH, false>(b, h1 - h0, dm, d0, h1, h2, dt, bad);
    ts = side_of<false>(F, METRIC(DYN, j0), bad);
  }
  for (int j = j0; j <= jn; j++) {
    const double h4 = f.tr[IX(W, ic, j + 2)], ha = f.tr[IX(W, ia, j)];
    const double d1 = h4 - h3;
    bad = bad || !in_range(h4) || !in_range(ha);
    const double a = UF(iu, j);
    const Metric mx = METRIC(DXE, j), my = METRIC(DYN, j);
    const XN xn = x_neighbours(h2, ha, lane);
    const Face FX = x_face<SCH, false>(vel_one(a), xn, h2, dt, bad);
    const Side tw = side_of<false>(FX, mx, bad);
    const double vn = VF(ic, j);
    bad = bad || !in_range(a) || !in_range(vn);
    const Vel b = vel_one(vn);
    const Face FY = y_face<SCH, false>(b, dm, d0, d1, h2, h3, dt, bad);
    const Side tn = side_of<false>(FY, my, bad);
    const Side ns = side_of<false>(FY, METRIC(DYN, j + 1), bad);
    bool slow;
    const double S = sum_faces<false>(tw, ts, tn, lane, FX.act, xn.m2, xn.m1, h2, slow);
    slow = __any_sync(FULL, bad) || slow;
    // Dt*TRACER*(UW(E)-UW(W))/DXE + Dt*TRACER*(VW(N)-VW(S))/DYN (calc.c:146-149)
    const double du = __shfl_sync(FULL, a, (lane + 1) & 31) - a, dv = vn - vs, tt = Dt * h2;
    const double p2 = two_products(tt, du, 0, mx, dv, 0, my);
    if (own) {
      double r;
      if (slow) r = tracer_cell_ool<SCH>(s, f, i, j);
      else r = (S + p2) - (s.polar ? 2.0 * Dt * PF(s, P_STR, IX(W, i, j)) : damp) * h2;
      out[IX(W, i, j)] = r;
    }
    ts = ns;
    vs = vn;
    h2 = h3;
    h3 = h4;
    dm = d0;
    d0 = d1;
  }
}

// BODYU, fast form.
template <int SCH, bool PL>
__device__ __forceinline__ void adv_u_strip(const DevState& s, const F7& f, double* out, int strip, int lane) {
  STRIP_SETUP
  const int ic1 = min(i + 1, nx + 2);
  // U at this lane's column, rows j and j+1, the differences of rows j-1 .. j+1,
  // and the sum of V at columns i, i+1 of row j-1
  double u2 = UF(ic, j0), u3 = UF(ic, j0 + 1), dm, d0, vs;
  bool bad = !in_range(u2) || !in_range(u3);
  Side ts;
  {
    const double u0 = UF(ic, j0 - 2), u1 = UF(ic, j0 - 1), a = VF(ic, j0 - 1), b = VF(ic1, j0 - 1);
    bad = bad || !in_range(u0) || !in_range(u1) || !in_range(a);
    vs = a + b;
    const Vel v = vel_pair(a, b, vs);
    dm = u2 - u1;
    d0 = u3 - u2;
    const Face F = y_face<SCH, true>(v, u1 - u0, dm, d0, u1, u2, dt, bad);
    ts = side_of<true>(F, METRIC(DYV, j0), bad);
  }
  for (int j = j0; j <= jn; j++) {
    const double u4 = UF(ic, j + 2), ua = UF(ia, j);
    const double d1 = u4 - u3;
    bad = bad || !in_range(u4) || !in_range(ua);
    // x face west of column i, row j: velocities u(i-1), u(i)
    const XN xn = x_neighbours(u2, ua, lane);
    const Face FX = x_face<SCH, true>(vel_pair(xn.m1, u2, xn.m1 + u2), xn, u2, dt, bad);
    const Side tw = side_of<true>(FX, METRIC(DXC, j), bad);
    // y face north of row j: velocities v(i, j), v(i+1, j)
    const double va = VF(ic, j), vb = VF(ic1, j), vn = va + vb;
    bad = bad || !in_range(va);  // vb is the next lane's
    const Metric my = METRIC(DYV, j);
    const Vel v = vel_pair(va, vb, vn);
    const Face FY = y_face<SCH, true>(v, dm, d0, d1, u2, u3, dt, bad);
    const Side tn = side_of<true>(FY, my, bad);
    const Side ns = side_of<true>(FY, METRIC(DYV, j + 1), bad);
    bool slow;
    const double S = sum_faces<true>(tw, ts, tn, lane, FX.act, xn.m2, xn.m1, u2, slow);
    slow = __any_sync(FULL, bad) || slow;
    // calc.c:198: u0*(uep-uwm)/(2 DXE) + u0*((vn0+vn1)/2 - (vs0+vs1)/2)/DYV; the
    // halving commutes with the difference (its operands are zero or at least 2^-902)
    const double ux = xn.p1 - xn.m1, vy = vn - vs;
    const double p2 = Dt * two_products(u2, ux, 0, METRIC(DXE2, j), vy, 0xfff00000u, my);
    if (own) {
      double r;
      if (slow) r = advu_cell_ool<SCH>(s, f, i, j);
      else r = S + p2;
      out[IX(W, i, j)] = r;
    }
    ts = ns;
    vs = vn;
    u2 = u3;
    u3 = u4;
    dm = d0;
    d0 = d1;
  }
}

// BODYV, fast form.
template <int SCH, bool PL>
__device__ __forceinline__ void adv_v_strip(const DevState& s, const F7& f, double* out, int strip, int lane) {
  STRIP_SETUP
  const int iu = min(i - 1, nx + 2);
  // V at this lane's column, rows j-1 .. j+1, the differences of rows j-1 ..
  // j+1; U at column i-1, row j
  double v1 = VF(ic, j0 - 1), v2 = VF(ic, j0), v3 = VF(ic, j0 + 1), dm, d0;
  double uw0 = UF(iu, j0);
  bool bad = !in_range(v1) || !in_range(v2) || !in_range(v3) || !in_range(uw0);
  Side ts;
  {
    const double v0 = VF(ic, j0 - 2);
    bad = bad || !in_range(v0);
    const Vel v = vel_pair(v1, v2, v1 + v2);
    dm = v2 - v1;
    d0 = v3 - v2;
    const Face F = y_face<SCH, true>(v, v1 - v0, dm, d0, v1, v2, dt, bad);
    ts = side_of<true>(F, METRIC(DYC, j0), bad);
  }
  for (int j = j0; j <= jn; j++) {
    const double v4 = VF(ic, j + 2), va = VF(ia, j);
    const double d1 = v4 - v3;
    bad = bad || !in_range(v4) || !in_range(va);
    const double uw1 = UF(iu, j + 1), uw = uw1 + uw0;
    bad = bad || !in_range(uw1);
    const Metric mx = METRIC(DXV, j);
    // x face west of column i, row j: velocities u(i-1, j+1), u(i-1, j)
    const XN xn = x_neighbours(v2, va, lane);
    const Face FX = x_face<SCH, true>(vel_pair(uw1, uw0, uw), xn, v2, dt, bad);
    const Side tw = side_of<true>(FX, mx, bad);
    // y face north of row j: velocities v(i, j), v(i, j+1)
    const Vel v = vel_pair(v2, v3, v2 + v3);
    const Face FY = y_face<SCH, true>(v, dm, d0, d1, v2, v3, dt, bad);
    const Side tn = side_of<true>(FY, METRIC(DYC, j), bad);
    const Side ns = side_of<true>(FY, METRIC(DYC, j + 1), bad);
    bool slow;
    const double S = sum_faces<true>(tw, ts, tn, lane, FX.act, xn.m2, xn.m1, v2, slow);
    slow = __any_sync(FULL, bad) || slow;
    // calc.c:235: v0*((ue0+ue1)/2 - (uw0+uw1)/2)/DXV + v0*(vnp-vsm)/(DYN+DYN), the
    // sums of u symmetric in their operands
    const double ue = __shfl_sync(FULL, uw, (lane + 1) & 31);
    const double ux = ue - uw, vy = v3 - v1;
    const Metric ms = METRIC(DYNS, j);
    slow = slow || ms.y == 0;  // row ny, where DYN(ny+1) lies beyond the pole
    const double p2 = Dt * two_products(v2, ux, 0xfff00000u, mx, vy, 0, ms);
    if (own) {
      double r;
      if (slow) r = advv_cell_ool<SCH>(s, f, i, j);
      else r = S + p2;
      out[IX(W, i, j)] = r;
    }
    ts = ns;
    uw0 = uw1;
    v1 = v2;
    v2 = v3;
    v3 = v4;
    dm = d0;
    d0 = d1;
  }
}
#undef STRIP_SETUP
#undef UF
#undef VF
#undef HF
// Self-check of the step's products and quotients: for each divisor b (recip:
// its sig_recip), `samples` numerators a drawn from a SplitMix64 stream (random
// significands over exponents 2^-950..2^60, both signs, and numerators whose
// quotient lies within a few ulps of a rounding midpoint), compared bit for
// bit with IEEE: a/b by div_rcp, and the integer-pipe operations on a and b
// (sig_mismatches); and the reciprocals that sig_div starts from, all 2^23.
__device__ __forceinline__ unsigned long long splitmix(unsigned long long& x) {
  unsigned long long z = (x += 0x9E3779B97F4A7C15ULL);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

__global__ void k_check_division(const double* div, const unsigned long long* recip, int n, long long samples,
                                 unsigned long long seed, unsigned long long* bad) {
  const long long total = (long long)n * samples;
  unsigned long long miss = 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const double b = div[t / samples];
    const double y = 1.0 / b;
    unsigned long long st = seed ^ (unsigned long long)t * 0xD1B54A32D192ED03ULL;
    const unsigned long long r1 = splitmix(st), r2 = splitmix(st);
    double a;
    if (r2 & 1) {  // random significand and exponent
      const unsigned long long e = 73 + (r2 >> 1) % 1010;  // 2^-950 .. 2^59
      a = __longlong_as_double((long long)((e << 52) | (r1 & 0xFFFFFFFFFFFFFULL) | (r2 & 2 ? 1ULL << 63 : 0)));
    } else {  // a = b * (q + half an ulp of q + small offset): quotient near a midpoint
      const unsigned long long e = 523 + (r2 >> 1) % 500;
      const double q = __longlong_as_double((long long)((e << 52) | (r1 & 0xFFFFFFFFFFFFFULL)));
      const double h = __longlong_as_double((long long)(((e - 53) << 52))) * (double)(((r2 >> 10) & 7) + 1) * 0.5;
      a = __dmul_rn(b, q + h);
    }
    const double want = a / b, got = div_rcp(a, b, y);
    if (dbits(want) != dbits(got)) miss++;
    miss += sig_mismatches(a, b, recip[t / samples]);
  }
  // every divisor against the numerators +-(2 - k ulp), k = 1..512: with the
  // divisor's significand also within a few ulps of 2 these are the pairs
  // where RN(a*y) strays more than one ulp from a/b and a wrong rounding is
  // not excluded by the case analysis alone
  const long long grid = (long long)n * 1024;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < grid;
       t += (long long)gridDim.x * blockDim.x) {
    const double b = div[t >> 10];
    const double y = 1.0 / b;
    const unsigned long long k = (unsigned long long)(t & 511), neg = (unsigned long long)((t >> 9) & 1);
    const double a = __longlong_as_double((long long)((0x3FFFFFFFFFFFFFFFULL - k) | (neg << 63)));
    const double want = a / b, got = div_rcp(a, b, y);
    if (dbits(want) != dbits(got)) miss++;
    miss += sig_mismatches(a, b, recip[t >> 10]);
  }
  for (unsigned u = blockIdx.x * blockDim.x + threadIdx.x; u < (1u << 23); u += gridDim.x * blockDim.x)
    if (!sig_rcp_close(__uint_as_float(0x3f800001u + u))) miss++;
  if (miss) atomicAdd(bad, miss);
}

// Self-check of sadd and ssub against the FP64 unit: operand pairs from a
// SplitMix64 stream, in classes that reach every branch of the adder: any two
// normal numbers; exponents within 64 of each other (alignment, carries,
// cancellation); b = -a give or take a few ulps (total and near-total
// cancellation); b a tie (an odd multiple of half an ulp of a); sums near
// the overflow and subnormal limits; zeros, subnormals, inf and NaN.
__device__ __forceinline__ double rnd_double(unsigned long long r, int e, bool neg) {
  return __longlong_as_double((long long)(((unsigned long long)e << 52) | (r & 0xFFFFFFFFFFFFFULL) |
                                          (neg ? 1ULL << 63 : 0ULL)));
}
__global__ void k_check_add(long long samples, unsigned long long seed, unsigned long long* bad) {
  unsigned long long miss = 0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < samples;
       t += (long long)gridDim.x * blockDim.x) {
    unsigned long long st = seed ^ (unsigned long long)t * 0xD1B54A32D192ED03ULL;
    const unsigned long long r1 = splitmix(st), r2 = splitmix(st), r3 = splitmix(st);
    const int cls = (int)(r3 % 8);
    double a, b;
    if (cls == 0) {
      a = rnd_double(r1, 1 + (int)((r3 >> 8) % 2046), r2 & 1);
      b = rnd_double(r2, 1 + (int)((r3 >> 20) % 2046), r2 & 2);
    } else if (cls <= 2) {
      const int e = 70 + (int)((r3 >> 8) % 1900);
      a = rnd_double(r1, e, r2 & 1);
      b = rnd_double(r2, e - (int)((r3 >> 20) % 64), r2 & 2);
    } else if (cls == 3) {
      a = rnd_double(r1, 3 + (int)((r3 >> 8) % 2040), r2 & 1);
      b = __longlong_as_double((dbits(a) ^ (long long)0x8000000000000000ULL) + (long long)((r2 >> 8) % 9) - 4);
    } else if (cls == 4) {  // |b| = k/2 ulp(a), k odd, with or without a few more low bits
      const int e = 60 + (int)((r3 >> 8) % 1900);
      a = rnd_double(r1, e, r2 & 1);
      const double k = (double)(2 * ((r2 >> 8) % 16) + 1);
      b = k * __longlong_as_double((long long)((unsigned long long)(e - 53) << 52));
      if (r2 & 4) b = __longlong_as_double(dbits(b) + (long long)((r2 >> 20) % 3) - 1);
      if (r2 & 2) b = -b;
    } else if (cls == 5) {  // near the top of the range
      a = rnd_double(r1, 2046 - (int)((r3 >> 8) % 3), r2 & 1);
      b = rnd_double(r2, 2046 - (int)((r3 >> 20) % 60), r2 & 2);
    } else if (cls == 6) {  // near the bottom: subnormal sums and operands
      a = rnd_double(r1, (int)((r3 >> 8) % 4), r2 & 1);
      b = rnd_double(r2, (int)((r3 >> 20) % 60), r2 & 2);
    } else {  // zeros, inf, NaN against anything
      const double sp[6] = {0.0, -0.0, __longlong_as_double(0x7ff0000000000000LL),
                            __longlong_as_double((long long)0xfff0000000000000ULL),
                            __longlong_as_double(0x7ff8000000000000LL), 1.0};
      a = sp[(r3 >> 8) % 6];
      b = (r2 & 1) ? sp[(r3 >> 20) % 6] : rnd_double(r2, 1 + (int)((r3 >> 24) % 2046), r2 & 2);
      if (r2 & 4) {
        const double t = a;
        a = b;
        b = t;
      }
    }
    const double s1 = a + b, s2 = sadd(a, b), d1 = a - b, d2 = ssub(a, b);
    const bool nan1 = (dbits(s1) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
    const bool nan2 = (dbits(d1) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
    if (nan1 ? !((dbits(s2) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL) : dbits(s1) != dbits(s2)) miss++;
    if (nan2 ? !((dbits(d2) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL) : dbits(d1) != dbits(d2)) miss++;
  }
  if (miss) atomicAdd(bad, miss);
}

// do_AdamsBashforth (calc.c:651-699) via copy_scaf/linop_scaf (sppde_core.c:247-298)
__global__ void k_ab(DevState s, int k, double* ab, const double* dn, const double* dm1, const double* dm2) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  if (k == 0) {
    ab[q] = dn[q];
  } else if (k == 1) {
    ab[q] = (3.0 / 2.0) * dn[q] + -(1.0 / 2.0) * dm1[q];
  } else {
    const double t = -(4.0 / 3.0) * dm1[q] + +(5.0 / 12.0) * dm2[q];
    ab[q] = (23.0 / 12.0) * dn[q] + 1.0 * t;
  }
}

// forall x += dx (core.c:175-177, 203-205)
__global__ void k_add(DevState s, double* x, const double* dx) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  x[q] = x[q] + dx[q];
}

// Writer-side halos. The reference refreshes a Laplacian field's halo with the
// single-rank update (every halo cell copies interior cell (wrap(i), wrap(j)))
// and then fixes the wall rows of the interior columns. Each halo cell's
// final value therefore comes from one interior cell (or is a constant), and
// the thread that computes that interior cell writes it:
//   x-halo columns and corners: the wrap;
//   halo rows of the interior columns, per field (band; a polar cap keeps the
//   wrap, it has no walls):
//     LE (laplacian_eta, laplacian.c:131-146): rows ny+1, ny+2 <- row ny,
//        row 0 <- row 1, row -1 <- row ny-1;
//     LU (laplacian.c:94-107): row ny+1 <- row ny, row 0 <- row 1, others wrap;
//     LV: rows ny+1 and 0 = 0, others wrap.
enum HaloKind { HK_WRAP, HK_LE, HK_LU, HK_LV };
constexpr int NOIMG = -1000000;
template <int K>
__device__ __forceinline__ void put_images(const DevState& s, double* f, int i, int j, double v) {
  const int W = s.W, nx = s.nx, ny = s.ny;
  f[IX(W, i, j)] = v;
  if (i > 2 && i < nx - 1 && j > 2 && j < ny - 1) return;
  const int xa = (i <= 2) ? i + nx : NOIMG, xb = (i >= nx - 1) ? i - nx : NOIMG;
  const int ya = (j <= 2) ? j + ny : NOIMG, yb = (j >= ny - 1) ? j - ny : NOIMG;
  if (xa != NOIMG) f[IX(W, xa, j)] = v;
  if (xb != NOIMG) f[IX(W, xb, j)] = v;
  if (ya != NOIMG) {
    if (xa != NOIMG) f[IX(W, xa, ya)] = v;
    if (xb != NOIMG) f[IX(W, xb, ya)] = v;
  }
  if (yb != NOIMG) {
    if (xa != NOIMG) f[IX(W, xa, yb)] = v;
    if (xb != NOIMG) f[IX(W, xb, yb)] = v;
  }
  if (K == HK_WRAP || s.polar != 0) {
    if (ya != NOIMG) f[IX(W, i, ya)] = v;
    if (yb != NOIMG) f[IX(W, i, yb)] = v;
  } else if (K == HK_LE) {
    if (j == ny) {
      f[IX(W, i, ny + 1)] = v;
      f[IX(W, i, ny + 2)] = v;
    }
    if (j == 1) f[IX(W, i, 0)] = v;
    if (j == ny - 1) f[IX(W, i, -1)] = v;
  } else if (K == HK_LU) {
    if (j == ny - 1) f[IX(W, i, -1)] = v;
    if (j == 1) f[IX(W, i, 0)] = v;
    if (j == ny) f[IX(W, i, ny + 1)] = v;
    if (j == 2) f[IX(W, i, ny + 2)] = v;
  } else {  // HK_LV
    if (j == ny - 1) f[IX(W, i, -1)] = v;
    if (j == 1) f[IX(W, i, 0)] = 0.0;
    if (j == ny) f[IX(W, i, ny + 1)] = 0.0;
    if (j == 2) f[IX(W, i, ny + 2)] = v;
  }
}

// laplacian_eta (laplacian.c:114-127), both passes in one: a warp takes 31
// columns and marches up `rows` rows; the psi west of a cell comes from the
// lane before (one lane more than cells), the xi south of it from the row
// before. psi and xi are zero on the halo (laplacian.c:116-118). In two
// launches, psi and xi through memory: 0.045 ms a level at 2048x1024; fused
// 0.036, and inside the eta kernel, which took 0.043 alone, 0.031.
struct LapEta {
  int c, cc;    // the lane's column, and the same kept inside the grid
  bool own;     // the lane's cell is one of the strip's
  double e0, xs;
  // rows from j0 on
  __device__ __forceinline__ void begin(const DevState& s, const double* e, int base, int j0, int lane) {
    const int W = s.W;
    c = base - 1 + lane;
    cc = min(c, s.nx);
    own = lane > 0 && c <= s.nx;
    e0 = e[IX(W, cc, j0)];
    xs = 0.0;
    if (j0 > 1) xs = mdiv(s, rmul(s.lap_ok, RW(s, R_KY, j0 - 1), e0 - e[IX(W, cc, j0 - 1)]), METRIC(DYC, j0 - 1));
  }
  // the value at row j (warp-wide)
  __device__ __forceinline__ double next(const DevState& s, const double* e, int j) {
    const int W = s.W;
    touch(e + IX(W, cc, min(j + 2, s.ny + 1)));
    const double ee = e[IX(W, cc + 1, j)], en = e[IX(W, cc, j + 1)];
    double psi = mdiv(s, rmul(s.lap_ok, RW(s, R_KX, j), ee - e0), METRIC(DXC, j));
    if (c == 0) psi = 0.0;
    const double pw = __shfl_up_sync(FULL, psi, 1);
    const double xi = mdiv(s, rmul(s.lap_ok, RW(s, R_KY, j), en - e0), METRIC(DYC, j));
    const double v = rmul(s.lap_ok, RW(s, R_KC, j), mdiv(s, psi - pw, METRIC(DXE, j)) + mdiv(s, xi - xs, METRIC(DYN, j)));
    e0 = en;
    xs = xi;
    return v;
  }
};
// One level, with its halo update and wall rows (laplacian.c:129-146): rows j0
// to jn of the 31 columns from base on.
__device__ __forceinline__ void lape_strip(const DevState& s, const double* e, double* eo, int base, int j0, int jn,
                                           int lane) {
  LapEta L;
  L.begin(s, e, base, j0, lane);
  for (int j = j0; j <= jn; j++) {
    const double v = L.next(s, e, j);
    if (L.own) put_images<HK_LE>(s, eo, L.c, j, v);
  }
}
// The first of the columns of a warp of the marching kernels' blocks.
__device__ __forceinline__ int march_base(int width) {
  return (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * width + 1;
}
__global__ void __launch_bounds__(TX, 16) k_lape(DevState s, const double* e, double* eo, int rows) {
  SW2G_PDL_ENTRY();
  const int j0 = blockIdx.y * rows + 1, base = march_base(FW);
  if (base <= s.nx) lape_strip(s, e, eo, base, j0, min(j0 + rows - 1, s.ny), threadIdx.x & 31);
}

// Deta_n += nu*Dt*L (calc.c:346-350); Du/Dv the same (core.c:258-266), with
// nu*Dt formed once on the host by the same multiplication. A term whose nu
// is a zero adds the product nudt*L, a zero when L is finite, and adding a
// zero to a finite nonzero x gives x; only a zero x (the sign of the sum) or a
// non-finite operand needs that term's arithmetic.
__device__ __forceinline__ bool zero_term_is_exact(double x, double L) {
  const long long xb = dbits(x) & 0x7fffffffffffffffLL;
  return xb != 0 && xb < 0x7ff0000000000000LL && dexp(L) != 0x7ff;
}
// Out of line, so that the rare case is a branch and not predicated FP64 work.
__device__ __noinline__ double add_product(double x, double nd, double v) { return x + nd * v; }

// NZ: bit t set when the order-t coefficient is nonzero (chosen at compile
// time: a skipped FP64 operation under a predicate still occupies the FP64 unit).
// NZ = 8: no hyperviscosity block at all (every nu zero: the reference skips it).
constexpr int kNoHyper = 8;
template <int NZ>
__device__ __forceinline__ double hyper_terms(const DevState& s, double x, double v2, double v4, double v6) {
  if constexpr (NZ == kNoHyper) {
    return x;
  } else {
    const double V[3] = {v2, v4, v6};
    const double nd[3] = {s.nu2dt, s.nu4dt, s.nu6dt};
#pragma unroll
    for (int t = 0; t < 3; t++) {
      const double v = V[t];
      if ((NZ >> t) & 1) x = x + rmul(s.nu_ok, nd[t], v);
      else if (!zero_term_is_exact(x, v)) x = add_product(x, nd[t], v);
    }
    return x;
  }
}
// The levels of Laplacian that run (calc.c:332-345); the others stay zero.
template <int NZ>
constexpr int kLevels = NZ == kNoHyper ? 0 : (NZ & 4) ? 3 : (NZ & 2) ? 2 : 1;
template <int NZ>
__device__ __forceinline__ double level(const double* l, int t, int q) {
  return t < kLevels<NZ> ? l[q] : 0.0;
}

template <int NZ>
__global__ void k_hyper_add(DevState s, double* d, const double* l2, const double* l4, const double* l6) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  if (!s.finite) {
    d[q] = d[q] + s.nu2dt * l2[q] + s.nu4dt * l4[q] + s.nu6dt * l6[q];
    return;
  }
  d[q] = hyper_terms<NZ>(s, d[q], l2[q], l4[q], l6[q]);
}

// The coefficient mask of the hyperviscosity terms (kNoHyper when every nu is zero).
int hyper_mask(const DevState& s) {
  if (s.nu2 == 0 && s.nu4 == 0 && s.nu6 == 0) return kNoHyper;
  return (s.nu2 != 0 ? 1 : 0) | (s.nu4 != 0 ? 2 : 0) | (s.nu6 != 0 ? 4 : 0);
}

void hyper_add(const DevState& s, dim3 g, cudaStream_t st, double* d, const double* l2, const double* l4,
               const double* l6) {
  const int m = (s.nu2dt != 0.0 ? 1 : 0) | (s.nu4dt != 0.0 ? 2 : 0) | (s.nu6dt != 0.0 ? 4 : 0);
  switch (m) {
    case 0: pdl_launch(k_hyper_add<0>, dim3(g), dim3(TX), st, s, d, l2, l4, l6); break;
    case 1: pdl_launch(k_hyper_add<1>, dim3(g), dim3(TX), st, s, d, l2, l4, l6); break;
    case 2: pdl_launch(k_hyper_add<2>, dim3(g), dim3(TX), st, s, d, l2, l4, l6); break;
    case 3: pdl_launch(k_hyper_add<3>, dim3(g), dim3(TX), st, s, d, l2, l4, l6); break;
    case 4: pdl_launch(k_hyper_add<4>, dim3(g), dim3(TX), st, s, d, l2, l4, l6); break;
    case 5: pdl_launch(k_hyper_add<5>, dim3(g), dim3(TX), st, s, d, l2, l4, l6); break;
    case 6: pdl_launch(k_hyper_add<6>, dim3(g), dim3(TX), st, s, d, l2, l4, l6); break;
    default: pdl_launch(k_hyper_add<7>, dim3(g), dim3(TX), st, s, d, l2, l4, l6); break;
  }
}

// do_eta_geofactor (calc.c:403-422)
__global__ void k_geofactor(DevState s, F7 f, double* ab) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  ab[q] -= (RW(s, R_GEO, j) * HH(i, j) * 0.5 * (VW(i, j) + VW(i, j - 1)));
}

// solve_pres_u/v + new_vels + dissipation_effect (core.c:217-231; calc.c:500-540, 357-400)
// x - (U*0)*Dt with U finite is x - (+-0): x itself unless x is a zero.
__device__ __noinline__ double minus_damping(double x, double U, double sigma, double Dt) { return x - U * sigma * Dt; }

// UD (a band with sigma = 0): the dissipation terms are zeros, subtracted
// only where the sum is zero or an operand is not finite.
// The new tendency of u (v): advection + pressure - damping.
template <bool UD>
__device__ __forceinline__ double u_tendency(const DevState& s, const double* e, double duadv, double U, int i, int j) {
  const int W = s.W, q = IX(W, i, j);
  const double mge = s.polar ? -PF(s, P_GE, q) * s.Dt : RW(s, R_MGEDT, j);  // -GE*Dt, calc.c:517
  const double a = duadv + mdiv(s, cmul(mge, e[IX(W, i + 1, j)] - e[q]), METRIC(DXC, j));
  if constexpr (UD) return zero_term_is_exact(a, U) ? a : minus_damping(a, U, s.sigma, s.Dt);
  return a - U * (s.polar ? PF(s, P_SU, q) : s.sigma) * s.Dt;  // calc.c:374-394
}
template <bool UD>
__device__ __forceinline__ double v_tendency(const DevState& s, const double* e, double dvadv, double V, int i, int j) {
  const int W = s.W, q = IX(W, i, j);
  const double mgn = s.polar ? -PF(s, P_GN, q) * s.Dt : RW(s, R_MGNDT, j);  // calc.c:538
  const double a = dvadv + mdiv(s, cmul(mgn, e[IX(W, i, j + 1)] - e[q]), METRIC(DYC, j + 1));
  if constexpr (UD) return zero_term_is_exact(a, V) ? a : minus_damping(a, V, s.sigma, s.Dt);
  return a - V * (s.polar ? PF(s, P_SV, q) : s.sigma) * s.Dt;
}
template <bool UD>
__global__ void k_pres_sum(DevState s, F7 f, const double* duadv, const double* dvadv, double* dun, double* dvn) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  if (!s.finite) {
    const double mge = s.polar ? -PF(s, P_GE, q) * s.Dt : RW(s, R_MGEDT, j);
    const double mgn = s.polar ? -PF(s, P_GN, q) * s.Dt : RW(s, R_MGNDT, j);
    dun[q] = duadv[q] + mge * (f.eta[IX(W, i + 1, j)] - f.eta[q]) / RW(s, R_DXC, j);
    dvn[q] = dvadv[q] + mgn * (f.eta[IX(W, i, j + 1)] - f.eta[q]) / RW(s, R_DYC, j + 1);
    dun[q] -= f.u[q] * (s.polar ? PF(s, P_SU, q) : s.sigma) * s.Dt;
    dvn[q] -= f.v[q] * (s.polar ? PF(s, P_SV, q) : s.sigma) * s.Dt;
    return;
  }
  dun[q] = u_tendency<UD>(s, f.eta, duadv[q], f.u[q], i, j);
  dvn[q] = v_tendency<UD>(s, f.eta, dvadv[q], f.v[q], i, j);
}

// laplacian_vels (laplacian.c:51-111), both passes in one: a warp takes 30
// columns (its first and last lane give the ze west and the di east of the
// others) and marches up `rows` rows, carrying ze and di and the products
// DXC*u and DXV*v from row to row (the same operands, formed once). The
// reference wraps ze and di in x and fixes their wall rows (laplacian.c:67-81):
// the values of columns 0 and nx+1 are those of columns nx and 1, evaluated
// there; ze is zero in row 0 and di in row ny+1 the wall difference of u, or
// on a polar cap, which has no walls, those of rows ny and 1. `images`: with
// the halo update and wall fixes of lu and lv (laplacian.c:91-107), which the
// next level reads. Bound by the FP64 unit (13 additions a cell, 70 % busy) and
// the issue slots. In two launches, ze and di through memory: 0.075 ms a level
// at 2048x1024; fused 0.072, and one launch less on small grids. Resident
// blocks 5 (117 registers), 8, 9 and 10: 0.089, 0.071, 0.072, 0.075 (at
// 4096x2048 0.324, 0.243, 0.237, 0.235).
constexpr int LVW = 30;
__device__ __forceinline__ void lapv_strip(const DevState& s, const double* uu, const double* vv, double* lu,
                                           double* lv, bool images, int base, int j0, int jn, int lane) {
  const int W = s.W, nx = s.nx, ny = s.ny;
  const int c = base - 1 + lane;
  const int sc = c == 0 ? nx : (c <= nx ? c : 1);  // where the column's ze and di are evaluated
  const bool own = lane > 0 && lane <= LVW && c <= nx;
  // ze and di at row j of the column, the products of u (rows j, j+1) and v (rows j-1, j) given
  auto zeta = [&](int j, double v0, double ve, double pu, double pu1) {
    return rmul(s.lap_ok, RW(s, R_IDXV, j), (ve - v0) - rmul(s.lap_ok, RW(s, R_IDYC, j + 1), pu1 - pu));
  };
  auto divg = [&](int j, double u0, double uw, double qs, double qv) {
    return rmul(s.lap_ok, RW(s, R_IDXE, j), (u0 - uw) + rmul(s.lap_ok, RW(s, R_IDYN, j), qv - qs));
  };
  auto PU = [&](int j, double u) { return rmul(s.lap_ok, RW(s, R_DXC, j), u); };
  auto QV = [&](int j, double v) { return rmul(s.lap_ok, RW(s, R_DXV, j), v); };
  auto u_at = [&](int i, int j) { return uu[IX(W, i, j)]; };
  auto v_at = [&](int i, int j) { return vv[IX(W, i, j)]; };
  double u0 = u_at(sc, j0), v0 = v_at(sc, j0);
  double pu = PU(j0, u0), qv = QV(j0, v0);
  double d = divg(j0, u0, u_at(sc - 1, j0), QV(j0 - 1, v_at(sc, j0 - 1)), qv);
  double zs = 0.0;
  if (j0 > 1) {
    zs = zeta(j0 - 1, v_at(sc, j0 - 1), v_at(sc + 1, j0 - 1), PU(j0 - 1, u_at(sc, j0 - 1)), pu);
  } else if (s.polar != 0) {
    zs = zeta(ny, v_at(sc, ny), v_at(sc + 1, ny), PU(ny, u_at(sc, ny)), PU(ny + 1, u_at(sc, ny + 1)));
  }
  for (int j = j0; j <= jn; j++) {
    // the next row's values, a row ahead (0.078 -> 0.070 ms; held in registers,
    // with fewer warps resident, 0.078)
    const int jp = min(j + 2, ny + 1);
    touch(uu + IX(W, sc, jp));
    touch(uu + IX(W, sc - 1, jp));
    touch(vv + IX(W, sc, jp));
    touch(vv + IX(W, sc + 1, j + 1));
    const double u1 = u_at(sc, j + 1), v1 = v_at(sc, j + 1);
    const double pu1 = PU(j + 1, u1);
    const double z = zeta(j, v0, v_at(sc + 1, j), pu, pu1);
    double qv1 = 0.0, dn;
    if (j < ny) {
      qv1 = QV(j + 1, v1);
      dn = divg(j + 1, u1, u_at(sc - 1, j + 1), qv, qv1);
    } else if (s.polar == 0) {  // laplacian.c:73
      dn = mdiv(s, u0 - u_at(sc - 1, ny), METRIC(DXE, ny));
    } else {
      dn = divg(1, u_at(sc, 1), u_at(sc - 1, 1), QV(0, v_at(sc, 0)), QV(1, v_at(sc, 1)));
    }
    const double zw = __shfl_up_sync(FULL, z, 1), de = __shfl_down_sync(FULL, d, 1);
    // (-a)*x + b*y = b*y - a*x
    const double xu = rmul(s.lap_ok, RW(s, R_IDXC, j), de - d) - rmul(s.lap_ok, RW(s, R_IDYN, j), z - zs);
    const double xv = rmul(s.lap_ok, RW(s, R_IDXV, j), z - zw) + rmul(s.lap_ok, RW(s, R_IDYC, j + 1), dn - d);
    if (own) {
      if (images) {
        put_images<HK_LU>(s, lu, c, j, xu);
        put_images<HK_LV>(s, lv, c, j, xv);
      } else {
        lu[IX(W, c, j)] = xu;
        lv[IX(W, c, j)] = xv;
      }
    }
    u0 = u1;
    v0 = v1;
    pu = pu1;
    qv = qv1;
    d = dn;
    zs = z;
  }
}

__global__ void __launch_bounds__(TX, 9) k_lapv(DevState s, const double* uu, const double* vv, double* lu, double* lv,
                                                int rows, bool images) {
  SW2G_PDL_ENTRY();
  const int j0 = blockIdx.y * rows + 1, base = march_base(LVW);
  if (base <= s.nx) lapv_strip(s, uu, vv, lu, lv, images, base, j0, min(j0 + rows - 1, s.ny), threadIdx.x & 31);
}

// solve_Coriolis_u (calc.c:542-569), in place
__global__ void k_coriolis_u(DevState s, double* u, const double* v, const double* duab) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  const double semi = 0.25 * (v[IX(W, i, j)] + v[IX(W, i + 1, j)] + v[IX(W, i, j - 1)] + v[IX(W, i + 1, j - 1)]);
  const double dtf = s.polar ? s.Dt * PF(s, P_FE, q) : RW(s, R_DTFE, j);  // Dt*FE, calc.c:563
  const double al = sadd(dtf, div_rcp(s.Dt * u[q] * RW(s, R_SINC, j), RW(s, R_RZC, j), RW(s, R_IRZC, j)));
  const double be = 0.25 * al * al;
  u[q] = (u[q] + duab[q] - be * u[q] + al * semi) / (1.0 + be);
}

// solve_Coriolis_v (calc.c:571-598), in place, reading the new u interior
__global__ void k_coriolis_v(DevState s, const double* u, double* v, const double* dvab) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  const double semi = 0.25 * (u[IX(W, i - 1, j + 1)] + u[IX(W, i, j + 1)] + u[IX(W, i, j)] + u[IX(W, i - 1, j)]);
  const double dtf = s.polar ? s.Dt * PF(s, P_FN, q) : RW(s, R_DTFN, j);  // Dt*FN, calc.c:592
  const double al = sadd(dtf, div_rcp(s.Dt * semi * RW(s, R_SINN, j), RW(s, R_RZN, j), RW(s, R_IRZN, j)));
  const double be = 0.25 * al * al;
  v[q] = (v[q] + dvab[q] - be * v[q] - al * semi) / (1.0 + be);
}

// check_stats_scaf (sppde_core.c:346-395) as the reference evaluates it: min and
// max start from the first interior value and skip NaNs after it, so the step
// aborts iff the first value is not finite or some value lies outside +-1e10.
// Tested on the bits (|x| > 1e10 and not NaN), for up to four fields at once.
__device__ __forceinline__ bool range_bad(double x, bool first) {
  const long long m = dbits(x) & 0x7fffffffffffffffLL;
  if (first) return m > 0x4202a05f20000000LL;  // beyond 1e10, inf or NaN
  return m > 0x4202a05f20000000LL && m <= 0x7ff0000000000000LL;
}
// From the third step on (AB3), the tail of each tendency is fused into one
// kernel per field, with the operations of the separate kernels in their
// order: the hyperviscosity terms (into the stored tendency), the
// Adams-Bashforth combination (calc.c:651-699, linop_scaf's two passes) and
//   eta: the geofactor (calc.c:403-422) and eta += D (core.c:203-205);
//   u, v: the Coriolis update (calc.c:542-598).
__device__ __forceinline__ double ab3(double dn, double dm1, double dm2) {
  const double t = cmul(5.0 / 12.0, dm2) - cmul(4.0 / 3.0, dm1);  // -(4/3)*dm1 + (5/12)*dm2
  return cmul(23.0 / 12.0, dn) + t;  // 1.0 * t is t
}
// v + (+0): v, except that -0 becomes +0 (the plain form's zero winds).
__device__ __forceinline__ double plus_pos_zero(double v) {
  return (dbits(v) == (long long)0x8000000000000000ULL) ? 0.0 : v;
}

// With `bad` given (a whole step, no forcing between its halves), the range
// check of the new value (core.c:309-312) is done here as well.
__device__ __forceinline__ void check_range(int* bad, double x, int i, int j) {
  if (bad && range_bad(x, i == 1 && j == 1)) atomicOr(bad, 1);
}

// The new eta of a cell (calc.c:403-422, core.c:203-210), given the tendency's
// hyperviscosity values.
template <int NZ, bool PL>
__device__ __forceinline__ void eta_ab3_cell(const DevState& s, const F7& f, double* eta, double* dn,
                                             const double* dm1, const double* dm2, double v2, double v4, double v6,
                                             int* bad, int i, int j) {
  const int W = s.W, q = IX(W, i, j);
  const double x = hyper_terms<NZ>(s, dn[q], v2, v4, v6);
  if constexpr (NZ != kNoHyper) dn[q] = x;
  double ab = ab3(x, dm1[q], dm2[q]);
  const double e = f.eta[q];
  if constexpr (PL) {
    const double h = e + s.depth;  // - hB with hB = +0 is exact
    ab -= smul(HALF(cmul(RW(s, R_GEO, j), h)), plus_pos_zero(f.v[q]) + plus_pos_zero(f.v[IX(W, i, j - 1)]));
  } else {
    ab -= smul(HALF(cmul(RW(s, R_GEO, j), HH(i, j))), VW(i, j) + VW(i, j - 1));
  }
  const double en = e + ab;
  put_images<HK_WRAP>(s, eta, i, j, en);  // with eta's halo update (core.c:206-210)
  check_range(bad, en, i, j);
}
template <int NZ, bool PL>
__global__ void k_eta_ab3(DevState s, F7 f, double* eta, double* dn, const double* dm1, const double* dm2,
                          const double* l2, const double* l4, const double* l6, int* bad) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  eta_ab3_cell<NZ, PL>(s, f, eta, dn, dm1, dm2, level<NZ>(l2, 0, q), level<NZ>(l4, 1, q), level<NZ>(l6, 2, q), bad,
                       i, j);
}
// The same with the last level of laplacian_eta (of the field e), which only
// the cell itself reads: neither it nor its halo goes through memory.
template <int NZ, bool PL>
__global__ void __launch_bounds__(TX, 16) k_eta_lap_ab3(DevState s, F7 f, double* eta, double* dn, const double* dm1,
                                                    const double* dm2, const double* l2, const double* l4,
                                                    const double* e, int* bad, int rows) {
  SW2G_PDL_ENTRY();
  constexpr int last = kLevels<NZ> - 1;
  const int W = s.W, j0 = blockIdx.y * rows + 1, jn = min(j0 + rows - 1, s.ny);
  const int base = march_base(FW);
  if (base > s.nx) return;
  LapEta L;
  L.begin(s, e, base, j0, threadIdx.x & 31);
  for (int j = j0; j <= jn; j++) {
    const double v = L.next(s, e, j);
    if (!L.own) continue;
    const int q = IX(W, L.c, j);
    const double v2 = last == 0 ? v : l2[q], v4 = last == 1 ? v : level<NZ>(l4, 1, q), v6 = last == 2 ? v : 0.0;
    eta_ab3_cell<NZ, PL>(s, f, eta, dn, dm1, dm2, v2, v4, v6, bad, L.c, j);
  }
}

// The tracer's update (calc.c:651-699, core.c:161-182): AB3, tracer += D and its
// halo update. As k_ab, k_add and k_halo in turn 0.031 ms at 1201x607, so
// 0.012.
__global__ void __launch_bounds__(TX, 16) k_tracer_ab3(DevState s, double* tr, const double* dn, const double* dm1,
                                                       const double* dm2, int* bad) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  const double t = tr[q] + ab3(dn[q], dm1[q], dm2[q]);
  put_images<HK_WRAP>(s, tr, i, j, t);
  check_range(bad, t, i, j);
}

template <int NZ, bool UD>
__global__ void __launch_bounds__(TX, 16) k_coriolis_u_ab3(DevState s, double* u, const double* v, const double* eta, const double* duadv,
                                 double* dn, const double* dm1, const double* dm2, const double* l2,
                                 const double* l4, const double* l6, int* bad) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  const double u0 = u[q];
  const double x = hyper_terms<NZ>(s, u_tendency<UD>(s, eta, duadv[q], u0, i, j), level<NZ>(l2, 0, q),
                                   level<NZ>(l4, 1, q), level<NZ>(l6, 2, q));
  dn[q] = x;
  const double duab = ab3(x, dm1[q], dm2[q]);
  const double semi = QUARTER(v[IX(W, i, j)] + v[IX(W, i + 1, j)] + v[IX(W, i, j - 1)] + v[IX(W, i + 1, j - 1)]);
  const double dtf = s.polar ? s.Dt * PF(s, P_FE, q) : RW(s, R_DTFE, j);
  const double al = dtf + mdiv(s, cmul(s.Dt, u0) * RW(s, R_SINC, j), METRIC(RZC, j));
  const double be = smul(QUARTER(al), al);
  const double un = quotient(((u0 + duab) - smul(be, u0)) + smul(al, semi), 1.0 + be);
  u[q] = un;
  check_range(bad, un, i, j);
}

template <int NZ, bool UD>
__global__ void __launch_bounds__(TX, 16) k_coriolis_v_ab3(DevState s, const double* u, double* v, const double* eta, const double* dvadv,
                                 double* dn, const double* dm1, const double* dm2, const double* l2,
                                 const double* l4, const double* l6, int* bad) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  const double v0 = v[q];
  const double x = hyper_terms<NZ>(s, v_tendency<UD>(s, eta, dvadv[q], v0, i, j), level<NZ>(l2, 0, q),
                                   level<NZ>(l4, 1, q), level<NZ>(l6, 2, q));
  dn[q] = x;
  const double dvab = ab3(x, dm1[q], dm2[q]);
  const double semi = QUARTER(u[IX(W, i - 1, j + 1)] + u[IX(W, i, j + 1)] + u[IX(W, i, j)] + u[IX(W, i - 1, j)]);
  const double dtf = s.polar ? s.Dt * PF(s, P_FN, q) : RW(s, R_DTFN, j);
  const double al = dtf + mdiv(s, cmul(s.Dt, semi) * RW(s, R_SINN, j), METRIC(RZN, j));
  const double be = smul(QUARTER(al), al);
  const double vn = quotient(((v0 + dvab) - smul(be, v0)) - smul(al, semi), 1.0 + be);
  v[q] = vn;
  // a band's row ny is a wall: do_channel zeroes it before the range check
  // (core.c:303-312), so the check sees +0 there
  if (s.polar != 0 || j != s.ny) check_range(bad, vn, i, j);
}

// Launch shape of the kernels that march: `width` columns per warp, and as
// many rows (a power of two up to `rows`) as still leave 24 warps for each SM,
// so that small grids spread over the chip. k_lapv takes up to 8 rows, the
// eta kernels 4: at 2048x1024 with 4, 8 and 16 rows k_lapv 0.073, 0.071 and
// 0.073 ms, k_lape 0.037, 0.038 and 0.043, k_eta_lap_ab3 0.077, 0.085, 0.092.
struct March {
  dim3 grid;
  int rows;
};
March march(const DevState& s, int width, int rows) {
  const int bx = (s.nx + width * (TX / 32) - 1) / (width * (TX / 32));
  while (rows > 1 && (long long)bx * (TX / 32) * ((s.ny + rows - 1) / rows) < 152 * 24) rows /= 2;
  return March{dim3(bx, (s.ny + rows - 1) / rows), rows};
}

// which: 0 eta (hyper + AB3 + geofactor + update), 1 u, 2 v (pressure, damping,
// hyper + AB3 + Coriolis); bad: the step's range flag when the range check is
// done here, else null; last_src: the field whose laplacian_eta is the last
// level, computed by the eta kernel, or null if that level is in Le already
template <int NZ>
void fused_tails(const DevState& s, dim3 g, cudaStream_t st, const F7& f, Fp64Buffers& b, int which, int* bad,
                 const double* last_src) {
  const bool ud = s.polar == 0 && s.sigma == 0.0;
  if (which == 0) {
    if constexpr (NZ != kNoHyper) {
      if (last_src) {
        const March m = march(s, FW, 4);
        auto k = s.plain ? k_eta_lap_ab3<NZ, true> : k_eta_lap_ab3<NZ, false>;
        pdl_launch(k, m.grid, dim3(TX), st, s, f, b.f[0], b.deta[0], b.deta[1], b.deta[2], b.Le[0], b.Le[1], last_src,
                   bad, m.rows);
        return;
      }
    }
    auto k = s.plain ? k_eta_ab3<NZ, true> : k_eta_ab3<NZ, false>;
    pdl_launch(k, g, dim3(TX), st, s, f, b.f[0], b.deta[0], b.deta[1], b.deta[2], b.Le[0], b.Le[1], b.Le[2], bad);
  } else if (which == 1) {
    auto k = ud ? k_coriolis_u_ab3<NZ, true> : k_coriolis_u_ab3<NZ, false>;
    pdl_launch(k, g, dim3(TX), st, s, b.f[1], b.f[2], b.f[0], b.duadv, b.du[0], b.du[1], b.du[2], b.L[0], b.L[2],
               b.L[4], bad);
  } else {
    auto k = ud ? k_coriolis_v_ab3<NZ, true> : k_coriolis_v_ab3<NZ, false>;
    pdl_launch(k, g, dim3(TX), st, s, b.f[1], b.f[2], b.f[0], b.dvadv, b.dv[0], b.dv[1], b.dv[2], b.L[1], b.L[3],
               b.L[5], bad);
  }
}
void fused_tail(const DevState& s, dim3 g, cudaStream_t st, const F7& f, Fp64Buffers& b, int which, int* bad,
                const double* last_src = nullptr) {
  switch (hyper_mask(s)) {
    case 0: fused_tails<0>(s, g, st, f, b, which, bad, last_src); break;
    case 1: fused_tails<1>(s, g, st, f, b, which, bad, last_src); break;
    case 2: fused_tails<2>(s, g, st, f, b, which, bad, last_src); break;
    case 3: fused_tails<3>(s, g, st, f, b, which, bad, last_src); break;
    case 4: fused_tails<4>(s, g, st, f, b, which, bad, last_src); break;
    case 5: fused_tails<5>(s, g, st, f, b, which, bad, last_src); break;
    case 6: fused_tails<6>(s, g, st, f, b, which, bad, last_src); break;
    case 7: fused_tails<7>(s, g, st, f, b, which, bad, last_src); break;
    default: fused_tails<kNoHyper>(s, g, st, f, b, which, bad, last_src); break;
  }
}

// Single-rank halo update (sppde_hupdate.c:274-342). The y pass then the x pass
// compose to: every halo cell copies the interior cell (wrapx(i), wrapy(j)).
// blockIdx.y selects the field: one launch wraps x and, when given, y.
__global__ void k_halo(double* x, double* y, int nx, int ny) {
  SW2G_PDL_ENTRY();
  const int W = nx + 4;
  const int nh = 4 * W + 4 * ny;  // 4 full halo rows + 4 halo columns over interior rows
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nh) return;
  if (blockIdx.y == 1) x = y;
  int i, j;
  if (t < 4 * W) {
    const int r = t / W;
    i = t - r * W - 1;
    j = (r < 2) ? r - 1 : ny + r - 1;  // rows -1, 0, ny+1, ny+2
  } else {
    const int u = t - 4 * W;
    const int c = u / ny;
    j = u - c * ny + 1;
    i = (c < 2) ? c - 1 : nx + c - 1;  // columns -1, 0, nx+1, nx+2
  }
  const int si = (i < 1) ? i + nx : ((i > nx) ? i - nx : i);
  const int sj = (j < 1) ? j + ny : ((j > ny) ? j - ny : j);
  x[IX(W, i, j)] = x[IX(W, si, sj)];
}

// do_channel (calc.c:600-649), polar 0: interior columns of the wall rows
__global__ void k_channel(int nx, int ny, double* u, double* v, double* wx, double* wy) {
  SW2G_PDL_ENTRY();
  const int W = nx + 4;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > nx) return;
  v[IX(W, i, 0)] = 0; v[IX(W, i, -1)] = 0;
  wy[IX(W, i, 0)] = 0; wy[IX(W, i, -1)] = 0;
  u[IX(W, i, 0)] = u[IX(W, i, 1)]; u[IX(W, i, -1)] = u[IX(W, i, 0)];
  wx[IX(W, i, 0)] = wx[IX(W, i, 1)]; wx[IX(W, i, -1)] = wx[IX(W, i, 0)];
  v[IX(W, i, ny)] = 0; v[IX(W, i, ny + 1)] = 0; v[IX(W, i, ny + 2)] = 0;
  wy[IX(W, i, ny)] = 0; wy[IX(W, i, ny + 1)] = 0; wy[IX(W, i, ny + 2)] = 0;
  u[IX(W, i, ny + 1)] = u[IX(W, i, ny)]; u[IX(W, i, ny + 2)] = u[IX(W, i, ny + 1)];
  wx[IX(W, i, ny + 1)] = wx[IX(W, i, ny)]; wx[IX(W, i, ny + 2)] = wx[IX(W, i, ny + 1)];
}

// A whole step's halo update of u and v followed by do_channel, in one launch
// (a band): the x-halo columns of the interior rows and the corners take the
// wrap, the interior columns of the wall rows do_channel's values. do_channel
// zeroes row ny of v, whose cells next to the seam the halo update copies
// first: one thread does both for them. winds: do_channel's rows of windx and
// windy, which it leaves as they are when they are +0.0 everywhere.
__global__ void k_halo_channel(int nx, int ny, double* u, double* v, double* wx, double* wy, bool winds) {
  SW2G_PDL_ENTRY();
  const int W = nx + 4;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  auto halo_col = [&](int c) { return c < 2 ? c - 1 : nx + c - 1; };  // columns -1, 0, nx+1, nx+2
  auto wrap = [&](int i) { return i < 1 ? i + nx : (i > nx ? i - nx : i); };
  if (t < nx) {  // do_channel (calc.c:600-649)
    const int i = t + 1;
    const double lo = u[IX(W, i, 1)], hi = u[IX(W, i, ny)];
    u[IX(W, i, 0)] = lo; u[IX(W, i, -1)] = lo;
    u[IX(W, i, ny + 1)] = hi; u[IX(W, i, ny + 2)] = hi;
    v[IX(W, i, 0)] = 0; v[IX(W, i, -1)] = 0;
    v[IX(W, i, ny + 1)] = 0; v[IX(W, i, ny + 2)] = 0;
    if (i > 2 && i < nx - 1) v[IX(W, i, ny)] = 0;
    if (winds) {
      const double wlo = wx[IX(W, i, 1)], whi = wx[IX(W, i, ny)];
      wx[IX(W, i, 0)] = wlo; wx[IX(W, i, -1)] = wlo;
      wx[IX(W, i, ny + 1)] = whi; wx[IX(W, i, ny + 2)] = whi;
      wy[IX(W, i, 0)] = 0; wy[IX(W, i, -1)] = 0;
      wy[IX(W, i, ny)] = 0; wy[IX(W, i, ny + 1)] = 0; wy[IX(W, i, ny + 2)] = 0;
    }
    return;
  }
  const int h = t - nx;
  if (h < 4 * (ny - 1)) {  // x halos of rows 1 .. ny-1
    const int c = h / (ny - 1), j = h - c * (ny - 1) + 1, i = halo_col(c), si = wrap(i);
    u[IX(W, i, j)] = u[IX(W, si, j)];
    v[IX(W, i, j)] = v[IX(W, si, j)];
  } else if (h == 4 * (ny - 1)) {  // row ny and the corners, sppde_hupdate.c:274-342
    const int rows[4] = {-1, 0, ny + 1, ny + 2}, from[4] = {ny - 1, ny, 1, 2};
    double vn[4];
    for (int c = 0; c < 4; c++) vn[c] = v[IX(W, wrap(halo_col(c)), ny)];
    for (int c = 0; c < 4; c++) {
      const int i = halo_col(c), si = wrap(i);
      u[IX(W, i, ny)] = u[IX(W, si, ny)];
      v[IX(W, i, ny)] = vn[c];
      for (int r = 0; r < 4; r++) {
        u[IX(W, i, rows[r])] = u[IX(W, si, from[r])];
        v[IX(W, i, rows[r])] = r == 1 ? vn[c] : v[IX(W, si, from[r])];
      }
    }
    for (int c = 0; c < 4; c++) v[IX(W, wrap(halo_col(c)), ny)] = 0;
  }
}

// compute_Dt maxima (calc.c:705-712): max |u+wx|/DXE and |v+wy|/DYN over the
// interior; NaNs never win the comparison, as in the reference's loop. A
// correctly rounded division by a positive number is non-decreasing in the
// numerator, so the largest quotient of a row is the quotient of its largest
// magnitude: the magnitudes are compared as integers (NaNs set to 0) and each
// warp divides once.
__device__ __forceinline__ long long mag_bits(double x) {
  const long long m = dbits(x) & 0x7fffffffffffffffLL;
  return (m > 0x7ff0000000000000LL) ? 0 : m;
}
// One block per row: the row's largest magnitudes, then its two quotients and
// two atomics (atomics on the same address from every warp of the grid would
// serialise in L2).
constexpr int CFL_T = 256;
__global__ void __launch_bounds__(CFL_T) k_cfl(DevState s, F7 f, unsigned long long* out) {
  SW2G_PDL_ENTRY();
  __shared__ long long red[2][CFL_T / 32];
  const int W = s.W;
  const int j = blockIdx.x + 1;
  long long bx = 0, by = 0;
  if (s.plain) {  // |u + (+0)| = |u|
#pragma unroll 4
    for (int i = threadIdx.x + 1; i <= s.nx; i += CFL_T) {
      bx = max(bx, mag_bits(f.u[IX(W, i, j)]));
      by = max(by, mag_bits(f.v[IX(W, i, j)]));
    }
  } else {
#pragma unroll 4
    for (int i = threadIdx.x + 1; i <= s.nx; i += CFL_T) {
      bx = max(bx, mag_bits(UW(i, j)));
      by = max(by, mag_bits(VW(i, j)));
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    bx = max(bx, __shfl_xor_sync(0xffffffffu, bx, o));
    by = max(by, __shfl_xor_sync(0xffffffffu, by, o));
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = bx;
    red[1][threadIdx.x >> 5] = by;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < CFL_T / 32; w++) {
      bx = max(bx, red[0][w]);
      by = max(by, red[1][w]);
    }
    const double mx = div_rcp(__longlong_as_double(bx), RW(s, R_DXE, j), RW(s, R_IDXE, j));
    const double my = div_rcp(__longlong_as_double(by), RW(s, R_DYN, j), RW(s, R_IDYN, j));
    if (mx > 0) atomicMax(out, (unsigned long long)dbits(mx));
    if (my > 0) atomicMax(out + 1, (unsigned long long)dbits(my));
  }
}

// The maxima of rows j0 to jn, columns i0 to i0 + CFLW - 1, on one warp (k_cfl otherwise).
// A row of any width on one warp held a launch up: 65536x32 2.23 ms a step, in pieces
// 0.71 (of 1024, 2048 and 4096 columns alike, and up to 4096 columns nothing changes).
constexpr int CFLW = 4096;
template <bool PL>
__device__ __forceinline__ void cfl_rows(const DevState& s, const F7& f, unsigned long long* out, int i0, int j0, int jn,
                                         int lane) {
  const int W = s.W, i1 = min(i0 + CFLW - 1, s.nx);
  for (int j = j0; j <= jn; j++) {
    long long bx = 0, by = 0;
#pragma unroll 4
    for (int i = i0 + lane; i <= i1; i += 32) {
      bx = max(bx, mag_bits(PL ? f.u[IX(W, i, j)] : UW(i, j)));
      by = max(by, mag_bits(PL ? f.v[IX(W, i, j)] : VW(i, j)));
    }
    for (int o = 16; o > 0; o >>= 1) {
      bx = max(bx, __shfl_xor_sync(FULL, bx, o));
      by = max(by, __shfl_xor_sync(FULL, by, o));
    }
    if (lane == 0) {
      const double mx = div_rcp(__longlong_as_double(bx), RW(s, R_DXE, j), RW(s, R_IDXE, j));
      const double my = div_rcp(__longlong_as_double(by), RW(s, R_DYN, j), RW(s, R_IDYN, j));
      if (mx > 0) atomicMax(out, (unsigned long long)dbits(mx));
      if (my > 0) atomicMax(out + 1, (unsigned long long)dbits(my));
    }
  }
}

// What a step computes from the old fields alone, in one launch: the CFL
// maxima, the bodies, and the first levels of the hyperviscosity's Laplacians.
// Every kind's strips are fk rows high; those of each kind follow those of the
// one before, all from one queue. kinds: four bits each, lowest first.
enum BodyKind { B_MASS, B_TRACER, B_ADV_U, B_ADV_V, B_LAPV, B_LAPE, B_CFL };
struct Bodies {
  double* out[4];  // of the bodies, by kind
  const double* le_src;
  double *Le, *Lu, *Lv;  // the Laplacians' first levels, of le_src and of (u, v)
  bool images;           // a second level of the velocities reads the first
  unsigned long long* cfl;
  unsigned kinds;
  int n;  // how many kinds
};
__host__ __device__ __forceinline__ int strip_columns(int kind, int nx) {
  return kind == B_CFL ? (nx + CFLW - 1) / CFLW : kind == B_LAPV ? (nx + LVW - 1) / LVW : (nx + FW - 1) / FW;
}
template <int SCH, bool PL, bool UD>
__global__ void __launch_bounds__(32 * FWARPS, FAST_MIN_BLOCKS)
    k_bodies(const __grid_constant__ DevState s, const __grid_constant__ F7 f, const __grid_constant__ Bodies o) {
  SW2G_PDL_ENTRY();
  const int lane = threadIdx.x & 31, rows = (s.ny + s.fk - 1) / s.fk;
  for (;;) {
    int strip = next_strip(s.strips, lane), k = 0, kind = 0, cols = 0;
    for (; k < o.n; k++) {
      kind = (o.kinds >> (4 * k)) & 15u;
      cols = strip_columns(kind, s.nx);
      if (strip < cols * rows) break;
      strip -= cols * rows;
    }
    if (k == o.n) break;
    const int j0 = strip / cols * s.fk + 1, jn = min(j0 + s.fk - 1, s.ny), x = strip % cols;
    switch (kind) {
      case B_MASS: mass_strip<SCH, PL, UD>(s, f, o.out[B_MASS], strip, lane); break;
      case B_TRACER: tracer_strip<SCH, PL>(s, f, o.out[B_TRACER], strip, lane); break;
      case B_ADV_U: adv_u_strip<SCH, PL>(s, f, o.out[B_ADV_U], strip, lane); break;
      case B_ADV_V: adv_v_strip<SCH, PL>(s, f, o.out[B_ADV_V], strip, lane); break;
      case B_LAPV: lapv_strip(s, f.u, f.v, o.Lu, o.Lv, o.images, x * LVW + 1, j0, jn, lane); break;
      case B_LAPE: lape_strip(s, o.le_src, o.Le, x * FW + 1, j0, jn, lane); break;
      default: cfl_rows<PL>(s, f, o.cfl, x * CFLW + 1, j0, jn, lane); break;
    }
  }
  strips_done(s.strips, lane);
}

struct RangeFields {
  const double* f[4];
  int n;
};
__global__ void k_range(DevState s, RangeFields r, int* bad) {
  SW2G_PDL_ENTRY();
  INTERIOR_IJ
  const int q = IX(W, i, j);
  const bool first = (i == 1 && j == 1);
  bool b = false;
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (k < r.n) b = b || range_bad(r.f[k][q], first);
  if (b) atomicOr(bad, 1);
}

#undef UW
#undef VW
#undef HH

// Launch of the fast bodies. Warps take strips of 31 columns x fk rows of each
// body from a queue (next_strip), and the grid is the blocks resident on the
// device at once (or fewer when there are fewer strips). A strip costs its rows
// and about one row more (the face south of its first row); the queue evens
// out the warps' different speeds, and the end of the launch, with part of the
// warps idle, costs about a strip's time (more in flows from rest, where the
// cells that need the literal code lie together). So the height is the one
// with the least (fk + 1) * (strips per resident warp + 1.2). With 0.3,
// 1.0 and 1.6 in place of 1.2: two forced steps from rest at 1024x512 2.41,
// 2.03 and 1.93 ms; four steps of a 500x500 cap 0.830, 0.795 and 0.794; four
// steps at 2048x1024 3.286, 3.290 and 3.318. One launch for the bodies in place
// of three or four: a step at 256x128 88 -> 80 us, at 2048x1024 0.364 ms of
// bodies -> 0.340; with the CFL maxima and the Laplacians' first levels 80 -> 72.
int choose_strip_rows(int columns, int ny, long long warps) {
  int best = 1;
  double least = 0;
  for (int fk = 1; fk <= 24; fk++) {
    const long long strips = (long long)columns * ((ny + fk - 1) / fk);
    const double cost = (fk + 1) * ((double)strips / (double)warps + 1.2);
    if (fk == 1 || cost < least) {
      least = cost;
      best = fk;
    }
  }
  return best;
}

// The blocks of a kernel that are resident on the current device at once.
constexpr int kMaxDevices = 64;
template <auto K>
long long resident_blocks() {
  static std::atomic<int> cap[kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) dev = 0;
  int c = cap[dev].load(std::memory_order_relaxed);
  if (!c) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, K, 32 * FWARPS, 0);
    c = (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
    cap[dev].store(c, std::memory_order_relaxed);
  }
  return c;
}

template <auto K>
void launch_strips(cudaStream_t st, const DevState& s0, const F7& f, const Bodies& o) {
  const long long full = resident_blocks<K>();
  DevState s = s0;
  int columns = 0;
  for (int k = 0; k < o.n; k++) columns += strip_columns((o.kinds >> (4 * k)) & 15, s.nx);
  s.fk = choose_strip_rows(columns, s.ny, full * FWARPS);
  const long long strips = (long long)columns * ((s.ny + s.fk - 1) / s.fk);
  const long long need = (strips + FWARPS - 1) / FWARPS;
  pdl_launch(K, dim3((int)(need < full ? need : full)), dim3(32 * FWARPS), st, s, f, o);
}

// One launch for all the bodies, or, for the literal kernels, one for each;
// returns how many.
template <int SCH>
int launch_bodies(dim3 g, cudaStream_t st, const DevState& s, const F7& f, const Bodies& o) {
  if constexpr (SCH != 3) {
    if (s.sig_ok) {  // Dt and the metric divisors in the range of the integer-pipe quotients
      if (!s.plain) launch_strips<k_bodies<SCH, false, false>>(st, s, f, o);
      else if (!s.polar && s.sigma == 0.0) launch_strips<k_bodies<SCH, true, true>>(st, s, f, o);
      else launch_strips<k_bodies<SCH, true, false>>(st, s, f, o);
      return 1;
    }
  }
  for (int k = 0; k < o.n; k++) {
    const int kind = (o.kinds >> (4 * k)) & 15;
    if (kind == B_CFL) {
      pdl_launch(k_cfl, dim3(s.ny), dim3(CFL_T), st, s, f, o.cfl);
      continue;
    }
    if (kind == B_LAPV || kind == B_LAPE) {
      const March m = kind == B_LAPV ? march(s, LVW, 8) : march(s, FW, 4);
      if (kind == B_LAPV) pdl_launch(k_lapv, m.grid, dim3(TX), st, s, f.u, f.v, o.Lu, o.Lv, m.rows, o.images);
      else pdl_launch(k_lape, m.grid, dim3(TX), st, s, o.le_src, o.Le, m.rows);
      continue;
    }
    auto kernel = kind == B_MASS     ? k_mass<SCH>
                  : kind == B_TRACER ? k_tracer<SCH>
                  : kind == B_ADV_U  ? k_adv_u<SCH>
                                     : k_adv_v<SCH>;
    pdl_launch(kernel, g, dim3(TX), st, s, f, o.out[kind]);
  }
  return o.n;
}

int bodies(int sch, dim3 g, cudaStream_t st, const DevState& s, const F7& f, const Bodies& o) {
  switch (sch) {
    case 0: return launch_bodies<0>(g, st, s, f, o);
    case 1: return launch_bodies<1>(g, st, s, f, o);
    case 2: return launch_bodies<2>(g, st, s, f, o);
    case 3: return launch_bodies<3>(g, st, s, f, o);
    case 4: return launch_bodies<4>(g, st, s, f, o);
    case 5: return launch_bodies<5>(g, st, s, f, o);
    case 6: return launch_bodies<6>(g, st, s, f, o);
    case 7: return launch_bodies<7>(g, st, s, f, o);
    case 8: return launch_bodies<8>(g, st, s, f, o);
    case 9: return launch_bodies<9>(g, st, s, f, o);
    default: return launch_bodies<kVanLeerSafe>(g, st, s, f, o);
  }
}

void rotate3(double** h) {
  double* t = h[2];
  h[2] = h[1];
  h[1] = h[0];
  h[0] = t;
}

}  // namespace

namespace {
// Forcing between steps (perturbs.c): field += scale * delta, or field =
// value where mask, over the interior cells.
__global__ void k_add_scaled(int nx, int ny, double* f, const double* d, double scale) {
  const int W = nx + 4;
  const int n = nx * ny;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int q = IX(W, t % nx + 1, t / nx + 1);
    f[q] += scale * d[q];
  }
}
__global__ void k_set_where(int nx, int ny, double* f, const double* val, const unsigned char* mask) {
  const int W = nx + 4;
  const int n = nx * ny;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int q = IX(W, t % nx + 1, t / nx + 1);
    if (mask[q]) f[q] = val[q];
  }
}
__global__ void k_scatter_cells(double* f, const int* __restrict__ cells, const double* __restrict__ values, int n) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
    f[cells[t]] = values ? values[t] : 0.0;
}
}  // namespace

void fp64_add_scaled(double* f, const double* d, double scale, int nx, int ny, cudaStream_t st) {
  const int n = nx * ny, blocks = (n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096;
  k_add_scaled<<<blocks, 256, 0, st>>>(nx, ny, f, d, scale);
  halo_wrap(f, nx, ny, st);
}

void fp64_set_where(double* f, const double* val, const unsigned char* mask, int nx, int ny, cudaStream_t st) {
  const int n = nx * ny, blocks = (n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096;
  k_set_where<<<blocks, 256, 0, st>>>(nx, ny, f, val, mask);
  halo_wrap(f, nx, ny, st);
}

void fp64_scatter_cells(double* f, const int* cells, const double* values, int n, cudaStream_t st) {
  if (n <= 0) return;
  const int blocks = (n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096;
  k_scatter_cells<<<blocks, 256, 0, st>>>(f, cells, values, n);
}

void fp64_channel(double* u, double* v, double* wx, double* wy, int nx, int ny, cudaStream_t st) {
  k_channel<<<(nx + 127) / 128, 128, 0, st>>>(nx, ny, u, v, wx, wy);
}

void fp64_range(const DevState& s, const double* const* fields, int n, int* bad, cudaStream_t st) {
  RangeFields r{};
  for (int k = 0; k < n && k < 4; k++) r.f[r.n++] = fields[k];
  const dim3 g((s.nx + TX - 1) / TX, s.ny);
  pdl_launch(k_range, g, dim3(TX), st, s, r, bad);
}

void fp64_check_add(long long samples, unsigned long long seed, unsigned long long* bad, cudaStream_t st) {
  k_check_add<<<152 * 8, 256, 0, st>>>(samples, seed, bad);
}

void fp64_check_division(const double* d_div, const unsigned long long* d_recip, int n, long long samples,
                         unsigned long long seed, unsigned long long* bad, cudaStream_t st) {
  k_check_division<<<152 * 8, 256, 0, st>>>(d_div, d_recip, n, samples, seed, bad);
}

void halo_wrap(double* x, int nx, int ny, cudaStream_t st) {
  const int nh = 4 * (nx + 4) + 4 * ny;
  pdl_launch(k_halo, dim3((nh + 255) / 256), dim3(256), st, x, x, nx, ny);
}
// Two fields in one launch.
void halo_wrap2(double* x, double* y, int nx, int ny, cudaStream_t st) {
  const int nh = 4 * (nx + 4) + 4 * ny;
  pdl_launch(k_halo, dim3(dim3((nh + 255) / 256, 2)), dim3(256), st, x, y, nx, ny);
}

// One reference time step; returns the number of kernels launched.
namespace {

// Launch bookkeeping shared by the two halves of a step: every tagged launch
// is timed while the timers are on, and counted.
#define LAUNCH(tag, ...)                          \
  do {                                            \
    if (tm && tm->on) tm->begin(tag, st);         \
    __VA_ARGS__;                                  \
    if (tm && tm->on) tm->end(st);                \
    nl++;                                         \
  } while (0)

// Whether the tails of the tendencies run as one kernel each: from the third
// step (AB3), unless a constant is not finite (which fails the first step).
bool tails_fused(const DevState& s, int k) { return k >= 2 && s.finite; }

// Head of a step: core.c:134-290, through the velocity halos.
// fused_checks: the range checks are done by the kernels that write the new
// values (a whole step, from the third step).
// The advection sweeps of u and v (core.c:212-215) run before the mass
// update: they read only u, v, the winds and the geometry, and write only
// their own tendencies, so the order changes no value, and a caller that
// copies eta in can overlap that copy with them (StepHooks).
int step_head(const DevState& s, Fp64Buffers& b, int sch, int k, bool tracer, StepChecks chk, int slot,
              cudaStream_t st, Timers* tm, bool fused_checks, bool whole, StepHooks hk) {
  int* const fbad = fused_checks ? chk.bad + slot : nullptr;
  const dim3 g((s.nx + TX - 1) / TX, s.ny);
  const bool fused = tails_fused(s, k);
  int nl = 0;
  auto F = [&]() { return F7{b.f[0], b.f[1], b.f[2], b.f[3], b.f[4], b.f[5], b.f[6]}; };
  const bool hyper = (s.nu2 != 0 || s.nu4 != 0 || s.nu6 != 0);

  // The Laplacians of the mass equation's hyperviscosity (calc.c:325-335,
  // laplacian.c:110-146). The reference zeroes Le before them (calc.c:325-327).
  // Here it is zeroed once at allocation: every level that runs rewrites all
  // cells of its Le (interior, halo wrap, wall rows), and levels that do not
  // run leave their Le zero.
  const int nlap = !hyper ? 0 : (s.nu6 != 0) ? 3 : (s.nu4 != 0) ? 2 : 1;
  auto lap_eta_source = [&](int q) -> const double* {
    // the reference passes u, not eta (calc.c:332)
    return q > 0 ? b.Le[q - 1] : s.lape_eta ? b.f[0] : b.f[1];
  };
  auto eta_laplacians = [&](int first, int levels) {
    const March m = march(s, FW, 4);
    for (int q = first; q < levels; q++)
      LAUNCH("lape", pdl_launch(k_lape, m.grid, dim3(TX), st, s, lap_eta_source(q), b.Le[q], m.rows));
  };
  // Reading u alone, and nothing that the kernels before their place in the
  // reference's order write, they run first when a caller copies the fields
  // in, which then overlaps the copies of v and eta with them (StepHooks);
  // otherwise they keep their place after the mass body.
  const bool laplacians_first = hyper && !s.lape_eta && hk.v_in;
  // From the third step the eta kernel computes the last level itself, except
  // where that level's source is eta, which the kernel changes.
  const bool last_in_eta = hyper && fused && !laplacians_first && !(s.lape_eta && nlap == 1);
  if (laplacians_first) eta_laplacians(0, nlap);
  if (hk.v_in) cudaStreamWaitEvent(st, hk.v_in, 0);

  // What reads old fields only, in one launch, the longest strips first: the
  // maxima of compute_Dt at the start of the step (core.c:155-159); the bodies
  // of u and v (core.c:212-215), of the tracer (core.c:161-182; skipped while
  // the tracer is identically +0, which the step then provably leaves
  // unchanged) and of the mass (core.c:184-210; calc.c:289-355); the first
  // levels of the Laplacians. A caller whose eta is still on its way in gets
  // what reads eta in a launch of its own behind that copy.
  const int nle = laplacians_first ? 0 : last_in_eta ? nlap - 1 : nlap;  // eta levels in kernels of their own
  Bodies o{{b.deta[0], b.dtr[0], b.duadv, b.dvadv}, nullptr, b.Le[0], b.L[0], b.L[1], nlap > 1, chk.cfl + 2 * slot, 0, 0};
  auto add_kind = [&](unsigned kind) { o.kinds |= kind << (4 * o.n++); };
  add_kind(B_CFL);
  add_kind(B_ADV_U);
  add_kind(B_ADV_V);
  if (tracer) add_kind(B_TRACER);
  if (!hk.eta_in) add_kind(B_MASS);
  if (hyper) add_kind(B_LAPV);
  if (nle > 0) {
    o.le_src = lap_eta_source(0);
    if (!hk.eta_in) add_kind(B_LAPE);
  }
  LAUNCH("bodies", nl += bodies(sch, g, st, s, F(), o) - 1);
  if (hk.eta_in) {
    cudaStreamWaitEvent(st, hk.eta_in, 0);
    o.kinds = B_MASS;
    o.n = 1;
    if (nle > 0) add_kind(B_LAPE);
    LAUNCH("mass", nl += bodies(sch, g, st, s, F(), o) - 1);
  }

  if (tracer) {
    if (fused) {
      LAUNCH("tracer_ab3", pdl_launch(k_tracer_ab3, g, dim3(TX), st, s, b.f[3], b.dtr[0], b.dtr[1], b.dtr[2], fbad));
      rotate3(b.dtr);
    } else {
      LAUNCH("ab", pdl_launch(k_ab, dim3(g), dim3(TX), st, s, k, b.dtrAB, b.dtr[0], b.dtr[1], b.dtr[2]));
      rotate3(b.dtr);
      LAUNCH("add", pdl_launch(k_add, dim3(g), dim3(TX), st, s, b.f[3], b.dtrAB));
      LAUNCH("halo", halo_wrap(b.f[3], s.nx, s.ny, st));
    }
  }
  if (hyper) {
    if (!laplacians_first) eta_laplacians(1, nle);
    if (!fused) LAUNCH("hyper_add", hyper_add(s, g, st, b.deta[0], b.Le[0], b.Le[1], b.Le[2]));
  }
  if (fused) {
    // writes eta's halo images too
    LAUNCH("eta_ab3", fused_tail(s, g, st, F(), b, 0, fbad, last_in_eta ? lap_eta_source(nlap - 1) : nullptr));
    rotate3(b.deta);
  } else {
    LAUNCH("ab", pdl_launch(k_ab, dim3(g), dim3(TX), st, s, k, b.detaAB, b.deta[0], b.deta[1], b.deta[2]));
    LAUNCH("geofactor", pdl_launch(k_geofactor, dim3(g), dim3(TX), st, s, F(), b.detaAB));
    rotate3(b.deta);
    LAUNCH("add", pdl_launch(k_add, dim3(g), dim3(TX), st, s, b.f[0], b.detaAB));
    LAUNCH("halo", halo_wrap(b.f[0], s.nx, s.ny, st));
  }
  if (hk.eta_out) cudaEventRecord(hk.eta_out, st);  // eta is final for this step

  // momentum (core.c:212-280), from the third step in the Coriolis kernels
  if (!fused) {
    auto pres_sum = s.polar == 0 && s.sigma == 0.0 ? k_pres_sum<true> : k_pres_sum<false>;
    LAUNCH("pres_sum", pdl_launch(pres_sum, dim3(g), dim3(TX), st, s, F(), b.duadv, b.dvadv, b.du[0], b.dv[0]));
  }
  if (hyper) {
    // As above: each level but the last rewrites every cell of its two L fields
    // (interior, halo wraps, wall fixes), the last their interior, which is all
    // that is read of it; L of levels not run stay zero.
    const March m = march(s, LVW, 8);
    for (int q = 1; q < nlap; q++)
      LAUNCH("lapv", pdl_launch(k_lapv, m.grid, dim3(TX), st, s, b.L[2 * q - 2], b.L[2 * q - 1], b.L[2 * q],
                                b.L[2 * q + 1], m.rows, q + 1 < nlap));
    if (!fused) {
      LAUNCH("hyper_add", hyper_add(s, g, st, b.du[0], b.L[0], b.L[2], b.L[4]));
      LAUNCH("hyper_add", hyper_add(s, g, st, b.dv[0], b.L[1], b.L[3], b.L[5]));
    }
  }
  if (fused) {
    // AB3 of u and v folded into the Coriolis updates (core.c:271-285); the v
    // tendency does not depend on the new u
    LAUNCH("coriolis_u", fused_tail(s, g, st, F(), b, 1, fbad));
    if (hk.u_out) cudaEventRecord(hk.u_out, st);  // u's interior is final
    LAUNCH("coriolis_v", fused_tail(s, g, st, F(), b, 2, fbad));
    rotate3(b.du);
    rotate3(b.dv);
  } else {
    LAUNCH("ab", pdl_launch(k_ab, dim3(g), dim3(TX), st, s, k, b.duAB, b.du[0], b.du[1], b.du[2]));
    LAUNCH("ab", pdl_launch(k_ab, dim3(g), dim3(TX), st, s, k, b.dvAB, b.dv[0], b.dv[1], b.dv[2]));
    rotate3(b.du);
    rotate3(b.dv);
    // Coriolis (core.c:282-285)
    LAUNCH("coriolis_u", pdl_launch(k_coriolis_u, dim3(g), dim3(TX), st, s, b.f[1], b.f[2], b.duAB));
    if (hk.u_out) cudaEventRecord(hk.u_out, st);
    LAUNCH("coriolis_v", pdl_launch(k_coriolis_v, dim3(g), dim3(TX), st, s, b.f[1], b.f[2], b.dvAB));
  }

  // halos (core.c:287-290)
  if (!whole) LAUNCH("halo", halo_wrap2(b.f[1], b.f[2], s.nx, s.ny, st));
  return nl;
}

// Tail of a step: the reference adds its time-dependent forcing before it
// (core.c:292-294); the halo refresh of tracer and eta that follows the
// forcing (core.c:296-300) is done by the forcing calls themselves, so the
// tail is do_channel and the range checks (core.c:303-312).
int step_tail(const DevState& s, Fp64Buffers& b, bool tracer, StepChecks chk, int slot, cudaStream_t st,
              Timers* tm, bool fused_checks, bool whole) {
  const dim3 g((s.nx + TX - 1) / TX, s.ny);
  const int gw = (s.nx + 127) / 128;
  int nl = 0;
  if (whole) LAUNCH("halo_channel", pdl_launch(k_halo_channel, dim3((s.nx + 4 * (s.ny - 1) + 1 + 127) / 128), dim3(128), st,
                                               s.nx, s.ny, b.f[1], b.f[2], b.f[4], b.f[5], s.plain == 0));
  else if (s.polar == 0) LAUNCH("channel", pdl_launch(k_channel, dim3(gw), dim3(128), st, s.nx, s.ny, b.f[1], b.f[2], b.f[4], b.f[5]));

  // range checks of tracer, eta, u, v (core.c:309-312); an all-zero tracer
  // passes trivially
  RangeFields r{};
  if (tracer) r.f[r.n++] = b.f[3];
  r.f[r.n++] = b.f[0];
  r.f[r.n++] = b.f[1];
  r.f[r.n++] = b.f[2];
  if (!fused_checks) LAUNCH("range", pdl_launch(k_range, dim3(g), dim3(TX), st, s, r, chk.bad + slot));
  return nl;
}
#undef LAUNCH

}  // namespace

int fp64_step(const DevState& s, Fp64Buffers& b, int sch, int k, bool tracer, StepChecks chk, int slot,
              cudaStream_t st, Timers* tm, int parts, StepHooks hk) {
  int nl = 0;
  const bool fused_checks = (parts == STEP_FULL) && tails_fused(s, k);
  const bool whole = (parts == STEP_FULL) && s.polar == 0;  // halos and do_channel in one launch
  if (parts & STEP_HEAD) nl += step_head(s, b, sch, k, tracer, chk, slot, st, tm, fused_checks, whole, hk);
  if (parts & STEP_TAIL) nl += step_tail(s, b, tracer, chk, slot, st, tm, fused_checks, whole);
  return nl;
}

// Compensated sums: each thread accumulates with Neumaier's method, then the
// (sum, error) pairs are combined along a tree with Knuth's TwoSum, so the
// result carries the rounding errors of every addition.
struct Pair {
  double hi, lo;
};
__device__ __forceinline__ Pair two_sum_add(Pair a, Pair b) {
  const double s = a.hi + b.hi;
  const double bb = s - a.hi;
  const double err = (a.hi - (s - bb)) + (b.hi - bb);
  return Pair{s, (a.lo + b.lo) + err};
}
__device__ __forceinline__ void neumaier(double& acc, double& cmp, double term) {
  const double t = acc + term;
  cmp += (fabs(acc) >= fabs(term)) ? ((acc - t) + term) : ((term - t) + acc);
  acc = t;
}
// Block-wide combine of three pairs per thread (blockDim a multiple of 32, <= 1024);
// thread 0 receives the totals.
__device__ __forceinline__ void block_combine3(Pair v[3]) {
  __shared__ double sh[3][2][32];
  for (int o = 16; o > 0; o >>= 1)
    for (int c = 0; c < 3; c++) {
      const Pair w{__shfl_down_sync(0xffffffffu, v[c].hi, o), __shfl_down_sync(0xffffffffu, v[c].lo, o)};
      v[c] = two_sum_add(v[c], w);
    }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0)
    for (int c = 0; c < 3; c++) { sh[c][0][warp] = v[c].hi; sh[c][1][warp] = v[c].lo; }
  __syncthreads();
  if (warp == 0) {
    for (int c = 0; c < 3; c++) v[c] = (lane < nw) ? Pair{sh[c][0][lane], sh[c][1][lane]} : Pair{0.0, 0.0};
    for (int o = 16; o > 0; o >>= 1)
      for (int c = 0; c < 3; c++) {
        const Pair w{__shfl_down_sync(0xffffffffu, v[c].hi, o), __shfl_down_sync(0xffffffffu, v[c].lo, o)};
        v[c] = two_sum_add(v[c], w);
      }
  }
}

// Energy per interior row (energy.c:36-41), compensated over i.
__global__ void k_energy_rows(DevState s, F7 f, double* out) {
  const int W = s.W;
  const int j = blockIdx.x + 1;
  double acc[3] = {0, 0, 0}, cmp[3] = {0, 0, 0};
  const double surf = RW(s, R_SURF, j), gcrow = RW(s, R_GC, j), depth = s.depth;
  for (int i = threadIdx.x + 1; i <= s.nx; i += blockDim.x) {
    const double gc = s.polar ? PF(s, P_GC, IX(W, i, j)) : gcrow;
#define UW(i, j) (f.u[IX(W, i, j)] + f.wx[IX(W, i, j)])
#define VW(i, j) (f.v[IX(W, i, j)] + f.wy[IX(W, i, j)])
#define HH(i, j) (f.eta[IX(W, i, j)] + s.depth - f.hb[IX(W, i, j)])
    const double uc = 0.5 * (UW(i, j) + UW(i - 1, j));
    const double vc = 0.5 * (VW(i, j) + VW(i, j - 1));
    const double w0 = f.wx[IX(W, i, j)], w1 = f.wy[IX(W, i, j)];
    const double h = HH(i, j);
    const double term[3] = {0.5 * h * (uc * uc + vc * vc) * surf - 0.5 * ((w0 * w0) + (w1 * w1)) * surf,
                            0.5 * gc * (h * h) * surf - 0.5 * gc * (depth * depth) * surf, h * surf};
#undef UW
#undef VW
#undef HH
    for (int c = 0; c < 3; c++) neumaier(acc[c], cmp[c], term[c]);
  }
  Pair v[3] = {{acc[0], cmp[0]}, {acc[1], cmp[1]}, {acc[2], cmp[2]}};
  block_combine3(v);
  if (threadIdx.x == 0)
    for (int c = 0; c < 3; c++) out[3 * (j - 1) + c] = v[c].hi + v[c].lo;
}

__global__ void k_energy_sum(const double* rows, int ny, double* out) {
  double acc[3] = {0, 0, 0}, cmp[3] = {0, 0, 0};
  for (int j = threadIdx.x; j < ny; j += blockDim.x)
    for (int c = 0; c < 3; c++) neumaier(acc[c], cmp[c], rows[3 * j + c]);
  Pair v[3] = {{acc[0], cmp[0]}, {acc[1], cmp[1]}, {acc[2], cmp[2]}};
  block_combine3(v);
  if (threadIdx.x == 0)
    for (int c = 0; c < 3; c++) out[c] = v[c].hi + v[c].lo;
}

void energy_rows(const DevState& s, const double* const* f, double* row_out, cudaStream_t st) {
  k_energy_rows<<<s.ny, 256, 0, st>>>(s, F7{f[0], f[1], f[2], f[3], f[4], f[5], f[6]}, row_out);
}

void energy_sum(const double* row_in, int ny, double* out3, cudaStream_t st) {
  k_energy_sum<<<1, 1024, 0, st>>>(row_in, ny, out3);
}

}  // namespace sw2g
