// qt_wsd.cu -- weighted simultaneous diagonalisation of the CDVR grids
// (LayerGrid with several matrices, src/DVR/TDDVR.cpp:72-88, around
// WeightedSimultaneousDiagonalization::calculate,
// src/Util/WeightedSimultaneousDiagonalization.cpp:5-378, and the Jacobi
// rotation helpers of src/Core/JacobiRotationFramework.cpp:4-164).
//
// One block of four warps per problem.  The iteration accepts or rejects
// optimiser steps on comparisons of nearly equal numbers, so its result is a
// discontinuous function of the inputs; this file therefore fixes one
// operation order, which the CPU restatement follows bit for bit:
//  * compiled with -fmad=false: no multiply-add is fused; a complex product
//    is (ac - bd) + i(ad + bc) (a Givens rotation's real c multiplies both
//    parts alone), sums run left to right; a sum over the
//    matrices of a problem is the pairwise tree of the values padded with
//    zeros to a power of two, and the measure adds its per-matrix traces in
//    index order;
//  * |z| is sqrt(re^2 + im^2); real(x / w) is (xr wr + xi wi) / (wr^2 + wi^2);
//    the rotated diagonals of a candidate rotation use the Hermitian form
//    c^2 A_pp + 2c Re(s A_pq) + |s|^2 A_qq (c is real);
//  * the optimiser's 3x3 eigenvector (Matrix::rDiag) comes from the largest
//    root of the characteristic polynomial of H scaled by a power of two
//    (binary32 Newton from the Gershgorin bound, then binary64 Newton from
//    that root plus 2^-17 with binary32 step quotients, until a step is
//    below 2^-30) and the largest cross product of two rows of H - lambda.
//
// Execution on this GPU: an FP64 instruction occupies its sub-partition's unit
// for 64 cycles, a dependent one follows after 73, a division takes 570 and a
// square root 620, whatever the number of active lanes, and the optimiser is
// one long dependency chain of them (about 2000 candidate evaluations of 120
// FP64 instructions each per problem, in sequence).  So:
//  * warp 0 (the master) runs the optimiser's scalar chain; every lane holds
//    the same values, and independent operations of the chain go to different
//    lanes of ONE instruction (results fetched by shuffles) instead of one
//    after another.  Comparisons, powers of two and conversions to and from
//    binary32 work on the bits: an integer instruction takes 4 cycles;
//  * all four warps evaluate the candidates (rotated diagonals of every matrix
//    at ten rotations, the tree sums) and run the Givens rotations and the
//    products of the off-diagonality measure.  During the optimisation the
//    other warps wait in a loop of their own for the master's next candidates,
//    two barriers per evaluation;
//  * the matrices live in shared memory when they fit (else in the task's
//    global scratch).
// Eight modes, bonds 7 (20 problems of 2..8 matrices): 19.2 -> 13.0 ms in this
// kernel, the whole sweep 21.8 -> 15.9 ms alone, against one thread of control
// for all warps, one FP64 instruction per comparison, pairs of matrices per
// lane and descriptors decoded at each use.
// All loops are bounded (at most 25 sweeps, 30 optimiser iterations, 64 step
// halvings per search, 40 + 100 Newton steps).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "qt_internal.h"

namespace qt {
namespace {

constexpr int kWsdThreads = 128;
constexpr unsigned kFull = 0xffffffffu;
constexpr double kDelta = 1E-5;  // step of the central differences
constexpr double kEps = 1E-3;    // the optimiser starts at s = (eps, -eps)
constexpr int kWsdSmemBudget = 220 * 1024;

__device__ __forceinline__ double2 cm(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 ca(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 cs(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cc(double2 a) { return make_double2(a.x, -a.y); }
// product with the real c of a rotation: (c x.re, c x.im)
__device__ __forceinline__ double2 rm(double2 c, double2 a) { return make_double2(c.x * a.x, c.x * a.y); }
__device__ __forceinline__ double cabs_(double2 a) { return sqrt(a.x * a.x + a.y * a.y); }
__device__ __forceinline__ double cdiv_re(double2 x, double2 w) {
  return (x.x * w.x + x.y * w.y) / (w.x * w.x + w.y * w.y);
}
__device__ __forceinline__ void bsync() { __syncthreads(); }
// the same barrier, reached by the master warp and by the others from different loops
__device__ __forceinline__ void role_sync() { asm volatile("barrier.sync 1, %0;" ::"n"(kWsdThreads) : "memory"); }

// binary64 -> binary32 by truncation of the significand; zero below 2^-126,
// infinity above the binary32 range (integer operations only)
__device__ __forceinline__ float f32_trunc(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), sign = hi & 0x80000000u, mag = hi & 0x7fffffffu;
  // the exponent's low nine bits and the significand, rebiased modulo 2^9
  unsigned r = (__funnelshift_l((unsigned)__double2loint(x), hi, 3) + 0x40000000u) | sign;
  if (mag < 0x38100000u) r = sign;
  if (mag >= 0x47f00000u) r = sign | 0x7f800000u;
  return __uint_as_float(r);
}
// binary32 -> binary64, exact for normal numbers; subnormals become zero
__device__ __forceinline__ double f64_of(float f) {
  const unsigned r = __float_as_uint(f), sign = r & 0x80000000u, mag = r & 0x7fffffffu;
  unsigned hi = sign | ((mag >> 3) + 0x38000000u), lo = r << 29;
  if (mag >= 0x7f800000u) hi = sign | 0x7ff00000u | ((mag & 0x7fffffu) >> 3);
  if (mag < 0x00800000u) {
    hi = sign;
    lo = 0;
  }
  return __hiloint2double((int)hi, (int)lo);
}

// a level's operation in one lane: the source lanes x | y << 5 (sign bit: of
// the addend's flip) and the masks of the factor and the addend.  A lane
// without an operation keeps its value as S - (+0), the zero from slot 5.
struct LaneOp {
  uint32_t src, gm, am;
};
constexpr int kEigLevels = 11;

struct Prob {
  int d, n;
  int lgG, m;     // G = 2^lgG lanes per tree over the matrices, m matrices per lane: G m = n padded to a power of two
  int chunk;   // matrices per pass of the off-diagonality measure
  double2* xw;  // n weighted matrices
  double2* xp;  // n plain (shifted) matrices
  double2* w;   // weight
  double2* T;   // transformation
  double2* tM;  // chunk x d^2: X T, then Y Y
  double2* tY;  // chunk x d^2: Y
  double2* blk;   // (n + 1) x 4: (pp, pq, qp, qq) of every matrix and of w at the current pair
  double2* cand0;  // 10 x 2: the first candidates of every pair
  double2* cand;  // 10 x 2: candidate ((c, |s|^2), s)
  double2* rot;   // the accepted rotation (c, s) of the pair
  double* sq;     // 2 x 10: sums of the squared rotated diagonals per candidate
  double* wd;     // 10 x 2: rotated diagonals of w per candidate
  double* tr;     // chunk x d: diagonal of W Z per matrix
  double* val;    // 2: broadcast values
  int* ctl;       // 1: the master's loop decision (0: done; 1, 2: evaluate cand0, cand)
  // the master's lanes:
  LaneOp eig[kEigLevels];    // the eigenproblem's levels
  double den, zh, zl;        // divisor of the central differences; 1 / den as zh + zl
  uint32_t diff;             // their terms: lanes of A, B, C, D (5 bits each), the sign of B
  double dx;                 // the candidate's offset from s in the lane's component
  double c0, sab0;           // c and |s| of the first candidate
  __device__ double2* X(int k) const { return xw + (int64_t)k * d * d; }
  __device__ double2* Xp(int k) const { return xp + (int64_t)k * d * d; }
};

// ---- master warp: the optimiser's scalar chain --------------------------------

// ---- lane-vectorised evaluation ------------------------------------------------
// An FP64 instruction occupies the SM sub-partition's FP64 unit for the same
// time whether or not it depends on the previous one, so the scalar chain
// costs one unit slot per instruction.  Independent multiplies, adds and
// subtracts of one level therefore go into ONE fused multiply-add across
// the lanes: x*y as fma(x, y, -0), x + y as fma(x, 1, y), x - y as
// fma(x, 1, -y) -- each rounds exactly once, like the separate operation
// (the -0 addend keeps the sign of a zero product).  A level's operands are
// shuffled from a slot vector S (lane l holds value #l); lane descriptors
// (three words per lane and level, in registers) name the source slots and
// mask the factor and the addend.

// -x and |x| on the sign bit (integer instructions, the IEEE results)
__device__ __forceinline__ double neg_bits(double x) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ull);
}
__device__ __forceinline__ double abs_bits(double x) {
  return __longlong_as_double(__double_as_longlong(x) & 0x7fffffffffffffffll);
}

enum { OP_SUB = 0, OP_MUL, OP_ADD, OP_ADDABS };
constexpr uint32_t lane_desc(int x, int y, int op) { return (uint32_t)x | ((uint32_t)y << 5) | ((uint32_t)op << 10); }
__device__ __forceinline__ LaneOp lane_op(uint32_t dsc, int lane) {
  if (dsc == 0) dsc = (uint32_t)lane | (5u << 5);
  const int op = (int)(dsc >> 10);
  LaneOp o;
  o.src = (dsc & 0x3ffu) | (op <= OP_MUL ? 0x80000000u : 0u);
  o.gm = op == OP_MUL ? 0xffffffffu : 0u;
  o.am = op == OP_MUL ? 0u : (op == OP_ADDABS ? 0x7fffffffu : 0xffffffffu);
  return o;
}
__device__ __forceinline__ double lane_level(double S, const LaneOp& o) {
  const double x = __shfl_sync(kFull, S, (int)(o.src & 31));
  const double y = __shfl_sync(kFull, S, (int)((o.src >> 5) & 31));
  const uint32_t yh = (uint32_t)__double2hiint(y), yl = (uint32_t)__double2loint(y);
  const uint32_t gh = (yh & o.gm) | (~o.gm & 0x3ff00000u);            // y or 1
  const uint32_t hh = (yh & o.am) ^ (o.src & 0x80000000u);            // -0 or +-y or |y|
  return __fma_rn(x, __hiloint2double((int)gh, (int)(yl & o.gm)), __hiloint2double((int)hh, (int)(yl & ~o.gm)));
}
// Comparisons of binary64 values by their bits (integer instructions; the
// same truth values as the floating-point comparison, NaN included):
// x < 0; x > 0; x > c for a constant c > 0
__device__ __forceinline__ unsigned long long bits_of(double x) { return (unsigned long long)__double_as_longlong(x); }
__device__ __forceinline__ bool is_negative(double x) {
  return bits_of(x) - 0x8000000000000001ull <= 0x7fefffffffffffffull;
}
__device__ __forceinline__ bool is_positive(double x) { return bits_of(x) - 1 <= 0x7fefffffffffffffull; }
__device__ __forceinline__ bool gt_pos(double x, double c) {
  return bits_of(x) - (bits_of(c) + 1) <= 0x7ff0000000000000ull - (bits_of(c) + 1);
}
// x < y of any two values; x > y of two that are not below zero (sums of squares) or NaN
__device__ __forceinline__ bool less(double x, double y) {
  const long long inf = 0x7ff0000000000000ll, mask = 0x7fffffffffffffffll;
  const long long a = __double_as_longlong(x), b = __double_as_longlong(y);
  const long long am = a & mask, bm = b & mask;
  return am <= inf && bm <= inf && (a < 0 ? -am : am) < (b < 0 ? -bm : bm);
}
__device__ __forceinline__ bool greater_pos(double x, double y) {
  const unsigned long long inf = 0x7ff0000000000000ull, a = bits_of(x), b = bits_of(y);
  return a > b && a <= inf && b <= inf;
}
// 2 x: the exponent of a normal number below 2^1023
__device__ __forceinline__ double twice(double x) {
  const unsigned h = (unsigned)__double2hiint(x);
  if ((h & 0x7fffffffu) - 0x00100000u < 0x7fd00000u) return __hiloint2double((int)(h + 0x00100000u), __double2loint(x));
  return (bits_of(x) << 1) == 0 ? x : x + x;
}
// a / 2 and a * 2 for a power of two a in the normal range: the exponent
__device__ __forceinline__ double half_pow2(double a) { return __longlong_as_double((long long)(bits_of(a) - (1ull << 52))); }
__device__ __forceinline__ double twice_pow2(double a) { return __longlong_as_double((long long)(bits_of(a) + (1ull << 52))); }

// p / dp as a call, so that the rare fallback of the Newton step is a branch
// and not an always-executed division
__device__ __noinline__ double exact_quotient(double p, double dp) { return p / dp; }

// Levels of the 3x3 eigenproblem (kEigLevels).  Slots at entry: 0 h00, 1 h01, 2 h11,
// 3 h02, 4 h12, 5 h22 (= 0).
enum { EL_C1 = 0, EL_C2, EL_C3, EL_C4, EL_C5, EL_E1, EL_E2, EL_E3, EL_E4, EL_E5, EL_E6 };
__constant__ uint32_t c_eig_lut[kEigLevels][32] = {
    // C1: the products of m and det, (h00 + h11), the Gershgorin rows' first sums
    {0, 0, 0, 0, 0, 0, 0, 0,
     lane_desc(0, 2, OP_MUL), lane_desc(1, 1, OP_MUL), lane_desc(0, 5, OP_MUL), lane_desc(3, 3, OP_MUL),
     lane_desc(2, 5, OP_MUL), lane_desc(4, 4, OP_MUL), lane_desc(1, 5, OP_MUL), lane_desc(4, 3, OP_MUL),
     lane_desc(1, 4, OP_MUL), lane_desc(2, 3, OP_MUL), lane_desc(0, 2, OP_ADD), lane_desc(0, 1, OP_ADDABS),
     lane_desc(2, 1, OP_ADDABS), lane_desc(5, 3, OP_ADDABS)},
    // C2: the three terms of m, the inner terms of det, tr, the Gershgorin rows
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0,
     lane_desc(8, 9, OP_SUB), lane_desc(10, 11, OP_SUB), lane_desc(12, 13, OP_SUB), lane_desc(14, 15, OP_SUB),
     lane_desc(16, 17, OP_SUB), lane_desc(18, 5, OP_ADD), lane_desc(19, 3, OP_ADDABS), lane_desc(20, 4, OP_ADDABS),
     lane_desc(21, 4, OP_ADDABS)},
    // C3: the outer products of det, the first sum of m, 2 tr
    {0, 0, 0, 0, 0, 0, 0, 0, lane_desc(0, 24, OP_MUL), lane_desc(1, 25, OP_MUL), lane_desc(3, 26, OP_MUL),
     lane_desc(22, 23, OP_ADD), lane_desc(27, 27, OP_ADD)},
    // C4
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, lane_desc(8, 9, OP_SUB), lane_desc(11, 24, OP_ADD)},
    // C5: det
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, lane_desc(13, 10, OP_ADD)},
    // E1: m00, m11, m22 (lambda in slot 31)
    {0, 0, 0, 0, 0, 0, lane_desc(0, 31, OP_SUB), lane_desc(2, 31, OP_SUB), lane_desc(5, 31, OP_SUB)},
    // E2: the products of the three cross products (slots 6 m00, 7 m11, 8 m22)
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0,
     lane_desc(1, 4, OP_MUL), lane_desc(3, 7, OP_MUL), lane_desc(3, 1, OP_MUL), lane_desc(6, 4, OP_MUL),
     lane_desc(6, 7, OP_MUL), lane_desc(1, 1, OP_MUL), lane_desc(1, 8, OP_MUL), lane_desc(3, 4, OP_MUL),
     lane_desc(3, 3, OP_MUL), lane_desc(6, 8, OP_MUL), lane_desc(7, 8, OP_MUL), lane_desc(4, 4, OP_MUL)},
    // E3: components c01 (9..11), c02 (12..14), c12 (15..17)
    {0, 0, 0, 0, 0, 0, 0, 0, 0,
     lane_desc(16, 17, OP_SUB), lane_desc(18, 19, OP_SUB), lane_desc(20, 21, OP_SUB), lane_desc(22, 23, OP_SUB),
     lane_desc(24, 25, OP_SUB), lane_desc(19, 18, OP_SUB), lane_desc(26, 27, OP_SUB), lane_desc(23, 22, OP_SUB),
     lane_desc(16, 17, OP_SUB)},
    // E4: their squares (18..26)
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0,
     lane_desc(9, 9, OP_MUL), lane_desc(10, 10, OP_MUL), lane_desc(11, 11, OP_MUL), lane_desc(12, 12, OP_MUL),
     lane_desc(13, 13, OP_MUL), lane_desc(14, 14, OP_MUL), lane_desc(15, 15, OP_MUL), lane_desc(16, 16, OP_MUL),
     lane_desc(17, 17, OP_MUL)},
    // E5: v0^2 + v1^2 of each (27..29)
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0,
     lane_desc(18, 19, OP_ADD), lane_desc(21, 22, OP_ADD), lane_desc(24, 25, OP_ADD)},
    // E6: the squared norms (0..2)
    {lane_desc(27, 20, OP_ADD), lane_desc(28, 23, OP_ADD), lane_desc(29, 26, OP_ADD)},
};

// Matrix::rDiag of the optimiser's symmetric 3x3 matrix (rfoBuildHessian,
// src/Core/JacobiRotationFramework.cpp:114-127: h00 = pre0 a^2, h01 = pre2 a^2,
// h11 = pre3 a^2, h02 = grad0 a, h12 = grad1 a, h22 = 0): the eigenvector of
// the largest eigenvalue as u0 = v0/v2, u1 = v1/v2 and v0^2 + v1^2 for |v| = 1.
// Whole warp 0, every lane the same inputs and outputs.
__device__ void eig3_top(const LaneOp (&lut)[kEigLevels], double p0, double p2, double p3, double g0, double g1,
                         double a, double* u0, double* u1, double* top2) {
  const int l = threadIdx.x & 31;
  double S = l == 0 ? p0 : (l == 1 ? p2 : (l == 2 ? p3 : (l == 3 ? g0 : (l == 4 ? g1 : 0.0))));
  {
    // times a^2 or a, then by 2^(1023 - e), e the largest biased exponent, so
    // that max |entry| is in [1, 2).  a is a power of two <= 1: where no
    // result leaves the normal range, all of it adds to the exponents
    const int ex = (int)(bits_of(S) >> 52) & 0x7ff;
    const bool zero = (bits_of(S) << 1) == 0;
    const int ea = ((int)(bits_of(a) >> 52) - 1023) * (l < 3 ? 2 : 1);
    const int e1 = zero ? 0 : ex + ea;
    const int e = __reduce_max_sync(kFull, e1);
    if (__all_sync(kFull, zero || (ex >= 1 && ex <= 2045 && e1 >= 1 && e1 + 1023 - e >= 1))) {
      if (!zero) S = __longlong_as_double(__double_as_longlong(S) + ((long long)(ea + 1023 - e) << 52));
    } else {
      S = S * a;
      S = S * (l < 3 ? a : 1.0);
      int es = l < 5 ? (int)(bits_of(S) >> 52) & 0x7ff : 0;
      es = __reduce_max_sync(kFull, es);
      if (es >= 1 && es <= 2045) S = S * __longlong_as_double((long long)(2046 - es) << 52);
      if (l >= 5) S = 0.0;
    }
  }
  const float fS = f32_trunc(S);
  // tr = (h00 + h11) + h22; m and det as three terms each; Gershgorin rows
  S = lane_level(S, lut[EL_C1]);
  // binary32 Newton from the Gershgorin bound: p(l) = -l^3 + tr l^2 - m l + det.
  // Its preparation and first steps run under the binary64 levels C1 .. C5
  const float f00 = __shfl_sync(kFull, fS, 0), f01 = __shfl_sync(kFull, fS, 1), f11 = __shfl_sync(kFull, fS, 2);
  const float f02 = __shfl_sync(kFull, fS, 3), f12 = __shfl_sync(kFull, fS, 4), f22 = 0.0f;
  const float ftr = f00 + f11 + f22;
  const float fm = (f00 * f11 - f01 * f01) + (f00 * f22 - f02 * f02) + (f11 * f22 - f12 * f12);
  const float fdet = f00 * (f11 * f22 - f12 * f12) - f01 * (f01 * f22 - f12 * f02) + f02 * (f01 * f12 - f11 * f02);
  S = lane_level(S, lut[EL_C2]);
  const float fg = f32_trunc(S);  // truncation keeps the order of the rows
  S = lane_level(S, lut[EL_C3]);
  float fl = __shfl_sync(kFull, fg, 28);
  const float fr1 = __shfl_sync(kFull, fg, 29), fr2 = __shfl_sync(kFull, fg, 30);
  if (fr1 > fl) fl = fr1;
  if (fr2 > fl) fl = fr2;
  auto newton32 = [&]() {  // one step; false when the iteration ends
    const float p = ((-fl + ftr) * fl - fm) * fl + fdet;
    const float dp = (-3.0f * fl + 2.0f * ftr) * fl - fm;
    if (!(dp < 0.0f)) return false;
    const float nx = fl - p / dp;
    if (!(nx < fl)) return false;
    fl = nx;
    return true;
  };
  bool more = newton32();
  S = lane_level(S, lut[EL_C4]);
  if (more) more = newton32();
  S = lane_level(S, lut[EL_C5]);
  for (int it = 2; more && it < 40; ++it) more = newton32();
  const double tr = __shfl_sync(kFull, S, 27), tr2 = __shfl_sync(kFull, S, 12);
  const double m = __shfl_sync(kFull, S, 14), det = __shfl_sync(kFull, S, 15);
  // binary64 Newton, monotone from above.  p = ((-lam + tr) lam - m) lam + det
  // in lane 0 and p' = (-3 lam + 2 tr) lam - m in lane 1, one instruction
  // per step of both chains; 3 lam in lane 2.
  double lam = f64_of(fl) + 0x1p-17;
  // (every step takes v as one factor, so that no selection waits for it)
  const double neg_m = neg_bits(m);
  const double k1 = l == 0 ? -1.0 : (l == 1 ? -3.0 : 3.0);
  const double a1 = l == 0 ? tr : -0.0, a2 = l == 1 ? tr2 : -0.0;
  const double a3 = l == 0 ? neg_m : -0.0, a4 = l == 0 ? -0.0 : neg_m;
  double pv;      // p in lane 0, p' in lane 1
  unsigned negs;  // bit 0: p < 0, bit 1: p' < 0
  auto pdp = [&]() {
    const double even = l == 1 ? 1.0 : lam, odd = l == 0 ? 1.0 : lam, last = l == 0 ? lam : 1.0;
    const double v1 = __fma_rn(k1, lam, a1);
    double v = __fma_rn(v1, even, a2);
    v = __fma_rn(v, odd, a3);
    v = __fma_rn(v, last, a4);
    pv = l == 0 ? __fma_rn(v, 1.0, det) : v;
    negs = __ballot_sync(kFull, is_negative(pv));
    return v1;  // 3 lam in lane 2
  };
  const double l3 = __shfl_sync(kFull, pdp(), 2);
  if (!((negs & 3) == 3 && less(tr, l3))) {
    lam = __shfl_sync(kFull, S, 28);  // the Gershgorin bound
    const double r1 = __shfl_sync(kFull, S, 29), r2 = __shfl_sync(kFull, S, 30);
    if (less(lam, r1)) lam = r1;
    if (less(lam, r2)) lam = r2;
    pdp();
  }
  for (int it = 0; it < 100; ++it) {
    if (!(negs & 2)) break;
    const float fv = f32_trunc(pv);
    double step = f64_of(__shfl_sync(kFull, fv, 0) / __shfl_sync(kFull, fv, 1));
    if (!((bits_of(step) & 0x7fffffffffffffffull) <= 0x4030000000000000ull))
      // |step| > 16 or NaN: the binary32 quotient left its range
      step = exact_quotient(__shfl_sync(kFull, pv, 0), __shfl_sync(kFull, pv, 1));
    const double nxt = lam - step;
    if (!(is_positive(step) && bits_of(nxt) != bits_of(lam))) break;  // nxt < lam
    lam = nxt;
    // step > 0 here: compare the bits with those of 2^-30
    if (bits_of(step) <= 0x3e10000000000000ull) break;
    pdp();
  }
  // eigenvector: the largest cross product of two rows of H - lambda
  if (l == 31) S = lam;
#pragma unroll
  for (int k = EL_E1; k <= EL_E6; ++k) S = lane_level(S, lut[k]);
  const double n01 = __shfl_sync(kFull, S, 0), n02 = __shfl_sync(kFull, S, 1), n12 = __shfl_sync(kFull, S, 2);
  int sel = 0;
  double nv = n01;
  if (greater_pos(n02, nv)) {
    sel = 1;
    nv = n02;
  }
  if (greater_pos(n12, nv)) sel = 2;
  // u0 = v0 / v2, u1 = v1 / v2, top2 = (v0^2 + v1^2) / |v|^2 in lanes 0, 1, 2
  const double num = __shfl_sync(kFull, S, l == 0 ? 9 + 3 * sel : (l == 1 ? 10 + 3 * sel : 27 + sel));
  const double den = __shfl_sync(kFull, S, l < 2 ? 11 + 3 * sel : sel);
  const double r = num / den;
  *u0 = __shfl_sync(kFull, r, 0);
  *u1 = __shfl_sync(kFull, r, 1);
  *top2 = __shfl_sync(kFull, r, 2);
}

// weightedJacobiDerivatives from the loss at the nine points (i, j) of the
// central differences (y[i + 3 j]): lane k takes numerator k as
// ((A + B) - C) - D (a difference x - y as x + (-y); subtracting +0 keeps
// every value) and one division by the lane's constant gives all five
// quotients: q0 = num zh + num zl is within an ulp of num / den, its remainder
// is exact, and the remainder times zh = fl(1 / den) corrects it to the rounded
// quotient (Markstein's theorem; four dependent operations of 73 cycles, a
// division takes 570).  Numbers near the ends of the range take the division.
// y: lane 1 + (i + 3 j) holds y[i + 3 j], lane 31 zero.
__device__ void grad_pre(const Prob& P, double y, double& g0, double& g1, double& p0, double& p2, double& p3) {
  const int l = threadIdx.x & 31;
  const double A = __shfl_sync(kFull, y, P.diff & 31);
  double B = __shfl_sync(kFull, y, (P.diff >> 5) & 31);
  double C = __shfl_sync(kFull, y, (P.diff >> 10) & 31);
  const double D = __shfl_sync(kFull, y, (P.diff >> 15) & 31);
  if (P.diff >> 20) B = neg_bits(B);
  if (l == 2 || l == 3) C = twice(C);
  const double num = ((A + B) - C) - D;
  const double q0 = __fma_rn(num, P.zh, num * P.zl);
  double r = __fma_rn(__fma_rn(neg_bits(q0), P.den, num), P.zh, q0);
  const unsigned e = (unsigned)(bits_of(num) >> 52) & 0x7ffu;
  if (e < 100 || e > 1900) r = (bits_of(num) << 1) == 0 ? num : exact_quotient(num, P.den);
  g0 = __shfl_sync(kFull, r, 0);
  g1 = __shfl_sync(kFull, r, 1);
  p0 = __shfl_sync(kFull, r, 2);
  p3 = __shfl_sync(kFull, r, 3);
  p2 = __shfl_sync(kFull, r, 4);
}

// Candidate 0 = (sqrt|1 - z0|, s) and the nine samples of the central
// differences around s (weightedJacobiDerivatives) into cand, one square
// root per lane (lanes 0..9); lane 10 takes sqrt(y0^2 + y1^2).  Returns each
// lane's root; z: its |x|^2 (lane 10: y0^2 + y1^2).
__device__ double put_candidates(const Prob& P, double2* cand, double z0, double sx, double sy, double y0, double y1,
                                 double& z) {
  const int l = threadIdx.x & 31, k = l & 15;
  // component 0 of s + ((i - 1) delta, (j - 1) delta) in lane k, component 1 in lane 16 + k; x + -0 keeps every x
  const double x = (k == 10 ? (l < 16 ? y0 : y1) : (l < 16 ? sx : sy)) + P.dx;
  const double x2 = x * x;
  z = x2 + __shfl_xor_sync(kFull, x2, 16);
  const double arg = 1 - (k == 0 ? z0 : z);
  const double r = sqrt(k == 10 ? z : abs_bits(arg));
  if (k <= 9) {
    if (l < 16) cand[2 * k] = make_double2(r, z);
    (l < 16 ? cand[2 * k + 1].x : cand[2 * k + 1].y) = x;
  }
  return r;
}

// ---- parallel phases (all warps) ------------------------------------------------

// rotatedDiagonals of a cached 2x2 block (pp, pq, qp, qq) of a Hermitian
// matrix for a real c: a0 = c^2 A_pp + 2c Re(s A_pq) + |s|^2 A_qq and
// a1 = c^2 A_qq - 2c Re(s A_pq) + |s|^2 A_pp (cc2 = c^2, c2 = 2c, ss2 = |s|^2)
__device__ __forceinline__ void rotated_diagonals(const double2* b, double cc2, double c2, double ss2, double2 s,
                                                  double& a0, double& a1) {
  const double2 apq = b[1];
  const double t = s.x * apq.x - s.y * apq.y;
  const double ct = c2 * t;
  a0 = (cc2 * b[0].x + ct) + ss2 * b[3].x;
  a1 = (cc2 * b[3].x - ct) + ss2 * b[0].x;
}

// The pairwise tree over the matrices, two sums at once: a lane's m (a power
// of two) consecutive leaves f(0..m-1) ..
template <class F>
__device__ __forceinline__ void local_tree(int m, F f, double& s0, double& s1) {
  f(0, s0, s1);
  if (m == 1) return;
  double b0, b1;
  f(1, b0, b1);
  s0 = s0 + b0;
  s1 = s1 + b1;
  if (m == 2) return;
  double st0[12], st1[12];  // finished subtrees of 2, 4, 8, .. leaves
  st0[0] = s0;
  st1[0] = s1;
  for (int i = 2; i < m; i += 2) {
    double a0, a1;
    f(i, a0, a1);
    f(i + 1, b0, b1);
    s0 = a0 + b0;
    s1 = a1 + b1;
    int lev = 0;
    for (int k = i >> 1; k & 1; k >>= 1, ++lev) {
      s0 = st0[lev] + s0;
      s1 = st1[lev] + s1;
    }
    st0[lev] = s0;
    st1[lev] = s1;
  }
}
// .. then the G lanes of a group (a power of two up to 32): the group's even
// lanes return the first sum, the odd ones the second, one addition per level
// for both.  Whole warp.
__device__ __forceinline__ double lane_tree(double s0, double s1, int G) {
  const bool odd = threadIdx.x & 1;
  const double other = __shfl_xor_sync(kFull, odd ? s0 : s1, 1);
  if (G == 1) return odd ? other : s0;  // lane 0's two sums in lanes 0 and 1
  double v = (odd ? s1 : s0) + other;
  for (int off = 2; off < G; off <<= 1) v = v + __shfl_xor_sync(kFull, v, off);
  return v;
}

// Ten candidates (all warps): G lanes per candidate add the
// squared rotated diagonals of the matrices, one more lane per candidate
// rotates w's.  An FP64 instruction costs the same for one lane as for 32, so
// up to eight matrices have a lane each, and the tree runs through shuffles.
// Pairs of matrices per lane with the tree's levels in shared memory, a
// barrier after each, took 4.6 k cycles per call for eight matrices, this
// form 1.9 k.  One copy of the code for all warps: the
// kernel's loop body is larger than the instruction cache next to the warps.
__device__ __forceinline__ void eval_items(const double2* blk, const double2* cand, double* sq, double* wd, int n, int lgG,
                                        int m) {
  const int G = 1 << lgG, lane = threadIdx.x & 31;
  const int total = 10 * G + 10;
  for (int it0 = threadIdx.x - lane; it0 < total; it0 += kWsdThreads) {
    const int it = it0 + lane;
    const bool isw = it >= 10 * G;
    const int j = isw ? min(it - 10 * G, 9) : it >> lgG, g = isw ? 0 : it & (G - 1);
    const double2 c = cand[2 * j], s = cand[2 * j + 1];
    const double cc2 = c.x * c.x, c2 = twice(c.x), ss2 = c.y;
    double s0, s1, w0 = 0.0, w1 = 0.0;
    local_tree(m, [&](int q, double& v0, double& v1) {
      const int k = isw ? n : g * m + q;
      v0 = v1 = 0.0;
      if (isw ? q == 0 : k < n) {
        double r0, r1;
        rotated_diagonals(blk + 4 * k, cc2, c2, ss2, s, r0, r1);
        if (q == 0) {
          w0 = r0;
          w1 = r1;
        }
        v0 = r0 * r0;
        v1 = r1 * r1;
      }
    }, s0, s1);
    const double v = lane_tree(s0, s1, G);
    if (isw) {
      if (it < total) {
        wd[2 * j] = w0;
        wd[2 * j + 1] = w1;
      }
    } else if (G == 1) {
      sq[j] = s0;
      sq[10 + j] = s1;
    } else if (g < 2) {
      sq[10 * g + j] = v;
    }
  }
}

// weightedJacobiLoc for the ten candidates in P.cand0 (which 1) or P.cand (2); xo0, xo1 = xold / w
// of the pair.  Master warp, with the other warps in their loop of
// rotations().  Returns the loss change of candidate j in lane j and
// xnum / xden (a division of the caller's, issued with the same instruction)
// in lane 20.
__device__ __forceinline__ double loc_many(const Prob& P, int which, double xo0, double xo1, double xnum, double xden) {
  const int l = threadIdx.x & 31;
  if (l == 0) P.ctl[0] = which;
  role_sync();
  eval_items(P.blk, which == 1 ? P.cand0 : P.cand, P.sq, P.wd, P.n, P.lgG, P.m);
  role_sync();
  // diff = (xnew0 / w0 - xold0 / w_pp) + (xnew1 / w1 - xold1 / w_qq), one division per lane
  double num = xnum, den = xden;
  if (l < 20) {
    const int c = l >= 10 ? 1 : 0, j = l - 10 * c;
    num = P.sq[l];
    den = P.wd[2 * j + c];
  }
  const double q = num / den;
  double t = q - (l < 10 ? xo0 : xo1);
  const double t1 = __shfl_sync(kFull, t, (l + 10) & 31);
  if ((bits_of(t) << 1) == 0) t = 0.0;  // 0 + t: a zero of either sign becomes +0
  return l < 10 ? t + t1 : q;
}

// calculateWeightedAngles: rational function optimisation of (c, s), into
// P.rot.  The loss of every new candidate is evaluated together with the nine
// samples of the central differences around it: if the candidate is accepted
// they are the next iteration's derivatives, if not the derivatives at the
// unchanged point are still valid -- the same numbers the reference
// recomputes.  Master warp.
__device__ void angles(const Prob& P, double xo0, double xo1) {
  const int lane = threadIdx.x & 31;
  const double eps = kEps, amin = 1E-12, amax = 1;
  double a = amax, diff_rel = 2 * eps * eps;
  double c0 = P.c0, s0 = eps, s1 = -eps, sab = P.sab0, loc_alt = 0;
  double cur = 0;  // loss changes of the current point (lane 0) and its samples (lanes 1..9)
  double g0 = 0, g1 = 0, p0 = 0, p2 = 0, p3 = 0;
  double cnew = 0, snew0 = 0, snew1 = 0, zab = 0, top2 = 0, xden = 1;
  int which = 1, iter = 0, guard = 0;
  for (;;) {
    const double res = loc_many(P, which, xo0, xo1, top2, xden);
    const double loc_new = __shfl_sync(kFull, res, 0);
    bool search = false;  // another step length at the same point
    if (which == 1) {
      which = 2;
      cur = res;
      loc_alt = loc_new;
    } else {
      diff_rel = __shfl_sync(kFull, res, 20);  // |trafo|^2 / (|s|^2 + eps^2)
      const double diff = loc_new - loc_alt;
      if (is_negative(diff)) {
        a = half_pow2(a);
      } else {
        if (bits_of(a) < bits_of(amax)) a = twice_pow2(a);  // a > 0
      }
      search = ++guard < 64 && gt_pos(a, amin) && is_negative(diff) && gt_pos(diff_rel, eps * eps);
      if (!search) {
        ++iter;
        if (gt_pos(a, amin) && is_positive(diff)) {
          c0 = cnew;
          s0 = snew0;
          s1 = snew1;
          sab = zab;
          loc_alt = loc_new;
          cur = res;
        }
      }
    }
    if (!search) {
      if (!(iter < 30 && gt_pos(diff_rel, eps * eps) && gt_pos(a, amin))) break;
      grad_pre(P, lane == 31 ? 0.0 : cur, g0, g1, p0, p2, p3);
      guard = 0;
    }
    double z = 1;
    for (int g2 = 0; gt_pos(a, amin) && gt_pos(z, 0.5) && g2 < 64; ++g2) {
      // rfoBuildHessian (src/Core/JacobiRotationFramework.cpp:114-127)
      double u0, u1;
      eig3_top(P.eig, p0, p2, p3, g0, g1, a, &u0, &u1, &top2);
      // ds = a u, snew = s + ds in lanes 0 and 1; zab = sqrt(snew0^2 + snew1^2)
      double v = a * (lane == 0 ? u0 : u1);
      v = (lane == 0 ? s0 : s1) + v;
      snew0 = __shfl_sync(kFull, v, 0);
      snew1 = __shfl_sync(kFull, v, 1);
      v = v * v;
      zab = sqrt(__shfl_sync(kFull, v, 0) + __shfl_sync(kFull, v, 1));
      z = zab * zab;
      if (gt_pos(z, 0.5)) a = half_pow2(a);
    }
    // lane 10: |s|^2 + eps^2 of the current point
    double zz;
    const double r = put_candidates(P, P.cand, z, snew0, snew1, sab, eps, zz);
    cnew = __shfl_sync(kFull, r, 0);
    xden = __shfl_sync(kFull, zz, 10);
  }
  if (lane == 0) {
    P.rot[0] = make_double2(c0, 0.0);
    P.rot[1] = make_double2(s0, s1);
    P.ctl[0] = 0;
  }
  role_sync();
}

// weightedJacobiRotations: every pair (i < j) in order; for each, the
// optimised rotation applied to every weighted matrix, to w and to T
__device__ void rotations(const Prob& P) {
  const int d = P.d, n = P.n, tid = threadIdx.x;
  for (int i = 0; i < d - 1; ++i)
    for (int j = i + 1; j < d; ++j) {
      if (tid < 32) {
        // xold / w of the pair, lanes 0 and 1; then the optimiser
        const int p2 = P.m << P.lgG, G = min(p2, 32), m = p2 / G;
        double s0, s1;
        local_tree(m, [&](int q, double& v0, double& v1) {
          const int k = tid * m + q;
          v0 = v1 = 0.0;
          if (tid < G && k < n) {
            const double x0 = P.X(k)[i + (int64_t)d * i].x, x1 = P.X(k)[j + (int64_t)d * j].x;
            v0 = x0 * x0;
            v1 = x1 * x1;
          }
        }, s0, s1);
        const double r = lane_tree(s0, s1, G) / (tid == 0 ? P.w[i + (int64_t)d * i].x : P.w[j + (int64_t)d * j].x);
        angles(P, __shfl_sync(kFull, r, 0), __shfl_sync(kFull, r, 1));
      } else {
        // the (i, j) blocks of every matrix and of w, then candidates until the master is done
        for (int e = tid - 32; e < 4 * (n + 1); e += kWsdThreads - 32) {
          const double2* A = (e >> 2) < n ? P.X(e >> 2) : P.w;
          P.blk[e] = A[(e & 2 ? j : i) + (int64_t)d * (e & 1 ? j : i)];
        }
        for (;;) {
          role_sync();
          const int which = P.ctl[0];
          if (!which) break;
          eval_items(P.blk, which == 1 ? P.cand0 : P.cand, P.sq, P.wd, n, P.lgG, P.m);
          role_sync();
        }
      }
      const double2 c = P.rot[0], s = P.rot[1];
      // givensRotation of every matrix and of w, columns i, j; givensTrafoRotation of T
      for (int e = tid; e < (n + 2) * d; e += kWsdThreads) {
        const int mi = e / d, r = e % d;
        if (mi <= n) {
          double2* B = mi < n ? P.X(mi) : P.w;
          const double2 bri = B[r + (int64_t)d * i], brj = B[r + (int64_t)d * j];
          B[r + (int64_t)d * i] = ca(rm(c, bri), cm(s, brj));
          B[r + (int64_t)d * j] = cs(rm(c, brj), cm(cc(s), bri));
        } else {
          const double2 ti = P.T[r + (int64_t)d * i], tj = P.T[r + (int64_t)d * j];
          P.T[r + (int64_t)d * i] = ca(rm(c, ti), cm(s, tj));
          P.T[r + (int64_t)d * j] = cs(rm(c, tj), cm(cc(s), ti));
        }
      }
      bsync();
      // rows i, j
      for (int e = tid; e < (n + 1) * d; e += kWsdThreads) {
        const int mi = e / d, r = e % d;
        double2* B = mi < n ? P.X(mi) : P.w;
        const double2 c0 = B[i + (int64_t)d * r], c1 = B[j + (int64_t)d * r];
        B[i + (int64_t)d * r] = ca(rm(c, c0), cm(cc(s), c1));
        B[j + (int64_t)d * r] = cs(rm(c, c1), cm(s, c0));
      }
      bsync();
    }
}

// measureWeightedOffDiagonality: sum_k Re tr(W (D_k - T^H X_k T)^2), the
// matrices `chunk` at a time, the elements of each product in parallel, each
// an ordered sum; the traces added in index order.  All threads get the sum.
__device__ double offdiag(const Prob& P) {
  const int d = P.d, n = P.n, tid = threadIdx.x;
  const int64_t dd = (int64_t)d * d;
  double total = 0;
  for (int k0 = 0; k0 < n; k0 += P.chunk) {
    const int cnt = P.chunk < n - k0 ? P.chunk : n - k0;
    for (int64_t e = tid; e < cnt * dd; e += kWsdThreads) {  // M = X T
      const int kk = (int)(e / dd);
      const int64_t ee = e % dd;
      const int i = (int)(ee % d), j = (int)(ee / d);
      const double2* X = P.Xp(k0 + kk);
      double2 acc = make_double2(0, 0);
      for (int l = 0; l < d; ++l) acc = ca(acc, cm(X[i + (int64_t)d * l], P.T[l + (int64_t)d * j]));
      P.tM[kk * dd + ee] = acc;
    }
    bsync();
    for (int64_t e = tid; e < cnt * dd; e += kWsdThreads) {  // Y = D - T^H M
      const int kk = (int)(e / dd);
      const int64_t ee = e % dd;
      const int i = (int)(ee % d), j = (int)(ee / d);
      const double2* M = P.tM + kk * dd;
      double2 acc = make_double2(0, 0);
      for (int l = 0; l < d; ++l) acc = ca(acc, cm(cc(P.T[l + (int64_t)d * i]), M[l + (int64_t)d * j]));
      double2 dg = make_double2(0, 0);
      if (i == j) dg = make_double2(cdiv_re(P.X(k0 + kk)[i + (int64_t)d * i], P.w[i + (int64_t)d * i]), 0);
      P.tY[kk * dd + ee] = cs(dg, acc);
    }
    bsync();
    for (int64_t e = tid; e < cnt * dd; e += kWsdThreads) {  // Z = Y Y
      const int kk = (int)(e / dd);
      const int64_t ee = e % dd;
      const int i = (int)(ee % d), j = (int)(ee / d);
      const double2* Y = P.tY + kk * dd;
      double2 acc = make_double2(0, 0);
      for (int l = 0; l < d; ++l) acc = ca(acc, cm(Y[i + (int64_t)d * l], Y[l + (int64_t)d * j]));
      P.tM[kk * dd + ee] = acc;
    }
    bsync();
    for (int e = tid; e < cnt * d; e += kWsdThreads) {  // Re (W Z)_ii
      const int kk = e / d, i = e % d;
      const double2* Z = P.tM + kk * dd;
      double2 acc = make_double2(0, 0);
      for (int l = 0; l < d; ++l) acc = ca(acc, cm(P.w[i + (int64_t)d * l], Z[l + (int64_t)d * i]));
      P.tr[e] = acc.x;
    }
    bsync();
    if (tid < 32) {  // trace of matrix k0 + b + lane, then the traces in index order
      for (int b = 0; b < cnt; b += 32) {
        double t = 0;
        if (b + tid < cnt)
          for (int i = 0; i < d; ++i) t += P.tr[(b + tid) * d + i];
        const int m = cnt - b < 32 ? cnt - b : 32;
        for (int q = 0; q < m; ++q) total += __shfl_sync(kFull, t, q);
      }
    }
  }
  if (tid == 0) P.val[0] = total;
  bsync();
  const double v = P.val[0];
  bsync();
  return v;
}

// shared memory of the fixed part of a problem with n matrices of order d
__host__ __device__ int64_t wsd_fixed_bytes(int n, int d) {
  const int64_t b = 16 * (4 * (int64_t)(n + 1) + 40 + 2) + 8 * (20 + 20 + (int64_t)n * d + 2) + 16;
  return (b + 15) / 16 * 16;
}

__global__ void __launch_bounds__(kWsdThreads, 1) k_wsd(const WSDTask* __restrict__ tasks,
                                                     const WSDTerm* __restrict__ terms, int64_t first,
                                                     int smem_bytes) {
  const WSDTask t = tasks[first + blockIdx.x];
  const int d = t.d, n = t.n;
  const int tid = threadIdx.x;
  const int64_t dd = (int64_t)d * d;
  extern __shared__ __align__(16) unsigned char wsd_smem[];
  Prob P;
  P.d = d;
  P.n = n;
  {
    int p2 = 1;
    while (p2 < n) p2 <<= 1;
    const int G = p2 <= 32 ? min(p2, 8) : 32;
    P.lgG = 31 - __clz(G);
    P.m = p2 / G;
  }
  P.blk = reinterpret_cast<double2*>(wsd_smem);
  P.cand0 = P.blk + 4 * (n + 1);
  P.cand = P.cand0 + 20;
  P.rot = P.cand + 20;
  P.sq = reinterpret_cast<double*>(P.rot + 2);
  P.wd = P.sq + 20;
  P.tr = P.wd + 20;
  P.val = P.tr + (int64_t)n * d;
  P.ctl = reinterpret_cast<int*>(P.val + 2);
  {
    const int l = tid & 31;
#pragma unroll
    for (int k = 0; k < kEigLevels; ++k) P.eig[k] = lane_op(c_eig_lut[k][l], l);
    // grad_pre's terms: y[i + 3 j] in lane 1 + i + 3 j, lane 31 zero
    P.den = l < 2 ? 2 * kDelta : (l < 4 ? kDelta * kDelta : 4 * kDelta * kDelta);
    P.zh = 1.0 / P.den;
    P.zl = __fma_rn(neg_bits(P.zh), P.den, 1.0) / P.den;
    const uint32_t A = l == 0 || l == 2 ? 6 : (l == 1 || l == 3 ? 8 : 9);
    const uint32_t B = l == 0 || l == 2 ? 4 : (l == 1 || l == 3 ? 2 : 1);
    const uint32_t C = l < 2 ? 31 : (l < 4 ? 5 : 3), D = l < 4 ? 31 : 7;
    P.diff = A | (B << 5) | (C << 10) | (D << 15) | ((l < 2 ? 1u : 0u) << 20);
    const int k = l & 15, q = l < 16 ? (k - 1) % 3 : (k - 1) / 3;
    P.dx = k < 1 || k > 9 ? -0.0 : (q == 0 ? -kDelta : (q == 1 ? 0.0 : kDelta));
    if (tid < 32) {
      double z;
      const double r = put_candidates(P, P.cand0, 2 * kEps * kEps, kEps, -kEps, kEps, -kEps, z);
      P.c0 = __shfl_sync(kFull, r, 0);
      P.sab0 = __shfl_sync(kFull, r, 10);
    }
  }
  // the matrices in shared memory when they fit, else in the task's scratch
  const int64_t fixed = wsd_fixed_bytes(n, d);
  const int64_t mats = (2 * (int64_t)n + 2) * dd * 16;
  const int64_t room = (int64_t)smem_bytes - fixed - mats;
  if (room >= 2 * dd * 16) {
    double2* base = reinterpret_cast<double2*>(wsd_smem + fixed);
    const int64_t fit = room / (2 * dd * 16);
    P.chunk = fit < n ? (int)fit : n;
    P.xw = base;
    P.xp = base + n * dd;
    P.w = base + 2 * n * dd;
    P.T = P.w + dd;
    P.tM = P.T + dd;
    P.tY = P.tM + P.chunk * dd;
  } else {
    P.chunk = 1;
    P.xw = t.scratch;
    P.xp = t.scratch + n * dd;
    P.w = t.scratch + 2 * n * dd;
    P.T = P.w + dd;
    P.tM = P.T + dd;
    P.tY = P.tM + dd;
  }
  // w = regularize(W), T = 1
  for (int64_t e = tid; e < dd; e += kWsdThreads) {
    double2 v = t.W[e];
    const int i = (int)(e % d), j = (int)(e / d);
    if (i == j) v.x += 1e-9 * exp(-cabs_(v) / 1e-9);
    P.w[e] = v;
    P.T[e] = make_double2(i == j ? 1.0 : 0.0, 0.0);
  }
  // shifts |tr X| (calculateShift), kept in the grid's imaginary parts until the end
  for (int k = tid; k < n; k += kWsdThreads) {
    const double2* X = terms[t.first + k].X;
    double2 tr = make_double2(0, 0);
    for (int i = 0; i < d; ++i) tr = ca(tr, X[i + (int64_t)d * i]);
    const double sh = cabs_(tr);
    t.grid[(int64_t)k * d].y = sh;
    P.tr[k] = sh;
  }
  bsync();
  // plain matrices shifted (shift)
  for (int64_t e = tid; e < n * dd; e += kWsdThreads) {
    const int k = (int)(e / dd);
    const int64_t ee = e % dd;
    double2 v = terms[t.first + k].X[ee];
    if (ee % (d + 1) == 0) v.x -= P.tr[k];
    P.Xp(k)[ee] = v;
  }
  bsync();
  // weightMatrices: (X w + w X) / 2
  for (int64_t e = tid; e < (int64_t)n * dd; e += kWsdThreads) {
    const int k = (int)(e / dd);
    const int i = (int)(e % dd % d), j = (int)(e % dd / d);
    const double2* x = P.Xp(k);
    double2 xw = make_double2(0, 0), wx = make_double2(0, 0);
    for (int l = 0; l < d; ++l) {
      xw = ca(xw, cm(x[i + (int64_t)d * l], P.w[l + (int64_t)d * j]));
      wx = ca(wx, cm(P.w[i + (int64_t)d * l], x[l + (int64_t)d * j]));
    }
    const double2 sum = ca(xw, wx);
    P.X(k)[i + (int64_t)d * j] = make_double2(0.5 * sum.x, 0.5 * sum.y);
  }
  bsync();
  double delta = offdiag(P);
  int iter = 0;
  bool converged = false;
  const double eps = 1e-5;
  while (!converged && iter < 25) {
    rotations(P);
    const double delta_last = delta;
    delta = offdiag(P);
    const double change = fabs(delta_last - delta);
    if (delta < eps || change < eps) converged = true;
    iter++;
  }
  // grid = Re(Xw(i,i) / w(i,i)) + shift; trafo = T^dagger
  for (int k = tid; k < n; k += kWsdThreads) {
    const double sh = t.grid[(int64_t)k * d].y;
    for (int i = 0; i < d; ++i)
      t.grid[(int64_t)k * d + i] = make_double2(cdiv_re(P.X(k)[i + (int64_t)d * i], P.w[i + (int64_t)d * i]) + sh, 0.0);
  }
  for (int64_t e = tid; e < dd; e += kWsdThreads) {
    const int i = (int)(e % d), j = (int)(e / d);
    t.trafo[e] = cc(P.T[j + (int64_t)d * i]);
  }
}

}  // namespace

cudaError_t launch_wsd(const WSDTask* tasks, const WSDTerm* terms, int64_t first, int64_t n, int max_n,
                       int max_d, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int64_t dd = (int64_t)max_d * max_d;
  const int64_t fixed = wsd_fixed_bytes(max_n, max_d);
  if (fixed > kWsdSmemBudget) return cudaErrorInvalidValue;
  // the largest problem's matrices and as many per-matrix product buffers as fit
  const int64_t mats = (2 * (int64_t)max_n + 2) * dd * 16;
  int64_t sm = fixed;
  if (fixed + mats + 2 * dd * 16 <= kWsdSmemBudget)
    sm = std::min<int64_t>(fixed + mats + 2 * (int64_t)max_n * dd * 16,
                           fixed + mats + (kWsdSmemBudget - fixed - mats) / (2 * dd * 16) * (2 * dd * 16));
  cudaError_t e = cudaFuncSetAttribute(k_wsd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  k_wsd<<<(unsigned)n, kWsdThreads, sm, s>>>(tasks, terms, first, (int)sm);
  return cudaGetLastError();
}

}  // namespace qt
