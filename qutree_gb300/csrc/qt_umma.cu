// qt_umma.cu -- the contractions of the mixed-precision plans on the
// fifth-generation tensor cores (tcgen05.mma, accumulators in tensor memory).
//
// Double-float plans (QT_PREC_DF64_TC): mode products, hole products and
// last-index accumulations run on one sum-of-products kernel (k_tcs, its
// design above it).  Every operand row is scaled by the power of two 2^-E
// of its largest exponent and cut into seven signed digits by error-free
// splits x_s = fl(fl(r + sigma_s) - sigma_s), sigma_s = 1.5 * 2^(16 - 7s):
// x_s is r rounded to a multiple of 2^(-7(s+1)), r - x_s is exact, the
// value's low word joins from s = 3.  The digit integers
// q_s = x_s 2^(7(s+1)) have |q_s| <= 128, so q_s 2^(-7s) is exact in bf16 and
// every digit product is exact.  Pairs with s + t <= 6 are summed in fp32
// accumulators, one per level L = s + t, as far as tensor memory holds them
// (the last taking the remaining levels together); the epilogue adds the
// levels in double-float and scales by 2^(E_row + F_column).
//
// Complex64 plans (QT_PREC_TF32X3): the mode products as split-TF32 (k_mp_tf):
// X and h (fp32) split into TF32 halves hi + lo; hi*hi + hi*lo + lo*hi
// accumulate in one fp32 sum per output (3 passes).
#include <cuda_runtime.h>

#include <cstdint>

#include "qt_arith.cuh"
#include "qt_internal.h"
#include "qt_tc05.cuh"

namespace qt {
namespace {

using namespace tc05;

constexpr int kRows = 128;                 // rows per tile (M)
constexpr int kDig = 7;                    // digits per value (double-float plans)
constexpr int kThreadsTc = 416;            // thirteen warps (roles per kernel below)
constexpr uint64_t kSpin = 2000000000ull;  // ns before a wait gives up (2 s)
constexpr int kChunkK = 16;                // k per ring stage

// a digit plane of one 16-k step: 128 rows x 16 k bf16 (core layout [kc][g][8][8])
constexpr int kOzAPlane = kRows * kChunkK * 2;        // 4096 bytes
constexpr int kOzAStage = kDig * 2 * kOzAPlane;       // 57344: seven digits, re and im
// TF: a TF32 plane of one stage: 128 rows x 16 k fp32 (core layout [kc][g][8][4])
constexpr int kTfAPlane = kRows * kChunkK * 4;        // 8192 bytes
constexpr int kTfAStage = 4 * kTfAPlane;              // hi_re, hi_im, lo_re, lo_im
constexpr int kTfBMax = 4 * 4 * 64 * 64;              // 65536: K 64, N 64
static_assert(kTfBMax <= kMpOzImageBytes, "operand image slot too small");

struct Bars {
  uint64_t full[2], empty[2], exready[2], exfree[2], tfull, tempty, bfull, drain;
  uint32_t tmem;
  int pad;
};

struct TfSmem {
  unsigned char b[kTfBMax];
  unsigned char a[2][kTfAStage];
  Bars bar;
};
static_assert(sizeof(TfSmem) <= 232448, "shared memory of the split-TF32 kernel exceeds 227 KB");

__device__ __forceinline__ float pow2f(int k) { return __int_as_float((k + 127) << 23); }
__device__ __forceinline__ float scale2(float v, int k) {
  if (k > 127) return (v * pow2f(127)) * pow2f(k - 127);
  if (k < -126) return (v * pow2f(-126)) * pow2f(k + 126);
  return v * pow2f(k);
}

// Digits of one double-float value v = hi + lo of a row whose largest biased
// exponent of hi parts is eb (|v| < 2^E, E = eb - 126).  The row is scaled
// to |v 2^-E| < 1 (exactly, by a power of two) and cut by error-free splits
// x_s = fl(fl(r + sigma_s) - sigma_s), sigma_s = 1.5 * 2^(16 - 7s): x_s is r
// rounded to the nearest multiple of 2^(-7(s+1)) and r - x_s is exact, so
// v 2^-E = x_0 + ... + x_6 + (remainder of at most 2^-49).  The low part
// joins from s = 3 (|lo| is below 2^-24 of the row scale); each digit is the
// exact sum of its hi and lo splits.  With q_s = x_s 2^(7(s+1)):
// |q_s| <= 128 -- integers of at most eight significant bits, exact in bf16.
// Stored is x_s itself (bf16), so that a product of digits s and t carries
// its level's weight 2^(-7(s+t+2)).
__device__ __forceinline__ float dsplit(float& r, float sigma) {
  const float x = __fsub_rn(__fadd_rn(r, sigma), sigma);
  r = __fsub_rn(r, x);
  return x;
}
__device__ __forceinline__ float digit_sigma(int s) { return __int_as_float(((127 + 16 - 7 * s) << 23) | 0x400000); }
// 2^(126 - eb), eb in 1..255 (subnormal from eb = 253 on): the row's scaling
__device__ __forceinline__ float row_factor(int eb) {
  const int k = 126 - eb;
  return __int_as_float(k >= -126 ? (k + 127) << 23 : 0x00800000 >> (-126 - k));
}
// |x| as an ordered integer; the biased exponent of a row whose largest one
// is m.  A row of zeros gets 126 (scale 1): its digits are zero whatever the
// scale, and the epilogue's common path keeps its rows.
__device__ __forceinline__ int fmag(float v) { return __float_as_int(v) & 0x7fffffff; }
__device__ __forceinline__ int row_exponent(int m) { return m == 0 ? 126 : max(1, m >> 23); }
// the seven digits x_s of hi + lo as floats (exact in bf16: their upper
// 16 bits are the bf16); f = row_factor of the row
__device__ __forceinline__ void digits_f32(float hi, float lo, float f, float d[kDig]) {
  float rh = __fmul_rn(hi, f), rl = __fmul_rn(lo, f);
#pragma unroll
  for (int s = 0; s < kDig; ++s) {
    float x = dsplit(rh, digit_sigma(s));
    if (s >= 3) x = __fadd_rn(x, dsplit(rl, digit_sigma(s)));
    d[s] = x;
  }
}
// the bf16 of two exact digits in one 32-bit word (a in the low half)
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// TF32 halves of x: hi = x rounded to 10 fraction bits, lo = x - hi (the
// tensor core reads the upper 19 bits of each 32-bit operand)
__device__ __forceinline__ void tf32_split(float x, uint32_t& hi, uint32_t& lo) {
  uint32_t h;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
  hi = h;
  const float r = __fsub_rn(x, __uint_as_float(h));
  uint32_t l;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(r));
  lo = l;
}

// byte offset, in a K-major core layout of `rows` rows, of row r at the
// 16-byte k-group kc
__device__ __forceinline__ int core_off(int r, int kc, int rows) {
  return kc * (rows / 8) * 128 + (r >> 3) * 128 + (r & 7) * 16;
}

// separate level accumulators that fit tensor memory (512 columns of 2 Np each)
__device__ __forceinline__ int levels_for(int Np) { return min(kDig, 512 / (2 * Np)); }

__device__ __forceinline__ void set_status(int* status, int code) {
  if (status) atomicCAS(status, 0, code);
}

// Write element (j, k) of H^T, value v, into the split-TF32 operand image
// [ks][hi_re, hi_im, lo_re, lo_im][core layout Np x 16 k] fp32.
__device__ __forceinline__ void put_image_tf(unsigned char* img, int Np, int j, int k, float4 v) {
  const int plane_bytes = Np * kChunkK * 4;
  const int ks = k / kChunkK, kk = k % kChunkK;
  const int off = core_off(j, kk / 4, Np) + (kk % 4) * 4;
  unsigned char* base = img + (size_t)ks * 4 * plane_bytes;
  uint32_t hr, lr, hi_, li;
  tf32_split(v.x, hr, lr);
  tf32_split(v.z, hi_, li);
  *reinterpret_cast<uint32_t*>(base + 0 * plane_bytes + off) = hr;
  *reinterpret_cast<uint32_t*>(base + 1 * plane_bytes + off) = hi_;
  *reinterpret_cast<uint32_t*>(base + 2 * plane_bytes + off) = lr;
  *reinterpret_cast<uint32_t*>(base + 3 * plane_bytes + off) = li;
}

// ---------------------------------------------------------------------------
// pre-pass of the split-TF32 mode products: the operand image of alpha h for
// every task of the stage, H^T rows j (N, padded to Np = 16 ceil(N / 16)),
// k < Kp zero-padded
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_mp_tf_h(const MPTask* __restrict__ tasks, const int* __restrict__ ids,
                                                 int64_t first) {
  const MPTask t = tasks[ids[first + blockIdx.x]];
  unsigned char* img = static_cast<unsigned char*>(t.oz_h);
  const float4* __restrict__ h = reinterpret_cast<const float4*>(t.h);
  const int K = t.a_in, N = t.a_out;
  const int Np = (N + 15) & ~15, Kp = (K + 15) & ~15;
  const bool one = t.alpha.x == 1.0 && t.alpha.y == 0.0;
  const float4 cf = C32::coef(t.alpha);
  for (int e = threadIdx.x; e < Np * Kp; e += blockDim.x) {
    const int j = e % Np, k = e / Np;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j < N && k < K) {
      v = h[j + (int64_t)N * k];
      if (!one) v = C32::mul(cf, v);
    }
    put_image_tf(img, Np, j, k, v);
  }
}

// ---------------------------------------------------------------------------
// One unit of work: 128 rows of a mode-product task.
// ---------------------------------------------------------------------------
struct TcUnit {
  int K, N, Np;              // reduction length, output columns (padded)
  const unsigned char* img;  // h operand image
  int64_t nrows;             // rows of the task
  const float4* in;          // the input tensor
  int64_t before;            // stride of the reduction index
  float4* out;
};

__device__ __forceinline__ TcUnit make_unit(const MPTask* tasks, int task) {
  const MPTask t = tasks[task];
  TcUnit u;
  u.K = t.a_in;
  u.N = t.a_out;
  u.Np = (u.N + 15) & ~15;
  u.img = static_cast<const unsigned char*>(t.oz_h);
  u.nrows = (int64_t)t.before * t.after;
  u.in = reinterpret_cast<const float4*>(t.in);
  u.before = t.before;
  u.out = reinterpret_cast<float4*>(t.out);
  return u;
}

// ---------------------------------------------------------------------------
// Split-TF32 mode products (complex64 plans).  out[b, j, c] =
// alpha sum_a h(j, a) in[b, a, c] is the GEMM Y = X H^T with rows r = (b, c)
// (K = a_in, N = a_out <= 64); four real MMAs per operand pair,
//   Y_re += X_re H_re^T - X_im H_im^T,   Y_im += X_re H_im^T + X_im H_re^T,
// the minus sign by the instruction's negate-A bit.  Roles (416 threads):
// warps 0-7 produce X's TF32 halves of each 16-k step into a two-stage ring
// (two threads per row, eight k each); warp 12 allocates tensor memory, loads
// the h image of the unit (bulk copies, once per change of task) and issues
// the MMAs from one thread; warps 8-11 read the accumulators (warp 8 + q:
// lanes 32q..) and write the outputs.  A CTA takes a contiguous range of
// 128-row tiles.  Every wait is bounded: a wait that runs out sets the status
// word, and the CTA drains its issued MMAs, frees tensor memory and returns.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreadsTc, 1) k_mp_tf(const MPTask* __restrict__ tasks,
                                                          const int2* __restrict__ tiles, int64_t tile0,
                                                          int64_t n_tiles, int* status) {
  extern __shared__ __align__(128) unsigned char tc_raw[];
  TfSmem& sm = *reinterpret_cast<TfSmem*>(tc_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t per = n_tiles / gridDim.x, extra = n_tiles % gridDim.x;
  const int64_t my0 = blockIdx.x * per + min((int64_t)blockIdx.x, extra);
  const int64_t my1 = my0 + per + (blockIdx.x < extra ? 1 : 0);

  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sm.bar.full[s], 256);
      mbar_init(&sm.bar.empty[s], 1);
    }
    mbar_init(&sm.bar.tfull, 1);
    mbar_init(&sm.bar.tempty, 128);
    mbar_init(&sm.bar.bfull, 1);
    mbar_init(&sm.bar.drain, 1);
    mbar_fence_init();
  }
  if (warp == 12) tmem_alloc(&sm.bar.tmem, 128u);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sm.bar.tmem;
  bool ok = true;

  if (warp < 8) {
    // ---------------- producers: two per row, eight k of every step each ----------------
    const int r = tid & (kRows - 1), h = tid >> 7;
    uint32_t q = 0;
    for (int64_t it = my0; it < my1 && ok; ++it) {
      const int2 tl = tiles[tile0 + it];
      const TcUnit U = make_unit(tasks, tl.x);
      const int K = U.K;
      const int64_t rg = (int64_t)tl.y * kRows + r;
      const bool valid = rg < U.nrows;
      const int64_t b = valid ? rg % U.before : 0, c = valid ? rg / U.before : 0;
      const float4* base = U.in + b + U.before * (int64_t)K * c;
      const int nks = (K + kChunkK - 1) / kChunkK;
      // this thread's eight values of step ks; the next step's loads are in
      // flight while the current one is split
      auto load8 = [&](float4 (&x)[8], int ks) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int a = ks * kChunkK + h * 8 + i;
          x[i] = (valid && a < K) ? __ldg(base + U.before * a) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      };
      float4 nx[8];
      load8(nx, 0);
      for (int ks = 0; ks < nks; ++ks, ++q) {
        const int s = q & 1;
        float4 x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = nx[i];
        if (ks + 1 < nks) load8(nx, ks + 1);
        if (!mbar_wait(&sm.bar.empty[s], ((q >> 1) & 1) ^ 1, kSpin)) {
          set_status(status, 1);
          ok = false;
          break;
        }
        unsigned char* A = sm.a[s];
        // fp32 values (complex64 storage keeps them in the hi words)
#pragma unroll
        for (int g2 = 0; g2 < 2; ++g2) {  // two 16-byte core rows of 4 k each
          uint32_t hr[4], hi_[4], lr[4], li[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            tf32_split(x[4 * g2 + i].x, hr[i], lr[i]);
            tf32_split(x[4 * g2 + i].z, hi_[i], li[i]);
          }
          const int off = core_off(r, 2 * h + g2, kRows);
          *reinterpret_cast<uint4*>(A + 0 * kTfAPlane + off) = make_uint4(hr[0], hr[1], hr[2], hr[3]);
          *reinterpret_cast<uint4*>(A + 1 * kTfAPlane + off) = make_uint4(hi_[0], hi_[1], hi_[2], hi_[3]);
          *reinterpret_cast<uint4*>(A + 2 * kTfAPlane + off) = make_uint4(lr[0], lr[1], lr[2], lr[3]);
          *reinterpret_cast<uint4*>(A + 3 * kTfAPlane + off) = make_uint4(li[0], li[1], li[2], li[3]);
        }
        fence_proxy_async();
        mbar_arrive(&sm.bar.full[s]);
      }
    }
  } else if (warp == 12) {
    // ---------------- MMA issue (one thread) and h loads ----------------
    if (lane == 0) {
      uint32_t q = 0, nb = 0, un = 0;
      const void* cur = nullptr;
      for (int64_t it = my0; it < my1 && ok; ++it, ++un) {
        const int2 tl = tiles[tile0 + it];
        const TcUnit U = make_unit(tasks, tl.x);
        const int K = U.K, Np = U.Np, nks = (K + kChunkK - 1) / kChunkK;
        const int plane_b = Np * kChunkK * 4;  // bytes of one h plane per step
        const uint32_t tpar = un & 1;
        if (U.img != cur) {
          // the previous unit's MMAs read the old h: wait until they completed
          if (un > 0 && !mbar_wait(&sm.bar.tfull, tpar ^ 1, kSpin)) {
            set_status(status, 2);
            ok = false;
            break;
          }
          const uint32_t bytes = (uint32_t)(nks * 4 * plane_b);
          mbar_arrive_expect_tx(&sm.bar.bfull, bytes);
          for (uint32_t o = 0; o < bytes; o += 32768u) {
            const uint32_t n = bytes - o < 32768u ? bytes - o : 32768u;
            bulk_g2s(sm.b + o, U.img + o, n, &sm.bar.bfull);
          }
          if (!mbar_wait(&sm.bar.bfull, nb & 1, kSpin)) {
            set_status(status, 3);
            ok = false;
            break;
          }
          ++nb;
          cur = U.img;
        }
        // the epilogue released the accumulators of the previous unit
        if (!mbar_wait(&sm.bar.tempty, tpar ^ 1, kSpin)) {
          set_status(status, 4);
          ok = false;
          break;
        }
        fence_after_sync();
        const uint32_t lboB = (uint32_t)(Np / 8) * 128;
        const uint32_t lboA4 = (kRows / 8) * 128;  // kc stride of a 16-k fp32 plane: [kc (4)][g][8][4]
        const uint32_t id = idesc_m128(2, Np, false), idn = idesc_m128(2, Np, true);
        uint32_t used = 0;  // 0 until the unit's first MMAs
        for (int ks = 0; ks < nks; ++ks, ++q) {
          const int s = q & 1;
          if (!mbar_wait(&sm.bar.full[s], (q >> 1) & 1, kSpin)) {
            set_status(status, 5);
            ok = false;
            break;
          }
          fence_after_sync();
          const uint32_t a0 = smem_u32(sm.a[s]);
          const uint32_t b0 = smem_u32(sm.b) + (uint32_t)(ks * 4 * plane_b);
#pragma unroll 1
          for (int h8 = 0; h8 < 2; ++h8) {  // two MMAs of k = 8 per step
            const uint32_t ao = (uint32_t)(2 * h8) * lboA4, bo = (uint32_t)(2 * h8) * lboB;
            const uint64_t ahr = desc_kmajor(a0 + 0 * kTfAPlane + ao, lboA4, 128);
            const uint64_t ahi = desc_kmajor(a0 + 1 * kTfAPlane + ao, lboA4, 128);
            const uint64_t alr = desc_kmajor(a0 + 2 * kTfAPlane + ao, lboA4, 128);
            const uint64_t ali = desc_kmajor(a0 + 3 * kTfAPlane + ao, lboA4, 128);
            const uint64_t bhr = desc_kmajor(b0 + 0 * plane_b + bo, lboB, 128);
            const uint64_t bhi = desc_kmajor(b0 + 1 * plane_b + bo, lboB, 128);
            const uint64_t blr = desc_kmajor(b0 + 2 * plane_b + bo, lboB, 128);
            const uint64_t bli = desc_kmajor(b0 + 3 * plane_b + bo, lboB, 128);
            const uint32_t dre = tmem, dim_ = tmem + (uint32_t)Np;
            const uint32_t f = used;  // 0 only for the first MMAs of the unit
            // lo x hi and hi x lo first, then hi x hi
            mma_tf32(dre, alr, bhr, id, f);
            mma_tf32(dim_, alr, bhi, id, f);
            mma_tf32(dre, ali, bhi, idn, 1);
            mma_tf32(dim_, ali, bhr, id, 1);
            mma_tf32(dre, ahr, blr, id, 1);
            mma_tf32(dim_, ahr, bli, id, 1);
            mma_tf32(dre, ahi, bli, idn, 1);
            mma_tf32(dim_, ahi, blr, id, 1);
            mma_tf32(dre, ahr, bhr, id, 1);
            mma_tf32(dim_, ahr, bhi, id, 1);
            mma_tf32(dre, ahi, bhi, idn, 1);
            mma_tf32(dim_, ahi, bhr, id, 1);
            used = 1;
          }
          commit(&sm.bar.empty[s]);  // the step is free once these MMAs completed
        }
        if (!ok) break;
        commit(&sm.bar.tfull);
      }
      // drain: every MMA issued by this thread completed before tensor memory is freed
      commit(&sm.bar.drain);
      if (!mbar_wait(&sm.bar.drain, 0, kSpin)) set_status(status, 6);
    }
  } else {
    // ---------------- epilogue: warp 8 + qd reads lanes 32 qd .. ----------------
    const int qd = warp - 8;
    const int r = 32 * qd + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(32 * qd) << 16);
    uint32_t un = 0;
    for (int64_t it = my0; it < my1 && ok; ++it, ++un) {
      const int2 tl = tiles[tile0 + it];
      const TcUnit U = make_unit(tasks, tl.x);
      const int N = U.N, Np = U.Np;
      if (!mbar_wait(&sm.bar.tfull, un & 1, kSpin)) {
        set_status(status, 7);
        ok = false;
        break;
      }
      fence_after_sync();
      const int64_t rg = (int64_t)tl.y * kRows + r;
      const bool live = rg < U.nrows;
      const int64_t ro = live ? rg % U.before + U.before * (int64_t)N * (rg / U.before) : 0;
      for (int j0 = 0; j0 < Np; j0 += 8) {
        __syncwarp();  // the tensor-memory loads below are warp-collective
        float vre[8], vim[8];
        tmem_ld8(lane_addr + (uint32_t)j0, vre);
        tmem_ld8(lane_addr + (uint32_t)(Np + j0), vim);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int j = j0 + i;
          if (live && j < N) U.out[ro + U.before * j] = make_float4(vre[i], 0.f, vim[i], 0.f);
        }
      }
      fence_before_sync();
      mbar_arrive(&sm.bar.tempty);
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 12) {
    fence_after_sync();
    tmem_dealloc(tmem, 128u);
  }
}

// ---------------------------------------------------------------------------
// Sums of products on the tensor cores (double-float plans): the hole
// products, the last-index accumulations and the mode products.  All compute,
// per output row m and column n,
//   D(m, n) = sum over units u of  sum_k X_u(m, k) W_u(n, k)     (complex)
// in units of at most 128 k, every unit with its own power-of-two scales per
// row of X_u (E_m) and per row of W_u (F_n):
//  * hole products S_t(i, j) = sum_k conj(A[k; i]) B_t[k; j]: the rows m are
//    the (task t, j) of a group of tasks that share A (X = B_t), n = i and
//    W = conj(A); the units are the chunks of the reduction, 64 k up to 32
//    columns, else 128;
//  * accumulations out[r, j] (+)= alpha sum_t sum_j' H_t(j, j') X_t[r, j']:
//    rows m = r (a block of 128), n = j, one unit per term t with X = X_t
//    and W = alpha H_t (alpha I for identity terms), up to 112 k;
//  * mode products C[b, j, c] = alpha sum_a h(j, a) B[b, a, c]: rows m = (b, c)
//    (a block of 128), n = j, one unit of up to 112 k.
// Beyond 64 columns an item is one column block (tc_blocks), and 48-column
// blocks take a unit in two halves (tcs_halve).
// The accumulator tile has 2 np columns, the real parts for n < np and the
// imaginary parts after them, so
//   Re D = Xr Wr - Xi Wi,   Im D = Xr Wi + Xi Wr
// are two MMAs of N = 2 np per digit pair: Xr x [Wr | Wi] and
// Xi x [-Wi | Wr].  W's image, written by a pre-pass per unit, stores the
// rows [-Wi | Wr | Wi] (np each) once per 16-k step and digit; the two
// operands are its rows np.. and 0.. .  The producers cut X's digits; the
// image steps arrive by bulk copies on the same barrier.  A level's sum is
// exact in fp32 where it has an accumulator of its own: digit 0 is at most
// 128 units, 1 and 2 at most 64, 3 at most 80, the others 128, so that 2 x 128
// products per pair stay below 2^24 units in levels 0..4, and 2 x 112 in 5 and
// 6.  With fewer than seven accumulators (levels_for; four for 128-k chunks up
// to 64 columns) the last one takes the remaining levels and is rounded.  The
// epilogue recombines the levels in double-float, scales by 2^(E_m + F_n) and
// adds them to the output in double-float (a work item's first unit stores, or
// adds to the old output where the accumulation asks for it).
// ---------------------------------------------------------------------------
constexpr int kTcsNStage = kDig * 3 * 64 * 32;  // W side of one 16-k step at np = 64

// Warps of the kernel: four producers; one MMA issuer and three exponent
// warps; eight of the epilogue.
constexpr int kTcsThreads = 512, kTcsExWarps = 3, kTcsEpWarps = 8;

enum { TCS_HP = 0, TCS_ACC = 1, TCS_MP = 2 };

struct TcsSmem {
  unsigned char a[2][kOzAStage];
  unsigned char n[2][kTcsNStage];
  Bars bar;
  int ex[2][kTcsExWarps][kRows];  // largest |X| of the rows of the two units in flight, per exponent warp
  int fx[8][64];                  // the unit's column exponents, one copy per epilogue warp
};
static_assert(sizeof(TcsSmem) <= 232448, "shared memory of the sum-of-products kernel exceeds 227 KB");

struct TcsArgs {
  const HPTask* hp;          // hole products: tasks, groups, partial tiles
  const HpTcGroup* groups;
  double2* ws;
  const AccTask* acc;        // accumulations: tasks and terms
  const AccTerm* terms;
  const MPTask* mp;          // mode products: tasks, tiles (task, 128-row block) and the pre-pass's tasks
  const int2* mp_tiles;
  const int* mp_tasks;
  const int4* items;         // HP (group, range z, first chunk, end chunk); ACC (task, block, units before, column block)
  int64_t item0, n_items;
  int64_t units;             // ACC: units of all items (weighted split over the CTAs)
  int* status;
};

// item `it` of the launch (mode products: (task, 128-row block, 0, column block))
template <int OP>
__device__ __forceinline__ int4 tcs_fetch(const TcsArgs& g, int64_t it) {
  if (OP == TCS_MP) {
    const int2 t = g.mp_tiles[g.item0 + it];
    return make_int4(t.x, t.y & ((1 << kMpTcBlockShift) - 1), 0, t.y >> kMpTcBlockShift);
  }
  return g.items[g.item0 + it];
}

// element k of row `row` of a hole-product operand of shape (before, a, after):
// k = b + before c, offset b + before row + before a c; walked in steps of one
struct KWalk {
  int b, c;
  __device__ __forceinline__ KWalk(int k, int before) : b(k - (k / before) * before), c(k / before) {}
  __device__ __forceinline__ int64_t off(int row, int before, int a) const {
    return b + (int64_t)before * row + (int64_t)before * a * c;
  }
  __device__ __forceinline__ void next(int before) {
    if (++b == before) {
      b = 0;
      ++c;
    }
  }
};

// the CTA's run of items: equal counts (HP: items of about equal length), or
// the items whose first unit falls into the CTA's equal share of all units
template <int OP>
__device__ __forceinline__ void tcs_range(const TcsArgs& g, int64_t& i0, int64_t& i1) {
  if (OP != TCS_ACC) {
    const int64_t per = g.n_items / gridDim.x, extra = g.n_items % gridDim.x;
    i0 = blockIdx.x * per + min((int64_t)blockIdx.x, extra);
    i1 = i0 + per + (blockIdx.x < extra ? 1 : 0);
    return;
  }
  auto first_at = [&](int64_t u) {  // first item with units-before >= u
    int64_t lo = 0, hi = g.n_items;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if ((int64_t)g.items[g.item0 + mid].z < u) lo = mid + 1;
      else hi = mid;
    }
    return lo;
  };
  i0 = first_at(g.units * blockIdx.x / gridDim.x);
  i1 = first_at(g.units * (blockIdx.x + 1) / gridDim.x);
}

// per item: its column block (padded columns np, real columns, first one),
// units, 16-k steps per unit and of the operand image
struct TcsItem {
  int np, ncols, c0, nunits, nks, isteps;
  int nl;     // level accumulators
  bool wide;  // more than kTcCols columns in all
  int half;   // 1: every term or chunk is two units, the second from step n0 on
  int n0;
  // unit u's term or chunk, its first 16-k step, its steps
  __device__ __forceinline__ int term(int u) const { return u >> half; }
  __device__ __forceinline__ int step0(int u) const { return u & half ? n0 : 0; }
  __device__ __forceinline__ int steps(int u) const { return !half ? nks : u & 1 ? nks - n0 : n0; }
};
// Bonds beyond 64 whose column blocks are wider than 40 (81..96: 48 columns)
// have room for five level accumulators only.  The tensor core truncates the
// sums into the last one, which holds levels 4..6, and the error grows with the
// number of MMAs on it: these units take half of the k.  Density matrices at
// bonds 88 and 96 against complex128: 4.8e-15 -> 3.4e-15 (multiply-adds 4.7e-15;
// six and seven accumulators 2.7e-15).
template <bool WIDE>
__device__ __forceinline__ void tcs_halve(TcsItem& v, int n) {
  v.wide = WIDE && n > kTcCols;
  v.half = v.wide && v.np > 40 && v.nks > 1 ? 1 : 0;
  v.n0 = (v.nks + 1) >> 1;
  v.nunits <<= v.half;
}
template <int OP, bool WIDE>
__device__ __forceinline__ TcsItem tcs_item(const TcsArgs& g, int4 itm) {
  TcsItem v;
  if (OP == TCS_HP) {
    const HpTcGroup& G = g.groups[itm.x];
    v.np = G.ap;
    v.ncols = G.nc;
    v.c0 = G.c0;
    v.nunits = itm.w - itm.z;
    v.nks = v.isteps = hp_tc_kc(G.ap) / kChunkK;
    // 128-k chunks of bonds up to 64 keep four accumulators (levels 0..2 exact up to 170 k)
    v.nl = v.nks > 4 && G.a <= kTcCols ? 4 : levels_for(G.ap);
    tcs_halve<WIDE>(v, G.a);
    return v;
  }
  int n, k;
  if (OP == TCS_ACC) {
    const AccTask& T = g.acc[itm.x];
    n = k = T.d;
    v.nunits = T.count;
  } else {
    const MPTask& t = g.mp[itm.x];
    n = t.a_out;
    k = t.a_in;
    v.nunits = 1;
  }
  v.np = tc_width(n);
  v.c0 = itm.w * v.np;
  v.ncols = min(v.np, n - v.c0);
  v.nks = (k + kChunkK - 1) / kChunkK;
  v.isteps = tc_steps(k);
  v.nl = levels_for(v.np);
  tcs_halve<WIDE>(v, n);
  return v;
}
// operand image of term or chunk u
template <int OP>
__device__ __forceinline__ const unsigned char* tcs_image(const TcsArgs& g, int4 itm, int u, const TcsItem& I) {
  const int64_t cb = hp_tc_chunk_bytes(I.np, I.isteps);
  if (OP == TCS_HP) return g.groups[itm.x].img + (size_t)(itm.z + u) * cb;
  if (OP == TCS_MP) return static_cast<const unsigned char*>(g.mp[itm.x].oz_h) + (size_t)itm.w * cb;
  return static_cast<const unsigned char*>(g.acc[itm.x].tc_img) + (size_t)(u + (I.nunits >> I.half) * itm.w) * cb;
}

// pre-pass: the image of W for one unit -- per 16-k step and digit a plane of
// 3 np rows, -Wi at row n, Wr at np + n, Wi at 2 np + n (rows past the last
// column zero) -- and the unit's row exponents F_n.  Thread (n, q) takes row
// n of the 8-k core rows q, q + 8, ...  HP units (group, chunk): W(i, k) = conj(A[k; i]);
// ACC units (task, term): W(j, k) = alpha H(j, k), alpha I for identity terms;
// MP units (task): W(j, k) = alpha h(j, k).
// What bounds it: a unit is one block, and most launches have fewer blocks than
// SMs, so its time is one thread's chain: the loads, then about 20 instructions
// per digit pair.  A thread takes 8 k and keeps them from the search for the
// row's largest element (16 k, loaded twice, by 256 threads: 15 to 19 us a
// launch; the 16-mode sweep 977 -> 875 us, the 64-mode one 7.80 -> 7.47 ms,
// bonds above 64 33.1 -> 32.4 ms, three states overlapped).
// Launches of more units than SMs gain from two blocks per SM (64 registers, a
// few spilled; at 88 to 116 one block: 64 modes 7.48 -> 7.40 ms).
constexpr int kTcsImgThreads = 512;
template <int OP>
__global__ void __launch_bounds__(kTcsImgThreads, 2) k_tcs_img(TcsArgs g, const int2* __restrict__ units, int64_t first) {
  int2 u = OP == TCS_MP ? make_int2(g.mp_tasks[first + blockIdx.x], 0) : units[first + blockIdx.x];
  const int n = threadIdx.x & 63, q = threadIdx.x >> 6;
  int np, ncols, c0, steps;  // the unit's column block and image
  unsigned char* img;
  if (OP == TCS_HP) {
    const HpTcGroup& G = g.groups[u.x];
    np = G.ap;
    ncols = G.nc;
    c0 = G.c0;
    steps = hp_tc_kc(np) / kChunkK;
    img = G.img + (size_t)u.y * hp_tc_chunk_bytes(np, steps);
  } else {
    int cb, cols, k;
    if (OP == TCS_MP) {
      cb = u.x >> kMpTcTaskShift;
      u.x &= (1 << kMpTcTaskShift) - 1;
      const MPTask& t = g.mp[u.x];
      cols = t.a_out;
      k = t.a_in;
      img = static_cast<unsigned char*>(t.oz_h);
    } else {
      const AccTask& T = g.acc[u.x];
      cb = u.y / T.count;
      cols = k = T.d;
      img = static_cast<unsigned char*>(T.tc_img);
    }
    np = tc_width(cols);
    c0 = cb * np;
    ncols = min(np, cols - c0);
    steps = tc_steps(k);
    img += (size_t)(OP == TCS_MP ? cb : u.y) * hp_tc_chunk_bytes(np, steps);
  }
  // the eight values of row n in core row hs
  auto load8 = [&](int hs, float4 (&v)[8]) {
    if (OP == TCS_HP) {
      const HpTcGroup& G = g.groups[u.x];
      const int K = G.before * G.after, k0 = u.y * hp_tc_kc(G.ap) + hs * 8;
      const float4* __restrict__ A = reinterpret_cast<const float4*>(G.A);
      KWalk w(min(k0, K), G.before);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n < ncols && k0 + kk < K) {
          x = __ldg(A + w.off(c0 + n, G.before, G.a));
          x.z = -x.z;
          x.w = -x.w;
        }
        v[kk] = x;
        w.next(G.before);
      }
    } else if (OP == TCS_MP) {
      const MPTask& t = g.mp[u.x];
      const float4 cf = DF64::coef(t.alpha);
      const bool one = t.alpha.x == 1.0 && t.alpha.y == 0.0;
      const float4* __restrict__ H = reinterpret_cast<const float4*>(t.h);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const int k = hs * 8 + kk;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n < ncols && k < t.a_in) {
          x = __ldg(H + c0 + n + (int64_t)t.a_out * k);
          if (!one) x = DF64::mul(cf, x);
        }
        v[kk] = x;
      }
    } else {
      const AccTask& T = g.acc[u.x];
      const AccTerm tm = g.terms[T.first + u.y % T.count];
      const double2 alpha = T.alpha_ptr ? *T.alpha_ptr : T.alpha;
      const float4 cf = DF64::coef(alpha);
      const float4* __restrict__ H = reinterpret_cast<const float4*>(tm.H);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const int k = hs * 8 + kk;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (n < ncols && k < T.d) {
          if (H) x = DF64::mul(cf, __ldg(H + c0 + n + (int64_t)T.d * k));
          else if (c0 + n == k) x = cf;
        }
        v[kk] = x;
      }
    }
  };
  __shared__ int fx[64];  // largest |W| of a row as an integer, then its exponent
  if (threadIdx.x < 64) fx[threadIdx.x] = 0;
  __syncthreads();
  // the largest |W| of this thread's core rows, the first one last: its values
  // stay in registers (up to 64 k a thread has no other)
  constexpr int kS = kTcsImgThreads / 64;
  const int last = 2 * steps - 1 - q, nhs = last >= 0 ? last / kS + 1 : 0;
  float4 v[8];
  int m = 0;
#pragma unroll 1
  for (int i = nhs - 1; i >= 0; --i) {
    load8(q + kS * i, v);
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) m = max(m, max(fmag(v[kk].x), fmag(v[kk].z)));
  }
  atomicMax(&fx[n], m);
  __syncthreads();
  if (n < np && nhs > 0) {
    const float f = row_factor(row_exponent(fx[n]));
    const int rows = 3 * np, plane = rows * 32;
#pragma unroll 1
    for (int i = 0;;) {
      const int hs = q + kS * i, c = hs & 1;
      unsigned char* base = img + (size_t)(hs >> 1) * kDig * plane;
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint32_t w[kDig][4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          float d0[kDig], d1[kDig];
          digits_f32(part ? v[2 * p].z : v[2 * p].x, part ? v[2 * p].w : v[2 * p].y, f, d0);
          digits_f32(part ? v[2 * p + 1].z : v[2 * p + 1].x, part ? v[2 * p + 1].w : v[2 * p + 1].y, f, d1);
#pragma unroll
          for (int d = 0; d < kDig; ++d) w[d][p] = pack_bf16(d0[d], d1[d]);
        }
#pragma unroll
        for (int d = 0; d < kDig; ++d) {
          unsigned char* pl = base + (size_t)d * plane;
          const uint4 x = make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
          if (part == 0) {
            *reinterpret_cast<uint4*>(pl + core_off(np + n, c, rows)) = x;
          } else {
            *reinterpret_cast<uint4*>(pl + core_off(n, c, rows)) =
                make_uint4(x.x ^ 0x80008000u, x.y ^ 0x80008000u, x.z ^ 0x80008000u, x.w ^ 0x80008000u);
            *reinterpret_cast<uint4*>(pl + core_off(2 * np + n, c, rows)) = x;
          }
        }
      }
      if (++i >= nhs) break;
      load8(q + kS * i, v);
    }
  }
  if (threadIdx.x < 64)
    reinterpret_cast<int*>(img + (size_t)steps * kDig * 3 * np * 32)[threadIdx.x] = row_exponent(fx[threadIdx.x]);
}

// pre-pass of the hole products: the biased row exponents E of the M side
// (the members' B rows j, 128 per item) over the item's chunk, into the
// group's table, so that the producers need not read every row twice.  Block
// (item, q) takes the rows 32 q .. 32 q + 31.  With before > 1 a row's k are
// contiguous in memory: a warp takes four rows at once, its lanes along k;
// with before == 1 consecutive rows are: lane l takes row 32 q + l, the
// eight warps an eighth of the chunk each.
__global__ void __launch_bounds__(256) k_hp_ex(TcsArgs g) {
  const int4 itm = g.items[g.item0 + blockIdx.x];
  const HpTcGroup& G = g.groups[itm.x];
  const int before = G.before, a = G.a, K = before * G.after, kc = hp_tc_kc(G.ap);
  const int k0 = itm.z * kc, k1 = min(K, k0 + kc);
  const int rows = G.n * a, m0 = 32 * (int)blockIdx.y;
  unsigned char* ex = G.ex + (size_t)itm.z * kRows;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (before > 1) {
    int e[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int m = m0 + warp + 8 * r;
      e[r] = 0;
      if (m < rows) {
        const int mi = m / a, j = m - mi * a;
        const float4* __restrict__ B = reinterpret_cast<const float4*>(g.hp[G.member[mi]].B);
#pragma unroll
        for (int s = 0; s < 4; ++s) {  // kc <= 128: four k per lane
          const int k = k0 + lane + 32 * s;
          if (k < k1) {
            const int c = k / before, b = k - c * before;
            const float4 x = __ldg(B + b + (int64_t)before * j + (int64_t)before * a * c);
            e[r] = max(e[r], max(fmag(x.x), fmag(x.z)));
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      int v = e[r];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
      if (lane == 0) ex[m0 + warp + 8 * r] = (uint8_t)row_exponent(v);
    }
  } else {
    __shared__ int part[8][32];
    const int m = m0 + lane;
    int e = 0;
    if (m < rows) {
      const int mi = m / a, j = m - mi * a;
      const float4* __restrict__ B = reinterpret_cast<const float4*>(g.hp[G.member[mi]].B);
      const int span = (k1 - k0 + 7) >> 3;
      const int ka = k0 + warp * span, kb = min(k1, ka + span);
      for (int k = ka; k < kb; ++k) {
        const float4 x = __ldg(B + j + (int64_t)a * k);
        e = max(e, max(fmag(x.x), fmag(x.z)));
      }
    }
    part[warp][lane] = e;
    __syncthreads();
    if (warp == 0) {
      int v = part[0][lane];
#pragma unroll
      for (int w = 1; w < 8; ++w) v = max(v, part[w][lane]);
      ex[m] = (uint8_t)row_exponent(v);
    }
  }
}

// Four columns of the accumulators (real parts from column 0 of `addr`, the
// imaginary parts np columns on), their levels added in double-float: levels
// 0..2 by two-sums, the others (at least one) into the low word.  Beyond 64
// (wide) level 3 by a two-sum too: in the low word it rounds to 2^-45 of the
// result, more than the double-float multiply-adds that these shapes replace
// (bonds 65..112: density matrices 8.6e-15 with it, 5.0e-15 by multiply-adds);
// up to 64 it would cost the 64-mode sweep 2%.  All threads of the warp.
__device__ __forceinline__ void tcs_levels(uint32_t addr, int np, int NL, bool wide, float (&v)[2][4],
                                           float (&l)[2][4]) {
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    float lv[kDig][4];
    const uint32_t a = addr + (uint32_t)(part * np);
#pragma unroll
    for (int L = 0; L < kDig; ++L)
      if (L < 4 || L < NL) tmem_ld4(a + (uint32_t)(L * 2 * np), lv[L]);
    tmem_wait_ld();
    if (wide) {
      float rest[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int L = kDig - 1; L >= 4; --L)
        if (L < NL) {
#pragma unroll
          for (int i = 0; i < 4; ++i) rest[i] = __fadd_rn(rest[i], lv[L][i]);
        }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float s, t, e1, e2, e3;
        df_two_sum(lv[0][i], lv[1][i], s, e1);
        df_two_sum(s, lv[2][i], t, e2);
        df_two_sum(t, lv[3][i], v[part][i], e3);
        l[part][i] = __fadd_rn(__fadd_rn(__fadd_rn(e3, e2), e1), rest[i]);
      }
      continue;
    }
    if (NL > 4) {
#pragma unroll
      for (int L = 4; L < kDig; ++L)
        if (L < NL) {
#pragma unroll
          for (int i = 0; i < 4; ++i) lv[3][i] = __fadd_rn(lv[3][i], lv[L][i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float s, e1, e2;
      df_two_sum(lv[0][i], lv[1][i], s, e1);
      df_two_sum(s, lv[2][i], v[part][i], e2);
      l[part][i] = __fadd_rn(__fadd_rn(e2, e1), lv[3][i]);
    }
  }
}

// 4 x 4 transpose of o among the four lanes of a quad: afterwards o[i] is what
// lane (lane & ~3) + i held in o[lane & 3]
__device__ __forceinline__ void quad_transpose(float4 (&o)[4], int lane) {
#pragma unroll
  for (int bit = 1; bit <= 2; bit <<= 1) {
    const bool up = lane & bit;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i & bit) continue;  // the pair (i, i | bit)
      const float4 send = up ? o[i] : o[i | bit];
      float4 got;
      got.x = __shfl_xor_sync(0xffffffffu, send.x, bit);
      got.y = __shfl_xor_sync(0xffffffffu, send.y, bit);
      got.z = __shfl_xor_sync(0xffffffffu, send.z, bit);
      got.w = __shfl_xor_sync(0xffffffffu, send.w, bit);
      if (up) o[i] = got;
      else o[i | bit] = got;
    }
  }
}
__device__ __forceinline__ float4* shfl_ptr(float4* p, int src) {
  return reinterpret_cast<float4*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(p), src));
}

// Row r of an item: element k of X at src + k stride (mode products and
// accumulations; hole products: src + b + before a c for k = b + before c), and
// whether the row exists.  u: the accumulation's term.
template <int OP>
__device__ __forceinline__ const float4* tcs_row(const TcsArgs& g, int4 itm, int u, int r, int64_t& stride) {
  if (OP == TCS_HP) {
    const HpTcGroup& G = g.groups[itm.x];
    const int mi = r / G.a;
    if (mi >= G.n) return nullptr;
    return reinterpret_cast<const float4*>(g.hp[G.member[mi]].B) + (int64_t)G.before * (r - mi * G.a);
  }
  const uint32_t rg = (uint32_t)itm.y * kRows + r;  // at most 2^31 rows
  if (OP == TCS_ACC) {
    const AccTask& T = g.acc[itm.x];
    stride = T.rows;
    return rg < (uint32_t)T.rows ? reinterpret_cast<const float4*>(g.terms[T.first + u].X) + rg : nullptr;
  }
  // mode product: row (b, c) of the input, its k-th element at b + before (k + a_in c)
  const MPTask& t = g.mp[itm.x];
  stride = t.before;
  const uint32_t before = (uint32_t)t.before;
  if (rg >= before * (uint32_t)t.after) return nullptr;
  const uint32_t c = rg / before;
  return reinterpret_cast<const float4*>(t.in) + (rg - c * before) + (int64_t)t.before * t.a_in * c;
}

// the row's largest |X| from the exponent warps' shares: a third of the k each,
// or, where a row's k are contiguous, every third row
__device__ __forceinline__ int tcs_row_max(const int (&ex)[kTcsExWarps][kRows], int r, bool along) {
  return along ? ex[r % kTcsExWarps][r] : max(max(ex[0][r], ex[1][r]), ex[2][r]);
}

// Roles (512 threads).
// Warps 0-3 produce X's digits, one thread per row of the tile, each 16-k step
// in two halves of eight k with the next half's loads in flight.
// Warp 4 allocates tensor memory and issues the MMAs from one thread; warps
// 5-7 find the rows' exponents of the units ahead (hole products: a pre-pass
// does).
// Warps 8-15 are the epilogue, warp w reading lanes 32 (w % 4).. (tensor
// memory's lane quarter of its sub-partition) for half (w - 8) / 4 of the
// columns: it adds a unit's levels, scales, and stores or adds to the outputs.
// Every wait is bounded (all lanes of a warp give up together): a wait that
// runs out sets the status word, and the CTA drains its issued MMAs, frees
// tensor memory and returns.
// What bounds it, per 128 x 64 unit of 64 k: a 16-k step (56 MMAs that read 57 KB
// of X's and 43 KB of W's digits from shared memory) takes 4.9 k cycles, all of
// it shared-memory bandwidth, and the epilogue 6 to 10 k cycles for each unit that
// it holds up the next unit's MMAs.  The rows' exponents need all of X before
// its first digit: in the producers, ahead of every unit, that pass took 9 to
// 15 k cycles; in warps of its own it runs under the previous unit (a CTA's
// mode products 22.1 -> 17.2 k cycles a unit; 64-mode wide sweep 41.1 -> 37.2 ms,
// 64-mode sweep 10.5 -> 10.1 ms, 16-mode 1.72 -> 1.67 ms).
template <int OP, bool WIDE>
__global__ void __launch_bounds__(kTcsThreads, 1) k_tcs(TcsArgs g) {
  extern __shared__ __align__(128) unsigned char tcs_raw[];
  TcsSmem& sm = *reinterpret_cast<TcsSmem*>(tcs_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int64_t my0, my1;
  tcs_range<OP>(g, my0, my1);
  int* status = g.status;

  if (tid == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sm.bar.full[s], 128);
      mbar_init(&sm.bar.empty[s], 1);
      mbar_init(&sm.bar.exready[s], kTcsExWarps);
      mbar_init(&sm.bar.exfree[s], 4 + kTcsEpWarps);
    }
    mbar_init(&sm.bar.tfull, 1);
    mbar_init(&sm.bar.tempty, kTcsEpWarps);
    mbar_init(&sm.bar.drain, 1);
    mbar_fence_init();
  }
  if (warp == 4) tmem_alloc(&sm.bar.tmem, 512u);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = sm.bar.tmem;
  bool ok = true;
  auto waited = [&](void* bar, uint32_t parity, int code) {  // whole warp
    if (__all_sync(0xffffffffu, mbar_wait(bar, parity, kSpin))) return true;
    set_status(status, code);
    ok = false;
    return false;
  };

  if (warp < 4) {
    // ---------------- producers: one per row ----------------
    const int r = tid;
    uint32_t q = 0, un = 0;
    for (int64_t it = my0; it < my1 && ok; ++it) {
      const int4 itm = tcs_fetch<OP>(g, it);
      const TcsItem I = tcs_item<OP, WIDE>(g, itm);
      const uint32_t nbytes = (uint32_t)(kDig * 3 * I.np * 32);
      int before = 0, K = 0;
      int64_t jump = 0;  // hole products: from the end of one run of b to the next
      if (OP == TCS_HP) {
        const HpTcGroup& G = g.groups[itm.x];
        before = G.before;
        K = before * G.after;
        jump = (int64_t)before * (G.a - 1);
      } else {
        K = OP == TCS_ACC ? g.acc[itm.x].d : g.mp[itm.x].a_in;
      }
      for (int u = 0; u < I.nunits; ++u, ++un) {
        const int buf = (int)(un & 1);
        int64_t stride = 1;
        const int t = I.term(u), s0 = I.step0(u), nks = I.steps(u);
        const float4* p = tcs_row<OP>(g, itm, t, r, stride);
        // the row's elements in order: `left` of them, the next one at p
        int left = 0, b = 0;
        if (OP == TCS_HP) {
          const int k0 = ((itm.z + t) * I.nks + s0) * kChunkK, c = k0 / before;
          b = k0 - c * before;
          if (p) {
            left = K - k0;
            p += b + (jump + before) * c;
          }
        } else if (p) {
          left = K - s0 * kChunkK;
          p += stride * (s0 * kChunkK);
        }
        auto load8 = [&](float4 (&x)[8]) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            x[i] = i < left ? __ldg(p) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (OP == TCS_HP) {
              ++p;
              if (++b == before) {
                b = 0;
                p += jump;
              }
            } else {
              p += stride;
            }
          }
          left -= 8;
        };
        float4 nx[8];
        load8(nx);
        int eb;
        if (OP == TCS_HP) {
          eb = __ldg(g.groups[itm.x].ex + (size_t)(itm.z + t) * kRows + r);
        } else {
          if (!waited(&sm.bar.exready[buf], (un >> 1) & 1, 18)) break;
          eb = row_exponent(tcs_row_max(sm.ex[buf], r, OP == TCS_MP && stride == 1));
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.bar.exfree[buf]);
        }
        const float rowf = row_factor(eb);
        const unsigned char* img = tcs_image<OP>(g, itm, t, I) + (size_t)s0 * nbytes;
        for (int ks = 0; ks < nks; ++ks, ++q) {
          const int s = q & 1;
          if (!waited(&sm.bar.empty[s], ((q >> 1) & 1) ^ 1, 11)) break;
          if (tid == 0) {
            // W's digits of this step; the copy completes on full[s] (it
            // finishes within microseconds, before any wait could run out)
            mbar_expect_tx(&sm.bar.full[s], nbytes);
            bulk_g2s(sm.n[s], img + (size_t)ks * nbytes, nbytes, &sm.bar.full[s]);
          }
          unsigned char* As = sm.a[s];
#pragma unroll 1
          for (int hh = 0; hh < 2; ++hh) {
            float4 x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = nx[i];
            if (ks + hh < nks) load8(nx);  // the next half: (ks, 1) or (ks + 1, 0)
            const int off = core_off(r, hh, kRows);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
              uint32_t w[kDig][4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                float d0[kDig], d1[kDig];
                digits_f32(part ? x[2 * i].z : x[2 * i].x, part ? x[2 * i].w : x[2 * i].y, rowf, d0);
                digits_f32(part ? x[2 * i + 1].z : x[2 * i + 1].x, part ? x[2 * i + 1].w : x[2 * i + 1].y, rowf, d1);
#pragma unroll
                for (int d = 0; d < kDig; ++d) w[d][i] = pack_bf16(d0[d], d1[d]);
              }
#pragma unroll
              for (int d = 0; d < kDig; ++d)
                *reinterpret_cast<uint4*>(As + (2 * d + part) * kOzAPlane + off) =
                    make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
            }
          }
          fence_proxy_async();
          mbar_arrive(&sm.bar.full[s]);
        }
        if (!ok) break;
      }
    }
  } else if (warp < 8) {
    if (warp == 4) {
      // ---------------- MMA issue (one thread) ----------------
      if (lane == 0) {
        uint32_t q = 0, un = 0;
        for (int64_t it = my0; it < my1 && ok; ++it) {
          const int4 itm = tcs_fetch<OP>(g, it);
          const TcsItem I = tcs_item<OP, WIDE>(g, itm);
          const int np = I.np, NL = I.nl;
          const uint32_t id = idesc_m128(1, 2 * np, false);
          const uint32_t lboA = (kRows / 8) * 128, lboN = (uint32_t)(3 * np / 8) * 128;
          const uint64_t pA = kOzAPlane >> 4, pN = (uint64_t)((3 * np * 32) >> 4);
          const uint64_t p1 = (uint64_t)((np / 8) * 128 >> 4);  // rows np..: [Wr | Wi]
          for (int u = 0; u < I.nunits && ok; ++u, ++un) {
            if (!mbar_wait(&sm.bar.tempty, (un & 1) ^ 1, kSpin)) {
              set_status(status, 14);
              ok = false;
              break;
            }
            fence_after_sync();
            for (int ks = 0, nks = I.steps(u); ks < nks; ++ks, ++q) {
              const int s = q & 1;
              if (!mbar_wait(&sm.bar.full[s], (q >> 1) & 1, kSpin)) {
                set_status(status, 15);
                ok = false;
                break;
              }
              fence_after_sync();
              const uint64_t dA = desc_kmajor(smem_u32(sm.a[s]), lboA, 128);
              const uint64_t dN = desc_kmajor(smem_u32(sm.n[s]), lboN, 128);
              const uint32_t first = ks == 0 ? 1u : 0u;
#pragma unroll
              for (int sd = 0; sd < kDig; ++sd) {
                const uint64_t ar = dA + (uint64_t)(2 * sd) * pA, ai = ar + pA;
#pragma unroll
                for (int td = 0; td + sd < kDig; ++td) {
                  const int L = sd + td < NL - 1 ? sd + td : NL - 1;
                  const uint64_t nb = dN + (uint64_t)td * pN;
                  const uint32_t d = tmem + (uint32_t)(L * 2 * np);
                  const uint32_t acc = (first && sd == 0 && td == L) ? 0u : 1u;
                  mma_bf16(d, ar, nb + p1, id, acc);  // Xr x [Wr | Wi]
                  mma_bf16(d, ai, nb, id, 1);         // Xi x [-Wi | Wr]
                }
              }
              commit(&sm.bar.empty[s]);
            }
            if (!ok) break;
            commit(&sm.bar.tfull);
          }
        }
        commit(&sm.bar.drain);
        if (!mbar_wait(&sm.bar.drain, 0, kSpin)) set_status(status, 16);
      }
    } else if (OP != TCS_HP) {
      // ---------------- exponents: the rows' largest |X| over the unit's k ----------------
      // (loads eight at a time in each of the three warps; the records they
      // need are read once per item, the next term's ahead of its unit)
      const int xw = warp - 5;
      uint32_t un = 0;
      for (int64_t it = my0; it < my1 && ok; ++it) {
        const int4 itm = tcs_fetch<OP>(g, it);
        const TcsItem I = tcs_item<OP, WIDE>(g, itm);
        int K;
        uint32_t nrows, before = 1;  // at most 2^31 rows
        int64_t stride;
        const float4* X;  // the item's tensor (accumulations: the term's)
        const AccTerm* terms = nullptr;
        if (OP == TCS_ACC) {
          const AccTask& T = g.acc[itm.x];
          K = T.d;
          nrows = (uint32_t)T.rows;
          stride = T.rows;
          terms = g.terms + T.first;
          X = reinterpret_cast<const float4*>(terms[0].X);
        } else {
          const MPTask& t = g.mp[itm.x];
          K = t.a_in;
          before = (uint32_t)t.before;
          nrows = before * (uint32_t)t.after;
          stride = t.before;
          X = reinterpret_cast<const float4*>(t.in);
        }
        const bool along = OP == TCS_MP && before == 1;  // a row's k are contiguous
        const uint32_t row0 = (uint32_t)itm.y * kRows;
        for (int u = 0; u < I.nunits; ++u, ++un) {
          const int buf = (int)(un & 1);
          const int k0 = I.step0(u) * kChunkK, k1 = WIDE ? min(K, k0 + I.steps(u) * kChunkK) : K;
          const float4* next =
              OP == TCS_ACC && u + 1 < I.nunits ? reinterpret_cast<const float4*>(terms[I.term(u + 1)].X) : X;
          // producers and epilogue of the unit two back have read this buffer
          if (!waited(&sm.bar.exfree[buf], ((un >> 1) & 1) ^ 1, 19)) break;
          int* ex = sm.ex[buf][xw];
          if (along) {
            // every third row, four at a time, the lanes along k
            for (int r0 = xw; r0 < kRows; r0 += 4 * kTcsExWarps) {
              int m[4] = {0, 0, 0, 0};
#pragma unroll 2
              for (int k = k0 + lane; k < k1; k += 32)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const uint32_t rg = row0 + r0 + kTcsExWarps * i;
                  const float4 x = rg < nrows ? __ldg(X + (int64_t)K * rg + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                  m[i] = max(m[i], max(fmag(x.x), fmag(x.z)));
                }
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int r = r0 + kTcsExWarps * i, v = __reduce_max_sync(0xffffffffu, m[i]);
                if (lane == i && r < kRows) ex[r] = v;
              }
            }
          } else {
            // a third of the k of every row, the lanes along the rows
            const int ka = k0 + xw * (k1 - k0) / kTcsExWarps, kb = k0 + (xw + 1) * (k1 - k0) / kTcsExWarps;
            const float4* p[4];
            int m[4] = {0, 0, 0, 0};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t rg = row0 + 32 * i + lane;
              int64_t o = rg;
              if (OP == TCS_MP) {
                const uint32_t c = rg / before;
                o = (int64_t)(rg - c * before) + (int64_t)before * K * c;
              }
              p[i] = rg < nrows ? X + o + stride * ka : nullptr;
            }
#pragma unroll 2
            for (int k = ka; k < kb; ++k)
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float4 x = p[i] ? __ldg(p[i] + stride * (k - ka)) : make_float4(0.f, 0.f, 0.f, 0.f);
                m[i] = max(m[i], max(fmag(x.x), fmag(x.z)));
              }
#pragma unroll
            for (int i = 0; i < 4; ++i) ex[32 * i + lane] = m[i];
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.bar.exready[buf]);
          X = next;
        }
      }
    }
  } else {
    // ---------------- epilogue: warps 8..15, lane quarter w % 4, column half (w - 8) / 4 ----------------
    const int qd = warp & 3, half = (warp - 8) >> 2;
    const int r = 32 * qd + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(32 * qd) << 16);
    int* fxw = sm.fx[warp - 8];
    uint32_t un = 0;
    for (int64_t it = my0; it < my1 && ok; ++it) {
      const int4 itm = tcs_fetch<OP>(g, it);
      const TcsItem I = tcs_item<OP, WIDE>(g, itm);
      const int np = I.np, NL = I.nl;
      const int c0 = half * (np >> 1), w = np >> 1;  // this warp's columns
      // output row r: element n at base[n * stride]
      float4* base = nullptr;
      int64_t stride = 1;
      bool add_first = false, along_k = false;
      if (OP == TCS_HP) {
        const HpTcGroup& G = g.groups[itm.x];
        const int mi = r / G.a, j = r - mi * G.a;
        if (mi < G.n) {
          const HPTask& t = g.hp[G.member[mi]];
          double2* dst = t.splits <= 1 ? t.S : g.ws + t.ws + (int64_t)itm.y * G.a * G.a;
          base = reinterpret_cast<float4*>(dst) + (int64_t)G.a * j;
        }
      } else if (OP == TCS_ACC) {
        const AccTask& T = g.acc[itm.x];
        const int64_t rg = (int64_t)itm.y * kRows + r;
        if (rg < T.rows) base = reinterpret_cast<float4*>(T.out) + rg;
        stride = T.rows;
        add_first = T.add != 0;
      } else {
        const MPTask& t = g.mp[itm.x];
        const int64_t rg = (int64_t)itm.y * kRows + r;
        if (rg < (int64_t)t.before * t.after)
          base = reinterpret_cast<float4*>(t.out) + rg % t.before + (int64_t)t.before * t.a_out * (rg / t.before);
        stride = t.before;
        add_first = t.add != 0;
        along_k = t.before == 1;
      }
      if (base) base += stride * (I.c0 + c0);
      const int ncols = I.ncols - c0;  // real columns of this warp's half (may be <= 0)
      for (int u = 0; u < I.nunits; ++u, ++un) {
        const int buf = (int)(un & 1);
        const bool store = u == 0 && !add_first;
        int er;
        if (OP == TCS_HP) {
          er = __ldg(g.groups[itm.x].ex + (size_t)(itm.z + I.term(u)) * kRows + r);
        } else {
          if (!waited(&sm.bar.exready[buf], (un >> 1) & 1, 20)) break;
          er = row_exponent(tcs_row_max(sm.ex[buf], r, along_k));
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.bar.exfree[buf]);
        }
        const int* fxg = reinterpret_cast<const int*>(tcs_image<OP>(g, itm, I.term(u), I) +
                                                      (size_t)I.isteps * kDig * 3 * np * 32);
        const int f0 = __ldg(fxg + lane), f1 = __ldg(fxg + 32 + lane);
        __syncwarp();
        fxw[lane] = f0 << 23;
        fxw[32 + lane] = f1 << 23;
        __syncwarp();
        // the common case: every scale 2^(E + F) of the warp's rows and the
        // unit's columns is a normal number and no operand is infinite or NaN
        const int fmax = max(__reduce_max_sync(0xffffffffu, f0), __reduce_max_sync(0xffffffffu, f1));
        const int fmin = min(__reduce_min_sync(0xffffffffu, f0), __reduce_min_sync(0xffffffffu, f1));
        const bool normal = __all_sync(
            0xffffffffu, !base || (er + fmin >= 126 && er + fmax <= 379 && er < 255 && fmax < 255));
        const int erow = (er - 125) << 23;  // + (F << 23): the bits of 2^(E - 126 + F - 126)
        if (!waited(&sm.bar.tfull, un & 1, 17)) break;
        fence_after_sync();
        // outputs contiguous along the columns (stride 1): a lane's 16-byte
        // stores would touch 32 lines; the quads transpose 4 x 4 blocks so
        // that a store covers eight rows of 64 bytes
        const bool along = stride == 1 && store && normal;  // uniform
        float4* qp[4];
        if (along) {
#pragma unroll
          for (int i = 0; i < 4; ++i) qp[i] = shfl_ptr(base, (lane & ~3) + i);
        }
        float4* p = base;
        for (int n0 = 0; n0 < w; n0 += 4, p += 4 * stride) {
          const int nc = min(4, ncols - n0);  // columns of the block that exist (uniform)
          if (nc <= 0) break;
          // the old outputs of these four columns: their loads in flight
          // together, under the tensor-memory reads
          float4 old[4];
          if (!store) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              old[e] = (base && e < nc) ? p[stride * e] : make_float4(0.f, 0.f, 0.f, 0.f);
          }
          __syncwarp();
          float v[2][4], l[2][4];  // recombined levels: re and im of the four columns
          tcs_levels(lane_addr + (uint32_t)(c0 + n0), np, NL, I.wide, v, l);
          if (along) {
            float4 o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float f = __int_as_float(erow + fxw[c0 + n0 + i]);
              o[i] = make_float4(__fmul_rn(v[0][i], f), __fmul_rn(l[0][i], f), __fmul_rn(v[1][i], f),
                                 __fmul_rn(l[1][i], f));
              df_norm(o[i].x, o[i].y);
              df_norm(o[i].z, o[i].w);
            }
            quad_transpose(o, lane);
            const int col = n0 + (lane & 3);
            if (col < ncols) {
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (qp[i]) qp[i][col] = o[i];
            }
            continue;
          }
          if (!base) continue;
          if (normal) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float f = __int_as_float(erow + fxw[c0 + n0 + i]);
              float4 o = make_float4(__fmul_rn(v[0][i], f), __fmul_rn(l[0][i], f), __fmul_rn(v[1][i], f),
                                     __fmul_rn(l[1][i], f));
              if (!store) {
                df_add(o.x, o.y, old[i].x, old[i].y);
                df_add(o.z, o.w, old[i].z, old[i].w);
              }
              df_norm(o.x, o.y);
              df_norm(o.z, o.w);
              if (i < nc) p[stride * i] = o;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (i >= nc) continue;
              const int fn = (int)((uint32_t)fxw[c0 + n0 + i] >> 23);
              const int sh = (er - 126) + (fn - 126);
              float4 o = make_float4(scale2(v[0][i], sh), scale2(l[0][i], sh), scale2(v[1][i], sh),
                                     scale2(l[1][i], sh));
              if (!store) {
                df_add(o.x, o.y, old[i].x, old[i].y);
                df_add(o.z, o.w, old[i].z, old[i].w);
              }
              df_norm(o.x, o.y);
              df_norm(o.z, o.w);
              if (er == 255 || fn == 255) {  // an Inf or NaN among the operands: propagate it
                const float nan = __int_as_float(0x7fffffff);
                o = make_float4(nan, nan, nan, nan);
              }
              p[stride * i] = o;
            }
          }
        }
        fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.bar.tempty);
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 4) {
    fence_after_sync();
    tmem_dealloc(tmem, 512u);
  }
}

int g_tc_sms = 0;

cudaError_t tc_grid(int64_t n_tiles, unsigned* grid) {
  if (!g_tc_sms) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    g_tc_sms = sms;
  }
  *grid = (unsigned)(n_tiles < g_tc_sms ? n_tiles : g_tc_sms);
  return cudaSuccess;
}

cudaError_t launch_tf(const MPTask* tasks, const int2* tiles, int64_t first_tile, int64_t n_tiles, int* status,
                      cudaStream_t s) {
  unsigned grid = 0;
  cudaError_t e = tc_grid(n_tiles, &grid);
  if (e != cudaSuccess) return e;
  const int sm = (int)sizeof(TfSmem);
  e = cudaFuncSetAttribute(k_mp_tf, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  if (e != cudaSuccess) return e;
  k_mp_tf<<<grid, kThreadsTc, sm, s>>>(tasks, tiles, first_tile, n_tiles, status);
  return cudaGetLastError();
}

// wide: some item has more than kTcCols columns
template <int OP>
cudaError_t launch_tcs(const TcsArgs& g, const int2* img_units, int64_t first_unit, int64_t n_units, bool wide,
                       cudaStream_t s) {
  if (n_units > 0) k_tcs_img<OP><<<(unsigned)n_units, kTcsImgThreads, 0, s>>>(g, img_units, first_unit);
  if (OP == TCS_HP) k_hp_ex<<<dim3((unsigned)g.n_items, kRows / 32), 256, 0, s>>>(g);
  unsigned grid = 0;
  cudaError_t e = tc_grid(g.n_items, &grid);
  if (e != cudaSuccess) return e;
  const int smem = (int)sizeof(TcsSmem);
  const auto kernel = wide ? k_tcs<OP, true> : k_tcs<OP, false>;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  kernel<<<grid, kTcsThreads, smem, s>>>(g);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_hp_tc(const HPTask* tasks, const HpTcGroup* groups, const int4* items, int64_t first_item,
                         int64_t n_items, const int2* img_units, int64_t first_unit, int64_t n_units,
                         double2* ws, bool wide, int* status, cudaStream_t s) {
  if (n_items <= 0) return cudaSuccess;
  TcsArgs g{};
  g.hp = tasks;
  g.groups = groups;
  g.ws = ws;
  g.items = items;
  g.item0 = first_item;
  g.n_items = n_items;
  g.status = status;
  return launch_tcs<TCS_HP>(g, img_units, first_unit, n_units, wide, s);
}

cudaError_t launch_mp_tcs(const MPTask* tasks, const int2* tiles, int64_t first_tile, int64_t n_tiles,
                          const int* tc_tasks, int64_t first_task, int64_t n_tasks, bool wide, int* status, cudaStream_t s) {
  if (n_tiles <= 0) return cudaSuccess;
  TcsArgs g{};
  g.mp = tasks;
  g.mp_tiles = tiles;
  g.mp_tasks = tc_tasks;
  g.item0 = first_tile;
  g.n_items = n_tiles;
  g.status = status;
  return launch_tcs<TCS_MP>(g, nullptr, first_task, n_tasks, wide, s);
}

cudaError_t launch_acc_tc(const AccTask* tasks, const AccTerm* terms, const int4* items, int64_t first_item,
                          int64_t n_items, int64_t units, const int2* img_units, int64_t first_unit,
                          int64_t n_units, bool wide, int* status, cudaStream_t s) {
  if (n_items <= 0) return cudaSuccess;
  TcsArgs g{};
  g.acc = tasks;
  g.terms = terms;
  g.items = items;
  g.item0 = first_item;
  g.n_items = n_items;
  g.units = units;
  g.status = status;
  return launch_tcs<TCS_ACC>(g, img_units, first_unit, n_units, wide, s);
}

cudaError_t launch_mp_tc(bool oz, const MPTask* tasks, const int2* tiles, int64_t first_tile, int64_t n_tiles,
                         const int* tc_tasks, int64_t first_task, int64_t n_tasks, bool wide, int* status, cudaStream_t s) {
  if (n_tiles <= 0) return cudaSuccess;
  if (oz) return launch_mp_tcs(tasks, tiles, first_tile, n_tiles, tc_tasks, first_task, n_tasks, wide, status, s);
  if (n_tasks > 0) k_mp_tf_h<<<(unsigned)n_tasks, 256, 0, s>>>(tasks, tc_tasks, first_task);
  return launch_tf(tasks, tiles, first_tile, n_tiles, status, s);
}

}  // namespace qt
