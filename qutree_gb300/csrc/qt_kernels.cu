// qt_kernels.cu -- complex128 kernels of the H.Psi sweep for sm_103a.
//
// GB300 executes FP64 at ~1.2 TFLOP/s (1/61 of its FP32 rate), so every
// complex128 contraction here is bound by the FP64 pipe, not by HBM: a
// complex multiply-add needs 4 DFMA but at most 32 bytes of operands, which
// L1/L2 deliver far faster than the DFMA units consume them.  The kernels are
// therefore plain SIMT loops with coalesced 16-byte complex loads, shared
// memory staging where an operand is reused by a whole tile, several
// independent accumulators per thread for instruction-level parallelism, and
// fixed summation orders (no atomics: results are bit-identical run to run).
//
// Batched launches: each kernel reads a task table and a tile table; block b
// processes tile b.  The planner (qt_plan.cpp) builds both once per tree.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <type_traits>

#include <cuda.h>

#include "qt_arith.cuh"
#include "qt_internal.h"

namespace qt {
namespace {

constexpr int kThreads = 256;
constexpr int kHpMaxDim = 112;  // largest bond the planner admits
constexpr int kAccRows = 64;
constexpr int kCvtPerThread = 8;  // 2048 elements per tile, as in the planner

__device__ __forceinline__ double2 cz() { return cz64(); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) { return cmul64(a, b); }
__device__ __forceinline__ void cfma(double2& acc, double2 a, double2 b) { cfma64(acc, a, b); }
__device__ __forceinline__ void cfmac(double2& acc, double2 a, double2 b) { cfmac64(acc, a, b); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return cadd64(a, b); }

__device__ __forceinline__ void shfl_from(double2& v, int src) {
  v.x = __shfl_sync(0xffffffffu, v.x, src & 31);
  v.y = __shfl_sync(0xffffffffu, v.y, src & 31);
}
__device__ __forceinline__ void shfl_from(float4& v, int src) {
  v.x = __shfl_sync(0xffffffffu, v.x, src & 31);
  v.y = __shfl_sync(0xffffffffu, v.y, src & 31);
  v.z = __shfl_sync(0xffffffffu, v.z, src & 31);
  v.w = __shfl_sync(0xffffffffu, v.w, src & 31);
}

// ---------------------------------------------------------------------------
// Mode-k product (matvec / matrixTensor).  A slot is (b, j0..j0+3, c): up to
// four outputs that share the input fiber in[b, :, c].  A thread takes NJ of
// a slot's outputs (block (tile, part): outputs j0 + NJ part ..): with NJ = 4
// one input load and four h loads feed four products per a; with NJ = 1 four
// times as many warps run a chain a quarter as long.  Slots run b fastest:
// along higher modes consecutive threads read consecutive input elements
// (coalesced) and share h; along mode 0 (before = 1) they read consecutive
// groups of h's rows and share the input fiber.  Every output is summed in
// the same order whatever NJ is.
// ---------------------------------------------------------------------------
template <class P, int NJ>
__global__ void __launch_bounds__(kThreads) k_mp(const MPTask* __restrict__ tasks,
                                                 const int2* __restrict__ tiles, int64_t tile0) {
  typedef typename P::S S;
  typedef typename P::A A;
  constexpr int U = 4 / NJ;  // steps of a whose loads are in flight together
  const int2 tl = tiles[tile0 + blockIdx.x];
  const MPTask t = tasks[tl.x];
  const S* __restrict__ in = reinterpret_cast<const S*>(t.in);
  const S* __restrict__ h = reinterpret_cast<const S*>(t.h);
  S* out = reinterpret_cast<S*>(t.out);
  const int nq = (t.a_out + 3) / 4;
  const int64_t before = t.before;
  const int64_t slot = (int64_t)tl.y + threadIdx.x;
  if (slot >= before * nq * t.after) return;
  const int64_t b = slot % before;
  const int64_t r = slot / before;
  const int j0 = 4 * (int)(r % nq) + NJ * (int)blockIdx.y;
  const int64_t c = r / nq;
  const int nj = t.a_out - j0 < NJ ? t.a_out - j0 : NJ;
  if (nj <= 0) return;
  const S* ip = in + b + before * t.a_in * c;  // in[b, a, c] = ip[before a]
  const bool unit = t.alpha.x == 1.0 && t.alpha.y == 0.0;
  const typename P::C alpha = P::coef(t.alpha);
  S res[NJ];
  if (t.diag) {
#pragma unroll
    for (int q = 0; q < NJ; ++q) {
      const int j = j0 + (q < nj ? q : 0);
      res[q] = P::mul(P::ld(h + j), P::ld(ip + before * j));
    }
  } else {
    A acc[NJ];
#pragma unroll
    for (int q = 0; q < NJ; ++q) acc[q] = P::zero();
    const S* hp = h + j0;  // h(j, a) = h[j + a_out a]
    const int64_t hs = t.a_out;
    int a = 0;
    for (; a + U <= t.a_in; a += U) {
      S x[U], h0[U][NJ];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        x[u] = P::ld(ip + before * u);
#pragma unroll
        for (int q = 0; q < NJ; ++q) h0[u][q] = P::ld(hp + hs * u + (q < nj ? q : 0));
      }
      ip += before * U;
      hp += hs * U;
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < NJ; ++q) {
          P::mac(acc[q], h0[u][q], x[u]);
          if ((a + u) & 1) P::norm(acc[q]);
        }
    }
    for (; a < t.a_in; ++a) {
      const S x = P::ld(ip);
      S h0[NJ];
#pragma unroll
      for (int q = 0; q < NJ; ++q) h0[q] = P::ld(hp + (q < nj ? q : 0));
      ip += before;
      hp += hs;
#pragma unroll
      for (int q = 0; q < NJ; ++q) {
        P::mac(acc[q], h0[q], x);
        if (a & 1) P::norm(acc[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < NJ; ++q) res[q] = P::fin(acc[q]);
  }
#pragma unroll
  for (int q = 0; q < NJ; ++q)
    if (q < nj) {
      const int64_t o = b + before * ((j0 + q) + (int64_t)t.a_out * c);
      const S v = unit ? res[q] : P::scale(alpha, res[q]);
      out[o] = t.add ? P::plus(out[o], v) : v;
    }
}

// One mode product passed by value (the primitive C ABI calls): one thread
// per output, in memory order, so that the stores and, for before > 1, the
// loads of `in` are coalesced and h is shared by the warp (before == 1: the
// other way round).  Bound: the FP64 pipe.  A complex multiply-add holds a
// sub-partition's FP64 unit for 256 cycles, far longer than its two operand
// loads, so four outputs per thread (as in k_mp) save nothing here and cost
// parallelism: 32 x 32 x 32 along any mode ran in 38.5 us on 32 blocks.
__device__ __forceinline__ void mp_single(const MPTask& t) {
  const int64_t e = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const int64_t before = t.before;
  if (e >= before * t.a_out * t.after) return;
  const int64_t b = e % before, r = e / before;
  const int64_t j = r % t.a_out, c = r / t.a_out;
  const double2* __restrict__ ip = t.in + b + before * t.a_in * c;
  const double2* __restrict__ hp = t.h + j;
  double2 acc = cz();
#pragma unroll 4
  for (int a = 0; a < t.a_in; ++a) cfma(acc, __ldg(hp + (int64_t)t.a_out * a), __ldg(ip + before * a));
  t.out[e] = t.add ? cadd(t.out[e], acc) : acc;
}
__global__ void __launch_bounds__(kThreads) k_mp_single(MPTask t) { mp_single(t); }

// ---------------------------------------------------------------------------
// Hole product (rhomat / contraction) of the primitive C ABI call:
// S(i, j) = sum_k conj(A[k; i]) B[k; j], k = (b, c).  A cluster of CTAs owns
// one output tile of up to 16 x 16 and splits the reduction: every CTA takes
// a contiguous range of k, its `groups` sets of ti x tj threads every
// groups-th row of it, one output per thread.  Rows are staged through
// shared memory 32 at a time (coalesced along b when before > 1, along the
// columns when before == 1).  The partial sums of the groups, then those of
// the CTAs (read through distributed shared memory) are added in a fixed
// order: no workspace, no atomics.  Bound: the FP64 pipe, one complex
// multiply-add per 256 cycles and sub-partition; so one output per thread
// and as many SMs as the shape gives.  64 x 64 outputs over 3712 rows ran in
// 4.4 ms on the four blocks of the former 32 x 32 tiles without a split.
// ---------------------------------------------------------------------------
constexpr int kHcTile = 16;   // outputs of a tile per side
constexpr int kHcRows = 32;   // staged rows
constexpr int kHcMaxCl = 8;   // CTAs of a cluster (portable size)
struct HcGeo {
  int ti, tj, nti, groups, cl;  // tile sides, tiles along i, thread groups, CTAs per tile
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
// all threads of the cluster; orders shared-memory accesses across its CTAs
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}
// element of the same shared-memory variable in CTA `rank` of the cluster
__device__ __forceinline__ double2 ld_cluster(const double2* p, uint32_t rank) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(a), "r"(rank));
  double2 v;
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(ra) : "memory");
  return v;
}

__global__ void __launch_bounds__(kThreads) k_hp_single(HPTask t, HcGeo g) {
  __shared__ double2 sA[kHcRows][kHcTile + 1], sB[kHcRows][kHcTile + 1];
  __shared__ double2 red[kThreads], part[kThreads];
  const int aA = t.a, aB = t.aB > 0 ? t.aB : t.a;
  const uint32_t rank = g.cl > 1 ? cluster_rank() : 0;
  const int tile = (int)(blockIdx.x / g.cl);
  const int i0 = (tile % g.nti) * g.ti, j0 = (tile / g.nti) * g.tj;
  const int mi = min(g.ti, aA - i0), mj = min(g.tj, aB - j0);
  // at most 2^31 rows (the operands have at most 2^31 elements)
  const uint32_t before = (uint32_t)t.before, K = before * (uint32_t)t.after;
  const uint32_t per = (K + g.cl - 1) / g.cl;
  const uint32_t kb = min(K, rank * per), ke = min(K, kb + per);
  const int nout = g.ti * g.tj, grp = threadIdx.x / nout, o = threadIdx.x - grp * nout;
  const int i = o % g.ti, j = o / g.ti;
  const bool active = grp < g.groups;
  double2 acc = cz();
  for (uint32_t k0 = kb; k0 < ke; k0 += kHcRows) {
    for (int e = threadIdx.x; e < 2 * kHcRows * kHcTile; e += kThreads) {
      const bool isA = e < kHcRows * kHcTile;
      const int ee = e & (kHcRows * kHcTile - 1);
      const int kk = before == 1 ? ee / kHcTile : ee % kHcRows;
      const int ii = before == 1 ? ee % kHcTile : ee / kHcRows;
      const uint32_t k = k0 + kk;
      double2 v = cz();
      if (k < ke && ii < (isA ? mi : mj)) {
        const uint32_t c = k / before, b = k - c * before;
        const int64_t col = (isA ? i0 : j0) + ii;
        v = __ldg((isA ? t.A : t.B) + b + (int64_t)before * (col + (int64_t)(isA ? aA : aB) * c));
      }
      (isA ? sA : sB)[kk][ii] = v;
    }
    __syncthreads();
    if (active) {
      const int nk = (int)min((uint32_t)kHcRows, ke - k0);
      for (int kk = grp; kk < nk; kk += g.groups) cfmac(acc, sA[kk][i], sB[kk][j]);
    }
    __syncthreads();
  }
  if (g.groups > 1) {
    red[threadIdx.x] = acc;
    __syncthreads();
    if (grp == 0)
      for (int q = 1; q < g.groups; ++q) acc = cadd(acc, red[q * nout + o]);
  }
  if (g.cl == 1) {
    if (grp == 0 && i < mi && j < mj) t.S[(i0 + i) + (int64_t)aA * (j0 + j)] = acc;
    return;
  }
  if (grp == 0) part[o] = acc;
  cluster_sync();
  for (int e = (int)rank + g.cl * (int)threadIdx.x; e < nout; e += g.cl * kThreads) {
    double2 s = ld_cluster(part + e, 0);
    for (int q = 1; q < g.cl; ++q) s = cadd(s, ld_cluster(part + e, (uint32_t)q));
    const int ie = e % g.ti, je = e / g.ti;
    if (ie < mi && je < mj) t.S[(i0 + ie) + (int64_t)aA * (j0 + je)] = s;
  }
  cluster_sync();  // no CTA leaves while its partial sums are being read
}

// ---------------------------------------------------------------------------
// Hole products of the sweep, split over the reduction index k.  A block owns
// one output tile of up to 64 x 64 and one range of kchunk rows of k; its
// thread (tx, ty) of the TA x TB grid owns the R x C outputs
// {tx + TA r} x {ty + TB c} (R, C in 1..4 chosen per task by the planner so
// that small tiles still occupy most of the 256 threads; one kernel per
// shape, launched once per shape present in a stage).  The operand rows
// move into shared memory 16 at a time with cp.async into two buffers: the
// next rows load while the current ones are consumed, one barrier per 16
// rows.  A task cut into several k ranges writes normalised partial tiles to
// the workspace; k_hp_sum adds them in range order (deterministic).
// ---------------------------------------------------------------------------
constexpr int kHpTile = 64;
constexpr int kHpRows = 16;
constexpr int kHpSmem = 2 * 2 * kHpRows * kHpTile * 16;  // two buffers of A and B rows: 64 KiB

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 16 : 0;  // 0: fill the 16 bytes with zeros, read nothing
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// one block: output tile tl.y, reduction range tl.z of task t
template <class P, int R, int C>
__device__ __forceinline__ void hp_split_tile(const HPTask& t, const int4 tl, typename P::S* __restrict__ ws) {
  typedef typename P::S S;
  typedef typename P::A A;
  extern __shared__ __align__(16) unsigned char hp_smem[];
  S* sm = reinterpret_cast<S*>(hp_smem);  // [buffer][A rows | B rows][kHpRows][kHpTile]
  const int aA = t.a, aB = t.aB > 0 ? t.aB : t.a;
  const int nti = (aA + kHpTile - 1) / kHpTile;
  const int ti0 = (tl.y % nti) * kHpTile, tj0 = (tl.y / nti) * kHpTile;
  const int mA = min(kHpTile, aA - ti0), mB = min(kHpTile, aB - tj0);
  const int TA = (mA + R - 1) / R, TB = (mB + C - 1) / C;
  const int before = t.before;
  const int64_t K = (int64_t)before * t.after;
  const int64_t kb = (int64_t)tl.z * t.kchunk;
  const int64_t ke = min(K, kb + (int64_t)t.kchunk);
  const S* __restrict__ Ap = reinterpret_cast<const S*>(t.A);
  const S* __restrict__ Bp = reinterpret_cast<const S*>(t.B);
  const int64_t sliceA = (int64_t)before * aA, sliceB = (int64_t)before * aB;
  const int tid = threadIdx.x;
  const bool active = tid < TA * TB;
  const int tx = active ? tid % TA : 0, ty = active ? tid / TA : 0;
  const int wA = R * TA, wB = C * TB;  // staged columns (zero beyond the tile; <= 64)
  const int nA = kHpRows * wA, nAB = kHpRows * (wA + wB);
  auto stage = [&](int buf, int64_t k0) {
    S* dA = sm + buf * 2 * kHpRows * kHpTile;
    S* dB = dA + kHpRows * kHpTile;
    for (int e = tid; e < nAB; e += kThreads) {
      const bool isA = e < nA;
      const int ee = isA ? e : e - nA;
      const int w = isA ? wA : wB;
      int kk, ii;
      if (before == 1) {  // consecutive columns are contiguous
        ii = ee % w;
        kk = ee / w;
      } else {  // consecutive rows are contiguous
        kk = ee % kHpRows;
        ii = ee / kHpRows;
      }
      const int64_t k = k0 + kk;
      const bool ok = k < ke && ii < (isA ? mA : mB);
      const S* src = isA ? Ap : Bp;
      if (ok) {
        const int64_t b = k % before, c = k / before;
        src += b + (int64_t)before * ((isA ? ti0 : tj0) + ii) + (isA ? sliceA : sliceB) * c;
      }
      cp_async16((isA ? dA : dB) + kk * kHpTile + ii, src, ok);
    }
    cp_async_commit();
  };
  A acc[R][C];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < C; ++c) acc[r][c] = P::zero();
  const int64_t nchunks = (ke - kb + kHpRows - 1) / kHpRows;
  if (nchunks > 0) stage(0, kb);
  for (int64_t ch = 0; ch < nchunks; ++ch) {
    cp_async_wait<0>();
    // chunk ch has landed, and every thread is done with buffer (ch + 1) & 1
    __syncthreads();
    if (ch + 1 < nchunks) stage((int)((ch + 1) & 1), kb + (ch + 1) * kHpRows);
    if (active) {
      const S* cA = sm + (ch & 1) * 2 * kHpRows * kHpTile;
      const S* cB = cA + kHpRows * kHpTile;
#pragma unroll 2
      for (int kk = 0; kk < kHpRows; ++kk) {
        S a[R], b[C];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = cA[kk * kHpTile + tx + TA * r];
#pragma unroll
        for (int c = 0; c < C; ++c) b[c] = cB[kk * kHpTile + ty + TB * c];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int c = 0; c < C; ++c) P::macc(acc[r][c], a[r], b[c]);
        if (kk & 1) {
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int c = 0; c < C; ++c) P::norm(acc[r][c]);
        }
      }
    }
  }
  if (!active) return;
  S* Sp = reinterpret_cast<S*>(t.S);
  const int64_t nS = (int64_t)aA * aB;
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int i = tx + TA * r, j = ty + TB * c;
      if (i < mA && j < mB) {
        const int64_t o = (ti0 + i) + (int64_t)aA * (tj0 + j);
        if (t.splits <= 1)
          Sp[o] = P::fin(acc[r][c]);
        else
          ws[t.ws + (int64_t)tl.z * nS + o] = P::fin(acc[r][c]);
      }
    }
}

// The register-tile shapes in three classes (hp_class) of about equal registers (rows x
// cols 1 x 1..4; 2 x 3, 2 x 4, 3 x 3; 3 x 4, 4 x 4): a stage's tiles of one
// class share a launch, so that the shapes of uneven bonds run side by side.
// One launch per shape, one after another with about two blocks per SM each,
// took 5.1 ms of a sweep of 64 uneven trees (bonds 6..24), 4.0 together.
template <class P, int CLASS>
__global__ void __launch_bounds__(kThreads, CLASS == 2 ? 2 : 3)
    k_hp(const HPTask* __restrict__ tasks, const int4* __restrict__ tiles, int64_t tile0,
         typename P::S* __restrict__ ws) {
  const int4 tl = tiles[tile0 + blockIdx.x];
  const HPTask t = tasks[tl.x];
  if (CLASS == 0) {
    switch (t.cols) {
      case 1: hp_split_tile<P, 1, 1>(t, tl, ws); break;
      case 2: hp_split_tile<P, 1, 2>(t, tl, ws); break;
      case 3: hp_split_tile<P, 1, 3>(t, tl, ws); break;
      default: hp_split_tile<P, 1, 4>(t, tl, ws);
    }
  } else if (CLASS == 1) {
    if (t.rows == 3) hp_split_tile<P, 3, 3>(t, tl, ws);
    else if (t.cols == 3) hp_split_tile<P, 2, 3>(t, tl, ws);
    else hp_split_tile<P, 2, 4>(t, tl, ws);
  } else {
    if (t.rows == 3) hp_split_tile<P, 3, 4>(t, tl, ws);
    else hp_split_tile<P, 4, 4>(t, tl, ws);
  }
}

// one task passed by value: block b covers output tile b % ntiles, range b / ntiles
template <class P, int R, int C>
__global__ void __launch_bounds__(kThreads, R * C > 9 ? 2 : 3)
    k_hp_one(HPTask t, int ntiles, typename P::S* __restrict__ ws) {
  hp_split_tile<P, R, C>(t, make_int4(0, (int)(blockIdx.x % ntiles), (int)(blockIdx.x / ntiles), 0), ws);
}

template <class P>
__global__ void __launch_bounds__(kThreads) k_hp_sum_one(HPTask t, const typename P::S* __restrict__ ws) {
  typedef typename P::S S;
  typedef typename P::A A;
  const int aB = t.aB > 0 ? t.aB : t.a;
  const int64_t n = (int64_t)t.a * aB;
  S* Sp = reinterpret_cast<S*>(t.S);
  for (int64_t e = (int64_t)blockIdx.x * kThreads + threadIdx.x; e < n; e += (int64_t)gridDim.x * kThreads) {
    A acc = P::zero();
    for (int z = 0; z < t.splits; ++z) P::add(acc, ws[t.ws + z * n + e]);
    Sp[e] = P::fin(acc);
  }
}

// S = sum over the k ranges of the partial tiles, in range order; kHpSumChunks
// blocks of 256 outputs per task (the loads of four ranges in flight).  In
// stages with wide tensor-core products (HPTask::comp) the low words' rounding
// errors are kept too: a hundred ranges, added without, cost the energy of an
// 8-mode tree with bonds 80..112 1e-14 -> 5e-14 of its value, with it 4e-15.
constexpr int kHpSumChunks = 16;
template <class P>
__global__ void __launch_bounds__(kThreads) k_hp_sum(const HPTask* __restrict__ tasks, int64_t task0,
                                                     const typename P::S* __restrict__ ws) {
  typedef typename P::S S;
  typedef typename P::A A;
  const HPTask t = tasks[task0 + blockIdx.x / kHpSumChunks];
  if (t.splits <= 1) return;
  const int aB = t.aB > 0 ? t.aB : t.a;
  const int64_t n = (int64_t)t.a * aB;
  S* Sp = reinterpret_cast<S*>(t.S);
  for (int64_t e = (int64_t)(blockIdx.x % kHpSumChunks) * kThreads + threadIdx.x; e < n;
       e += (int64_t)kHpSumChunks * kThreads) {
    A acc = P::zero();
    if constexpr (std::is_same<P, DF64>::value) {
      if (t.comp) {
        float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int z = 0; z < t.splits; ++z) DF64::add_comp(acc, c, ws[t.ws + z * n + e]);
        acc.y = __fadd_rn(acc.y, c.x);
        acc.w = __fadd_rn(acc.w, c.z);
        Sp[e] = P::fin(acc);
        continue;
      }
    }
#pragma unroll 4
    for (int z = 0; z < t.splits; ++z) P::add(acc, ws[t.ws + z * n + e]);
    Sp[e] = P::fin(acc);
  }
}

// ---------------------------------------------------------------------------
// Last-mode accumulation (multStateAB summed over terms):
//   out[r, j] (+)= alpha * sum_t sum_j' H_t(j, j') X_t[r, j'].
// 64 rows x 16 columns per block; a warp covers 32 consecutive rows (coalesced
// X loads) of 4 columns (H loads broadcast across the warp).
// ---------------------------------------------------------------------------
template <class P>
__global__ void __launch_bounds__(kThreads) k_acc(const AccTask* __restrict__ tasks,
                                                  const AccTerm* __restrict__ terms,
                                                  const int4* __restrict__ tiles, int64_t tile0) {
  typedef typename P::S S;
  typedef typename P::A A;
  const int4 tl = tiles[tile0 + blockIdx.x];
  const AccTask t = tasks[tl.x];
  const int r = tl.y + threadIdx.x % kAccRows;
  const int jb = tl.z + (threadIdx.x / kAccRows) * 4;
  const bool rv = r < t.rows;
  const int d = t.d;
  if (jb >= d) return;  // the whole warp lies past the last column
  const int nq = d - jb < 4 ? d - jb : 4;  // uniform across the warp
  const int64_t rows = t.rows;
  A acc[4] = {P::zero(), P::zero(), P::zero(), P::zero()};
  for (int s = 0; s < t.count; ++s) {
    const AccTerm T = terms[t.first + s];
    const S* X = reinterpret_cast<const S*>(T.X);
    if (T.H == nullptr) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = jb + q;
        if (rv && j < d) P::add(acc[q], P::ld(X + r + rows * j));
      }
    } else {
      const S* H = reinterpret_cast<const S*>(T.H);
      const S* hrow[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) hrow[q] = H + (jb + q < d ? jb + q : 0);
      if (nq == 4) {
        for (int jp = 0; jp < d; ++jp) {
          const S x = rv ? P::ld(X + r + rows * jp) : P::zero();
#pragma unroll
          for (int q = 0; q < 4; ++q) P::mac(acc[q], P::ld(hrow[q] + (int64_t)d * jp), x);
          if (jp & 1) {
#pragma unroll
            for (int q = 0; q < 4; ++q) P::norm(acc[q]);
          }
        }
      } else {
        for (int jp = 0; jp < d; ++jp) {
          const S x = rv ? P::ld(X + r + rows * jp) : P::zero();
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (q < nq) P::mac(acc[q], P::ld(hrow[q] + (int64_t)d * jp), x);
          if (jp & 1) {
#pragma unroll
            for (int q = 0; q < 4; ++q) P::norm(acc[q]);
          }
        }
      }
    }
  }
  const double2 alpha64 = t.alpha_ptr ? *t.alpha_ptr : t.alpha;
  const typename P::C alpha = P::coef(alpha64);
  S* out = reinterpret_cast<S*>(t.out);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int j = jb + q;
    if (rv && j < d) {
      const S v = P::scale(alpha, P::fin(acc[q]));
      S* p = out + r + rows * j;
      *p = t.add ? P::plus(*p, v) : v;
    }
  }
}

// The same with NQ = 1 or 2 of a thread's four columns (block (tile, part)),
// for stages that would leave SMs idle.  A thread sums all terms of a node,
// a chain of count x d steps, and with few warps in flight the loads' latency
// is what a step costs: the steps run in batches of U, the next batch's loads
// (of the next term after a term's last) in flight under the current one's
// multiply-adds.  Every output is summed in the order of k_acc.
template <class P, int NQ>
__global__ void __launch_bounds__(kThreads) k_acc_few(const AccTask* __restrict__ tasks,
                                                      const AccTerm* __restrict__ terms,
                                                      const int4* __restrict__ tiles, int64_t tile0) {
  typedef typename P::S S;
  typedef typename P::A A;
  constexpr int U = 4;
  const int4 tl = tiles[tile0 + blockIdx.x];
  const AccTask t = tasks[tl.x];
  const int r = tl.y + threadIdx.x % kAccRows;
  const int jb = tl.z + (threadIdx.x / kAccRows) * 4 + NQ * (int)blockIdx.y;
  const bool rv = r < t.rows;
  const int d = t.d;
  if (jb >= d) return;  // the whole warp lies past the last column
  const int nq = d - jb < NQ ? d - jb : NQ;  // uniform across the warp
  const int64_t rows = t.rows;
  const int rc = rv ? r : 0;
  A acc[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) acc[q] = P::zero();

  struct Batch {  // steps jp .. of term s; an identity term (H null) is one batch
    S x[U], h[U][NQ];
    int jp;
    bool ident;
  };
  int s = 0, jp = 0;  // the next batch to load
  AccTerm T = {nullptr, nullptr}, Tn = {nullptr, nullptr};
  if (t.count > 0) T = terms[t.first];
  if (t.count > 1) Tn = terms[t.first + 1];
  auto load = [&](Batch& B) {
    const S* X = reinterpret_cast<const S*>(T.X) + rc;
    const S* H = reinterpret_cast<const S*>(T.H);
    B.jp = jp;
    B.ident = H == nullptr;
    if (B.ident) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) B.h[0][q] = P::ld(X + rows * (jb + (q < nq ? q : 0)));
      jp = d;
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = jp + u < d ? jp + u : d - 1;  // past the end: loaded, not used
        B.x[u] = P::ld(X + rows * k);
#pragma unroll
        for (int q = 0; q < NQ; ++q) B.h[u][q] = P::ld(H + (q < nq ? jb + q : 0) + (int64_t)d * k);
      }
      jp += U;
    }
    if (jp >= d) {
      jp = 0;
      ++s;
      T = Tn;
      if (s + 1 < t.count) Tn = terms[t.first + s + 1];
    }
  };
  auto sum = [&](const Batch& B) {
    if (B.ident) {
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (rv && q < nq) P::add(acc[q], B.h[0][q]);
      return;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (B.jp + u >= d) break;
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (q < nq) P::mac(acc[q], B.h[u][q], B.x[u]);
      if ((B.jp + u) & 1) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) P::norm(acc[q]);
      }
    }
  };
  if (t.count > 0) {
    Batch b0, b1;
    load(b0);
    for (;;) {
      const bool more1 = s < t.count;
      if (more1) load(b1);
      sum(b0);
      if (!more1) break;
      const bool more0 = s < t.count;
      if (more0) load(b0);
      sum(b1);
      if (!more0) break;
    }
  }
  const double2 alpha64 = t.alpha_ptr ? *t.alpha_ptr : t.alpha;
  const typename P::C alpha = P::coef(alpha64);
  S* out = reinterpret_cast<S*>(t.out);
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int j = jb + q;
    if (rv && j < d) {
      const S v = P::scale(alpha, P::fin(acc[q]));
      S* p = out + r + rows * j;
      *p = t.add ? P::plus(*p, v) : v;
    }
  }
}

// out = sum_t c_t M_t (d x d), one element per thread; blockIdx.y is the
// block of 256 elements.  A chain of `count` dependent sums per element: with
// one block per matrix (16 elements a thread at d = 64) the ten stages of
// the 64-mode sweep took 390 us, 122 this way.
template <class P>
__global__ void __launch_bounds__(kThreads) k_lin(const LinTask* __restrict__ tasks,
                                                  const LinTerm* __restrict__ terms, int64_t task0) {
  typedef typename P::S S;
  const LinTask t = tasks[task0 + blockIdx.x];
  const int e = (int)blockIdx.y * kThreads + threadIdx.x;
  if (e >= t.d * t.d) return;
  typename P::A acc = P::zero();
#pragma unroll 4
  for (int s = 0; s < t.count; ++s) {
    const LinTerm T = terms[t.first + s];
    P::cmac(acc, P::coef(T.c), P::ld(reinterpret_cast<const S*>(T.M) + e));
    P::norm(acc);
  }
  reinterpret_cast<S*>(t.out)[e] = P::fin(acc);
}

// out(i, j) = sum_t sum_k A_t(i, k) op(B_t)(k, j).  A block owns 8 x 8
// outputs: warp w column 8 bj + w, lane l row 8 bi + (l & 7), lane group
// q = l >> 3 the indices k = q mod 4.  So a chain is a quarter of the terms'
// steps (a node's projected matrix sums all its terms: 150 x 64 steps on the
// 64-mode tree), and the block reads each 128-byte piece of A and B once for
// eight outputs.  A tile of the table (256 outputs) stands for up to kMmBlocks
// blocks; the planner puts the longest sums first.  One output and all four k
// groups per thread, nodes in address order (the longest sums last): 720 us on
// the 64-mode sweep; 405 this way.
constexpr int kMmBlocks = 6;  // >= ceil(d/8)^2 / ceil(d^2/256) for d <= kHpMaxDim
template <class P>
__global__ void __launch_bounds__(kThreads) k_mm(const MMTask* __restrict__ tasks, const MMTerm* __restrict__ terms,
                                                 const int2* __restrict__ tiles, int64_t tile0) {
  typedef typename P::S S;
  const int2 tl = tiles[tile0 + blockIdx.x];
  const MMTask t = tasks[tl.x];
  const int d = t.d, nb = (d + 7) >> 3, blk = (tl.y >> 8) * kMmBlocks + (int)blockIdx.y;
  if (blk >= nb * nb) return;
  const int lane = threadIdx.x & 31, q = lane >> 3;
  const int oi = 8 * (blk % nb) + (lane & 7), oj = 8 * (blk / nb) + (int)(threadIdx.x >> 5);
  if (oj >= d) return;  // the whole warp
  const int i = min(oi, d - 1);
  typename P::A acc = P::zero();
  const int64_t bs = t.trans_b ? d : 1;  // B element (k, j): B[j + d k] or B[k + d j]
  const int64_t sa = 4 * (int64_t)d, sb = 4 * bs;
  for (int s = 0; s < t.count; ++s) {
    const MMTerm T = terms[t.first + s];
    const S* A = reinterpret_cast<const S*>(T.A) + i + (int64_t)d * q;
    const S* B = reinterpret_cast<const S*>(T.B) + (t.trans_b ? oj : (int64_t)d * oj) + bs * q;
    int k = 0;
#pragma unroll 4
    for (; k + 3 < d; k += 4) {
      P::mac(acc, P::ld(A), P::ld(B));
      A += sa;
      B += sb;
      if (k & 4) P::norm(acc);
    }
    if (q == 0)
      for (; k < d; ++k) {
        P::mac(acc, P::ld(A), P::ld(B));
        A += d;
        B += bs;
      }
    P::norm(acc);
  }
  const S f = P::fin(acc);
#pragma unroll
  for (int o = 1; o < 4; ++o) {
    S v = f;
    shfl_from(v, lane + 8 * o);
    if (q == 0) P::add(acc, v);
  }
  if (q == 0 && oi < d) reinterpret_cast<S*>(t.out)[oi + d * oj] = P::fin(acc);
}

// Energy-gradient preparation: M3 = Eout - E rho per node, alpha = 1/S00.
template <class P>
__global__ void __launch_bounds__(kThreads) k_grad(const GradTask* __restrict__ tasks, int64_t task0) {
  typedef typename P::S S;
  const GradTask t = tasks[task0 + blockIdx.x];
  const double E = t.h00->x / t.s00->x;
  const typename P::C mE = P::coef(make_double2(-E, 0.0));
  const S* eout = reinterpret_cast<const S*>(t.eout);
  const S* rho = reinterpret_cast<const S*>(t.rho);
  S* m3 = reinterpret_cast<S*>(t.m3);
  for (int e = threadIdx.x; e < t.d * t.d; e += kThreads) {
    typename P::A acc = eout ? P::ld(eout + e) : P::zero();
    P::cmac(acc, mE, P::ld(rho + e));
    m3[e] = P::fin(acc);
  }
  if (t.write_alpha && threadIdx.x == 0) *t.alpha = make_double2(1.0 / t.s00->x, 0.0);
}

// Precision conversions: dir 0 complex128 -> double-float, dir 1 back.
__global__ void __launch_bounds__(kThreads) k_cvt(const CvtTask* __restrict__ tasks,
                                                  const int2* __restrict__ tiles, int64_t tile0) {
  const int2 tl = tiles[tile0 + blockIdx.x];
  const CvtTask t = tasks[tl.x];
  // all loads of the thread first (eight 16-byte loads in flight), then convert
  if (t.dir == 0) {
    double2 v[kCvtPerThread];
#pragma unroll
    for (int q = 0; q < kCvtPerThread; ++q) {
      const int64_t i = tl.y + threadIdx.x + (int64_t)q * kThreads;
      v[q] = i < t.n ? __ldg(reinterpret_cast<const double2*>(t.src) + i) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int q = 0; q < kCvtPerThread; ++q) {
      const int64_t i = tl.y + threadIdx.x + (int64_t)q * kThreads;
      if (i < t.n) {
        const float2 r = df_split(v[q].x), m = df_split(v[q].y);
        reinterpret_cast<float4*>(t.dst)[i] = make_float4(r.x, r.y, m.x, m.y);
      }
    }
  } else {
    float4 w[kCvtPerThread];
#pragma unroll
    for (int q = 0; q < kCvtPerThread; ++q) {
      const int64_t i = tl.y + threadIdx.x + (int64_t)q * kThreads;
      w[q] = i < t.n ? __ldg(reinterpret_cast<const float4*>(t.src) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < kCvtPerThread; ++q) {
      const int64_t i = tl.y + threadIdx.x + (int64_t)q * kThreads;
      if (i < t.n)
        reinterpret_cast<double2*>(t.dst)[i] =
            make_double2((double)w[q].x + (double)w[q].y, (double)w[q].z + (double)w[q].w);
    }
  }
}

// ---------------------------------------------------------------------------
// Inverse of a Hermitian positive definite d x d matrix by the symmetric sweep
// operator, in place: A (shared memory, column-major, lower triangle) becomes
// -A^-1 (lower triangle).  Step k takes column c of the current matrix and
// p = 1 / c_k: A_ij -= c_i conj(c_j) p, A_ik = c_i p, A_kk = -p.  The pivots
// are those of the Cholesky factorisation; the first that is not positive
// ends the sweep (false, uniform over the block, A void).  d^3 / 2 complex
// multiply-adds (Gauss-Jordan on [A | I] without the symmetry: 2 d^3) and one
// barrier per step: the threads that update column k + 1 also write it to
// the other column buffer.  256 threads as 16 x 16 (i, j); c: 2 d elements.
// Bound: FP64 issue for d >= 32 (complex128), the barrier and the pivot's
// reciprocal below.
// ---------------------------------------------------------------------------
template <class P>
__device__ bool herm_sweep_inverse(typename P::S* A, int d, typename P::S* c) {
  typedef typename P::S S;
  __shared__ typename P::R pr[2];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int i = threadIdx.x; i < d; i += kThreads) c[i] = A[i];
  if (threadIdx.x == 0) pr[0] = P::rrecip(A[0]);
  for (int k = 0; k < d; ++k) {
    __syncthreads();
    const S* cur = c + (k & 1) * d;
    S* nxt = c + ((k + 1) & 1) * d;
    if (!P::positive(cur[k])) return false;
    const typename P::R p = pr[k & 1];
    if (k + 1 < d && tx == ((k + 1) & 15) && ty == tx) {
      // the owner of the next pivot first: its reciprocal runs under the others' updates
      typename P::A a = A[k + 1 + d * (k + 1)];
      P::mac(a, cur[k + 1], P::neg(P::conj_scale(cur[k + 1], p)));
      pr[(k + 1) & 1] = P::rrecip(P::fin(a));
    }
    for (int j = ty; j < d; j += 16) {
      const S cj = cur[j];
      const S w = P::conj_scale(cj, p);
      const S nw = P::neg(w);
      const int i0 = j - ((j - tx) & 15);  // the thread's rows i >= j: first multiple step at or above j
      for (int i = i0 < j ? i0 + 16 : i0; i < d; i += 16) {
        S v;
        if (j == k) {
          v = i == k ? P::neg(P::real(p)) : P::conj(P::conj_scale(cur[i], p));
        } else if (i == k) {
          v = w;
        } else {
          typename P::A a = A[i + d * j];
          P::mac(a, cur[i], nw);
          v = P::fin(a);
        }
        A[i + d * j] = v;
        if (j == k + 1) nxt[i] = v;
        else if (i == k + 1) nxt[j] = P::conj(v);
      }
    }
  }
  __syncthreads();
  return true;
}

// ---------------------------------------------------------------------------
// Regularised inverse of a Hermitian matrix (SpectralDecompositionTree::
// calculate + invert): parallel cyclic Jacobi with a round-robin pairing
// (every round rotates d/2 disjoint index pairs at once), then
//   rhoinv = U diag(1 / (w + eps*exp(-w/eps))) U^dagger.
// One block per matrix; A lives in shared memory, U in global scratch.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void rr_pair(int m, int r, int i, int& p, int& q) {
  // circle method over m (even) indices, round r in [0, m-1), pair i in [0, m/2)
  if (i == 0) {
    p = r;
    q = m - 1;
  } else {
    p = (r + i) % (m - 1);
    q = (r - i + (m - 1)) % (m - 1);
  }
  if (p > q) {
    int x = p;
    p = q;
    q = x;
  }
}

// Cyclic Jacobi on the Hermitian d x d matrix A (shared memory): A becomes
// diagonal (the eigenvalues), U (global) the eigenvectors, A_in = U A U^dagger.
// Scratch: rot / ph (np each), pq (2 np), red_off / red_diag (kThreads each).
__device__ void herm_jacobi(double2* A, double2* U, int d, double2* rot, double2* ph, int* pq,
                            double* red_off, double* red_diag) {
  const int m = d + (d & 1);
  const int np = m / 2;
  for (int e = threadIdx.x; e < d * d; e += kThreads) U[e] = make_double2((e % d) == (e / d) ? 1.0 : 0.0, 0.0);
  __syncthreads();
  for (int sweep = 0; sweep < 40; ++sweep) {
    double off = 0.0, dg = 0.0;
    for (int e = threadIdx.x; e < d * d; e += kThreads) {
      const double v = A[e].x * A[e].x + A[e].y * A[e].y;
      if (e % d == e / d)
        dg += v;
      else
        off += v;
    }
    red_off[threadIdx.x] = off;
    red_diag[threadIdx.x] = dg;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) {
        red_off[threadIdx.x] += red_off[threadIdx.x + s];
        red_diag[threadIdx.x] += red_diag[threadIdx.x + s];
      }
      __syncthreads();
    }
    const double toff = red_off[0], tdiag = red_diag[0];
    __syncthreads();
    if (!(toff > 1e-30 * tdiag) || toff == 0.0) break;
    for (int r = 0; r < m - 1; ++r) {
      for (int i = threadIdx.x; i < np; i += kThreads) {
        int p, q;
        rr_pair(m, r, i, p, q);
        double c = 1.0, s = 0.0;
        double2 e = make_double2(1.0, 0.0);
        if (q < d) {
          const double2 apq = A[p + d * q];
          const double ab = hypot(apq.x, apq.y);
          if (ab > 0.0) {
            e = make_double2(apq.x / ab, apq.y / ab);
            const double theta = 0.5 * atan2(2.0 * ab, A[q + d * q].x - A[p + d * p].x);
            c = cos(theta);
            s = sin(theta);
          }
        }
        rot[i] = make_double2(c, s);
        ph[i] = e;
        pq[2 * i] = p;
        pq[2 * i + 1] = q;
      }
      __syncthreads();
      // columns: A <- A G, U <- U G
      for (int idx = threadIdx.x; idx < np * d; idx += kThreads) {
        const int i = idx / d, k = idx % d;
        const int p = pq[2 * i], q = pq[2 * i + 1];
        if (q >= d || rot[i].y == 0.0) continue;
        const double c = rot[i].x, s = rot[i].y;
        const double2 e = ph[i];
        const double2 se = make_double2(s * e.x, s * e.y);    // s*e
        const double2 sce = make_double2(s * e.x, -s * e.y);  // s*conj(e)
        double2 akp = A[k + d * p], akq = A[k + d * q];
        double2 np_ = make_double2(c * akp.x, c * akp.y);
        double2 t2 = cmul(sce, akq);
        np_.x -= t2.x;
        np_.y -= t2.y;
        double2 nq = cmul(se, akp);
        nq.x += c * akq.x;
        nq.y += c * akq.y;
        A[k + d * p] = np_;
        A[k + d * q] = nq;
        double2 ukp = U[k + (int64_t)d * p], ukq = U[k + (int64_t)d * q];
        np_ = make_double2(c * ukp.x, c * ukp.y);
        t2 = cmul(sce, ukq);
        np_.x -= t2.x;
        np_.y -= t2.y;
        nq = cmul(se, ukp);
        nq.x += c * ukq.x;
        nq.y += c * ukq.y;
        U[k + (int64_t)d * p] = np_;
        U[k + (int64_t)d * q] = nq;
      }
      __syncthreads();
      // rows: A <- G^dagger A
      for (int idx = threadIdx.x; idx < np * d; idx += kThreads) {
        const int i = idx / d, k = idx % d;
        const int p = pq[2 * i], q = pq[2 * i + 1];
        if (q >= d || rot[i].y == 0.0) continue;
        const double c = rot[i].x, s = rot[i].y;
        const double2 e = ph[i];
        const double2 se = make_double2(s * e.x, s * e.y);
        const double2 sce = make_double2(s * e.x, -s * e.y);
        const double2 apk = A[p + d * k], aqk = A[q + d * k];
        double2 np_ = make_double2(c * apk.x, c * apk.y);
        double2 t2 = cmul(se, aqk);
        np_.x -= t2.x;
        np_.y -= t2.y;
        double2 nq = cmul(sce, apk);
        nq.x += c * aqk.x;
        nq.y += c * aqk.y;
        A[p + d * k] = np_;
        A[q + d * k] = nq;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < np; i += kThreads) {
        const int p = pq[2 * i], q = pq[2 * i + 1];
        if (q < d && rot[i].y != 0.0) {
          A[p + d * q] = cz();
          A[q + d * p] = cz();
        }
      }
      __syncthreads();
    }
  }
}

// Whether the Hermitian matrix with lower triangle U (global memory,
// overwritten) has a Cholesky factorisation; uniform over the block.
__device__ bool cholesky_succeeds(double2* U, int d) {
  for (int k = 0; k < d; ++k) {
    const double dk = U[k + (int64_t)d * k].x;
    if (!(dk > 0.0)) return false;
    const double l = sqrt(dk);
    __syncthreads();
    for (int i = k + threadIdx.x; i < d; i += kThreads) {
      const double2 v = U[i + (int64_t)d * k];
      U[i + (int64_t)d * k] = make_double2(v.x / l, v.y / l);
    }
    __syncthreads();
    // trailing update of the lower triangle: U(i,j) -= L(i,k) conj(L(j,k))
    const int rem = d - k - 1;
    for (int e = threadIdx.x; e < rem * rem; e += kThreads) {
      const int i = k + 1 + e % rem, j = k + 1 + e / rem;
      if (j > i) continue;
      const double2 li = U[i + (int64_t)d * k], lj = U[j + (int64_t)d * k];
      double2 u = U[i + (int64_t)d * j];
      cfma(u, make_double2(-li.x, -li.y), make_double2(lj.x, -lj.y));
      U[i + (int64_t)d * j] = u;
    }
    __syncthreads();
  }
  return true;
}

__device__ __forceinline__ void eig_body(const EigTask& t, double eps) {
  extern __shared__ double2 smem[];
  const int d = t.d;
  const int m = d + (d & 1);
  const int np = m / 2;
  double2* A = smem;                      // d*d
  double2* rot = A + (int64_t)d * d;      // np entries: (c, s)
  double2* ph = rot + np;                 // np entries: e
  double2* fw = ph + np;                  // m entries: f(eigenvalue) in .x
  int* pq = (int*)(fw + m);               // 2*np
  __shared__ double red_off[kThreads], red_diag[kThreads];
  double2* U = t.U;
  auto load = [&](double2* dst) {  // the Hermitian part
    for (int e = threadIdx.x; e < d * d; e += kThreads) {
      const int i = e % d, j = e / d;
      const double2 aij = t.rho[i + (int64_t)d * j], aji = t.rho[j + (int64_t)d * i];
      dst[e] = (i == j) ? make_double2(aij.x, 0.0)
                        : make_double2(0.5 * (aij.x + aji.x), 0.5 * (aij.y - aji.y));
    }
    __syncthreads();
  };
  load(A);
  // If every eigenvalue w exceeds 40 eps, eps*exp(-w/eps) changes 1/w by less
  // than 2e-19 relative and the regularised inverse is the plain inverse.  Two
  // certificates, the second only where the first leaves the question open:
  //  * |rho^-1|_F <= 1 / (40 eps), since w >= 1 / |rho^-1|_F;
  //  * a Cholesky factorisation of rho - 100 eps I (backward error about
  //    d 2^-53 |rho|, far below 50 eps for eps = 1e-10 and normalised states).
  //    With |rho^-1|_F > sqrt(d) / (100 eps) some w is below 100 eps: it would
  //    fail (rank-deficient densities, which need the eigenvalues anyway).
  __shared__ double2 col_s[2 * kHpMaxDim];
  if (herm_sweep_inverse<F64>(A, d, col_s)) {
    double n2 = 0.0;
    for (int e = threadIdx.x; e < d * d; e += kThreads) {
      const int i = e % d, j = e / d;
      if (i < j) continue;
      const double2 x = A[e];
      n2 += (i == j ? 1.0 : 2.0) * (x.x * x.x + x.y * x.y);
    }
    red_off[threadIdx.x] = n2;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) red_off[threadIdx.x] += red_off[threadIdx.x + s];
      __syncthreads();
    }
    const double lim = 1.0 / (40.0 * eps), open = 1.0 / (100.0 * eps);
    bool plain = red_off[0] <= lim * lim;
    if (!plain && red_off[0] <= d * (open * open)) {
      load(U);
      for (int i = threadIdx.x; i < d; i += kThreads) U[i + (int64_t)d * i].x -= 100.0 * eps;
      __syncthreads();
      plain = cholesky_succeeds(U, d);
    }
    if (plain) {
      for (int e = threadIdx.x; e < d * d; e += kThreads) {
        const int i = e % d, j = e / d;
        const double2 x = i >= j ? A[e] : A[j + d * i];
        t.rhoinv[e] = i == j ? make_double2(-x.x, 0.0) : make_double2(-x.x, i > j ? -x.y : x.y);
      }
      return;
    }
  }
  __syncthreads();
  load(A);
  herm_jacobi(A, U, d, rot, ph, pq, red_off, red_diag);
  for (int i = threadIdx.x; i < d; i += kThreads) {
    const double w = A[i + d * i].x;
    fw[i].x = 1.0 / (w + eps * exp(-w / eps));
  }
  __syncthreads();
  for (int e = threadIdx.x; e < d * d; e += kThreads) {
    const int i = e % d, j = e / d;
    double2 acc = cz();
    for (int k = 0; k < d; ++k) {
      const double2 uik = U[i + (int64_t)d * k];
      const double2 ujk = U[j + (int64_t)d * k];
      const double f = fw[k].x;
      // acc += uik * f * conj(ujk)
      cfma(acc, make_double2(uik.x * f, uik.y * f), make_double2(ujk.x, -ujk.y));
    }
    t.rhoinv[e] = acc;
  }
}

__global__ void __launch_bounds__(kThreads) k_eig(const EigTask* __restrict__ tasks, int64_t task0,
                                                  double eps) {
  const EigTask t = tasks[task0 + blockIdx.x];
  eig_body(t, eps);
}

// ---------------------------------------------------------------------------
// Projector pieces of LayerDerivative (projectOut + rho^-1), per node, in the
// arithmetic of the plan:
//   X  = S^-1
//   P  = X D
//   M2 = -(rhoinv P^T)
// so that the derivative is dPsi = alpha ((H Phi) rhoinv^T + Phi M2^T).
// S = Phi^dagger Phi is Hermitian positive definite: X comes from the sweep
// operator; a pivot that is not positive (linearly dependent columns) sends
// the node to Gauss-Jordan with partial pivoting.  Row m of P gives column m
// of M2, so the blocks (node, part) of a node share the rows of P: each
// inverts S itself (no exchange) and takes every parts-th row.
// ---------------------------------------------------------------------------
// X = S^-1 by Gauss-Jordan with partial pivoting (warp-parallel pivot
// search); W (d x d) is scratch
template <class P>
__device__ void pivoted_inverse(const typename P::S* Sin, typename P::S* W, typename P::S* X, int d) {
  typedef typename P::S S;
  typedef typename P::A A;
  __shared__ S fcol[kHpMaxDim];
  __shared__ int piv;
  __shared__ S pinv;
  for (int e = threadIdx.x; e < d * d; e += kThreads) {
    W[e] = Sin[e];
    S z = P::zero();
    if ((e % d) == (e / d)) z = P::coef(make_double2(1.0, 0.0));
    X[e] = z;
  }
  __syncthreads();
  for (int col = 0; col < d; ++col) {
    if (threadIdx.x < 32) {  // pivot: largest |S(r, col)|, r >= col
      double bv = -1.0;
      int best = col;
      for (int r = col + threadIdx.x; r < d; r += 32) {
        const double m = P::mag2(W[r + d * col]);
        if (m > bv) bv = m, best = r;
      }
      for (int off = 16; off > 0; off >>= 1) {
        const double ov = __shfl_down_sync(0xffffffffu, bv, off);
        const int ob = __shfl_down_sync(0xffffffffu, best, off);
        if (ov > bv || (ov == bv && ob < best)) bv = ov, best = ob;
      }
      if (threadIdx.x == 0) piv = best;
    }
    __syncthreads();
    const int pr = piv;
    if (pr != col) {
      for (int j = threadIdx.x; j < d; j += kThreads) {
        S x = W[col + d * j];
        W[col + d * j] = W[pr + d * j];
        W[pr + d * j] = x;
        x = X[col + d * j];
        X[col + d * j] = X[pr + d * j];
        X[pr + d * j] = x;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) pinv = P::recip(W[col + d * col]);
    __syncthreads();
    const S pv = pinv;
    for (int j = threadIdx.x; j < d; j += kThreads) {
      W[col + d * j] = P::mul(W[col + d * j], pv);
      X[col + d * j] = P::mul(X[col + d * j], pv);
    }
    __syncthreads();
    for (int r = threadIdx.x; r < d; r += kThreads) fcol[r] = P::neg(W[r + d * col]);
    __syncthreads();
    for (int e = threadIdx.x; e < d * d; e += kThreads) {
      const int r = e % d, j = e / d;
      if (r == col) continue;
      const S f = fcol[r];
      if (j > col) {
        A w = W[e];
        P::mac(w, f, W[col + d * j]);
        W[e] = P::fin(w);
      }
      A x = X[e];
      P::mac(x, f, X[col + d * j]);
      X[e] = P::fin(x);
    }
    __syncthreads();
  }
}

template <class P>
__global__ void __launch_bounds__(kThreads) k_proj(const ProjTask* __restrict__ tasks, int64_t task0) {
  typedef typename P::S S;
  typedef typename P::A A;
  extern __shared__ __align__(16) unsigned char proj_smem[];
  const ProjTask t = tasks[task0 + blockIdx.x];
  const int d = t.d;
  S* X = reinterpret_cast<S*>(proj_smem);
  __shared__ __align__(16) unsigned char col_raw[2 * kHpMaxDim * sizeof(S)];
  const S* Sin = reinterpret_cast<const S*>(t.S);
  S* Pm = reinterpret_cast<S*>(t.P);
  int part = blockIdx.y, parts = gridDim.y;
  for (int e = threadIdx.x; e < d * d; e += kThreads) X[e] = Sin[e];
  __syncthreads();
  if (herm_sweep_inverse<P>(X, d, reinterpret_cast<S*>(col_raw))) {
    for (int e = threadIdx.x; e < d * d; e += kThreads) {  // X = -(lower triangle), mirrored
      const int i = e % d, j = e / d;
      if (i < j) continue;
      const S x = P::neg(X[e]);
      X[e] = x;
      if (i > j) X[j + d * i] = P::conj(x);
    }
  } else {
    if (part > 0) return;  // one block of the node (the outcome is the same in all): the scratch is the node's
    parts = 1;
    S* W = Pm;
    S* Xg = reinterpret_cast<S*>(t.Sinv);
    __syncthreads();
    pivoted_inverse<P>(Sin, W, Xg, d);
    for (int e = threadIdx.x; e < d * d; e += kThreads) X[e] = Xg[e];
  }
  __syncthreads();
  // this block's rows of P = X D: rows part, part + parts, ...
  const S* __restrict__ D = reinterpret_cast<const S*>(t.D);
  const int mine = (d - part + parts - 1) / parts;
  for (int e = threadIdx.x; e < mine * d; e += kThreads) {
    const int i = part + parts * (e % mine), j = e / mine;
    A acc = P::zero();
#pragma unroll 4
    for (int k = 0; k < d; ++k) {
      P::mac(acc, X[i + d * k], P::ld(D + k + d * j));
      if (k & 1) P::norm(acc);
    }
    Pm[i + d * j] = P::fin(acc);
  }
  __syncthreads();
  // M2 = -rhoinv P^T, the columns m that these rows give
  const S* __restrict__ Ri = reinterpret_cast<const S*>(t.rhoinv);
  S* M2 = reinterpret_cast<S*>(t.M2);
  for (int e = threadIdx.x; e < mine * d; e += kThreads) {
    const int j = e % d, m = part + parts * (e / d);
    A acc = P::zero();
#pragma unroll 4
    for (int k = 0; k < d; ++k) {
      P::mac(acc, P::ld(Ri + j + d * k), Pm[m + d * k]);
      if (k & 1) P::norm(acc);
    }
    M2[j + d * m] = P::neg(P::fin(acc));
  }
}

__global__ void k_identity(double2* m, int d, int prec) {
  for (int e = threadIdx.x; e < d * d; e += blockDim.x) {
    const bool diag = (e % d) == (e / d);
    if (prec >= 1)
      reinterpret_cast<float4*>(m)[e] = make_float4(diag ? 1.f : 0.f, 0.f, 0.f, 0.f);
    else
      m[e] = make_double2(diag ? 1.0 : 0.0, 0.0);
  }
}

// Eight independent FMA chains per thread; one store per thread keeps the
// chains live.  Every store index is < gridDim.x * blockDim.x.
__global__ void __launch_bounds__(kThreads) k_fp64_fma(double* out, int iters, double a, double b) {
  double acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = threadIdx.x + i;
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = fma(acc[i], a, b);
  }
  double s = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) s += acc[i];
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

// The double-float complex multiply-add of the chain kernels (DF64::mac,
// renormalised every second step) on eight register accumulators per thread:
// the ceiling of double-float arithmetic on this GPU, no memory traffic.
// Every product reads another accumulator (acc[i] += a * acc[i ^ 4]), so
// nothing is loop-invariant; |a| = 1e-3 keeps the values finite.  One store
// per thread, index < gridDim.x * blockDim.x.
__global__ void __launch_bounds__(kThreads) k_df64_mac(float4* out, int iters, float4 a, float4 b) {
  float4 acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = make_float4(threadIdx.x + i, 0.f, b.x * i, 0.f);
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      DF64::mac(acc[i], a, acc[i ^ 4]);
      if (it & 1) DF64::norm(acc[i]);
    }
  }
  float4 s = acc[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) s = DF64::plus(s, acc[i]);
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

inline int64_t eig_smem_bytes(int d) {
  const int m = d + (d & 1);
  const int np = m / 2;
  return 16 * ((int64_t)d * d + 2 * np + m) + 8 * (int64_t)np + 16;
}

__global__ void __launch_bounds__(kThreads) k_axpy(double2* out, const double2* x, double2 a,
                                                   const double2* y, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
    double2 v = x[i];
    cfma(v, a, y[i]);
    out[i] = v;
  }
}
}  // namespace

// ---------------------------------------------------------------------------
// Krylov vector helpers of the SCF sweep (complex128).
// k_dot: out = sum_i conj(a_i) b_i in one block; every thread sums a fixed
// strided subset in order, then a fixed-order tree in shared memory, so the
// result is reproducible run to run.
// k_lincomb: out_i = sum_t c_t v_t,i over up to kLinCombMax vectors.
// ---------------------------------------------------------------------------
constexpr int kDotThreads = 512;
constexpr int64_t kDotParts = 256;

__global__ void __launch_bounds__(kDotThreads) k_dot(const double2* __restrict__ a,
                                                     const double2* __restrict__ b, int64_t n,
                                                     double2* __restrict__ out) {
  __shared__ double2 red[kDotThreads];
  double2 acc = cz();
  for (int64_t i = threadIdx.x; i < n; i += kDotThreads) {
    if (b)
      cfmac(acc, a[i], b[i]);
    else
      acc = cadd(acc, a[i]);
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = kDotThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] = cadd(red[threadIdx.x], red[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0];
}

__global__ void __launch_bounds__(kThreads) k_lincomb(double2* __restrict__ out, LinComb lc, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
    double2 acc = cz();
    for (int t = 0; t < lc.count; ++t) cfma(acc, lc.c[t], lc.v[t][i]);
    out[i] = acc;
  }
}

// first pass: block b sums its contiguous slice in a fixed order
__global__ void __launch_bounds__(kDotThreads) k_dot_part(const double2* __restrict__ a,
                                                          const double2* __restrict__ b, int64_t n,
                                                          int64_t slice, double2* __restrict__ part) {
  __shared__ double2 red[kDotThreads];
  const int64_t lo = (int64_t)blockIdx.x * slice, hi = min(n, lo + slice);
  double2 acc = cz();
  for (int64_t i = lo + threadIdx.x; i < hi; i += kDotThreads) cfmac(acc, a[i], b[i]);
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = kDotThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] = cadd(red[threadIdx.x], red[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// complex128 <-> double-float copy of n elements (dir 0: to double-float)
__global__ void __launch_bounds__(kThreads) k_convert(void* __restrict__ dst, const void* __restrict__ src,
                                                      int64_t n, int dir) {
  for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
    if (dir == 0) {
      const double2 v = reinterpret_cast<const double2*>(src)[i];
      const float2 r = df_split(v.x), m = df_split(v.y);
      reinterpret_cast<float4*>(dst)[i] = make_float4(r.x, r.y, m.x, m.y);
    } else {
      const float4 v = reinterpret_cast<const float4*>(src)[i];
      reinterpret_cast<double2*>(dst)[i] = make_double2((double)v.x + (double)v.y, (double)v.z + (double)v.w);
    }
  }
}

// One step of the Lanczos recursion of the SCF driver, its scalars on the
// device: l < 0 starts it (V_0 = psi / |psi|), l >= 0 takes h = H V_l
// (LanczosStep::kout, in the plan's arithmetic) and forms
//   al_l = Re <V_l, h>,  w = h - al_l V_l - be_{l-1} V_{l-1},  be_l = |w|,
//   V_{l+1} = w / be_l,
// the last step (l + 1 == size) only al_l.  The new vector also goes to the
// effective Hamiltonian's input kin.  A residual below `breakdown` times the
// largest |al|, be ends the space (res[kLzStop] = l + 1; later steps return at
// once).  A cluster of up to eight CTAs; every dot product is summed as
// k_dot_part and k_dot do it (slices of 8192 or more by 512 threads and a
// tree, then a tree over the slices), slices shared out over the CTAs, the
// partial sums read through distributed shared memory.  One launch in place
// of eight with two waits of the host between them; per step 80 us of an
// 8-mode tree's ~110 went there.  The host learns of the end through
// host_stop and queues no further products.
__device__ __forceinline__ double ld_cluster_d(const double* p, uint32_t rank) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(a), "r"(rank));
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];\n" : "=d"(v) : "r"(ra) : "memory");
  return v;
}
__device__ __forceinline__ double lz_tree(double v, double* red) {
  // the tree of k_dot; its last five levels within the first warp
  red[threadIdx.x] = v;
  __syncthreads();
  for (int w = kDotThreads / 2; w >= 32; w >>= 1) {
    if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < 32) {
    double r = red[threadIdx.x];
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) r += __shfl_down_sync(0xffffffffu, r, w);
    if (threadIdx.x == 0) red[0] = r;
  }
  __syncthreads();
  const double r = red[0];
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kDotThreads) k_lanczos(LanczosStep t, int cl) {
  __shared__ double red[kDotThreads];
  __shared__ double part[2][kDotParts];
  if (t.l >= 0 && t.res[kLzStop] != 0.0) return;  // the same in every CTA
  const int rank = cl > 1 ? (int)cluster_rank() : 0;
  // the sum over all slices of each thread's running products (sum(i)), in two stages
  auto dot = [&](int which, auto sum) {
    for (int p = rank; p < t.parts; p += cl) {
      const int64_t lo = p * t.slice, hi = min(t.n, lo + t.slice);
      double acc = 0.0;
      for (int64_t i = lo + threadIdx.x; i < hi; i += kDotThreads) sum(i, acc);
      const double v = lz_tree(acc, red);
      if (t.parts == 1) return v;  // (one CTA)
      if (threadIdx.x == 0) part[which][p / cl] = v;
    }
    if (cl > 1) cluster_sync();
    else __syncthreads();
    const int p = threadIdx.x;
    double v = 0.0;
    if (p < t.parts) v = cl > 1 ? ld_cluster_d(&part[which][p / cl], (uint32_t)(p % cl)) : part[which][p];
    return lz_tree(v, red);
  };
  auto each = [&](auto f) {
    for (int p = rank; p < t.parts; p += cl) {
      const int64_t lo = p * t.slice, hi = min(t.n, lo + t.slice);
      for (int64_t i = lo + threadIdx.x; i < hi; i += kDotThreads) f(i);
    }
  };
  auto emit = [&](int64_t i, double2 v) {  // the new Krylov vector, also as the input of the next product
    t.next[i] = v;
    if (t.df) {
      const float2 r = df_split(v.x), m = df_split(v.y);
      reinterpret_cast<float4*>(t.kin)[i] = make_float4(r.x, r.y, m.x, m.y);
    } else {
      reinterpret_cast<double2*>(t.kin)[i] = v;
    }
  };
  auto add2 = [](double& acc, double2 a, double2 b) { acc = fma(a.y, b.y, fma(a.x, b.x, acc)); };
  const bool writer = rank == 0 && threadIdx.x == 0;
  if (t.l < 0) {
    const double s = dot(0, [&](int64_t i, double& acc) { add2(acc, t.v[i], t.v[i]); });
    const double c = 1.0 / sqrt(s);
    each([&](int64_t i) { emit(i, make_double2(c * t.v[i].x, c * t.v[i].y)); });
    if (writer) {
      t.res[kLzStop] = 0.0;
      t.res[kLzNorm2] = s;
    }
  } else {
    const double al = dot(0, [&](int64_t i, double& acc) {
      double2 h;
      if (t.df) {
        const float4 f = reinterpret_cast<const float4*>(t.kout)[i];
        h = make_double2((double)f.x + (double)f.y, (double)f.z + (double)f.w);
      } else {
        h = reinterpret_cast<const double2*>(t.kout)[i];
      }
      t.w[i] = h;
      add2(acc, t.v[i], h);
    });
    if (writer) t.res[t.l] = al;
    if (!t.last) {
      const double be = t.prev ? t.res[kLzBeta + t.l - 1] : 0.0;
      const double s = dot(1, [&](int64_t i, double& acc) {
        double2 w = t.w[i];
        const double2 v = t.v[i];
        w.x = fma(-al, v.x, w.x);
        w.y = fma(-al, v.y, w.y);
        if (t.prev) {
          const double2 u = t.prev[i];
          w.x = fma(-be, u.x, w.x);
          w.y = fma(-be, u.y, w.y);
        }
        t.w[i] = w;
        add2(acc, w, w);
      });
      const double nrm = sqrt(fmax(s, 0.0));
      double scale = fabs(al);
      for (int q = 0; q < t.l; ++q) scale = fmax(scale, fmax(fabs(t.res[q]), t.res[kLzBeta + q]));
      const bool stop = nrm <= t.breakdown * scale;
      if (writer) {
        t.res[kLzBeta + t.l] = s == s ? nrm : s;  // fmax drops a NaN
        if (stop) {
          t.res[kLzStop] = t.l + 1;
          *t.host_stop = 1;
        }
      }
      if (!stop) {
        const double c = 1.0 / nrm;
        each([&](int64_t i) { emit(i, make_double2(c * t.w[i].x, c * t.w[i].y)); });
      }
    }
  }
  if (cl > 1) cluster_sync();  // no CTA leaves while its partial sums are being read
}

cudaError_t launch_lanczos(const LanczosStep& step, cudaStream_t s) {
  LanczosStep t = step;
  // the slices of launch_dot
  int64_t parts = std::min<int64_t>(kDotParts, std::max<int64_t>(1, (t.n + 8191) / 8192));
  t.slice = (t.n + parts - 1) / parts;
  t.parts = (int)std::max<int64_t>(1, (t.n + t.slice - 1) / t.slice);
  int cl = 1;
  while (cl < 8 && cl < t.parts) cl *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cl);
  cfg.blockDim = dim3(kDotThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)cl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_lanczos, t, cl);
}

cudaError_t launch_convert(void* dst, const void* src, int64_t n, int dir, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int blocks = (int)std::min<int64_t>((n + kThreads - 1) / kThreads, 152 * 8);
  k_convert<<<blocks, kThreads, 0, s>>>(dst, src, n, dir);
  return cudaGetLastError();
}

cudaError_t launch_dot(const double2* a, const double2* b, int64_t n, double2* out, cudaStream_t s) {
  // slices of >= 8192 elements, at most kDotParts of them; the partial sums
  // go to out[1 ..] and are added in order by one block into out[0]
  int64_t parts = std::min<int64_t>(kDotParts, std::max<int64_t>(1, (n + 8191) / 8192));
  const int64_t slice = (n + parts - 1) / parts;
  parts = std::max<int64_t>(1, (n + slice - 1) / slice);
  k_dot_part<<<(unsigned)parts, kDotThreads, 0, s>>>(a, b, n, slice, out + 1);
  k_dot<<<1, kDotThreads, 0, s>>>(out + 1, nullptr, parts, out);
  return cudaGetLastError();
}

cudaError_t launch_hp_one_shape(const HPTask& t, int ntiles, double2* ws, cudaStream_t s);

cudaError_t launch_hp_split(const HPTask& task, double2* ws, int64_t ws_elems, cudaStream_t s) {
  HPTask t = task;
  const int aB = t.aB > 0 ? t.aB : t.a;
  if (t.a > kHpMaxDim || aB > kHpMaxDim || t.a < 1 || aB < 1) return cudaErrorInvalidValue;
  hp_shape(std::min(std::max(t.a, aB), kHpTile), &t.rows, &t.cols);
  const int ntiles = ((t.a + kHpTile - 1) / kHpTile) * ((aB + kHpTile - 1) / kHpTile);
  const int64_t K = (int64_t)t.before * t.after;
  int64_t kc = std::max<int64_t>(256, (K * ntiles + 4 * 152 - 1) / (4 * 152));
  kc = (kc + kHpRows - 1) / kHpRows * kHpRows;
  int64_t splits = (K + kc - 1) / kc;
  const int64_t per = (int64_t)t.a * aB;
  if (splits > 1 && splits * per > ws_elems) {  // fewer, longer ranges to fit the workspace
    splits = std::max<int64_t>(1, ws_elems / per);
    kc = (K + splits - 1) / splits;
    splits = (K + kc - 1) / kc;
  }
  t.splits = (int)splits;
  t.kchunk = (int)std::min<int64_t>(K, kc);
  t.ws = 0;
  cudaError_t e = launch_hp_one_shape(t, ntiles, ws, s);
  if (e != cudaSuccess) return e;
  if (t.splits > 1) k_hp_sum_one<F64><<<(unsigned)std::min<int64_t>(64, (per + kThreads - 1) / kThreads), kThreads, 0, s>>>(t, ws);
  return cudaGetLastError();
}

cudaError_t launch_lincomb(double2* out, const LinComb& lc, int64_t n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (lc.count < 0 || lc.count > kLinCombMax) return cudaErrorInvalidValue;
  const int64_t want = (n + kThreads - 1) / kThreads;
  const int blocks = (int)std::min<int64_t>(want, 152 * 8);
  k_lincomb<<<blocks, kThreads, 0, s>>>(out, lc, n);
  return cudaGetLastError();
}

cudaError_t launch_axpy(double2* out, const double2* x, double2 a, const double2* y, int64_t n,
                        cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t want = (n + kThreads - 1) / kThreads;
  const int blocks = (int)std::min<int64_t>(want, (int64_t)sms * 8);
  k_axpy<<<blocks, kThreads, 0, s>>>(out, x, a, y, n);
  return cudaGetLastError();
}

cudaError_t probe_df64_peak(cudaStream_t s, double* tflops) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int blocks = sms * 8, iters = 2048;
  float4* buf = nullptr;
  e = cudaMallocAsync((void**)&buf, sizeof(float4) * blocks * kThreads, s);
  if (e != cudaSuccess) return e;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const float4 a = make_float4(1e-3f, 1e-11f, 2e-4f, -1e-12f), b = make_float4(0.5f, 0.f, 0.f, 0.f);
  k_df64_mac<<<blocks, kThreads, 0, s>>>(buf, iters, a, b);  // warm-up
  cudaEventRecord(e0, s);
  k_df64_mac<<<blocks, kThreads, 0, s>>>(buf, iters, a, b);
  cudaEventRecord(e1, s);
  e = cudaEventSynchronize(e1);
  float ms = 0;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(buf, s);
  cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  // 8 flops (complex128-equivalent) per complex multiply-add
  *tflops = 8.0 * 8.0 * iters * (double)blocks * kThreads / (ms * 1e-3) / 1e12;
  return cudaGetLastError();
}

cudaError_t probe_fp64_peak(cudaStream_t s, double* tflops) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int blocks = sms * 8, iters = 4096;
  double* buf = nullptr;
  e = cudaMallocAsync((void**)&buf, sizeof(double) * blocks * kThreads, s);
  if (e != cudaSuccess) return e;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  k_fp64_fma<<<blocks, kThreads, 0, s>>>(buf, iters, 0.999, 0.001);  // warm-up
  cudaEventRecord(e0, s);
  k_fp64_fma<<<blocks, kThreads, 0, s>>>(buf, iters, 0.999, 0.001);
  cudaEventRecord(e1, s);
  e = cudaEventSynchronize(e1);
  float ms = 0;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(buf, s);
  cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  *tflops = 2.0 * 8.0 * iters * (double)blocks * kThreads / (ms * 1e-3) / 1e12;
  return cudaGetLastError();
}

template <class P, int CLASS>
cudaError_t launch_hp_class(const HPTask* tasks, const int4* tiles, int64_t first, int64_t n, typename P::S* ws,
                            cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(k_hp<P, CLASS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kHpSmem);
  if (e != cudaSuccess) return e;
  k_hp<P, CLASS><<<(unsigned)n, kThreads, kHpSmem, s>>>(tasks, tiles, first, ws);
  return cudaSuccess;
}

template <int R, int C>
cudaError_t launch_hp_one_rc(const HPTask& t, int ntiles, double2* ws, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(k_hp_one<F64, R, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, kHpSmem);
  if (e != cudaSuccess) return e;
  k_hp_one<F64, R, C><<<(unsigned)((int64_t)ntiles * t.splits), kThreads, kHpSmem, s>>>(t, ntiles, ws);
  return cudaSuccess;
}

cudaError_t launch_hp_one_shape(const HPTask& t, int ntiles, double2* ws, cudaStream_t s) {
  switch (t.rows * 8 + t.cols) {
    case 1 * 8 + 1: return launch_hp_one_rc<1, 1>(t, ntiles, ws, s);
    case 1 * 8 + 2: return launch_hp_one_rc<1, 2>(t, ntiles, ws, s);
    case 1 * 8 + 3: return launch_hp_one_rc<1, 3>(t, ntiles, ws, s);
    case 1 * 8 + 4: return launch_hp_one_rc<1, 4>(t, ntiles, ws, s);
    case 2 * 8 + 3: return launch_hp_one_rc<2, 3>(t, ntiles, ws, s);
    case 2 * 8 + 4: return launch_hp_one_rc<2, 4>(t, ntiles, ws, s);
    case 3 * 8 + 3: return launch_hp_one_rc<3, 3>(t, ntiles, ws, s);
    case 3 * 8 + 4: return launch_hp_one_rc<3, 4>(t, ntiles, ws, s);
    case 4 * 8 + 4: return launch_hp_one_rc<4, 4>(t, ntiles, ws, s);
    default: return cudaErrorInvalidValue;
  }
}


// ---------------------------------------------------------------------------
// CDVR kernels (complex128)
// ---------------------------------------------------------------------------
// Strided complex contraction (TCTask): one block per 32 x 32 output tile,
// k in chunks of 16 staged through shared memory.  Operand tiles are read
// along whichever of their two indices has unit stride.
constexpr int kTcK = 16;
__global__ void __launch_bounds__(kThreads) k_tc(const TCTask* __restrict__ tasks,
                                                 const int4* __restrict__ tiles, int64_t tile0) {
  const int4 tl = tiles[tile0 + blockIdx.x];
  const TCTask t = tasks[tl.x];
  const int64_t M = (int64_t)t.M0 * t.M1, N = (int64_t)t.N0 * t.N1, K = (int64_t)t.K0 * t.K1;
  const int64_t mb = (int64_t)tl.y * kTcTile, nb = (int64_t)tl.z * kTcTile;
  __shared__ double2 As[kTcK][kTcTile + 1];
  __shared__ double2 Bs[kTcK][kTcTile + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double2 acc[2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j] = cz();
  const bool a_mfast = t.am0 == 1 || t.M0 * (int64_t)t.M1 == 1;
  const bool b_nfast = t.bn0 == 1 || t.N0 * (int64_t)t.N1 == 1;
  for (int64_t k0 = 0; k0 < K; k0 += kTcK) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int e = threadIdx.x + r * kThreads;  // 512 elements of each tile
      int mi, ki;
      if (a_mfast) {
        mi = e & 31;
        ki = e >> 5;
      } else {
        ki = e & 15;
        mi = e >> 4;
      }
      const int64_t m = mb + mi, k = k0 + ki;
      double2 v = cz();
      if (m < M && k < K) {
        const int64_t m0 = m % t.M0, m1 = m / t.M0, kk0 = k % t.K0, kk1 = k / t.K0;
        v = t.A[m0 * t.am0 + m1 * t.am1 + kk0 * t.ak0 + kk1 * t.ak1];
        if (t.conjA) v.y = -v.y;
      }
      As[ki][mi] = v;
      int ni, kj;
      if (b_nfast) {
        ni = e & 31;
        kj = e >> 5;
      } else {
        kj = e & 15;
        ni = e >> 4;
      }
      const int64_t nn = nb + ni, kb = k0 + kj;
      double2 w = cz();
      if (nn < N && kb < K) {
        const int64_t n0 = nn % t.N0, n1 = nn / t.N0, kk0 = kb % t.K0, kk1 = kb / t.K0;
        w = t.B[kk0 * t.bk0 + kk1 * t.bk1 + n0 * t.bn0 + n1 * t.bn1];
        if (t.conjB) w.y = -w.y;
      }
      Bs[kj][ni] = w;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kTcK; ++kk) {
      const double2 a0 = As[kk][ty * 2], a1 = As[kk][ty * 2 + 1];
      const double2 b0 = Bs[kk][tx * 2], b1 = Bs[kk][tx * 2 + 1];
      cfma(acc[0][0], a0, b0);
      cfma(acc[0][1], a0, b1);
      cfma(acc[1][0], a1, b0);
      cfma(acc[1][1], a1, b1);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int64_t m = mb + ty * 2 + i, nn = nb + tx * 2 + j;
      if (m >= M || nn >= N) continue;
      const int64_t off = (m % t.M0) * t.cm0 + (m / t.M0) * t.cm1 + (nn % t.N0) * t.cn0 + (nn / t.N0) * t.cn1;
      const double2 v = cmul(t.alpha, acc[i][j]);
      if (t.add) {
        const double2 o = t.C[off];
        t.C[off] = make_double2(o.x + v.x, o.y + v.y);
      } else {
        t.C[off] = v;
      }
    }
}

__device__ double2 block_sum2(double2 v, double2* red) {
  red[threadIdx.x] = v;
  __syncthreads();
  for (int s = kThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      red[threadIdx.x].x += red[threadIdx.x + s].x;
      red[threadIdx.x].y += red[threadIdx.x + s].y;
    }
    __syncthreads();
  }
  const double2 r = red[0];
  __syncthreads();
  return r;
}

// out = gramSchmidt(in + noise) (include/Core/Tensor_Implementation.h:805-853):
// per column, up to 15 passes of projection on the previous columns and
// normalisation, while the summed |overlap| of a pass exceeds 1e-12.
__global__ void __launch_bounds__(kThreads) k_gs(const GSTask* __restrict__ tasks, int64_t task0) {
  const GSTask t = tasks[task0 + blockIdx.x];
  __shared__ double2 red[kThreads];
  const int64_t rows = t.rows;
  const int64_t tot = rows * t.cols;
  for (int64_t e = threadIdx.x; e < tot; e += kThreads) {
    const double2 a = t.in[e], z = t.noise[e];
    t.out[e] = make_double2(a.x + z.x, a.y + z.y);
  }
  __syncthreads();
  double2* A = t.out;
  for (int n = 0; n < t.cols; ++n) {
    double2* an = A + rows * n;
    for (int iter = 0; iter < 15; ++iter) {
      double accum = 0;
      for (int m = 0; m < n; ++m) {
        const double2* am = A + rows * m;
        double2 part = cz();
        for (int64_t i = threadIdx.x; i < rows; i += kThreads) cfmac(part, am[i], an[i]);
        const double2 ov = block_sum2(part, red);
        accum += sqrt(ov.x * ov.x + ov.y * ov.y);
        for (int64_t i = threadIdx.x; i < rows; i += kThreads) {
          const double2 x = cmul(ov, am[i]);
          an[i] = make_double2(an[i].x - x.x, an[i].y - x.y);
        }
        __syncthreads();
      }
      double2 part = cz();
      for (int64_t i = threadIdx.x; i < rows; i += kThreads) part.x += an[i].x * an[i].x + an[i].y * an[i].y;
      const double nrm = block_sum2(part, red).x;
      if (nrm != 0.0) {
        const double sc = sqrt(nrm);
        for (int64_t i = threadIdx.x; i < rows; i += kThreads) an[i] = make_double2(an[i].x / sc, an[i].y / sc);
      }
      __syncthreads();
      if (!(accum > 1e-12)) break;
    }
  }
}

inline int64_t eigf_smem_bytes(int d) { return eig_smem_bytes(d) + 4 * (int64_t)(d + 1) + 16; }

// spectral functions of a Hermitian matrix (EigFTask)
__global__ void __launch_bounds__(kThreads) k_eigf(const EigFTask* __restrict__ tasks, int64_t task0) {
  extern __shared__ double2 smem[];
  const EigFTask t = tasks[task0 + blockIdx.x];
  const int d = t.d;
  const int m = d + (d & 1);
  const int np = m / 2;
  double2* A = smem;
  double2* rot = A + (int64_t)d * d;
  double2* ph = rot + np;
  double2* fw = ph + np;
  int* pq = (int*)(fw + m);
  int* perm = pq + 2 * np;
  __shared__ double red_off[kThreads], red_diag[kThreads];
  for (int e = threadIdx.x; e < d * d; e += kThreads) {
    const int i = e % d, j = e / d;
    const double2 aij = t.A[i + (int64_t)d * j], aji = t.A[j + (int64_t)d * i];
    A[e] = (i == j) ? make_double2(aij.x, 0.0) : make_double2(0.5 * (aij.x + aji.x), 0.5 * (aij.y - aji.y));
  }
  __syncthreads();
  herm_jacobi(A, t.U, d, rot, ph, pq, red_off, red_diag);
  __syncthreads();
  const double2* U = t.U;
  if (t.fn == 4) {
    if (threadIdx.x == 0) {  // ascending order of the eigenvalues
      for (int i = 0; i < d; ++i) perm[i] = i;
      for (int i = 0; i < d; ++i) {
        int best = i;
        for (int j = i + 1; j < d; ++j)
          if (A[perm[j] + d * perm[j]].x < A[perm[best] + d * perm[best]].x) best = j;
        const int x = perm[i];
        perm[i] = perm[best];
        perm[best] = x;
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < d * d; e += kThreads) {
      const int i = e % d, j = e / d;
      const double2 u = U[j + (int64_t)d * perm[i]];
      t.out[e] = make_double2(u.x, -u.y);
    }
    for (int i = threadIdx.x; i < d; i += kThreads) t.vals[i] = make_double2(A[perm[i] + d * perm[i]].x, 0.0);
    return;
  }
  const double eps = t.eps;
  for (int i = threadIdx.x; i < d; i += kThreads) {
    const double w = A[i + d * i].x;
    double f;
    if (t.fn == 0) {
      f = 1.0 / (w + eps * exp(-w / eps));
    } else {
      const double g = sqrt(fmax(w, 0.0));
      if (t.fn == 1)
        f = g;
      else if (t.fn == 2)
        f = 1.0 / (g + eps * exp(-g / eps));
      else
        f = g + eps * exp(-g / eps);
    }
    fw[i].x = f;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < d * d; e += kThreads) {
    const int i = e % d, j = e / d;
    double2 acc = cz();
    for (int k = 0; k < d; ++k) {
      const double2 uik = U[i + (int64_t)d * k];
      const double2 ujk = U[j + (int64_t)d * k];
      const double fk = fw[k].x;
      cfma(acc, make_double2(uik.x * fk, uik.y * fk), make_double2(ujk.x, -ujk.y));
    }
    t.out[e] = acc;
  }
}

// polynomial potential on grid tensors (VPotTask): terms in order, each
// product left to right, nothing fused (the CPU restatement does the same)
__global__ void __launch_bounds__(kThreads) k_vpot(const VPotTask* __restrict__ tasks,
                                                   const VCoord* __restrict__ coords,
                                                   const int2* __restrict__ tiles, int64_t tile0,
                                                   const PotTerm* __restrict__ terms,
                                                   const PotFactor* __restrict__ factors, int n_terms) {
  const int2 tl = tiles[tile0 + blockIdx.x];
  const VPotTask t = tasks[tl.x];
  const int64_t e = (int64_t)tl.y + threadIdx.x;
  if (e >= t.n) return;
  int idx[6];
  int64_t r = e;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    if (k < t.order) {
      idx[k] = (int)(r % t.dims[k]);
      r /= t.dims[k];
    } else {
      idx[k] = 0;
    }
  }
  double v = 0.0;
  for (int q = 0; q < n_terms; ++q) {
    const PotTerm pt = terms[q];
    double tv = pt.c;
    for (int fct = pt.first; fct < pt.first + pt.count; ++fct) {
      const PotFactor pf = factors[fct];
      const VCoord c = coords[t.first + pf.mode];
      const double x = c.grid[idx[c.index]].x;
      for (int p = 0; p < pf.power; ++p) tv = __dmul_rn(tv, x);
    }
    v = __dadd_rn(v, tv);
  }
  t.out[e] = make_double2(v, 0.0);
}

// local part of the correction tensor (DVLTask)
__global__ void __launch_bounds__(kThreads) k_dvl(const DVLTask* __restrict__ tasks,
                                                  const int2* __restrict__ tiles, int64_t tile0) {
  const int2 tl = tiles[tile0 + blockIdx.x];
  const DVLTask t = tasks[tl.x];
  const int64_t d = t.d;
  const int64_t e = (int64_t)tl.y + threadIdx.x;
  if (e >= d * d * d * d) return;
  const int64_t l1 = e % d, i0 = e / d % d, m1 = e / (d * d) % d, i3 = e / (d * d * d);
  double2 v = cz();
  if (i0 == i3) {
    const int64_t bef = t.bef;
    for (int64_t b = 0; b < bef; ++b) {
      const double2 a = t.cup[b + bef * l1];
      const double2 x = cmul(make_double2(a.x, -a.y), t.vnode[b + bef * i0]);
      cfma(v, x, t.cup[b + bef * m1]);
    }
  }
  if (l1 == m1 && i0 == i3) {
    const double2 ve = t.vedge[l1 + d * i0];
    v = make_double2(v.x - ve.x, v.y - ve.y);
  }
  t.dv[e] = v;
}

// out = (add ? out : 0) + v * in, elementwise (EWTask)
__global__ void __launch_bounds__(kThreads) k_ew(const EWTask* __restrict__ tasks,
                                                 const int2* __restrict__ tiles, int64_t tile0) {
  const int2 tl = tiles[tile0 + blockIdx.x];
  const EWTask t = tasks[tl.x];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int64_t e = (int64_t)tl.y + threadIdx.x + (int64_t)q * kThreads;
    if (e >= t.n) continue;
    double2 r = cmul(t.v[e], t.in[e]);
    if (t.add) {
      const double2 o = t.out[e];
      r = make_double2(r.x + o.x, r.y + o.y);
    }
    t.out[e] = r;
  }
}

// outputs per thread of a mode-product or accumulation stage of `tiles` tiles:
// one (four blocks per tile) while four per thread would leave SMs with fewer
// than two blocks, two up to twice that.  Stages of an 8-mode complex128
// sweep: mode products 151 -> 115 us, accumulations 110 -> 57; of a 12-mode
// double-float one (bonds 13..19): 282 -> 207 and 195 -> 133.  Beyond, one
// output per thread costs loads: the mode products of 64 uneven trees 2.93 -> 3.81 ms,
// accumulations at bonds 58..96 34 -> 45 ms.
inline int outputs_per_thread(int64_t tiles) { return tiles <= 2 * 152 ? 1 : tiles <= 4 * 152 ? 2 : 4; }

template <class P>
cudaError_t launch_stage_p(const Stage& st, const DevTables& t, double eps, int max_eig_d,
                           cudaStream_t s) {
  switch (st.kind) {
    case ST_MP:
      if (st.n_tiles > 0) {
        const unsigned n = (unsigned)st.n_tiles;
        switch (outputs_per_thread(st.n_tiles)) {
          case 1: k_mp<P, 1><<<dim3(n, 4), kThreads, 0, s>>>(t.mp, t.mp_tiles, st.first_tile); break;
          case 2: k_mp<P, 2><<<dim3(n, 2), kThreads, 0, s>>>(t.mp, t.mp_tiles, st.first_tile); break;
          default: k_mp<P, 4><<<n, kThreads, 0, s>>>(t.mp, t.mp_tiles, st.first_tile);
        }
      }
      if (st.noz > 0) {
        cudaError_t e = launch_mp_tc(std::is_same<P, DF64>::value, t.mp, t.mp_oz_tiles, st.oz0, st.noz,
                                     t.mp_oz_tasks, st.ozt0, st.nozt, st.tc_wide, t.status, s);
        if (e != cudaSuccess) return e;
      }
      break;
    case ST_HP: {
      typedef typename P::S S;
      // the segments (one register-tile shape each) lie class by class
      for (int g = st.seg0; g < st.seg0 + st.nseg;) {
        const int cls = hp_class(t.hp_segs[g].x, t.hp_segs[g].y);
        const int64_t first = t.hp_segs[g].z;
        int64_t n = 0;
        for (; g < st.seg0 + st.nseg && hp_class(t.hp_segs[g].x, t.hp_segs[g].y) == cls; ++g) n += t.hp_segs[g].w;
        S* ws = reinterpret_cast<S*>(t.hp_ws);
        cudaError_t e = cls == 0   ? launch_hp_class<P, 0>(t.hp, t.hp_tiles, first, n, ws, s)
                        : cls == 1 ? launch_hp_class<P, 1>(t.hp, t.hp_tiles, first, n, ws, s)
                                   : launch_hp_class<P, 2>(t.hp, t.hp_tiles, first, n, ws, s);
        if (e != cudaSuccess) return e;
      }
      if (st.nhti > 0) {
        if (!std::is_same<P, DF64>::value) return cudaErrorInvalidValue;  // the planner emits none
        cudaError_t e = launch_hp_tc(t.hp, t.hp_tc_groups, t.hp_tc_items, st.hti0, st.nhti, t.hp_tc_imgs, st.htu0,
                                     st.nhtu, reinterpret_cast<double2*>(t.hp_ws), st.tc_wide, t.status, s);
        if (e != cudaSuccess) return e;
      }
      if (st.aux)
        k_hp_sum<P><<<(unsigned)(st.n_tasks * kHpSumChunks), kThreads, 0, s>>>(t.hp, st.first_task,
                                                             reinterpret_cast<const S*>(t.hp_ws));
      break;
    }
    case ST_ACC:
      if (st.n_tiles > 0) {
        const unsigned n = (unsigned)st.n_tiles;
        switch (outputs_per_thread(st.n_tiles)) {
          case 1: k_acc_few<P, 1><<<dim3(n, 4), kThreads, 0, s>>>(t.acc, t.acc_terms, t.acc_tiles, st.first_tile); break;
          case 2: k_acc_few<P, 2><<<dim3(n, 2), kThreads, 0, s>>>(t.acc, t.acc_terms, t.acc_tiles, st.first_tile); break;
          default: k_acc<P><<<n, kThreads, 0, s>>>(t.acc, t.acc_terms, t.acc_tiles, st.first_tile);
        }
      }
      if (st.nati > 0) {
        if (!std::is_same<P, DF64>::value) return cudaErrorInvalidValue;  // the planner emits none
        cudaError_t e = launch_acc_tc(t.acc, t.acc_terms, t.acc_tc_items, st.ati0, st.nati, st.atc_units,
                                      t.acc_tc_imgs, st.atu0, st.natu, st.tc_wide, t.status, s);
        if (e != cudaSuccess) return e;
      }
      break;
    case ST_LIN:
      // max_eig_d bounds every matrix
      k_lin<P><<<dim3((unsigned)st.n_tasks, (unsigned)((max_eig_d * max_eig_d + kThreads - 1) / kThreads)), kThreads, 0, s>>>(
          t.lin, t.lin_terms, st.first_task);
      break;
    case ST_MM:
      k_mm<P><<<dim3((unsigned)st.n_tiles, kMmBlocks), kThreads, 0, s>>>(t.mm, t.mm_terms, t.mm_tiles, st.first_tile);
      break;
    case ST_EIG: {
      const int64_t sm = eig_smem_bytes(max_eig_d);
      cudaError_t e = cudaFuncSetAttribute(k_eig, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sm);
      if (e != cudaSuccess) return e;
      k_eig<<<(unsigned)st.n_tasks, kThreads, sm, s>>>(t.eig, st.first_task, eps);
      break;
    }
    case ST_PROJ: {
      // max_eig_d (<= kHpMaxDim) bounds every node's bond.  Up to four blocks
      // per node while the stage leaves SMs idle: the rows of P are shared
      // out, the inversion is repeated (64-mode sweep, bonds 32..64: 510 us with
      // one block per node, 387 with two; 16 modes: 76 -> 57 with four).
      const int sm = max_eig_d * max_eig_d * 16;
      cudaError_t e = cudaFuncSetAttribute(k_proj<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
      if (e != cudaSuccess) return e;
      const unsigned parts = (unsigned)std::max<int64_t>(1, std::min<int64_t>(4, 2 * 152 / st.n_tasks));
      k_proj<P><<<dim3((unsigned)st.n_tasks, parts), kThreads, sm, s>>>(t.proj, st.first_task);
      break;
    }
    case ST_CVT:
      k_cvt<<<(unsigned)st.n_tiles, kThreads, 0, s>>>(t.cvt, t.cvt_tiles, st.first_tile);
      break;
    case ST_GRAD:
      k_grad<P><<<(unsigned)st.n_tasks, kThreads, 0, s>>>(t.grad, st.first_task);
      break;
    case ST_TC:
      k_tc<<<(unsigned)st.n_tiles, kThreads, 0, s>>>(t.tc, t.tc_tiles, st.first_tile);
      break;
    case ST_GS:
      k_gs<<<(unsigned)st.n_tasks, kThreads, 0, s>>>(t.gs, st.first_task);
      break;
    case ST_EIGF: {
      const int64_t sm = eigf_smem_bytes(max_eig_d);
      cudaError_t e = cudaFuncSetAttribute(k_eigf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      if (e != cudaSuccess) return e;
      k_eigf<<<(unsigned)st.n_tasks, kThreads, sm, s>>>(t.eigf, st.first_task);
      break;
    }
    case ST_WSD:
      return launch_wsd(t.wsd, t.wsd_terms, st.first_task, st.n_tasks, t.wsd_max_n, t.wsd_max_d, s);
    case ST_VPOT:
      k_vpot<<<(unsigned)st.n_tiles, kThreads, 0, s>>>(t.vpot, t.vcoords, t.vpot_tiles, st.first_tile,
                                                       t.pot_terms, t.pot_factors, t.n_pot_terms);
      break;
    case ST_DVL:
      k_dvl<<<(unsigned)st.n_tiles, kThreads, 0, s>>>(t.dvl, t.dvl_tiles, st.first_tile);
      break;
    case ST_EW:
      k_ew<<<(unsigned)st.n_tiles, kThreads, 0, s>>>(t.ew, t.ew_tiles, st.first_tile);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_stage(const Stage& st, const DevTables& t, double eps, int max_eig_d,
                         int prec, cudaStream_t s) {
  switch (prec) {
    case 1: return launch_stage_p<DF64>(st, t, eps, max_eig_d, s);
    case 2: return launch_stage_p<C32>(st, t, eps, max_eig_d, s);
    default: return launch_stage_p<F64>(st, t, eps, max_eig_d, s);
  }
}

cudaError_t launch_set_identity(double2* m, int d, int prec, cudaStream_t s) {
  k_identity<<<1, kThreads, 0, s>>>(m, d, prec);
  return cudaGetLastError();
}

cudaError_t launch_single_mp(const MPTask& task, cudaStream_t s, void*) {
  const int64_t n = (int64_t)task.before * task.a_out * task.after;
  const int64_t blocks = (n + kThreads - 1) / kThreads;
  if (blocks == 0) return cudaSuccess;
  k_mp_single<<<(unsigned)blocks, kThreads, 0, s>>>(task);
  return cudaGetLastError();
}

cudaError_t launch_single_hp(const HPTask& task, cudaStream_t s, void*) {
  const int aA = task.a, aB = task.aB > 0 ? task.aB : task.a;
  if (aA < 1 || aB < 1) return cudaSuccess;
  HcGeo g;
  g.nti = (aA + kHcTile - 1) / kHcTile;
  const int ntj = (aB + kHcTile - 1) / kHcTile;
  g.ti = (aA + g.nti - 1) / g.nti;  // tiles of equal sides
  g.tj = (aB + ntj - 1) / ntj;
  g.groups = std::min(kThreads / (g.ti * g.tj), kHcRows);
  const int64_t tiles = (int64_t)g.nti * ntj, K = (int64_t)task.before * task.after;
  // more CTAs per tile while they find SMs (152) and at least 16 rows each
  g.cl = 1;
  while (g.cl < kHcMaxCl && tiles * g.cl < 152 && K >= 32 * g.cl) g.cl *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * g.cl));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)g.cl;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_hp_single, task, g);
}

// ---------------------------------------------------------------------------
// Allocation-free density inverse.
//
// Callers that may not allocate device memory themselves (code running while
// a CUDA stream is being captured, where cudaMalloc/cudaFree are not
// allowed; latency-critical loops that cannot afford the implicit device
// synchronisation of cudaFree; hosts whose device memory is owned by a pool
// allocator that forbids side allocations) get the regularised inverses of
// density matrices they already hold on the device without handing the
// library any workspace.  The Jacobi eigenvector matrices live in the
// file-scope array below instead of a cudaMalloc'd arena:
//   - capacity kStaticEigElems complex elements (8 MiB): n_mats * d * d
//     must not exceed 524288, e.g. 128 matrices of 64 x 64;
//   - every GPU that loads the library holds these 8 MiB until the process
//     exits;
//   - all calls share the one array and it keeps the last call's contents.
//     The kernel writes every scratch element before reading it (U starts as
//     the identity), so nothing needs clearing between calls; two calls that
//     overlap on the GPU (different streams, contexts or host threads) race
//     on the array and must be ordered by the caller.
// Host code cannot use the array's name as a device address, so the address
// is looked up with cudaGetSymbolAddress (with that device current) on the
// first call that a device sees, and again on the first call after the
// device's context was replaced (cudaDeviceReset).  Those first calls must
// happen outside any stream capture; inside one they fail with
// cudaErrorStreamCaptureUnsupported instead of using a stale address.
// ---------------------------------------------------------------------------
constexpr int64_t kStaticEigElems = (int64_t)(8 << 20) / 16;
static __device__ __align__(256) double2 g_eig_scratch[kStaticEigElems];

namespace {

constexpr int kMaxDevices = 64;

// The array's device address, cached per device together with the identity
// of the CUDA context it was looked up in.  A device reset (cudaDeviceReset)
// destroys the primary context and the module with it; the next context may
// load the module at another address.  Context handles can be reused after a
// reset, context IDs (cuCtxGetId) are unique for the life of the process, so
// the cache is keyed by the ID.
struct ScratchAddr {
  unsigned long long ctx_id = 0;
  double2* addr = nullptr;
};
ScratchAddr g_eig_scratch_addr[kMaxDevices];
std::mutex g_eig_scratch_mutex;

typedef CUresult (*PfnCtxGetCurrent)(CUcontext*);
typedef CUresult (*PfnCtxGetId)(CUcontext, unsigned long long*);

// ID of the calling thread's current CUDA context (0 and an error if unknown)
cudaError_t current_ctx_id(unsigned long long* id) {
  static PfnCtxGetCurrent get_current = nullptr;
  static PfnCtxGetId get_id = nullptr;
  if (!get_current || !get_id) {
    void* f1 = nullptr;
    void* f2 = nullptr;
    cudaDriverEntryPointQueryResult q1, q2;
    cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1);
    if (e == cudaSuccess) e = cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2);
    if (e != cudaSuccess) return e;
    if (q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !f1 || !f2)
      return cudaErrorNotSupported;
    get_current = (PfnCtxGetCurrent)f1;
    get_id = (PfnCtxGetId)f2;
  }
  CUcontext ctx = nullptr;
  if (get_current(&ctx) != CUDA_SUCCESS || !ctx) return cudaErrorDeviceUninitialized;
  if (get_id(ctx, id) != CUDA_SUCCESS) return cudaErrorDeviceUninitialized;
  return cudaSuccess;
}

// U[b] = g_eig_scratch + b*d*d; matrix b of the batch is one block
__global__ void __launch_bounds__(kThreads) k_eig_strided(const double2* __restrict__ rho,
                                                          double2* __restrict__ rhoinv, double2* U,
                                                          int d, double eps) {
  const int64_t o = (int64_t)blockIdx.x * d * d;
  EigTask t;
  t.rho = rho + o;
  t.rhoinv = rhoinv + o;
  t.U = U + o;
  t.d = d;
  t.pad = 0;
  eig_body(t, eps);
}

}  // namespace

int64_t static_eig_capacity() { return kStaticEigElems; }

cudaError_t launch_rho_inverse_static(const double2* rho, double2* rhoinv, int n_mats, int d,
                                      double eps, cudaStream_t s) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  double2* scratch = nullptr;
  {
    unsigned long long id = 0;
    e = current_ctx_id(&id);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(g_eig_scratch_mutex);
    ScratchAddr& cache = g_eig_scratch_addr[dev];
    if (!cache.addr || cache.ctx_id != id) {
      // set-up once per device and context, with that device current; it
      // may load the module, so it must not happen inside a stream capture
      cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
      e = cudaStreamIsCapturing(s, &cs);
      if (e != cudaSuccess) return e;
      if (cs != cudaStreamCaptureStatusNone) return cudaErrorStreamCaptureUnsupported;
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_eig_scratch);
      if (e != cudaSuccess) return e;
      cache.addr = (double2*)p;
      cache.ctx_id = id;
    }
    scratch = cache.addr;
  }
  const int64_t sm = eig_smem_bytes(d);
  e = cudaFuncSetAttribute(k_eig_strided, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  k_eig_strided<<<(unsigned)n_mats, kThreads, sm, s>>>(rho, rhoinv, scratch, d, eps);
  return cudaGetLastError();
}


// ---------------------------------------------------------------------------
// Householder QR of node tensors (qrOrthogonal, complex128 on the FP64 pipe).
// A (m x n, column-major: the node tensor as a (lastBefore x d_up) matrix) is
// replaced by its thin Q = H_0 ... H_{s-1} [I; 0], s = min(m, n), and R (n x n,
// column-major, upper triangular) is written.  Reflector j,
// H_j = I - tau_j v_j v_j^H, maps x = A[j:m, j] to alpha e_1 with
// alpha = -e^{i arg x_0} |x| (the Eigen choice).
//
// A cluster of CTAs owns a node, each CTA a contiguous block of its rows (in
// shared memory when they fit, else in place).  Step j is one pass over the
// rows below j for all dot products with x = A[j+1:m, j] (columns k > j: to
// update them; k < j: the Gram matrix of the reflectors), one exchange of the
// CTAs' partial sums through distributed shared memory, and the update:
//   w_k = v^H a_k = x^H a_k + conj(v_0) a_jk,   a_k -= tau v w_k,
// where |x|^2 is the sum for k = j, and row j comes from its CTA; tau = 2 / |v|^2
// of the v that is stored.  Then
// Q = [I; 0] - V M with the compact form M = T V_top^H, (T^-1)_il = v_i^H v_l
// for i < l and 1 / tau_i on the diagonal, solved by back substitution
// (columns shared out over the CTAs), and one product per row, the identity
// added last.  No atomics, fixed orders of addition.
//
// Bound: the FP64 pipe, 10 m n^2 DFMA over the cluster's SMs, and per step a
// chain of about 3 us (sums, exchange, square root, divisions).  One block per
// node ran the 31 nodes of a 16-mode tree (bonds 32) in 13.5 ms.
// ---------------------------------------------------------------------------
constexpr int kQrBuf = 16;  // rows of V staged at a time when the block is in global memory
__device__ __forceinline__ void qr_sync(int cl) {
  if (cl > 1)
    cluster_sync();
  else
    __syncthreads();
}

__global__ void __launch_bounds__(kThreads) k_house_qr(const QRTask* __restrict__ tasks, int cl, int slab_smem) {
  extern __shared__ __align__(16) unsigned char qr_raw[];
  const QRTask t = tasks[blockIdx.x / cl];
  const int m = t.m, n = t.n, steps = min(m, n);
  const int tid = threadIdx.x;
  const int rank = cl > 1 ? (int)cluster_rank() : 0;
  const int rp = (m + cl - 1) / cl;                       // rows per CTA
  const int r0 = min(m, rank * rp), nr = min(m, r0 + rp) - r0;
  double2* sh = reinterpret_cast<double2*>(qr_raw);
  double2* part = sh;             // [2][n] this CTA's sums (read by the cluster)
  double2* rowj = part + 2 * n;   // [2][n] row j, in its CTA (read by the cluster)
  double2* tw = rowj + 2 * n;     // [n] tau w_k
  double2* red = tw + n;          // [kThreads]
  double2* slab = red + kThreads; // the CTA's rows, or kQrBuf rows of V
  __shared__ double s_tau[kHpMaxDim];
  __shared__ double2 s_alpha[kHpMaxDim];
  double2* X = slab_smem ? slab : t.A + r0;  // element (i, k) of the block at X[i + ld k]
  const int64_t ld = slab_smem ? (rp | 1) : m;
  if (slab_smem)
    for (int e = tid; e < nr * n; e += kThreads) {
      const int i = e % nr, k = e / nr;
      X[i + ld * k] = t.A[r0 + i + (int64_t)m * k];
    }
  int ch = 1;  // dot products: n column slots x ch row lanes (a power of two)
  while (2 * ch * n <= kThreads) ch *= 2;
  __syncthreads();
  for (int j = 0; j < steps; ++j) {
    const int par = j & 1, lo = max(0, j - r0);  // first row of the block at or below row j
    // partial x^H a_k over the block's rows > j
    {
      const int k = tid % n, c = tid / n;
      double2 acc = cz();
      if (c < ch) {
        const double2* x = X + ld * j;
        const double2* a = X + ld * k;
        for (int i = max(0, j + 1 - r0) + c; i < nr; i += ch) cfmac(acc, x[i], a[i]);
        red[tid] = acc;
      }
      for (int h = ch / 2; h > 0; h /= 2) {
        __syncthreads();
        if (c < h) red[tid] = cadd(red[tid], red[tid + h * n]);
      }
      __syncthreads();
      if (tid < n) part[par * n + tid] = red[tid];
      if (j >= r0 && j < r0 + nr && tid < n) rowj[par * n + tid] = X[(j - r0) + ld * tid];
    }
    qr_sync(cl);
    // total sums (CTAs in a fixed tree) and row j
    double2 row = cz();
    {
      const int k = tid % n, c = tid / n;
      if (cl > 1) {
        int q = 1;  // threads per column, a power of two
        while (2 * q * n <= kThreads && 2 * q <= cl) q *= 2;
        if (c < q) {
          double2 v = cz();
          for (int r = c; r < cl; r += q) v = cadd(v, ld_cluster(part + par * n + k, (uint32_t)r));
          red[tid] = v;
        }
        for (int h = q / 2; h > 0; h /= 2) {
          __syncthreads();
          if (c < h) red[tid] = cadd(red[tid], red[tid + h * n]);
        }
        if (tid < n) row = ld_cluster(rowj + par * n + tid, (uint32_t)(j / rp));
      } else if (tid < n) {
        red[tid] = part[par * n + tid];
        row = rowj[par * n + tid];
      }
    }
    if (tid == j) red[kThreads - 1] = red[j];  // |x|^2 below x_0 (the slot is free: n <= kHpMaxDim)
    if (tid == j) tw[j] = row;                     // x_0
    __syncthreads();
    if (tid < 32) {  // the scalars, roots and divisions in separate lanes
      const double below = red[kThreads - 1].x;
      const double2 x0 = tw[j];
      const double a2 = x0.x * x0.x + x0.y * x0.y;
      const double rt = sqrt(tid == 0 ? below + a2 : a2);
      const double nrm = __shfl_sync(0xffffffffu, rt, 0), ax0 = __shfl_sync(0xffffffffu, rt, 1);
      const double q = (tid == 0 ? x0.x : x0.y) / ax0;
      double2 ph = make_double2(__shfl_sync(0xffffffffu, q, 0), __shfl_sync(0xffffffffu, q, 1));
      if (!(ax0 > 0.0)) ph = make_double2(1.0, 0.0);
      const double2 al = make_double2(-ph.x * nrm, -ph.y * nrm);
      const double2 v0 = make_double2(x0.x - al.x, x0.y - al.y);
      const double vn2 = below + (v0.x * v0.x + v0.y * v0.y);
      if (tid == 0) {
        s_tau[j] = vn2 > 0.0 ? 2.0 / vn2 : 0.0;
        s_alpha[j] = al;
      }
    }
    __syncthreads();
    const double tau = s_tau[j];
    const double2 al = s_alpha[j], x0 = tw[j];
    const double2 v0 = make_double2(x0.x - al.x, x0.y - al.y);
    if (tid < n && tid != j) {
      double2 w = red[tid];
      cfmac(w, v0, row);
      if (tid > j)
        tw[tid] = make_double2(tau * w.x, tau * w.y);
      else if (rank == 0)
        t.R[j + (int64_t)n * tid] = make_double2(w.x, -w.y);  // v_k^H v_j, parked below R's diagonal
    }
    if (j >= r0 && j < r0 + nr && tid == j) X[(j - r0) + ld * j] = v0;
    __syncthreads();
    const int nk = n - 1 - j;
    if (nk > 0) {
      const int rows = kThreads / nk;  // row lanes per column
      const int k = j + 1 + tid % nk, c = tid / nk;
      if (c < rows) {
        const double2* v = X + ld * j;
        double2* a = X + ld * k;
        const double2 f = make_double2(-tw[k].x, -tw[k].y);
        for (int i = lo + c; i < nr; i += rows) cfma(a[i], v[i], f);
      }
    }
    __syncthreads();
  }
  // R's upper triangle (final in the rows above the diagonal; the diagonal is alpha)
  for (int e = tid; e < n * n; e += kThreads) {
    const int i = e % n, k = e / n;
    if (i > k) continue;
    if (i >= r0 && i < r0 + nr)
      t.R[e] = i < k ? X[(i - r0) + ld * k] : s_alpha[i];
    else if (i >= m && rank == 0)
      t.R[e] = cz();
  }
  // the reflectors' top rows for the other CTAs
  if (slab_smem)
    for (int e = tid; e < min(nr, max(0, n - r0)) * steps; e += kThreads) {
      const int w = min(nr, n - r0), i = e % w, k = e / w;
      t.A[r0 + i + (int64_t)m * k] = X[i + ld * k];
    }
  qr_sync(cl);
  // M = T V_top^H (steps x n) into Qs, columns rank, rank + cl, ...
  {
    const int cb = min(kThreads / steps, kThreads / 2), i = tid % steps, c = tid / steps;
    for (int c0 = 0; rank + cl * c0 < n; c0 += cb) {
      const int k = rank + cl * (c0 + c);
      const bool act = c < cb && k < n;
      double2 acc = cz();
      if (act && i <= k && k < m) {
        acc = t.A[k + (int64_t)m * i];
        acc.y = -acc.y;
      }
      for (int l = steps - 1; l >= 0; --l) {
        double2* mr = red + (l & 1) * (kThreads / 2);
        if (act && i == l) {
          const double2 v = make_double2(s_tau[l] * acc.x, s_tau[l] * acc.y);
          mr[c] = v;
          t.Qs[l + (int64_t)steps * k] = v;
        }
        __syncthreads();
        if (act && i < l) {
          const double2 g = t.R[l + (int64_t)n * i];
          cfma(acc, make_double2(-g.x, -g.y), mr[c]);
        }
      }
      __syncthreads();
    }
  }
  qr_sync(cl);
  if (rank == 0)
    for (int e = tid; e < n * n; e += kThreads)
      if (e % n > e / n) t.R[e] = cz();
  // Q = [I; 0] - V M, row by row
  const int span = slab_smem ? nr : kQrBuf;
  for (int b0 = 0; b0 < nr; b0 += span) {
    const int nb = min(span, nr - b0);
    const double2* v = X;
    int64_t lv = ld;
    if (!slab_smem) {
      for (int e = tid; e < nb * steps; e += kThreads) slab[e] = X[b0 + e % nb + ld * (e / nb)];
      __syncthreads();
      v = slab;
      lv = nb;
    }
    for (int e = tid; e < nb * n; e += kThreads) {
      const int i = e % nb, k = e / nb, row = r0 + b0 + i;
      double2 acc = cz();
      const int last = min(row, steps - 1);  // v_l is zero above row l
#pragma unroll 4
      for (int l = 0; l <= last; ++l) {
        const double2 x = v[i + lv * l];
        cfma(acc, make_double2(-x.x, -x.y), t.Qs[l + (int64_t)steps * k]);
      }
      if (row == k) acc.x += 1.0;
      t.A[row + (int64_t)m * k] = acc;
    }
    __syncthreads();
  }
}

// mode products of several tensors, one thread per output as k_mp_single;
// blockIdx.y is the task
__global__ void __launch_bounds__(kThreads) k_mp_each(const MPTask* __restrict__ tasks) {
  mp_single(tasks[blockIdx.y]);
}

cudaError_t launch_mp_each(const MPTask* tasks, int n_tasks, int64_t max_outputs, cudaStream_t s) {
  if (n_tasks <= 0 || max_outputs <= 0) return cudaSuccess;
  k_mp_each<<<dim3((unsigned)((max_outputs + kThreads - 1) / kThreads), (unsigned)n_tasks), kThreads, 0, s>>>(tasks);
  return cudaGetLastError();
}

// CTAs per node: the most (a power of two, at most 16, or 8 where clusters of
// 16 do not fit) that leave every CTA at least 32 rows and the launch at most
// 152 CTAs.
cudaError_t launch_house_qr(const void* tasks, int n_tasks, int max_m, int max_n, cudaStream_t s) {
  if (n_tasks <= 0) return cudaSuccess;
  const int fixed = 5 * max_n + kThreads;  // shared elements beside the rows
  constexpr int kMaxSmem = 227 * 1024 - 4096;  // the static arrays take the rest
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kThreads);
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaError_t e = cudaFuncSetAttribute(k_house_qr, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_house_qr, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  int cl = 1;
  while (cl < 16 && (int64_t)2 * cl * n_tasks <= 152 && max_m >= 64 * cl) cl *= 2;
  for (;; cl /= 2) {
    const int64_t rp = (max_m + cl - 1) / cl;
    const int64_t in_smem = 16 * (fixed + (rp | 1) * max_n);
    const int slab = in_smem <= kMaxSmem;
    cfg.dynamicSmemBytes = (size_t)(slab ? in_smem : 16 * (fixed + (int64_t)kQrBuf * max_n));
    cfg.gridDim = dim3((unsigned)(n_tasks * cl));
    at[0].val.clusterDim.x = (unsigned)cl;
    int fit = 1;
    if (cl > 8) {
      if (cudaOccupancyMaxActiveClusters(&fit, k_house_qr, &cfg) != cudaSuccess) {
        cudaGetLastError();
        fit = 0;
      }
    }
    if (fit < 1) continue;
    return cudaLaunchKernelEx(&cfg, k_house_qr, static_cast<const QRTask*>(tasks), cl, slab);
  }
}

}  // namespace qt
