// Brute-force ground truth of the B200 Vamana hot path: the k <= 32 nearest base
// points of every query, distance then id (FP64 distances for float data, exact
// integers otherwise).
//
//   k_gt_prep  : squared norms; for float data the two BF16 halves of every row
//   k_gt_tc    : queries x base on the tensor cores (tcgen05), per-query
//                candidate lists from the accumulators
//   k_gt_merge : the lists of a query merged; float candidates get their FP64
//                distance here
//   k_gt_partial / k_gt_merge_parts : FP64 over every point, for the float
//                queries the screen cannot bound
//
// Every (query, point) value is one multiply-add and a comparison beside the
// product itself, so the work is a GEMM whose accumulators are consumed on
// chip.  A CTA keeps one tile of queries in shared memory and streams base
// tiles of 128 points; one thread issues the tcgen05.mma of a tile while the
// epilogue warps read the other TMEM buffer: thread r of a query tile owns
// query r (TMEM lane r), keeps its threshold in a register and appends the few
// values that pass to the query's list in global memory.  The (query tile, base
// tile) steps are split evenly over one CTA per SM.
//
// Integer data: one score per pair, 2 q.p - |p|^2 (L2) or q.p (MIPS), exact in
// 32 bits; the list keeps the k best.  Float data: rows are split x = hi + lo
// (two BF16 values, |x - hi - lo| <= 2^-17 |x|) and the score is hi.hi + hi.lo
// + lo.hi in FP32, whose distance from the true one is at most e (gt_error);
// the list keeps every value within 2 e of the k-th best, which holds the true
// k best, and only those get the FP64 distance of the definition.  A query
// whose list overflows, or whose bound is not finite, is computed in FP64
// against every point.
//
// Measured on B200, all kernels of a call: 10,000 x 1M x 128 uint8, k = 32: 144
// ms (mma.sync tiles of 16 queries a warp) -> 4.34 ms (norms 0.09, sample 0.47,
// thresholds 0.02, lists 3.68, merge 0.08); 1000 x 400k x 200 float inner product:
// 185 ms (FP64 on the CUDA cores, one row per lane) -> 1.17 ms (halves 0.16, sample
// 0.14, lists 0.77, merge 0.09).  What bounds it now: the epilogue (two
// instructions a value, and the lists), not the products (0.6 ms of the uint8
// call at the measured GEMM rate).
#include <cfloat>
#include <climits>
#include <cstdio>
#include <mutex>

#include <cuda.h>
#include <cuda_bf16.h>

#include "dd_common.cuh"
#include "kernel_util.cuh"
#include "kernels.cuh"
#include "prune_core.cuh"

namespace ddk {

// ============================================================ exact FP64 form
template <int MT>
__device__ __forceinline__ double exact_dist64(const uint8_t* q, const uint8_t* x, uint32_t d) {
  const float* a = (const float*)q;
  const float* b = (const float*)x;
  double acc = 0.0;
  for (uint32_t t = 0; t < d; t++) {
    if (MT == DD_L2) {
      double df = __dsub_rn((double)a[t], (double)__ldg(b + t));
      acc = __dadd_rn(acc, __dmul_rn(df, df));
    } else {
      acc = __dsub_rn(acc, __dmul_rn((double)a[t], (double)__ldg(b + t)));
    }
  }
  return acc;
}

// warp-distributed sorted top-k (k <= 32): lane i holds the i-th best (dist, id)
__device__ __forceinline__ void topk_insert(double& bd, uint32_t& bi, uint32_t k, double dv,
                                            uint32_t iv, bool cand) {
  const uint32_t lane = lane_id();
  uint32_t mask = __ballot_sync(0xffffffffu, cand);
  while (mask) {
    int src = __ffs(mask) - 1;
    mask &= mask - 1;
    double cd = __shfl_sync(0xffffffffu, dv, src);
    uint32_t ci = __shfl_sync(0xffffffffu, iv, src);
    double kd = __shfl_sync(0xffffffffu, bd, k - 1);
    uint32_t ki = __shfl_sync(0xffffffffu, bi, k - 1);
    if (!((cd < kd) || (cd == kd && ci < ki))) continue;
    bool before = (lane < k) && ((bd < cd) || (bd == cd && bi < ci));
    uint32_t pos = __popc(__ballot_sync(0xffffffffu, before));
    double ud = __shfl_up_sync(0xffffffffu, bd, 1);
    uint32_t ui = __shfl_up_sync(0xffffffffu, bi, 1);
    if (lane == pos) { bd = cd; bi = ci; }
    else if (lane > pos) { bd = ud; bi = ui; }
  }
}

// grid (blocks of 8 listed queries, chunks); each warp keeps a top-k of its chunk
template <int MT>
__global__ void __launch_bounds__(256) k_gt_partial(IndexView ix, const uint8_t* queries, uint64_t qstride,
                                                    const uint32_t* list, uint32_t count, uint32_t k,
                                                    uint32_t nchunks, double* part_d,
                                                    uint32_t* part_i) {
  __shared__ __align__(16) uint8_t qbuf[8][1024];
  const uint32_t wic = threadIdx.x >> 5, lane = lane_id();
  const uint64_t i = (uint64_t)blockIdx.x * 8 + wic;
  if (i >= count) return;
  load_vec(qbuf[wic], queries + (uint64_t)list[i] * qstride, r16((uint64_t)ix.d * 4));
  __syncwarp();
  const uint64_t chunk = (ix.n + nchunks - 1) / nchunks;
  const uint64_t c0 = (uint64_t)blockIdx.y * chunk;
  const uint64_t c1 = min(ix.n, c0 + chunk);
  double bd = INFINITY;
  uint32_t bi = DD_NONE;
  for (uint64_t base = c0; base < c1; base += 32) {
    uint64_t p = base + lane;
    double dv = INFINITY;
    uint32_t iv = DD_NONE;
    if (p < c1) {
      dv = exact_dist64<MT>(qbuf[wic], ix.points + p * ix.stride, ix.d);
      iv = (uint32_t)p;
    }
    double td = __shfl_sync(0xffffffffu, bd, k - 1);
    uint32_t ti = __shfl_sync(0xffffffffu, bi, k - 1);
    topk_insert(bd, bi, k, dv, iv, (dv < td) || (dv == td && iv < ti));
  }
  if (lane < k) {
    uint64_t o = (i * nchunks + blockIdx.y) * k + lane;
    part_d[o] = bd;
    part_i[o] = bi;
  }
}

__global__ void k_gt_merge_parts(const double* part_d, const uint32_t* part_i, const uint32_t* list,
                                 uint32_t count, uint32_t k, uint32_t nchunks, uint32_t* ids,
                                 float* dists) {
  const uint32_t lane = lane_id();
  const uint64_t i = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= count) return;
  double bd = INFINITY;
  uint32_t bi = DD_NONE;
  const uint64_t tot = (uint64_t)nchunks * k;
  for (uint64_t base = 0; base < tot; base += 32) {
    uint64_t e = base + lane;
    double dv = e < tot ? part_d[i * tot + e] : INFINITY;
    uint32_t iv = e < tot ? part_i[i * tot + e] : DD_NONE;
    double td = __shfl_sync(0xffffffffu, bd, k - 1);
    uint32_t ti = __shfl_sync(0xffffffffu, bi, k - 1);
    topk_insert(bd, bi, k, dv, iv, (dv < td) || (dv == td && iv < ti));
  }
  if (lane < k) {
    const uint64_t q = list[i];
    ids[q * k + lane] = bi;
    dists[q * k + lane] = (float)bd;
  }
}

// ============================================================ sizes
constexpr uint32_t kGtTile = 128;      // base points of a tile (accumulator columns)
constexpr uint32_t kGtBlockBytes = 128;             // bytes of a row in one k-block
constexpr uint32_t kGtTileBytes = kGtTile * kGtBlockBytes;
// entries of a query's list of one segment; a compaction leaves at most 8 fewer.
// The lists are in global memory (L2): appends are stores that nothing waits
// for, and with the sample's thresholds about 50 values come to a list, so that
// it is hardly ever compacted.  (In shared memory a list held 48: some warp
// compacted one in most steps, and the step's TMEM buffer waited for it: the
// lists of the uint8 call above took 4.3 ms instead of 3.7.)
constexpr uint32_t kGtCap = 128;
// |p|^2 of the rows past n, and the scores that no point lies below and no such
// row reaches (integer rows of 1024 bytes: scores above -2^27)
constexpr int kGtIntPad = 1 << 30, kGtIntNone = -(1 << 29);
constexpr float kGtFloatPad = 3e38f, kGtFloatNone = -1.5e38f;

struct GtShape {
  bool f32;
  uint32_t nkb;       // k-blocks of a row (float: hi and lo side by side)
  uint32_t ksteps;    // 32-byte mma steps of a row
  uint32_t mtiles;    // 128-query tiles a CTA holds
  uint32_t rows;      // queries of a CTA tile
  uint32_t stages;    // base tiles in flight
  uint32_t smem;
  uint32_t dp;        // float: elements of a converted row
  uint64_t slab, nslabs, qtiles, btiles, grid, per, segs;  // of a slab
  uint64_t groups, gtiles;  // sample groups (0: no sample) and their base tiles
};
// The first thresholds: the scores of kGtGroups groups of sampled base tiles
// are reduced to each group's largest, and the k-th largest of those is a
// score that at least k points reach.  A list that starts from nothing takes
// about k ln(points / k) values of its segment, one that starts from the
// sample's threshold a fraction of that, and lists are dearer than products.
// Whole host calls, 10,000 x 1M x 128 uint8 and 1000 x 400k x 200 float: without a
// sample 26.4 and 9.04 ms, with 1/16 of the base 9.2 and 1.22, 1/8 4.85 and 1.22,
// 1/5 4.74 and 1.24, 1/4 4.83 and 1.30.
// A base of few tiles is sampled whole, a group a tile (99 x 67,546 x 87 uint8
// 1.48 ms without the sample); one of fewer than k tiles is not.
constexpr uint32_t kGtGroups = 128, kGtSampleOf = 5;

static GtShape gt_shape(const IndexView& ix, uint64_t nq, uint32_t k, const GtLimits& lim) {
  GtShape s{};
  s.f32 = ix.dtype == DD_F32;
  s.dp = (ix.d + 15) & ~15u;
  const uint32_t row = s.f32 ? 4 * s.dp : (uint32_t)((ix.d + 31) & ~31u);  // bytes multiplied
  s.nkb = (row + kGtBlockBytes - 1) / kGtBlockBytes;
  s.ksteps = row / 32;
  // two query tiles share a base tile where the row is one k-block (the
  // epilogue of 128 queries would ask more of L2 than it gives)
  s.mtiles = (!s.f32 && s.nkb == 1) ? 2 : 1;
  s.rows = 128 * s.mtiles;
  // queries | the epilogue warps' norms; 1 KB is static (barriers)
  const uint32_t fixed = s.mtiles * s.nkb * kGtTileBytes + s.rows * 16;
  s.stages = std::min<uint32_t>(8, (226 * 1024 - fixed) / kGtTileBytes);
  s.smem = fixed + s.stages * kGtTileBytes;
  s.slab = s.f32 ? std::min<uint64_t>(ix.n, lim.slab) : ix.n;
  s.nslabs = (ix.n + s.slab - 1) / s.slab;
  s.qtiles = (nq + s.rows - 1) / s.rows;
  s.btiles = (s.slab + kGtTile - 1) / kGtTile;
  const uint64_t total = s.qtiles * s.btiles;
  s.grid = std::min<uint64_t>(lim.grid, total);
  s.per = (total + s.grid - 1) / s.grid;
  s.segs = (s.btiles - 1) / s.per + 2;
  s.groups = s.btiles >= k ? std::min<uint64_t>(kGtGroups, s.btiles) : 0;
  s.gtiles = std::max<uint64_t>(1, s.btiles / (kGtSampleOf * kGtGroups));
  return s;
}

// offsets of one device workspace
struct GtWork {
  uint64_t pnorm, qnorm, scal, over, over_list, gmax, thr0, cnt, ent_v, ent_i, bhalf, qhalf, total;
  uint64_t zero0, zero1;  // bytes [zero0, zero1) start as zeros
};

static GtWork gt_work(const IndexView& ix, uint64_t nq, const GtShape& s) {
  GtWork w{};
  uint64_t off = 0;
  auto take = [&](uint64_t bytes) {
    const uint64_t o = off;
    off += (bytes + 1023) & ~(uint64_t)1023;
    return o;
  };
  const uint64_t lists = s.nslabs * s.qtiles * s.segs * s.rows;
  w.zero0 = off;
  w.scal = take(64);  // [0] largest |p|^2 bits, [1] overflowed queries, [2] error bits
  w.over = take(4 * nq);
  w.cnt = take(4 * lists);
  w.gmax = take(s.groups ? 4ull * nq * kGtGroups : 0);
  w.zero1 = off;
  w.thr0 = take(4 * nq);
  w.over_list = take(4 * nq);
  w.qnorm = take(4 * nq);
  w.pnorm = take(4 * s.btiles * kGtTile);
  w.ent_v = take(4 * lists * kGtCap);
  w.ent_i = take(4 * lists * kGtCap);
  if (s.f32) {
    w.bhalf = take(2ull * s.slab * 2 * s.dp);
    w.qhalf = take(2ull * nq * 2 * s.dp);
  }
  w.total = off;
  return w;
}

uint64_t groundtruth_work_bytes(const IndexView& ix, uint64_t nq, uint32_t k, const GtLimits& lim) {
  return gt_work(ix, nq, gt_shape(ix, nq, k, lim)).total;
}

// ============================================================ preparation
// norms[i] of rows [0, n) (zeros for MIPS), the pad value up to npad; float
// rows also go to half[i] = hi[dp] | lo[dp] (BF16).  One warp a row.
template <int DT>
__global__ void __launch_bounds__(256) k_gt_prep(const uint8_t* rows, uint64_t stride, uint64_t n,
                                                 uint64_t npad, uint32_t d, uint32_t dp, bool l2,
                                                 bool is_base, void* norms, uint32_t* pmax,
                                                 __nv_bfloat16* half) {
  const uint32_t lane = lane_id();
  uint32_t best = 0;
  for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < npad;
       i += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    if (DT == DD_F32) {
      double acc = 0.0;
      if (i < n) {
        const float* r = (const float*)(rows + i * stride);
        __nv_bfloat16* h = half + i * 2 * dp;
        __nv_bfloat16* l = h + dp;
        for (uint32_t t = lane; t < dp; t += 32) {
          const float x = t < d ? __ldg(r + t) : 0.f;
          const __nv_bfloat16 b = __float2bfloat16_rn(x);
          h[t] = b;
          l[t] = __float2bfloat16_rn(__fsub_rn(x, __bfloat162float(b)));
          acc = fma((double)x, (double)x, acc);
        }
      }
      for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      const float f = (float)acc;
      // a base row's norm enters its score for L2 only; a query's bounds its error
      if (lane == 0)
        ((float*)norms)[i] = i >= n ? kGtFloatPad : (is_base && !l2 ? 0.f : f);
      if (i < n) best = max(best, __float_as_uint(f) & 0x7fffffffu);
    } else {
      uint32_t acc = 0;
      if (i < n && l2) {
        const uint4* r = (const uint4*)(rows + i * stride);
        for (uint32_t t = lane; t < (d + 15) / 16; t += 32) {
          const uint4 v = __ldg(r + t);
          if (DT == DD_U8) {
            acc = __dp4a(v.x, v.x, acc); acc = __dp4a(v.y, v.y, acc);
            acc = __dp4a(v.z, v.z, acc); acc = __dp4a(v.w, v.w, acc);
          } else {
            int a = (int)acc;
            a = __dp4a((int)v.x, (int)v.x, a); a = __dp4a((int)v.y, (int)v.y, a);
            a = __dp4a((int)v.z, (int)v.z, a); a = __dp4a((int)v.w, (int)v.w, a);
            acc = (uint32_t)a;
          }
        }
      }
      for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) ((int*)norms)[i] = i < n ? (int)acc : kGtIntPad;
    }
  }
  if (DT == DD_F32 && is_base && lane == 0 && best) atomicMax(pmax, best);
}

// How far the float score of any base point can lie from the exact one (of the
// query with norm qn, base norms up to P).  Rounding to 8 bits leaves |lo| <=
// 2^-8 |x| and, below the last bit of lo, a residue of at most 2^-17 |x|, so
// lo.lo' (2^-16) and two residues (2^-17 each) are left out of the three bf16
// products: 1.01 2^-15 of sum |q_i p_i| <= |q| |p|.  The tensor core adds at
// most 3 d products in FP32 (each addition 2^-23 of the absolute sum, which the
// splitting raises by less than 2%), |p|^2 and the final multiply-add round once
// each; 2% and an absolute term for subnormal products are added.  The FP64
// distances the result is ordered by are far inside that margin of the real ones.
// Measured over 1 to 256 dimensions and seven distributions of 5,000 to 400,000
// rows (Gaussian, positive, unit, clustered, far from 0, cancelling, of 24 binary
// orders): at most 0.65 of the bound at d = 1, 0.3 from d = 16 and 0.15 from 100.
__device__ __forceinline__ float gt_error(float qn2, float pn2, uint32_t d, bool l2) {
  const float q = sqrtf(qn2) * 1.0001f, P = sqrtf(pn2) * 1.0001f;
  const float c = 1.01f * 0x1p-15f + 1.02f * (float)(3 * d + 64) * 0x1p-23f;
  const float dot = q * P;
  const float e = l2 ? 2.f * dot * c + 0x1p-22f * (2.f * dot + P * P) : dot * (c + 0x1p-22f);
  const float room = 4.f * dot + 4.f * P * P;  // no score can overflow
  return room < 1e38f ? 1.02f * e + (float)d * 2e-37f * (1.f + q + P) : INFINITY;
}

// ============================================================ tcgen05 plumbing
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for a phase, for 2^32 cycles (about two seconds) at most: then the
// kernel's abort flag is set, every later wait returns at once, the loops run
// out and the host reads the error word.
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort) {
  if (mbar_try(bar, parity)) return;
  const long long t0 = clock64();
  while (!mbar_try(bar, parity)) {
    if (*abort) return;
    if (clock64() - t0 > (1ll << 32)) {
      *abort = 1u;
      return;
    }
  }
}
__device__ __forceinline__ void tma_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x,
                                         int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];" ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
// K-major operand in 128-byte swizzled rows: 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
template <bool F32>
__device__ __forceinline__ void umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if (F32)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t (&v)[32], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
        "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
        "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr));
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ============================================================ k_gt_tc
struct GtArgs {
  uint64_t nq, n;          // queries; base rows of this slab
  uint64_t id0;            // first base id of the slab
  uint32_t d, k;
  uint32_t nkb, ksteps, stages;
  uint32_t btiles, per, segs;
  uint64_t list0;          // first list row of this slab
  uint32_t idesc;
  const void* pnorm;
  const float* qnorm;      // float data
  const uint32_t* pmax;    // float data: bits of the largest |p|^2
  uint32_t* over;          // float data: queries the screen gave up
  uint32_t* cnt;
  uint32_t* ent_v;         // [list tile][kGtCap][rows]
  uint32_t* ent_i;
  uint32_t* err;
  // sample launch: tile i of the sample is base tile i * gstride, its group i / gtiles
  uint32_t gtiles, gstride;
  uint32_t* gmax;          // [nq][kGtGroups] gt_rank_bits of the groups' largest scores
  const uint32_t* thr0;    // first thresholds (null: none)
};

// Score order as unsigned integers: larger is better
template <bool F32>
__device__ __forceinline__ uint32_t gt_rank_bits(uint32_t v) {
  if (!F32) return v ^ 0x80000000u;
  return (v & 0x80000000u) ? ~v : v | 0x80000000u;
}

template <bool F32>
__device__ __forceinline__ uint32_t gt_from_rank(uint32_t b) {
  if (!F32) return b ^ 0x80000000u;
  return (b & 0x80000000u) ? b & 0x7fffffffu : ~b;
}

// the threshold that keeps every point that may be among the k best when k
// points reach `kth`: to be beaten (int) or reached (float, bound 2 e = err2)
template <bool F32>
__device__ __forceinline__ uint32_t gt_threshold(uint32_t kth, float err2) {
  if (!F32) return kth;
  const float f = __uint_as_float(kth);
  return __float_as_uint(f - (err2 + fabsf(f) * 0x1p-22f));
}

// SAMPLE: only the largest score of every group of sampled tiles
template <bool F32, int MT, int MTILES, bool SAMPLE>
__global__ void __launch_bounds__(MTILES * 128 + 64, 1)
    k_gt_tc(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap bmap,
            GtArgs g) {
  constexpr uint32_t ROWS = 128 * MTILES;
  constexpr uint32_t EW = 4 * MTILES;  // epilogue warps; then the producer, then the issuer
  constexpr int KB = F32 ? 64 : 128;  // elements of a k-block
  constexpr uint32_t FULL = 0xffffffffu;
  extern __shared__ __align__(1024) uint8_t smem_gt[];
  __shared__ __align__(8) uint64_t bars[2 + 8 + 8 + 4];
  __shared__ uint32_t s_tmem, s_abort;
  const uint32_t tid = threadIdx.x, wid = tid >> 5, lane = lane_id();
  // the swizzle pattern follows the address: tiles start on 1024 bytes
  uint8_t* base = smem_gt;
  if (smem_u32(base) & 1023u) {
    if (tid == 0) dd_set_error(g.err, DD_ETIMEOUT);
    return;
  }
  const uint32_t qs = smem_u32(base);                                   // query blocks
  const uint32_t bs = qs + MTILES * g.nkb * kGtTileBytes;               // base stages
  uint8_t* after = base + (MTILES * g.nkb + g.stages) * kGtTileBytes;
  uint32_t* pn_s = (uint32_t*)after;         // [EW][128] norms of the current tile
  const uint32_t b0 = smem_u32(bars);
  auto bar_q = [&](uint32_t i) { return b0 + 8 * i; };            // 0 loaded, 1 free
  auto bar_full = [&](uint32_t s) { return b0 + 8 * (2 + s); };
  auto bar_empty = [&](uint32_t s) { return b0 + 8 * (10 + s); };
  auto bar_tfull = [&](uint32_t b) { return b0 + 8 * (18 + b); };
  auto bar_tempty = [&](uint32_t b) { return b0 + 8 * (20 + b); };
  if (tid == 0) {
    mbar_init(bar_q(0), 1);
    mbar_init(bar_q(1), 1);
    for (uint32_t s = 0; s < g.stages; s++) {
      mbar_init(bar_full(s), 1);
      mbar_init(bar_empty(s), 1);
    }
    for (uint32_t b = 0; b < 2; b++) {
      mbar_init(bar_tfull(b), 1);
      mbar_init(bar_tempty(b), EW);
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  constexpr uint32_t TCOLS = 256 * MTILES;  // two buffers of MTILES x 128 columns
  if (wid == EW + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_tmem)),
                 "r"(TCOLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  volatile uint32_t* abort = &s_abort;
  const uint64_t t0 = (uint64_t)blockIdx.x * g.per;
  const uint64_t t1 = min(t0 + g.per, (uint64_t)((g.nq + ROWS - 1) / ROWS) * g.btiles);
  const uint32_t nt = t1 > t0 ? (uint32_t)(t1 - t0) : 0u;  // this CTA's steps
  // every role walks (query tile, base tile) from here
  uint32_t qt = (uint32_t)(t0 / g.btiles), bt = (uint32_t)(t0 % g.btiles);
  auto next_step = [&]() {
    if (++bt == g.btiles) {
      bt = 0;
      qt++;
    }
  };

  if (wid == EW) {
    // ---- producer: one thread
    if (lane == 0) {
      uint32_t st = 0, ph = 0, nseg = 0;
      for (uint32_t t = 0; t < nt; t++, next_step()) {
        if (t == 0 || bt == 0) {
          // a new query tile: once the products of the last one are done
          if (nseg) mbar_wait(bar_q(1), (nseg - 1) & 1u, abort);
          mbar_expect(bar_q(0), MTILES * g.nkb * kGtTileBytes);
          for (uint32_t m = 0; m < MTILES; m++)
            for (uint32_t kb = 0; kb < g.nkb; kb++)
              tma_tile(qs + (m * g.nkb + kb) * kGtTileBytes, &qmap, bar_q(0), (int)kb * KB,
                       (int)(qt * ROWS + 128 * m));
          nseg++;
        }
        for (uint32_t kb = 0; kb < g.nkb; kb++) {
          mbar_wait(bar_empty(st), ph ^ 1u, abort);
          mbar_expect(bar_full(st), kGtTileBytes);
          tma_tile(bs + st * kGtTileBytes, &bmap, bar_full(st), (int)kb * KB,
                   (int)((SAMPLE ? bt * g.gstride : bt) * kGtTile));
          if (++st == g.stages) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
    }
  } else if (wid == EW + 1) {
    // ---- issuer: one thread
    if (lane == 0) {
      uint32_t st = 0, ph = 0, nseg = 0, buf = 0, tph = 0;
      // descriptors count 16-byte units: a k-step is 2, a tile 1024
      constexpr uint32_t TILE16 = kGtTileBytes / 16;
      const uint64_t qd0 = umma_desc(qs), bd0 = umma_desc(bs);
      const uint32_t half = g.ksteps / 2;  // float: steps of hi, then of lo
      for (uint32_t t = 0; t < nt; t++, next_step()) {
        if (t == 0 || bt == 0) {
          mbar_wait(bar_q(0), nseg & 1u, abort);
          nseg++;
        }
        mbar_wait(bar_tempty(buf), tph ^ 1u, abort);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem + buf * MTILES * 128;
        uint32_t left = g.ksteps, i = 0;
        for (uint32_t kb = 0; kb < g.nkb; kb++) {
          mbar_wait(bar_full(st), ph, abort);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t bd = bd0 + st * TILE16;
#pragma unroll
          for (uint32_t s = 0; s < 4; s++) {
            if (s < left) {
              if (!F32) {
                const uint64_t ad = qd0 + kb * TILE16 + 2 * s;
#pragma unroll
                for (uint32_t m = 0; m < MTILES; m++)
                  umma<F32>(acc + m * 128, ad + m * g.nkb * TILE16, bd + 2 * s, g.idesc,
                            (kb | s) ? 1u : 0u);
              } else {
                // base hi meets the queries' hi and lo, base lo their hi
                const uint32_t j = i < half ? i : i - half, j2 = i + half;
                umma<F32>(acc, qd0 + (j >> 2) * TILE16 + 2 * (j & 3), bd + 2 * s, g.idesc,
                          (kb | s) ? 1u : 0u);
                if (i < half)
                  umma<F32>(acc, qd0 + (j2 >> 2) * TILE16 + 2 * (j2 & 3), bd + 2 * s, g.idesc, 1u);
                i++;
              }
            }
          }
          left -= min(left, 4u);
          umma_commit(bar_empty(st));
          if (++st == g.stages) {
            st = 0;
            ph ^= 1u;
          }
        }
        umma_commit(bar_tfull(buf));
        if (t + 1 == nt || bt + 1 == g.btiles) umma_commit(bar_q(1));
        buf ^= 1u;
        if (buf == 0) tph ^= 1u;
      }
    }
  } else {
    // ---- epilogue: one thread per query
    const uint32_t m = wid >> 2;             // query tile of this warp
    const uint32_t r = tid;                  // list row (m * 128 + TMEM lane)
    const uint32_t tl = (wid & 3u) * 32u;    // this warp's TMEM lanes
    uint32_t* pn_w = pn_s + wid * 128;
    uint32_t buf = 0, tph = 0;
    uint32_t cnt = 0;
    uint64_t tile = 0;          // the segment's list tile
    uint32_t *lv = nullptr, *li = nullptr;  // its scores and ids, [kGtCap][ROWS]
    uint32_t thr = 0;       // the score a value must beat (int) or reach (float), as bits
    float err2 = 0.f;
    bool dead = true;       // no query, or given up
    auto passes = [&](uint32_t v) -> bool {
      return F32 ? __uint_as_float(v) >= __uint_as_float(thr) : (int)v > (int)thr;
    };
    // the rows of this warp in `rows`: sorted, the k best (float: and all
    // within 2 e of the k-th) kept, the threshold renewed
    auto compact = [&](uint32_t rows) {
      for (; rows; rows &= rows - 1) {
        const uint32_t src = __ffs(rows) - 1;
        const uint32_t rr = wid * 32 + src;
        const uint32_t c = __shfl_sync(FULL, cnt, src);
        const float e2 = __shfl_sync(FULL, err2, src);
        constexpr int PER = kGtCap / 32;
        uint32_t v[PER], id[PER], rk[PER];
#pragma unroll
        for (int j = 0; j < PER; j++) {
          const uint32_t e = lane + 32 * j;
          v[j] = e < c ? lv[e * ROWS + rr] : 0u;
          id[j] = e < c ? li[e * ROWS + rr] : 0u;
          rk[j] = 0;
        }
#pragma unroll 4
        for (uint32_t e = 0; e < c; e++) {
          const uint32_t ov = lv[e * ROWS + rr], oi = li[e * ROWS + rr];
#pragma unroll
          for (int j = 0; j < PER; j++) {
            const uint32_t a = gt_rank_bits<F32>(ov), b = gt_rank_bits<F32>(v[j]);
            rk[j] += (a > b || (a == b && oi < id[j])) ? 1u : 0u;
          }
        }
        uint32_t kth = 0;
        bool mine = false;
#pragma unroll
        for (int j = 0; j < PER; j++)
          if (lane + 32 * j < c && rk[j] == g.k - 1) {
            mine = true;
            kth = v[j];
          }
        const uint32_t who = __ballot_sync(FULL, mine);
        uint32_t nthr = F32 ? __float_as_uint(kGtFloatNone) : (uint32_t)kGtIntNone;
        if (who) {
          kth = __shfl_sync(FULL, kth, __ffs(who) - 1);
          nthr = gt_threshold<F32>(kth, e2);
        }
        __syncwarp();
        uint32_t kept = 0;
#pragma unroll
        for (int j = 0; j < PER; j++) {
          const bool keep = lane + 32 * j < c &&
                            (F32 ? __uint_as_float(v[j]) >= __uint_as_float(nthr) : rk[j] < g.k);
          if (keep) {
            lv[rk[j] * ROWS + rr] = v[j];
            li[rk[j] * ROWS + rr] = id[j];
          }
          kept += __popc(__ballot_sync(FULL, keep));
        }
        __syncwarp();
        if (lane == src) {
          cnt = kept;
          if (who) thr = F32 ? __float_as_uint(fmaxf(__uint_as_float(thr), __uint_as_float(nthr)))
                             : (uint32_t)max((int)thr, (int)nthr);
          if (kept > kGtCap - 8) {  // float: too many within the bound
            dead = true;
            cnt = 0;
          }
          if (dead) thr = F32 ? __float_as_uint(INFINITY) : 0x7fffffffu;
        }
      }
    };
    const uint4* pnorm4 = (const uint4*)g.pnorm;
    auto norms_of = [&](uint32_t b) {
      return __ldg(pnorm4 + (uint64_t)(SAMPLE ? b * g.gstride : b) * 32 + lane);
    };
    uint4 pn_next = nt ? norms_of(bt) : make_uint4(0, 0, 0, 0);
    uint32_t gbest = 0;  // sample: largest score so far of the current group (rank bits)
    for (uint32_t t = 0; t < nt; t++, next_step()) {
      const uint64_t q = (uint64_t)qt * ROWS + r;
      if (t == 0 || bt == 0) {
        const uint64_t seg = blockIdx.x - ((uint64_t)qt * g.btiles) / g.per;
        tile = g.list0 / ROWS + qt * g.segs + seg;
        lv = g.ent_v + tile * kGtCap * ROWS;
        li = g.ent_i + tile * kGtCap * ROWS;
        cnt = 0;
        dead = q >= g.nq;
        if (F32 && !dead) {
          err2 = 2.f * gt_error(g.qnorm[q], __uint_as_float(*g.pmax), g.d, MT == DD_L2);
          if (!(err2 < INFINITY)) dead = true;
        }
        thr = F32 ? __float_as_uint(dead ? INFINITY : kGtFloatNone)
                  : (dead ? 0x7fffffffu : (uint32_t)kGtIntNone);
        if (!SAMPLE && !dead && g.thr0) thr = g.thr0[q];
      }
      __syncwarp();
      *(uint4*)(pn_w + 4 * lane) = pn_next;
      if (t + 1 < nt) pn_next = norms_of(bt + 1 == g.btiles ? 0 : bt + 1);
      __syncwarp();
      mbar_wait(bar_tfull(buf), tph, abort);
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t id_t = (uint32_t)g.id0 + bt * kGtTile;
      const uint32_t acc = tmem + (buf * MTILES + m) * 128 + (tl << 16);
      // one 32-column block is in flight while the other is looked at
      uint32_t va[32], vb[32];
      auto look = [&](uint32_t (&v)[32], uint32_t cb) {
#pragma unroll
        for (int h = 0; h < 4; h++) {
          bool any;
          const uint4 pa = *(const uint4*)(pn_w + 32 * cb + 8 * h);
          const uint4 pb = *(const uint4*)(pn_w + 32 * cb + 8 * h + 4);
          const uint32_t pn8[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
          if (F32) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const float pn = __uint_as_float(pn8[j]);
              const float s = __fmaf_rn(MT == DD_L2 ? 2.f : 1.f, __uint_as_float(v[8 * h + j]), -pn);
              v[8 * h + j] = __float_as_uint(s);
              mx = fmaxf(mx, s);
            }
            any = mx >= __uint_as_float(thr);
            if (SAMPLE) gbest = max(gbest, gt_rank_bits<F32>(__float_as_uint(mx)));
          } else {
            int mx = INT_MIN;
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const int s = (MT == DD_L2 ? 2 : 1) * (int)v[8 * h + j] - (int)pn8[j];
              v[8 * h + j] = (uint32_t)s;
              mx = max(mx, s);
            }
            any = mx > (int)thr;
            if (SAMPLE) gbest = max(gbest, gt_rank_bits<F32>((uint32_t)mx));
          }
          if (!SAMPLE && __any_sync(FULL, any)) {
#pragma unroll
            for (int j = 0; j < 8; j++)
              if (passes(v[8 * h + j])) {
                lv[cnt * ROWS + r] = v[8 * h + j];
                li[cnt * ROWS + r] = id_t + 32 * cb + 8 * h + j;
                cnt++;
              }
            __syncwarp();
            compact(__ballot_sync(FULL, cnt > kGtCap - 8));
          }
        }
      };
      tmem_ld32(va, acc);
      tmem_wait_ld();
#pragma unroll 1
      for (uint32_t cb = 0; cb < 4; cb += 2) {
        tmem_ld32(vb, acc + 32 * cb + 32);
        look(va, cb);
        tmem_wait_ld();
        if (cb == 0) tmem_ld32(va, acc + 64);
        look(vb, cb + 1);
        if (cb == 0) tmem_wait_ld();
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_tempty(buf));
      buf ^= 1u;
      if (buf == 0) tph ^= 1u;
      if (SAMPLE) {
        if (t + 1 == nt || (bt + 1) % g.gtiles == 0) {
          if (q < g.nq) atomicMax(&g.gmax[q * kGtGroups + bt / g.gtiles], gbest);
          gbest = 0;
        }
      } else if (t + 1 == nt || bt + 1 == g.btiles) {
        g.cnt[tile * ROWS + r] = cnt;
        if (F32 && dead && q < g.nq) g.over[q] = 1u;
        __syncwarp();
      }
    }
  }
  __syncthreads();
  if (s_abort && tid == 0) dd_set_error(g.err, DD_ETIMEOUT);
  if (s_abort)  // copies and products still in flight end before the memory is given up
    for (int i = 0; i < 1000; i++) __nanosleep(2000);
  __syncwarp();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (wid == EW + 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS));
}

// One warp per query: the k-th largest of its groups' largest scores
template <bool F32, int MT>
__global__ void __launch_bounds__(256) k_gt_first(const uint32_t* gmax, uint64_t nq, uint32_t k,
                                                  const float* qnorm, const uint32_t* pmax,
                                                  uint32_t d, uint32_t* thr0) {
  const uint32_t lane = lane_id();
  const uint64_t q = (uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (q >= nq) return;
  constexpr int PER = kGtGroups / 32;
  uint32_t v[PER], above[PER];
#pragma unroll
  for (int j = 0; j < PER; j++) {
    v[j] = gmax[q * kGtGroups + 32 * j + lane];
    above[j] = 0;
  }
#pragma unroll
  for (int j = 0; j < PER; j++)
    for (int s = 0; s < 32; s++) {
      const uint32_t o = __shfl_sync(0xffffffffu, v[j], s);
#pragma unroll
      for (int i = 0; i < PER; i++) above[i] += o > v[i] ? 1u : 0u;
    }
  // the smallest value with fewer than k above it
  uint32_t best = 0xffffffffu;
#pragma unroll
  for (int j = 0; j < PER; j++)
    if (above[j] < k) best = min(best, v[j]);
  best = __reduce_min_sync(0xffffffffu, best);
  if (lane == 0) {
    const uint32_t kth = gt_from_rank<F32>(best);
    if (F32)
      thr0[q] = gt_threshold<F32>(
          kth, 2.f * gt_error(qnorm[q], __uint_as_float(*pmax), d, MT == DD_L2));
    else
      thr0[q] = kth - 1u;  // a score must beat it
  }
}

// One warp per query: the lists of all slabs and segments.  Integer scores give
// the distance at once.  Float candidates: the k-th best score of all lists
// first, then the FP64 distance of those within 2 e of it, which also shows how far
// their scores were off: gt_error counts on the tensor core's additions, whose
// precision is not documented, so a query with one score beyond e goes to the FP64
// form.
template <bool F32, int MT>
__global__ void __launch_bounds__(256) k_gt_merge(IndexView ix, const uint8_t* queries,
                                                  uint64_t qstride, uint64_t nq, uint32_t k,
                                                  uint32_t rows, uint32_t segs, uint64_t nslabs,
                                                  uint64_t qtiles, const uint32_t* cnt,
                                                  const uint32_t* ent_v, const uint32_t* ent_i,
                                                  const void* qnorm, const uint32_t* over,
                                                  uint32_t* scal, uint32_t* over_list,
                                                  uint32_t* ids, float* dists) {
  __shared__ __align__(16) uint8_t qbuf[8][1024];
  const uint32_t lane = lane_id(), wic = threadIdx.x >> 5;
  const uint64_t q = (uint64_t)blockIdx.x * 8 + wic;
  if (q >= nq) return;
  if (F32) {
    if (over[q]) {
      if (lane == 0) over_list[atomicAdd(&scal[1], 1u)] = (uint32_t)q;
      return;
    }
    load_vec(qbuf[wic], queries + q * qstride, r16((uint64_t)ix.d * 4));
    __syncwarp();
  }
  const uint64_t qt = q / rows, r = q % rows;
  const uint64_t nt = nslabs * segs;  // list i: slab i / segs, segment i % segs
  auto tile_of = [&](uint64_t i) { return ((i / segs) * qtiles + qt) * segs + i % segs; };
  double bd = INFINITY;
  uint32_t bi = DD_NONE;
  float cut = -INFINITY;
  float err = 0.f;   // float data: how far a score may be from the exact one
  double qn64 = 0.0; // L2: |q|^2, which the exact score is relative to
  bool off = false;  // a score was farther from it
  if (F32) {
    // lane i: the i-th best score (as its negative, ascending)
    double sd = INFINITY;
    uint32_t si = DD_NONE;
    for (uint64_t i = 0; i < nt; i++) {
      const uint64_t tile = tile_of(i);
      const uint32_t c = cnt[tile * rows + r];
      for (uint32_t b = 0; b < c; b += 32) {
        const uint32_t e = b + lane;
        const double v =
            e < c ? -(double)__uint_as_float(ent_v[(tile * kGtCap + e) * rows + r]) : INFINITY;
        const double td = __shfl_sync(0xffffffffu, sd, k - 1);
        topk_insert(sd, si, k, v, e, v < td);
      }
    }
    const double kth = __shfl_sync(0xffffffffu, sd, k - 1);
    err = gt_error(((const float*)qnorm)[q], __uint_as_float(scal[0]), ix.d, MT == DD_L2);
    if (kth < INFINITY)
      cut = __uint_as_float(gt_threshold<true>(__float_as_uint((float)-kth), 2.f * err));
    if (MT == DD_L2) {
      for (uint32_t t = lane; t < ix.d; t += 32) {
        const double x = (double)((const float*)qbuf[wic])[t];
        qn64 = fma(x, x, qn64);
      }
      for (int o = 16; o; o >>= 1) qn64 += __shfl_xor_sync(0xffffffffu, qn64, o);
    }
  }
  // pending candidates, one per lane, evaluated when 32 are there
  uint32_t have = 0, pend = DD_NONE;
  float pscore = 0.f;
  auto evaluate = [&]() {
    const bool on = lane < have;
    const double dv = on ? exact_dist64<MT>(qbuf[wic], ix.points + (uint64_t)pend * ix.stride, ix.d)
                         : INFINITY;
    const uint32_t iv = on ? pend : DD_NONE;
    const double exact = MT == DD_L2 ? qn64 - dv : -dv;
    off |= on && !(fabs((double)pscore - exact) <= (double)err);
    const double td = __shfl_sync(0xffffffffu, bd, k - 1);
    const uint32_t ti = __shfl_sync(0xffffffffu, bi, k - 1);
    topk_insert(bd, bi, k, dv, iv, (dv < td) || (dv == td && iv < ti));
    have = 0;
  };
  for (uint64_t i = 0; i < nt; i++) {
    const uint64_t tile = tile_of(i);
    const uint32_t c = cnt[tile * rows + r];
    for (uint32_t b = 0; b < c; b += 32) {
      const uint32_t e = b + lane;
      const uint32_t v = e < c ? ent_v[(tile * kGtCap + e) * rows + r] : 0u;
      const uint32_t iv = e < c ? ent_i[(tile * kGtCap + e) * rows + r] : DD_NONE;
      if (F32) {
        uint32_t m = __ballot_sync(0xffffffffu, e < c && __uint_as_float(v) >= cut);
        for (; m; m &= m - 1) {
          const uint32_t id = __shfl_sync(0xffffffffu, iv, __ffs(m) - 1);
          const uint32_t sc = __shfl_sync(0xffffffffu, v, __ffs(m) - 1);
          if (lane == have) {
            pend = id;
            pscore = __uint_as_float(sc);
          }
          if (++have == 32) evaluate();
        }
      } else {
        const double dv =
            e < c ? (double)(MT == DD_L2 ? ((const int*)qnorm)[q] - (int)v : -(int)v) : INFINITY;
        const double td = __shfl_sync(0xffffffffu, bd, k - 1);
        const uint32_t ti = __shfl_sync(0xffffffffu, bi, k - 1);
        topk_insert(bd, bi, k, dv, iv, (dv < td) || (dv == td && iv < ti));
      }
    }
  }
  if (F32 && have) evaluate();
  if (F32 && __any_sync(0xffffffffu, off)) {  // the bound does not hold: FP64 over every point
    if (lane == 0) over_list[atomicAdd(&scal[1], 1u)] = (uint32_t)q;
    return;
  }
  if (lane < k) {
    ids[q * k + lane] = bi;
    dists[q * k + lane] = (float)bd;
  }
}

// ============================================================ host side
typedef CUresult (*encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                              const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static encode_fn tensor_map_encoder() {
  static std::mutex mu;
  static encode_fn fn = nullptr;
  std::lock_guard<std::mutex> lk(mu);
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
        qr == cudaDriverEntryPointSuccess)
      fn = (encode_fn)p;
  }
  return fn;
}

// rows of `row_elems` elements; boxes of 128 rows x 128 bytes, swizzled; what
// lies outside reads as zeros
static bool gt_tensor_map(CUtensorMap* m, bool f32, const void* p, uint64_t row_elems, uint64_t rows,
                          uint64_t row_bytes) {
  encode_fn enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dim[2] = {row_elems, rows};
  const cuuint64_t str[1] = {row_bytes};
  const cuuint32_t box[2] = {f32 ? 64u : 128u, kGtTile}, es[2] = {1, 1};
  return enc(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2,
             const_cast<void*>(p), dim, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool F32, int MT, int MTILES>
static void gt_launch(const GtShape& s, const CUtensorMap& qm, const CUtensorMap& bm, GtArgs g,
                      uint32_t* thr0, int max_grid, cudaStream_t st) {
  if (s.groups && g.id0 == 0) {  // the first slab's sample serves all slabs
    GtArgs a = g;
    a.gtiles = (uint32_t)s.gtiles;
    a.btiles = (uint32_t)(s.groups * s.gtiles);
    a.gstride = (uint32_t)(s.btiles / a.btiles);
    const uint64_t total = s.qtiles * a.btiles, grid = std::min<uint64_t>(max_grid, total);
    a.per = (uint32_t)((total + grid - 1) / grid);
    set_smem(k_gt_tc<F32, MT, MTILES, true>, s.smem);
    k_gt_tc<F32, MT, MTILES, true><<<(unsigned)grid, MTILES * 128 + 64, s.smem, st>>>(qm, bm, a);
    k_gt_first<F32, MT><<<(unsigned)((g.nq + 7) / 8), 256, 0, st>>>(g.gmax, g.nq, g.k, g.qnorm,
                                                                    g.pmax, g.d, thr0);
  }
  g.thr0 = s.groups ? thr0 : nullptr;
  set_smem(k_gt_tc<F32, MT, MTILES, false>, s.smem);
  k_gt_tc<F32, MT, MTILES, false><<<(unsigned)s.grid, MTILES * 128 + 64, s.smem, st>>>(qm, bm, g);
}

// queries: nq device rows, qstride bytes apart (a multiple of 64), zero padded.
// work: groundtruth_work_bytes.  (*over)[0] (device, after the stream has run): how
// many queries launch_groundtruth_exact must still compute; (*over)[1]: the
// error bits of these launches (the index's word keeps what other calls left).
bool launch_groundtruth(const IndexView& ix, const uint8_t* queries, uint64_t qstride, uint64_t nq,
                        uint32_t k, uint32_t* ids, float* dists, uint8_t* work, const GtLimits& lim,
                        cudaStream_t st, uint32_t** over) {
  const GtShape s = gt_shape(ix, nq, k, lim);
  const GtWork w = gt_work(ix, nq, s);
  const bool l2 = ix.metric == DD_L2;
  cudaMemsetAsync(work + w.zero0, 0, w.zero1 - w.zero0, st);
  uint32_t* scal = (uint32_t*)(work + w.scal);
  *over = scal + 1;
  const int qgrid = (int)std::min<uint64_t>((nq + 7) / 8, 148 * 8);
  const int bgrid = (int)std::min<uint64_t>((s.btiles * kGtTile + 7) / 8, 148 * 8);
  CUtensorMap qm, bm;
  GtArgs g{};
  g.nq = nq;
  g.d = ix.d;
  g.k = k;
  g.nkb = s.nkb;
  g.ksteps = s.ksteps;
  g.stages = s.stages;
  g.btiles = (uint32_t)s.btiles;
  g.per = (uint32_t)s.per;
  g.segs = (uint32_t)s.segs;
  g.pnorm = work + w.pnorm;
  g.qnorm = (const float*)(work + w.qnorm);
  g.pmax = scal;
  g.over = (uint32_t*)(work + w.over);
  g.cnt = (uint32_t*)(work + w.cnt);
  g.ent_v = (uint32_t*)(work + w.ent_v);
  g.ent_i = (uint32_t*)(work + w.ent_i);
  g.err = scal + 2;
  g.gmax = (uint32_t*)(work + w.gmax);
  uint32_t* thr0 = (uint32_t*)(work + w.thr0);
  const uint32_t shape_bits = ((kGtTile >> 3) << 17) | ((128u >> 4) << 24);
  auto* bhalf = (__nv_bfloat16*)(work + w.bhalf);
  auto* qhalf = (__nv_bfloat16*)(work + w.qhalf);
  if (s.f32) {
    g.idesc = (1u << 4) | (1u << 7) | (1u << 10) | shape_bits;  // bf16 x bf16 -> f32
    k_gt_prep<DD_F32><<<qgrid, 256, 0, st>>>(queries, qstride, nq, nq, ix.d, s.dp, l2, false,
                                             work + w.qnorm, nullptr, qhalf);
    if (!gt_tensor_map(&qm, true, qhalf, 2 * s.dp, nq, 4ull * s.dp)) return false;
  } else {
    const uint32_t sg = ix.dtype == DD_I8 ? 1u : 0u;
    g.idesc = (2u << 4) | (sg << 7) | (sg << 10) | shape_bits;  // s8/u8 -> s32
    if (ix.dtype == DD_I8)
      k_gt_prep<DD_I8><<<qgrid, 256, 0, st>>>(queries, qstride, nq, nq, ix.d, 0, l2, false,
                                              work + w.qnorm, nullptr, nullptr);
    else
      k_gt_prep<DD_U8><<<qgrid, 256, 0, st>>>(queries, qstride, nq, nq, ix.d, 0, l2, false,
                                              work + w.qnorm, nullptr, nullptr);
    if (!gt_tensor_map(&qm, false, queries, qstride, nq, qstride)) return false;
  }
  if (s.f32)  // the bound needs the largest norm of all slabs
    for (uint64_t sl = 0; sl + 1 < s.nslabs; sl++)
      k_gt_prep<DD_F32><<<bgrid, 256, 0, st>>>(ix.points + (sl + 1) * s.slab * ix.stride, ix.stride,
                                               std::min<uint64_t>(s.slab, ix.n - (sl + 1) * s.slab),
                                               std::min<uint64_t>(s.slab, ix.n - (sl + 1) * s.slab),
                                               ix.d, s.dp, l2, true, work + w.pnorm, scal, bhalf);
  for (uint64_t sl = 0; sl < s.nslabs; sl++) {
    const uint64_t first = sl * s.slab, rows = std::min<uint64_t>(s.slab, ix.n - first);
    const uint8_t* pts = ix.points + first * ix.stride;
    g.n = rows;
    g.id0 = first;
    g.list0 = sl * s.qtiles * s.segs * s.rows;
    const uint64_t npad = s.btiles * kGtTile;
    if (s.f32) {
      k_gt_prep<DD_F32><<<bgrid, 256, 0, st>>>(pts, ix.stride, rows, npad, ix.d, s.dp, l2, true,
                                               work + w.pnorm, scal, bhalf);
      if (!gt_tensor_map(&bm, true, bhalf, 2 * s.dp, rows, 4ull * s.dp)) return false;
      if (l2) gt_launch<true, DD_L2, 1>(s, qm, bm, g, thr0, lim.grid, st);
      else gt_launch<true, DD_MIPS, 1>(s, qm, bm, g, thr0, lim.grid, st);
    } else {
      if (ix.dtype == DD_I8)
        k_gt_prep<DD_I8><<<bgrid, 256, 0, st>>>(pts, ix.stride, rows, npad, ix.d, 0, l2, true,
                                                work + w.pnorm, nullptr, nullptr);
      else
        k_gt_prep<DD_U8><<<bgrid, 256, 0, st>>>(pts, ix.stride, rows, npad, ix.d, 0, l2, true,
                                                work + w.pnorm, nullptr, nullptr);
      if (!gt_tensor_map(&bm, false, pts, ix.stride, rows, ix.stride)) return false;
      if (s.mtiles == 2) {
        if (l2) gt_launch<false, DD_L2, 2>(s, qm, bm, g, thr0, lim.grid, st);
        else gt_launch<false, DD_MIPS, 2>(s, qm, bm, g, thr0, lim.grid, st);
      } else {
        if (l2) gt_launch<false, DD_L2, 1>(s, qm, bm, g, thr0, lim.grid, st);
        else gt_launch<false, DD_MIPS, 1>(s, qm, bm, g, thr0, lim.grid, st);
      }
    }
  }
  const unsigned mgrid = (unsigned)((nq + 7) / 8);
#define MERGE(F, M)                                                                            \
  k_gt_merge<F, M><<<mgrid, 256, 0, st>>>(ix, queries, qstride, nq, k, s.rows, (uint32_t)s.segs, \
                                          s.nslabs, s.qtiles, g.cnt, g.ent_v, g.ent_i, g.qnorm, \
                                          g.over, scal, (uint32_t*)(work + w.over_list), ids,  \
                                          dists);
  if (s.f32 && l2) { MERGE(true, DD_L2) }
  else if (s.f32) { MERGE(true, DD_MIPS) }
  else if (l2) { MERGE(false, DD_L2) }
  else { MERGE(false, DD_MIPS) }
#undef MERGE
  return true;
}

uint32_t groundtruth_exact_chunks(const IndexView& ix) {
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(256, ix.n / 4096));
}

// FP64 over every point for `count` queries of the screen's overflow list,
// from entry `first`; parts: count x chunks x k doubles, then as many ids
void launch_groundtruth_exact(const IndexView& ix, const uint8_t* queries, uint64_t qstride,
                              uint64_t nq, uint32_t first, uint32_t count, uint32_t k,
                              uint32_t* ids, float* dists, const uint8_t* work,
                              const GtLimits& lim, uint8_t* parts, cudaStream_t st) {
  const GtWork w = gt_work(ix, nq, gt_shape(ix, nq, k, lim));
  const uint32_t* list = (const uint32_t*)(work + w.over_list) + first;
  const uint32_t nchunks = groundtruth_exact_chunks(ix);
  double* pd = (double*)parts;
  uint32_t* pi = (uint32_t*)(pd + (uint64_t)count * nchunks * k);
  const dim3 grid((count + 7) / 8, nchunks);
  if (ix.metric == DD_L2)
    k_gt_partial<DD_L2><<<grid, 256, 0, st>>>(ix, queries, qstride, list, count, k, nchunks, pd, pi);
  else
    k_gt_partial<DD_MIPS><<<grid, 256, 0, st>>>(ix, queries, qstride, list, count, k, nchunks, pd, pi);
  k_gt_merge_parts<<<(count + 7) / 8, 256, 0, st>>>(pd, pi, list, count, k, nchunks, ids, dists);
}

}  // namespace ddk
