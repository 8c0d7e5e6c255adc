// Reverse-edge kernels of the B200 Vamana hot path.
//
//   k_apply_rows  : update_neighbors of the batch (src/bsp_index.hpp:354-357)
//   k_rev_split   : fast form: one thread per target appends, or lists the
//                   target for one of the prunes
//   k_rev_short   : robustPrune of a full row that gained a few entries, one
//                   warp per listed target: only pairs with a new entry
//   k_reverse     : one warp per target: append, or robustPrune when the row
//                   would overflow R (src/bsp_index.hpp:384-407)
//   k_reverse_big : targets with more candidates than a warp's shared memory
//                   holds, one CTA each
// The grouping of (target, source) pairs by target is semisort.cu.
#include <cfloat>
#include <cstdio>

#include "dd_common.cuh"
#include "kernel_util.cuh"
#include "kernels.cuh"
#include "prune_core.cuh"
#include "search_core.cuh"
#include "sort_emul.cuh"

namespace ddk {

// row_key (may be null): the rows' distances go beside them (new_key)
__global__ void k_apply_rows(uint32_t* graph, const uint32_t* new_out, float* row_key,
                             const float* new_key, uint64_t floor, uint64_t nvec, uint32_t Rp) {
  // rows are Rp uint32 = Rp/4 uint4; batch rows are contiguous in the graph
  const uint4* src = (const uint4*)new_out;
  uint4* dst = (uint4*)(graph + floor * Rp);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec;
       i += (uint64_t)gridDim.x * blockDim.x) {
    dst[i] = src[i];
    if (row_key) ((float4*)(row_key + floor * Rp))[i] = ((const float4*)new_key)[i];
  }
}

// per-warp shared layout of the reverse kernel
struct RevLayout {
  uint32_t tv, cid, ckey, ws, total;
};
__host__ __device__ inline RevLayout rev_layout(uint32_t d, int dtype, uint32_t Rp, bool tensor) {
  RevLayout r;
  uint32_t off = 0;
  uint32_t esz = dtype == DD_F32 ? 4 : 1;
  const uint32_t sel_bytes = greedy_sel_bytes(d, dtype, Rp, tensor);
  r.tv = off; off += r16((uint64_t)d * esz);
  r.cid = off; off += r16(4ull * kRevCandCap);
  r.ckey = off; off += r16(4ull * kRevCandCap);
  r.ws = off; off += prune_ws_bytes_sel(kRevCandCap, sel_bytes);
  r.total = off;
  return r;
}

// The segment of sorted pairs for one target: [start, end) of rs.st / rs.sv.
__device__ __forceinline__ void segment_of(const ReverseScratch& rs, uint32_t k, uint32_t& start,
                                           uint32_t& end) {
  start = rs.heads[k];
  end = (k + 1 < rs.counters[1]) ? rs.heads[k + 1] : rs.counters[0];
}

// the reverse prune's greedy loads the next chunk's rows ahead (with kept
// row distances no candidate row is read before the greedy)
constexpr bool kRevPrefetch = true;

// Append the sources of segment [start, end) (already in batch order), or
// prune when the row would exceed R (one warp; s + deg <= kRevCandCap).
// Returns the number of candidates pruned (0: appended).
template <int DT, int MT, bool TC>
__device__ uint32_t reverse_one(const IndexView& ix, const RoundArgs& ra, const ReverseScratch& rs,
                            uint32_t t, uint32_t start, uint32_t s, uint32_t deg, uint32_t clean,
                            uint8_t* tv, PruneSmem Pm) {
  const uint32_t lane = lane_id();
  uint32_t* row = ix.graph + (uint64_t)t * ix.Rp;
  // the row's distances to t, kept beside the graph (fast form)
  float* rk = (ra.new_key && ra.row_key) ? ra.row_key + (uint64_t)t * ix.Rp : nullptr;
  const uint32_t* sk = rs.sv + start;
  if (s + deg <= ix.R) {
    for (uint32_t j = lane; j < s; j += 32) {
      row[deg + j] = (uint32_t)(ra.floor + sk[j] / ix.Rp);
      if (rk) rk[deg + j] = ra.new_key[sk[j]];
    }
    if (ra.row_meta && lane == 0) ra.row_meta[t] = deg + s + (clean << 16);
    __syncwarp();
    return 0;
  }
  if (!rk) {  // otherwise no distance to t is computed here
    const uint32_t qb = r16((uint64_t)ix.d * ElemSize<DT>::v);
    load_vec(tv, ix.points + (uint64_t)t * ix.stride, qb);
    __syncwarp();
  }
  // a source's distance to t is the one its own prune selected t with (the
  // distances are symmetric bit for bit: (a-b)^2 = (b-a)^2, a*b = b*a, same
  // summation order), when the insert prune kept it
  for (uint32_t j = lane; j < s; j += 32) {
    uint32_t c = (uint32_t)(ra.floor + sk[j] / ix.Rp);
    Pm.cid[j] = c;
    Pm.ckey[j] = ra.new_key ? ra.new_key[sk[j]]
                            : Dist<DT, MT>::eval(tv, ix.points + (uint64_t)c * ix.stride, ix.d);
  }
  for (uint32_t j = lane; j < deg; j += 32) {
    uint32_t c = row[j];
    Pm.cid[s + j] = c;
    Pm.ckey[s + j] = rk ? rk[j] : Dist<DT, MT>::eval(tv, ix.points + (uint64_t)c * ix.stride, ix.d);
  }
  __syncwarp();
  const uint32_t m = s + deg;
  warp_std_sort(Pm, m, s, clean);
  const uint32_t nsel = warp_greedy_select_fast<DT, MT, kRevPrefetch, TC>(
      ix.points, ix.stride, ix.d, t, Pm, m, ra.alpha, ix.R, row, ix.Rp, Pm.sel, rk);
  if (ra.row_meta && lane == 0) ra.row_meta[t] = nsel | (nsel << 16);
  return m;
}

template <int DT, int MT, bool TC>
__global__ void __launch_bounds__(kRevWarps * 32, 8) k_reverse(IndexView ix, RoundArgs ra, ReverseScratch rs) {
  extern __shared__ uint4 smem_raw[];
  const RevLayout L = rev_layout(ix.d, DT, ix.Rp, TC);
  const uint32_t wic = threadIdx.x >> 5, lane = lane_id();
  uint8_t* base = (uint8_t*)smem_raw + (size_t)wic * L.total;
  PruneSmem Pm = prune_ws((uint32_t*)(base + L.cid), (float*)(base + L.ckey), base + L.ws,
                          kRevCandCap);
  Pm.sel = (uint4*)(base + L.ws + prune_sel_offset(kRevCandCap));
  uint32_t nprune = 0, ncand = 0;
  auto tally = [&](uint32_t m) {
    nprune += m ? 1u : 0u;
    ncand += m;
  };
  auto report = [&]() {
    if (lane == 0 && nprune) {
      atomicAdd(&rs.counters[2], nprune);
      atomicAdd(&rs.counters[3], ncand);
    }
  };
  if (rs.split) {  // the general prune list, by work queue
    const uint32_t N = rs.counters[7];
    uint64_t cur = 0;
    for (uint64_t i = warp_next_item(&rs.counters[9], cur, 0); i < N;
         i = warp_next_item(&rs.counters[9], cur, 0)) {
      uint32_t start, end;
      segment_of(rs, rs.list[rs.list_cap - 1 - i], start, end);
      const uint32_t t = rs.st[start], meta = ra.row_meta[t];
      tally(reverse_one<DT, MT, TC>(ix, ra, rs, t, start, end - start, meta & 0xffffu, meta >> 16,
                                    base + L.tv, Pm));
      __syncwarp();
    }
    report();
    return;
  }
  const uint32_t T = rs.counters[1];
  for (uint32_t k = blockIdx.x * kRevWarps + wic; k < T; k += gridDim.x * kRevWarps) {
    uint32_t start, end;
    segment_of(rs, k, start, end);
    const uint32_t t = rs.st[start];
    const uint32_t s = end - start;
    const uint32_t meta = ra.row_meta ? ra.row_meta[t] : 0u;
    const uint32_t deg =
        ra.row_meta ? meta & 0xffffu : row_degree(ix.graph + (uint64_t)t * ix.Rp, ix.Rp);
    if (s + deg > kRevCandCap) {
      if (lane == 0) {
        atomicMax(&rs.counters[5], s + deg);  // largest candidate list of the round
        rs.big[atomicAdd(&rs.counters[4], 1u)] = k;
      }
      continue;  // handled by k_reverse_big
    }
    tally(reverse_one<DT, MT, TC>(ix, ra, rs, t, start, s, deg, meta >> 16, base + L.tv, Pm));
  }
  report();
}

// ---------------------------------------------------------------- fast form
// k_rev_split: one thread per target of the round.  The row's degree comes
// from row_meta, so an append (s + deg <= R) is a handful of 4-byte writes;
// the other targets are listed for the prune that fits them.
__device__ __forceinline__ void list_push(uint32_t* count, uint32_t* list, uint64_t stride_cap,
                                          bool back, bool mine, uint32_t v) {
  const uint32_t b = __ballot_sync(0xffffffffu, mine);
  if (!b) return;
  uint32_t at = 0;
  if (lane_id() == (uint32_t)__ffs(b) - 1) at = atomicAdd(count, __popc(b));
  at = __shfl_sync(0xffffffffu, at, __ffs(b) - 1) + __popc(b & lanemask_lt());
  if (mine) list[back ? stride_cap - 1 - at : at] = v;
}

__global__ void __launch_bounds__(256) k_rev_split(IndexView ix, RoundArgs ra, ReverseScratch rs) {
  const uint32_t T = rs.counters[1];
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t k0 = (uint64_t)blockIdx.x * blockDim.x; k0 < T; k0 += step) {
    const uint64_t k = k0 + threadIdx.x;
    bool brief = false, general = false, big = false;
    if (k < T) {
      uint32_t start, end;
      segment_of(rs, (uint32_t)k, start, end);
      const uint32_t t = rs.st[start], s = end - start;
      const uint32_t meta = ra.row_meta[t];
      const uint32_t deg = meta & 0xffffu, clean = meta >> 16;
      const uint32_t m = s + deg;
      if (m <= ix.R) {
        const uint64_t r0 = (uint64_t)t * ix.Rp + deg;
        for (uint32_t j = 0; j < s; j++) {
          const uint32_t key = rs.sv[start + j];
          ix.graph[r0 + j] = (uint32_t)(ra.floor + key / ix.Rp);
          ra.row_key[r0 + j] = ra.new_key[key];
        }
        ra.row_meta[t] = meta + s;
      } else if (m > kRevCandCap) {
        big = true;
        atomicMax(&rs.counters[5], m);
      } else if (m <= kRevShortCap && m - clean <= kRevShortNew) {
        brief = true;
      } else {
        general = true;
      }
    }
    list_push(&rs.counters[6], rs.list, 0, false, brief, (uint32_t)k);
    list_push(&rs.counters[7], rs.list, rs.list_cap, true, general, (uint32_t)k);
    list_push(&rs.counters[4], rs.big, 0, false, big, (uint32_t)k);
  }
}

// k_rev_short: robustPrune of a target whose row holds the selection of an
// earlier prune (clean entries, kept in its order) and gained u <= 32 others
// (new sources and sources appended since), m <= 128 candidates in all.
//
// No selected entry of a prune is occluded by another one before it, and
// neither the pair's distance nor the later entry's distance to the target has
// changed (all are symmetric and kept bit for bit), so among clean entries no
// occlusion can happen again; between clean entries of equal distance the
// test is the same in both orders.  Only pairs with at least one other entry
// e are computed: the mask M_e of the sorted positions x that occlude e (x
// before e) or that e occludes (x after e).  The walk then visits the others
// in order: e survives unless an entry alive before it is in M_e, and a
// surviving e removes the entries of M_e after it.  That is the reference's
// greedy rule (include/index.h:100-118): an entry is selected iff no selected
// one before it occludes it.
//
// With the default parameter file's 2% rounds a full row of 64 gains 2.7
// entries between prunes: 5 x 16 row tiles against one column tile instead of
// the whole 67 x 67 triangle.  Integer data: rows come straight from global
// memory in fragment order (lane (g, t) of an 8-row group loads bytes 16 t ..
// 16 t + 15 of each 64, and the k index is permuted alike for both operands),
// so nothing is staged and a warp needs 4 KB of shared memory.
//
// Bound by instruction issue (55% of slots, ~3000 instructions a prune; DRAM
// 2%) and by the instruction cache.  On B200, all reverse edges of a build,
// with the split, the lazily sorted hub lists and the ballot-word partitions
// against one warp per target before: 1M x 100 int8 in 2% rounds 87 -> 44 ms
// of kernel time (build 208 -> 165 ms), 100k x 64 f32 15.3 -> 6.4 ms (30.7 ->
// 20.7), 4M x 128 uint8 107 -> 78 ms, overlapped (655 -> 637).  u <= 32 and
// m <= 128 because the masks and the new entries then fit one lane each and
// four words; beyond that the pairs saved no longer pay for the second pass.
struct ShortSmem {
  uint32_t cid[kRevShortCap];
  float ckey[kRevShortCap];
  int posL[kRevShortCap], posR[kRevShortCap];  // sort scratch
  uint32_t occ[kRevShortNew][4];               // M_e, 128 position bits
  int2 nq[kRevShortCap];   // per position: |x|^2 and |x|^2 - T (L2); 0 and -T (MIPS)
  int stack[64];
  uint32_t leafbits[4];
  uint32_t npos[kRevShortNew];                 // sorted positions of the others
};

template <int DT, int MT>
__device__ __forceinline__ void short_masks_mma(const IndexView& ix, double alpha, ShortSmem& S,
                                                uint32_t m, uint32_t u) {
  const uint32_t lane = lane_id(), g = lane >> 2, t = lane & 3;
  const uint32_t FULL = 0xffffffffu;
  const double inv_alpha = 1.0 / alpha;
  for (uint32_t i = lane; i < m; i += 32) {
    const int T = occlusion_threshold(alpha, inv_alpha, S.ckey[i]);
    const int nn = MT == DD_L2 ? __ldg(ix.norms + (S.cid[i] & ~DD_VBIT)) : 0;
    S.nq[i] = make_int2(nn, nn - T);
  }
  __syncwarp();
  const bool wide = ix.stride > 64;  // rows of 128 bytes (two 64-byte halves), else 64
  auto load_row = [&](uint32_t pos, uint4 (&r)[2]) {
    r[0] = r[1] = make_uint4(0, 0, 0, 0);
    if (pos < m) {
      const uint4* src =
          (const uint4*)(ix.points + (uint64_t)(S.cid[pos] & ~DD_VBIT) * ix.stride) + t;
      r[0] = __ldg(src);
      if (wide) r[1] = __ldg(src + 4);
    }
  };
  for (uint32_t e0 = 0; e0 < u; e0 += 8) {
    uint4 b[2];
    load_row(e0 + g < u ? S.npos[e0 + g] : m, b);
    // this lane's two columns (others e0 + 2t, + 1)
    uint32_t pe[2];
    int2 ne[2];
#pragma unroll
    for (int c = 0; c < 2; c++) {
      pe[c] = e0 + 2 * t + c < u ? S.npos[e0 + 2 * t + c] : m;
      ne[c] = pe[c] < m ? S.nq[pe[c]] : make_int2(0, 0);
    }
    for (uint32_t i0 = 0; i0 < m; i0 += 16) {
      uint4 a0[2], a1[2];
      load_row(i0 + g, a0);
      load_row(i0 + g + 8, a1);
      int acc[4] = {0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < 2; j++) {
        if (j == 0 || wide) {
          const uint32_t x[4] = {a0[j].x, a1[j].x, a0[j].y, a1[j].y};
          mma_k32<DT>(acc, x, b[j].x, b[j].y);
          const uint32_t y[4] = {a0[j].z, a1[j].z, a0[j].w, a1[j].w};
          mma_k32<DT>(acc, y, b[j].z, b[j].w);
        }
      }
      uint32_t v = 0;  // column c's 16 row bits at 16 c
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint32_t x = i0 + g + 8 * h;
        const int2 nx = x < m ? S.nq[x] : make_int2(0, 0);
#pragma unroll
        for (int c = 0; c < 2; c++) {
          // x before e: d <= T_e; x after e: d <= T_x
          const int dot = MT == DD_L2 ? 2 * acc[2 * h + c] : acc[2 * h + c];
          const int need = x < pe[c] ? nx.x + ne[c].y : nx.y + ne[c].x;
          if (x < m && x != pe[c] && dot >= need) v |= 1u << (16 * c + 8 * h + g);
        }
      }
      v |= __shfl_xor_sync(FULL, v, 4);
      v |= __shfl_xor_sync(FULL, v, 8);
      v |= __shfl_xor_sync(FULL, v, 16);
      if (g == 0) {
        ((uint16_t*)S.occ[e0 + 2 * t])[i0 >> 4] = (uint16_t)v;
        ((uint16_t*)S.occ[e0 + 2 * t + 1])[i0 >> 4] = (uint16_t)(v >> 16);
      }
    }
  }
  __syncwarp();
}

// the same masks with the reference's own arithmetic: one position per lane
// against each other entry (rows of at most RegRow words in registers)
template <int DT, int MT>
__device__ __forceinline__ void short_masks_lanes(const IndexView& ix, double alpha, ShortSmem& S,
                                                  uint32_t m, uint32_t u) {
  constexpr int NVM = RegRow<DT>::NVM;
  const uint32_t lane = lane_id();
  const uint32_t nv = row_words16(ix.d, DT);
  for (uint32_t c = 0; c * 32 < m; c++) {
    const uint32_t x = 32 * c + lane;
    const bool in = x < m;
    const uint8_t* rx = ix.points + (uint64_t)(in ? S.cid[x] & ~DD_VBIT : 0u) * ix.stride;
    const double kx = in ? (double)S.ckey[x] : 0.0;
    uint4 row[NVM];
    if (nv <= (uint32_t)NVM) {
#pragma unroll
      for (int k = 0; k < NVM; k++)
        row[k] = (in && (uint32_t)k < nv) ? __ldg((const uint4*)rx + k) : make_uint4(0, 0, 0, 0);
    }
    for (uint32_t e = 0; e < u; e++) {
      const uint32_t pe = S.npos[e];
      const uint8_t* re = ix.points + (uint64_t)(S.cid[pe] & ~DD_VBIT) * ix.stride;
      float dsp = 0.f;
      if (nv <= (uint32_t)NVM) dsp = dist_reg<DT, MT, NVM>((const uint4*)re, row, ix.d, nv);
      else if (in) dsp = Dist<DT, MT>::eval(re, rx, ix.d);
      const double key = x < pe ? (double)S.ckey[pe] : kx;
      const uint32_t b =
          __ballot_sync(0xffffffffu, in && x != pe && __dmul_rn(alpha, (double)dsp) <= key);
      if (lane == 0) S.occ[e][c] = b;
    }
  }
  __syncwarp();
}

constexpr uint32_t kShortWarps = 4;

template <int DT, int MT>
__global__ void __launch_bounds__(kShortWarps * 32, DT == DD_F32 ? 4 : 7)
    k_rev_short(IndexView ix, RoundArgs ra, ReverseScratch rs) {
  __shared__ __align__(16) ShortSmem smem[kShortWarps];
  const uint32_t FULL = 0xffffffffu;
  const uint32_t lane = lane_id();
  ShortSmem& S = smem[threadIdx.x >> 5];
  PruneSmem Pm{};
  Pm.cid = S.cid;
  Pm.ckey = S.ckey;
  Pm.posL = S.posL;
  Pm.posR = S.posR;
  Pm.stack = S.stack;
  Pm.leafbits = S.leafbits;
  const uint32_t N = rs.counters[6];
  uint32_t nprune = 0, ncand = 0;
  uint64_t cur = 0;
  for (uint64_t it = warp_next_item(&rs.counters[8], cur, 0); it < N;
       it = warp_next_item(&rs.counters[8], cur, 0)) {
    uint32_t start, end;
    segment_of(rs, rs.list[it], start, end);
    const uint32_t t = rs.st[start], meta = ra.row_meta[t];
    const uint32_t s = end - start, deg = meta & 0xffffu, clean = meta >> 16, m = s + deg;
    uint32_t* row = ix.graph + (uint64_t)t * ix.Rp;
    float* rk = ra.row_key + (uint64_t)t * ix.Rp;
    // sources, then the row; DD_VBIT marks the entries that are not clean
    for (uint32_t j = lane; j < s; j += 32) {
      const uint32_t key = rs.sv[start + j];
      S.cid[j] = (uint32_t)(ra.floor + key / ix.Rp) | DD_VBIT;
      S.ckey[j] = ra.new_key[key];
    }
    for (uint32_t j = lane; j < deg; j += 32) {
      S.cid[s + j] = row[j] | (j < clean ? 0u : DD_VBIT);
      S.ckey[s + j] = rk[j];
    }
    __syncwarp();
    warp_std_sort<kRevShortCap>(Pm, m, s, clean);
    uint32_t alive[4], u = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const uint32_t i = 32 * c + lane;
      const uint32_t id = i < m ? S.cid[i] : t;
      const bool other = i < m && (id & DD_VBIT);
      alive[c] = __ballot_sync(FULL, (id & ~DD_VBIT) != t);
      const uint32_t ob = __ballot_sync(FULL, other);
      if (other) S.npos[u + __popc(ob & lanemask_lt())] = i;
      u += __popc(ob);
    }
    __syncwarp();
    if (DT != DD_F32 && greedy_uses_mma(ix.d, DT)) short_masks_mma<DT, MT>(ix, ra.alpha, S, m, u);
    else short_masks_lanes<DT, MT>(ix, ra.alpha, S, m, u);
    for (uint32_t e = 0; e < u; e++) {
      const uint32_t pe = S.npos[e], we = pe >> 5;
      const uint4 M = *(const uint4*)S.occ[e];
      const uint32_t Mw[4] = {M.x, M.y, M.z, M.w};
      uint32_t hit = 0, self = 0;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const uint32_t before = (uint32_t)c < we ? FULL
                                : ((uint32_t)c == we ? (1u << (pe & 31)) - 1u : 0u);
        hit |= 32u * c < m ? Mw[c] & alive[c] & before : 0u;
        self |= (uint32_t)c == we ? alive[c] & (1u << (pe & 31)) : 0u;
      }
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const uint32_t upto = (uint32_t)c < we ? FULL
                              : ((uint32_t)c == we ? (2u << (pe & 31)) - 1u : 0u);
        if (hit || !self) alive[c] &= (uint32_t)c == we ? ~(1u << (pe & 31)) : FULL;
        else alive[c] &= 32u * c < m ? ~(Mw[c] & ~upto) : FULL;
      }
    }
    // the first R entries alive, in order
    uint32_t nsel = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const uint32_t at = nsel + __popc(alive[c] & lanemask_lt());
      if (((alive[c] >> lane) & 1u) && at < ix.R) {
        row[at] = S.cid[32 * c + lane] & ~DD_VBIT;
        rk[at] = S.ckey[32 * c + lane];
      }
      nsel += __popc(alive[c]);
    }
    nsel = min(nsel, ix.R);
    for (uint32_t j = nsel + lane; j < ix.Rp; j += 32) row[j] = DD_NONE;
    if (lane == 0) {
      ra.row_meta[t] = nsel | (nsel << 16);
      nprune++;
      ncand += m;
    }
    __syncwarp();
  }
  if (nprune) {  // lane 0
    atomicAdd(&rs.counters[2], nprune);
    atomicAdd(&rs.counters[3], ncand);
  }
}

// Targets with more than kRevCandCap candidates: one CTA each, candidates in
// this CTA's global workspace slice.  The greedy walk stops at the R-th
// selection, usually after a small part of a hub's list (a start point
// collects up to 186k sources of a million-point round), so the list is sorted
// lazily, front to back: the introsort's ranges are independent of each other
// once they are split, so the leftmost range is split until about kBigBatch
// elements of finished short ranges stand at the front, those are sorted, and
// the walk takes them; the ranges to their right wait on the stack and are
// split only if the walk gets there.  A walk that ends early costs about two
// passes over the list instead of log2 of them.  Ranges longer than cta_range
// are partitioned by the whole CTA, shorter ones by single warps; then all
// threads finish the leaves.
//
// The walk takes one candidate per thread: each is tested against the rows
// selected before the batch (shared memory, read by broadcast; its own row in
// registers), then the warps resolve their candidates in order, and the later
// warps test each warp's new selections together.
//
// The short ranges are recorded in `ranges` (room for cap/8 + 64 records).
// Ranges longer than K at one recursion depth are disjoint and the depth is
// at most 2 log2(m), so there are at most (m / K) * 2 log2(m) + 1 records:
// K = 256 keeps that within m/8 + 1 for m <= 65536, K = 1024 for every m
// below 2^32.
__device__ __forceinline__ int big_cta_range(uint32_t m) { return m <= 65536u ? 256 : 1024; }
constexpr int kBigStackInts = 3 * 72;
constexpr int kBigBatch = 2048;

template <int DT, int MT>
__global__ void __launch_bounds__(kBigThreads) k_reverse_big(IndexView ix, RoundArgs ra, ReverseScratch rs) {
  constexpr int NVM = RegRow<DT>::NVM;
  constexpr uint32_t FULL = 0xffffffffu;
  extern __shared__ uint4 sel[];  // selected rows: Rp x nv words (rows of at most NVM words)
  __shared__ __align__(16) uint8_t tv[1024];
  __shared__ uint32_t sh[32];
  __shared__ int cstack[kBigStackInts];
  __shared__ int wstack[kBigThreads / 32][kBigStackInts];
  __shared__ uint32_t s_deg, s_nsmall, s_next, s_nsel;
  __shared__ uint32_t s_selid[kMaxRp];
  const uint32_t tid = threadIdx.x, lane = lane_id(), wid = tid >> 5;
  const uint32_t nv = row_words16(ix.d, DT);
  const uint64_t cap = rs.gcap;
  const uint64_t slot = blockIdx.x;
  uint32_t* cid = rs.gcand + slot * cap;
  float* ckey = rs.gkey + slot * cap;
  int* posL = rs.gpos + slot * 2 * cap;
  int* posR = posL + cap;
  uint32_t* bits = rs.gbits + slot * (cap / 32 + 2);
  int* ranges = rs.granges + slot * 3 * (cap / 8 + 64);
  const uint32_t nbig = rs.counters[4];
  ddsort::Arr<uint32_t> A{cid, ckey};
  for (uint32_t e = blockIdx.x; e < nbig; e += gridDim.x) {
    const uint32_t k = rs.big[e];
    uint32_t start, end;
    segment_of(rs, k, start, end);
    const uint32_t t = rs.st[start];
    const uint32_t s = end - start;
    uint32_t* row = ix.graph + (uint64_t)t * ix.Rp;
    float* rk = (ra.new_key && ra.row_key) ? ra.row_key + (uint64_t)t * ix.Rp : nullptr;
    if (wid == 0) {
      uint32_t dg = row_degree(row, ix.Rp);
      if (lane == 0) s_deg = dg;
    }
    const uint32_t qb = r16((uint64_t)ix.d * ElemSize<DT>::v);
    for (uint32_t j = tid; j < qb / 16; j += blockDim.x)
      ((uint4*)tv)[j] = __ldg((const uint4*)(ix.points + (uint64_t)t * ix.stride) + j);
    __syncthreads();
    const uint32_t deg = s_deg;
    const uint32_t m = s + deg;
    if ((uint64_t)m > cap) {  // cannot happen: s <= batch size, cap = batch + Rp
      if (tid == 0) dd_set_error(ix.err, DD_ESEG_CAP);
      __syncthreads();
      continue;
    }
    for (uint32_t j = tid; j < s; j += blockDim.x) {
      const uint32_t key = rs.sv[start + j];
      uint32_t c = (uint32_t)(ra.floor + key / ix.Rp);
      cid[j] = c;
      ckey[j] = ra.new_key ? ra.new_key[key]
                           : Dist<DT, MT>::eval(tv, ix.points + (uint64_t)c * ix.stride, ix.d);
    }
    for (uint32_t j = tid; j < deg; j += blockDim.x) {
      uint32_t c = row[j];
      cid[s + j] = c;
      ckey[s + j] = rk ? rk[j] : Dist<DT, MT>::eval(tv, ix.points + (uint64_t)c * ix.stride, ix.d);
    }
    for (uint32_t w = tid; w < (m + 31) / 32; w += blockDim.x) bits[w] = 0;
    if (tid == 0) {
      s_nsel = 0;
      cstack[0] = 0;
      cstack[1] = (int)m;
      cstack[2] = 2 * ddsort::floor_log2((int)m);
    }
    __syncthreads();
    const int cta_range = big_cta_range(m);
    int sp = 3;
    uint32_t nsel = 0;
    while (sp > 0 && nsel < ix.R) {
      // ---- sort emulation, phase 1: split the front, long ranges by the whole CTA
      const int front = cstack[sp - 3];
      int back = front;
      if (tid == 0) {
        s_nsmall = 0;
        s_next = 0;
      }
      while (sp > 0 && back - front < kBigBatch) {
        int depth = cstack[sp - 1], last = cstack[sp - 2], first = cstack[sp - 3];
        sp -= 3;
        __syncthreads();
        while (last - first > cta_range && depth > 0) {
          --depth;
          const int mid = first + (last - first) / 2;
          if (tid == 0) ddsort::move_median_to_first(A, first, first + 1, mid, last - 1);
          __syncthreads();
          const int cut = cta_partition_rank(A, first + 1, last, posL, posR, sh);
          if (tid == 0) {
            cstack[sp] = cut;
            cstack[sp + 1] = last;
            cstack[sp + 2] = depth;
          }
          sp += 3;
          last = cut;
          __syncthreads();
        }
        if (tid == 0) {  // the rest of this range goes to a warp
          int r = (int)s_nsmall++;
          ranges[3 * r] = first;
          ranges[3 * r + 1] = last;
          ranges[3 * r + 2] = depth;
        }
        back = last;
        __syncthreads();
      }
      // ---- phase 2: short ranges, one warp each (disjoint scratch: posL + first)
      while (true) {
        uint32_t r = 0;
        if (lane == 0) r = atomicAdd(&s_next, 1u);
        r = __shfl_sync(FULL, r, 0);
        if (r >= s_nsmall) break;
        const int first = ranges[3 * r], last = ranges[3 * r + 1], depth = ranges[3 * r + 2];
        warp_partition_loop(A, first, last, depth, wstack[wid], bits, posL + first, posR + first,
                            true);
      }
      __syncthreads();
      // ---- phase 3: leaves
      for (int q = front + (int)tid; q < back; q += (int)blockDim.x)
        if (bits[q >> 5] & (1u << (q & 31)))
          ddsort::insertion_sort_range(A, q, ddsort::leaf_end(bits, q, back));
      __syncthreads();
      // ---- greedy selection (the row of t is rewritten; its old entries are in cid)
      for (int c0 = front; c0 < back && nsel < ix.R; c0 += (int)blockDim.x) {
        const int j = c0 + (int)tid;
        const uint32_t cj = j < back ? cid[j] : DD_NONE;
        bool alive = cj != DD_NONE && cj != t;
        const float fk = alive ? ckey[j] : 0.f;
        const double kj = (double)fk;
        const uint8_t* rj = ix.points + (uint64_t)(alive ? cj : 0u) * ix.stride;
        uint4 reg[NVM];
        if (nv <= (uint32_t)NVM) {
#pragma unroll
          for (int w = 0; w < NVM; w++)
            reg[w] = (alive && (uint32_t)w < nv) ? __ldg((const uint4*)rj + w)
                                                 : make_uint4(0, 0, 0, 0);
        }
        auto occlude = [&](uint32_t q) {  // by the q-th selected row
          float dsp = 0.f;
          if (nv <= (uint32_t)NVM) dsp = dist_reg<DT, MT, NVM>(sel + (uint64_t)q * nv, reg, ix.d, nv);
          else if (alive)
            dsp = Dist<DT, MT>::eval(ix.points + (uint64_t)s_selid[q] * ix.stride, rj, ix.d);
          if (__dmul_rn(ra.alpha, (double)dsp) <= kj) alive = false;
        };
        for (uint32_t q = 0; q < nsel && __any_sync(FULL, alive); q++) occlude(q);
        uint32_t seen = nsel;
        for (uint32_t w = 0; w < blockDim.x / 32; w++) {
          if (wid == w) {
            uint32_t rem = __ballot_sync(FULL, alive);
            while (rem && nsel < ix.R) {
              const uint32_t i = (uint32_t)__ffs(rem) - 1;
              if (lane == i) {
                row[nsel] = cj;
                if (rk) rk[nsel] = fk;
                s_selid[nsel] = cj;
                if (nv <= (uint32_t)NVM) {
#pragma unroll
                  for (int x = 0; x < NVM; x++)
                    if ((uint32_t)x < nv) sel[(uint64_t)nsel * nv + x] = reg[x];
                }
                alive = false;  // selected: not a candidate any more
              }
              __syncwarp();
              if (__any_sync(FULL, alive)) occlude(nsel);
              nsel++;
              rem = __ballot_sync(FULL, alive);
            }
            if (lane == 0) s_nsel = nsel;
          }
          __syncthreads();
          nsel = s_nsel;
          if (wid > w)
            for (uint32_t q = seen; q < nsel && __any_sync(FULL, alive); q++) occlude(q);
          seen = nsel;
          __syncthreads();
          if (nsel >= ix.R) break;
        }
      }
    }
    for (uint32_t j = nsel + tid; j < ix.Rp; j += blockDim.x) row[j] = DD_NONE;
    if (tid == 0) {
      if (ra.row_meta) ra.row_meta[t] = nsel | (nsel << 16);
      atomicAdd(&rs.counters[2], 1u);
      atomicAdd(&rs.counters[3], m);
    }
    __syncthreads();
  }
}

void launch_apply_rows(const IndexView& ix, const RoundArgs& ra, cudaStream_t st) {
  uint64_t nvec = (uint64_t)ra.B * ix.Rp / 4;
  if (!nvec) return;
  int grid = (int)std::min<uint64_t>((nvec + 255) / 256, 4096);
  k_apply_rows<<<grid, 256, 0, st>>>(ix.graph, ra.new_out, ra.new_key ? ra.row_key : nullptr,
                                     ra.new_key, ra.floor, nvec, ix.Rp);
}

__global__ void __launch_bounds__(256) k_clear_clean(uint32_t* row_meta, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    row_meta[i] &= 0xffffu;
}

void launch_clear_clean(uint32_t* row_meta, uint64_t n, cudaStream_t st) {
  k_clear_clean<<<(int)std::min<uint64_t>((n + 255) / 256, 4096), 256, 0, st>>>(row_meta, n);
}

// |x|^2 of every row: eight lanes a row, zero padding contributes nothing
template <int DT>
__global__ void __launch_bounds__(256) k_row_norms(const uint8_t* points, uint64_t stride,
                                                   uint64_t n, uint32_t words, int* norms) {
  const uint32_t sub = threadIdx.x & 7;
  for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3; i < ((n + 3) & ~3ull);
       i += ((uint64_t)gridDim.x * blockDim.x) >> 3) {
    uint32_t acc = 0;
    if (i < n)
      for (uint32_t w = sub; w < words; w += 8) {
        const uint4 v = __ldg((const uint4*)(points + i * stride) + w);
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
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    acc += __shfl_xor_sync(0xffffffffu, acc, 4);
    if (i < n && sub == 0) norms[i] = (int)acc;
  }
}

void launch_row_norms(const IndexView& ix, int* norms, cudaStream_t st) {
  const int grid = (int)std::min<uint64_t>((ix.n * 8 + 255) / 256, 148 * 16);
  const uint32_t words = row_words16(ix.d, ix.dtype);
  if (ix.dtype == DD_U8) k_row_norms<DD_U8><<<grid, 256, 0, st>>>(ix.points, ix.stride, ix.n, words, norms);
  else k_row_norms<DD_I8><<<grid, 256, 0, st>>>(ix.points, ix.stride, ix.n, words, norms);
}

void launch_reverse(const IndexView& ix, const RoundArgs& ra, const ReverseScratch& rs,
                    bool tensor, cudaStream_t st, int sm_count, const ReverseFork& fork) {
  if (!ra.B) return;
  RevLayout L = rev_layout(ix.d, ix.dtype, ix.Rp, tensor);
  const size_t sm = (size_t)L.total * kRevWarps;
  const uint32_t nv = row_words16(ix.d, ix.dtype);
  const size_t bsm = nv <= reg_row_max_words(ix.dtype) ? (size_t)ix.Rp * nv * 16 : 0;
  // split rounds: the hub targets' few CTAs, the general prunes and the short
  // prunes touch different rows and share the GPU
  const bool fast = rs.split;
  cudaStream_t big_st = fast ? fork.aux[0] : st, gen_st = fast ? fork.aux[1] : st;
  if (fast) {
    const int grid = (int)std::min<uint64_t>(((uint64_t)ra.B * ix.Rp + 255) / 256, 148 * 8);
    k_rev_split<<<grid, 256, 0, st>>>(ix, ra, rs);
    cudaEventRecord(fork.forked, st);
    for (cudaStream_t a : fork.aux) cudaStreamWaitEvent(a, fork.forked, 0);
  }
#define CALL2(DT, MT, TC)                                                             \
  set_smem(k_reverse_big<DT, MT>, bsm);                                               \
  set_smem(k_reverse<DT, MT, TC>, sm);                                                \
  if (fast) k_reverse_big<DT, MT><<<kBigSlots, kBigThreads, bsm, big_st>>>(ix, ra, rs); \
  k_reverse<DT, MT, TC><<<sm_count * occupancy(k_reverse<DT, MT, TC>, kRevWarps * 32, sm), \
                          kRevWarps * 32, sm, gen_st>>>(ix, ra, rs);                  \
  if (fast)                                                                           \
    k_rev_short<DT, MT><<<sm_count * occupancy(k_rev_short<DT, MT>, kShortWarps * 32, 0), \
                          kShortWarps * 32, 0, st>>>(ix, ra, rs);                     \
  else                                                                                \
    k_reverse_big<DT, MT><<<kBigSlots, kBigThreads, bsm, big_st>>>(ix, ra, rs);
#define CALL(DT, MT)                                                                  \
  if (tensor) { CALL2(DT, MT, true); } else { CALL2(DT, MT, false); }
  DD_DISPATCH_DM(ix.dtype, ix.metric, CALL);
#undef CALL
#undef CALL2
  if (fast) {
    for (int i = 0; i < 2; i++) {
      cudaEventRecord(fork.joined[i], fork.aux[i]);
      cudaStreamWaitEvent(st, fork.joined[i], 0);
    }
  }
}

}  // namespace ddk
