// Beam-search kernels of the B200 Vamana hot path.
//
//   k_search : one warp per batch point: beam_search on the round-start
//              graph; the visited list goes to the point's global slice
//              (include/index.h:274-278; src/bsp_index.hpp:259-268)
// The query searches are in k_query.cu.
#include <cfloat>
#include <cstdio>

#include "dd_common.cuh"
#include "kernel_util.cuh"
#include "kernels.cuh"
#include "prune_core.cuh"
#include "search_core.cuh"
#include "sort_emul.cuh"

namespace ddk {

// Per-warp shared memory of the search kernels:
//   build search: qv | frontier | step candidates | hash table; the visited
//     list goes to the point's slice of a global array (read by k_prune).
//   query / debug: qv | frontier | step candidates | visited | evicted | hash.
// With h24 the hash table stores 24-bit ids (3 bytes a slot instead of 4),
// which is exact whenever every id is below 0xFFFFFF.
WarpLayout make_search_layout(uint32_t d, int dtype, int metric, uint32_t L, uint32_t Rp,
                              uint32_t vcap, bool build, bool h24, bool keep_vis, bool fastf, bool hash_global) {
  WarpLayout w{};
  uint32_t esz = dtype == DD_F32 ? 4 : 1;
  uint32_t off = 0;
  w.qv = off; off += r16((uint64_t)d * esz);
  // the fast searches keep one 64-bit key per entry of a padded frontier (a
  // query's id and distance arrays, which it may fall back to, fit in it)
  w.nf = !fastf || L > (build ? 128u : 256u) ? 0 : (L <= 64 ? 64 : (L <= 128 ? 128 : 256));
  w.fr_id = off;
  w.fr_d = off + r16(4ull * L);
  off += w.nf ? 8 * w.nf : 2 * r16(4ull * L);
  w.c_id = off; off += r16(4ull * Rp);
  w.c_d = off; off += r16(4ull * Rp);
  w.s_id = off; off += r16(4ull * Rp);
  w.s_d = off; off += w.nf && build ? 0 : r16(4ull * Rp);
  w.term = off; off += w.nf && build && dtype == DD_F32 && metric == DD_L2 ? kFloatTermBytes : 0;
  w.vcap = vcap;
  w.ccap = vcap + Rp;
  w.fastf = (build && fastf) ? 1u : 0u;
  w.hbits = w.fastf ? fast_hash_bits(L) : hash_bits_for(L);
  w.h24 = h24 ? 1u : 0u;
  const uint32_t hash_bytes =
      r16(w.fastf ? fast_table_bytes(w.hbits) : hash_table_bytes(w.hbits, h24));
  if (build) {
    w.vis_id = w.vis_d = 0;  // global
    w.ws = off;
    off += hash_bytes;
  } else {
    w.keep_vis = keep_vis ? 1u : 0u;
    if (keep_vis) {
      w.vis_id = off; off += r16(4ull * vcap);
      w.vis_d = off; off += r16(4ull * vcap);
    }
    w.ws = off; off += 128;  // filter of the evicted ids
    if (keep_vis) {          // the debug search keeps its evicted list here too
      w.ev = off; off += r16(4ull * vcap);
    }
    w.hash_global = hash_global ? 1u : 0u;
    w.hash_words = hash_bytes / 4;
    if (!hash_global) off += hash_bytes;
  }
  w.total = r16(off);
  return w;
}

// |query|^2 of a staged integer query (16-byte words, zero padded), every lane
template <int DT>
__device__ __forceinline__ int query_norm(const uint8_t* qv, uint32_t d) {
  if (DT == DD_F32) return 0;
  const uint32_t lane = lane_id();
  uint32_t s = 0;
  if (lane < (d + 3) / 4) {
    const uint32_t v = ((const uint32_t*)qv)[lane];
    s = DT == DD_U8 ? __dp4a(v, v, 0u) : (uint32_t)__dp4a((int)v, (int)v, 0);
  }
  return (int)__reduce_add_sync(0xffffffffu, s);
}

// build search: visited list in the global slice vis_g (vcap ids then vcap dists)
__device__ __forceinline__ SearchSmem carve_build(uint8_t* base, const WarpLayout& w, uint32_t* vis_g) {
  SearchSmem S;
  S.qv = base + w.qv;
  S.fr_id = (uint32_t*)(base + w.fr_id);
  S.fr_d = (float*)(base + w.fr_d);
  S.c_id = (uint32_t*)(base + w.c_id);
  S.c_d = (float*)(base + w.c_d);
  S.s_id = (uint32_t*)(base + w.s_id);
  S.s_d = (float*)(base + w.s_d);
  S.vis_id = vis_g;
  S.vis_d = (float*)(vis_g + w.vcap);
  S.ev_id = nullptr;
  S.ev_bloom = nullptr;
  S.hash = (uint32_t*)(base + w.ws);
  S.h24 = (int)w.h24;
  S.term = (float*)(base + w.term);
  return S;
}

// ============================================================ build round
// k_search: one warp per batch point runs beam_search on the round-start graph
// and leaves its visited list in the point's global slice
// (include/index.h:274-278; src/bsp_index.hpp:259-268).
// FASTF: the fast form's seen filter and, for L <= 128, warp_build_search with
// capped registers.  Integer data: 64, so that four CTAs of up to 8 warps fit an
// SM (4M x 128 uint8 searches 374 ms, with 72 registers 380, with 80 401);
// float L2: 72, four CTAs of 7 warps (100k x 64: 8.26 ms, 64 registers 8.52);
// float inner product: 80, three CTAs of 8 warps (400k x 200: 98.6 ms, 64
// registers 100.4).
template <int DT, int MT>
struct SearchBounds {
  static constexpr int threads = DT == DD_F32 && MT == DD_L2 ? 224 : 256;
  static constexpr int ctas = DT == DD_F32 && MT == DD_MIPS ? 3 : 4;
};
template <int DT, int MT, int FPL, int CPL, bool FASTF>
__global__ void __launch_bounds__((FASTF && FPL == 4) ? SearchBounds<DT, MT>::threads : 512,
                                  (FASTF && FPL == 4) ? SearchBounds<DT, MT>::ctas : 1)
    k_search(IndexView ix, RoundArgs ra, WarpLayout lay) {
  extern __shared__ uint4 smem_raw[];
  const uint32_t wpc = blockDim.x >> 5;
  const uint32_t wic = threadIdx.x >> 5;
  const uint64_t gw = (uint64_t)blockIdx.x * wpc + wic;
  uint8_t* base = (uint8_t*)smem_raw + (size_t)wic * lay.total;
  SearchParams P;
  P.points = ix.points; P.stride = (uint32_t)ix.stride; P.graph = ix.graph; P.Rp = ix.Rp; P.n = ix.n;
  P.d = ix.d; P.start = ra.start; P.L = ra.L; P.k = 0; P.cut = 0.0; P.limit = ix.n;
  P.degree_limit = ix.R; P.hbits = lay.hbits; P.vcap = lay.vcap; P.ecap = 0; P.query_mode = 0;
  P.keep_visited = 1; P.err = ix.err;
  P.screen = ix.screen; P.sstride = ix.sstride; P.snorm = ix.snorm; P.fgroup_lg = ix.fgroup_lg; P.norms = ix.norms;
  const uint32_t qb = r16((uint64_t)ix.d * ElemSize<DT>::v);
  uint64_t cur = gw;
  const uint64_t step = (uint64_t)gridDim.x * wpc;
  for (uint64_t b = warp_next_item(ra.qsearch, cur, step); b < ra.B;
       b = warp_next_item(ra.qsearch, cur, step)) {
    const uint32_t p = (uint32_t)(ra.floor + b);
    SearchSmem S = carve_build(base, lay, ra.vis_all + b * 2ull * lay.vcap);
    load_vec(S.qv, ix.points + (uint64_t)p * ix.stride, qb);
    __syncwarp();
    if (FASTF && FPL == 4) S.qn = query_norm<DT>(S.qv, ix.d);
    SearchOut o;
    if (FASTF && FPL == 4)
      o = lay.nf == 64 ? warp_build_search<DT, MT, 2, CPL>(P, S, p)
                       : warp_build_search<DT, MT, 4, CPL>(P, S, p);
    else
      o = warp_beam_search<DT, MT, FPL, CPL, FASTF>(P, S, p);
    if (lane_id() == 0) {
      ra.stat_vis[b] = o.vis_n;
      if (ra.stat_cmps) ra.stat_cmps[b] = o.cmps;
    }
    __syncwarp();
  }
}

LaunchPlan plan_search(const IndexView& ix, const WarpLayout& lay, uint32_t L) {
  LaunchPlan p{1, 1};
#define CALL4(DT, MT, F, C)                                                          \
  p = lay.fastf ? plan_warp_kernel(k_search<DT, MT, F, C, true>, lay.total)          \
                : plan_warp_kernel(k_search<DT, MT, F, C, false>, lay.total);
#define CALL(DT, MT) DD_DISPATCH_FC(L, ix.Rp, DT, MT, CALL4)
  DD_DISPATCH_DM(ix.dtype, ix.metric, CALL);
#undef CALL
#undef CALL4
  return p;
}

std::vector<LaunchPlan> search_plan_candidates(const IndexView& ix, const WarpLayout& lay,
                                               uint32_t L) {
  std::vector<LaunchPlan> v;
#define CALL4(DT, MT, F, C)                                                          \
  v = lay.fastf ? warp_kernel_candidates(k_search<DT, MT, F, C, true>, lay.total)    \
                : warp_kernel_candidates(k_search<DT, MT, F, C, false>, lay.total);
#define CALL(DT, MT) DD_DISPATCH_FC(L, ix.Rp, DT, MT, CALL4)
  DD_DISPATCH_DM(ix.dtype, ix.metric, CALL);
#undef CALL
#undef CALL4
  return v;
}

void launch_search(const IndexView& ix, const RoundArgs& ra, const WarpLayout& lay,
                   const LaunchPlan& plan, int grid, cudaStream_t st) {
  const size_t sm = (size_t)lay.total * plan.warps_per_cta;
#define CALL5(DT, MT, F, C, X)                                                       \
  set_smem(k_search<DT, MT, F, C, X>, sm);                                           \
  k_search<DT, MT, F, C, X><<<grid, plan.warps_per_cta * 32, sm, st>>>(ix, ra, lay);
#define CALL4(DT, MT, F, C)                                                          \
  if (lay.fastf) { CALL5(DT, MT, F, C, true); } else { CALL5(DT, MT, F, C, false); }
#define CALL(DT, MT) DD_DISPATCH_FC(ra.L, ix.Rp, DT, MT, CALL4)
  DD_DISPATCH_DM(ix.dtype, ix.metric, CALL);
#undef CALL
#undef CALL5
#undef CALL4
}

}  // namespace ddk
