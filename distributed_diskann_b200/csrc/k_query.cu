// Query searches of the B200 Vamana hot path.
//
//   k_query  : searchAll (include/utils/beamSearch.h:314-346), mixed L
//   k_beam   : beam_search with the full frontier and visited outputs
#include <cfloat>
#include <cstdio>

#include "dd_common.cuh"
#include "kernel_util.cuh"
#include "kernels.cuh"
#include "search_core.cuh"

namespace ddk {

// query / debug layout: everything in shared memory
// global_hash / global_ev: this warp's global slices (hash_global layouts; the
// evicted list of layouts without keep_vis)
__device__ __forceinline__ SearchSmem carve_query(uint8_t* base, const WarpLayout& w,
                                                  uint32_t* global_hash = nullptr,
                                                  uint32_t* global_ev = nullptr) {
  SearchSmem S;
  S.qv = base + w.qv;
  S.fr_id = (uint32_t*)(base + w.fr_id);
  S.fr_d = (float*)(base + w.fr_d);
  S.c_id = (uint32_t*)(base + w.c_id);
  S.c_d = (float*)(base + w.c_d);
  S.s_id = (uint32_t*)(base + w.s_id);
  S.s_d = (float*)(base + w.s_d);
  S.vis_id = w.keep_vis ? (uint32_t*)(base + w.vis_id) : nullptr;
  S.vis_d = w.keep_vis ? (float*)(base + w.vis_d) : nullptr;
  S.ev_bloom = (uint32_t*)(base + w.ws);
  S.ev_id = w.keep_vis ? (uint32_t*)(base + w.ev) : global_ev;
  S.hash = w.hash_global ? global_hash
                         : (uint32_t*)(base + w.ws + 128 + (w.keep_vis ? r16(4ull * w.vcap) : 0));
  S.h24 = (int)w.h24;
  S.term = (float*)(base + w.term);
  return S;
}

// ============================================================ queries
template <int DT, int MT, int FPL, int CPL>
__global__ void __launch_bounds__(512) k_query(IndexView ix, QueryArgs qa, WarpLayout lay) {
  extern __shared__ uint4 smem_raw[];
  cudaTriggerProgrammaticLaunchCompletion();  // the next class may start where there is room
  const uint32_t wpc = blockDim.x >> 5, wic = threadIdx.x >> 5, lane = lane_id();
  const uint64_t gw = (uint64_t)blockIdx.x * wpc + wic;
  // large seen tables (beam widths above 128) live in this warp's global slice
  const SearchSmem S =
      carve_query((uint8_t*)smem_raw + (size_t)wic * lay.total, lay,
                  lay.hash_global ? qa.hash_scratch + gw * (uint64_t)lay.hash_words : nullptr,
                  qa.ev_scratch + gw * (uint64_t)qa.ev_cap);
  const uint32_t qb = r16((uint64_t)ix.d * ElemSize<DT>::v);
  const uint64_t nitems = qa.cls_items ? (uint64_t)*qa.cls_count : qa.nq;
  uint64_t cur = gw;
  const uint64_t step = (uint64_t)gridDim.x * wpc;
  for (uint64_t it = warp_next_item(qa.cls_queue, cur, step); it < nitems;
       it = warp_next_item(qa.cls_queue, cur, step)) {
    const uint64_t q = qa.cls_items ? qa.cls_items[it] : it;
    SearchParams P;
    uint32_t Lq = qa.Ls[q];
    if (Lq == 0 || Lq > qa.Lvalid || Lq < qa.k) {
      if (lane == 0) dd_set_error(ix.err, DD_ECAND_CAP);
      Lq = qa.Lvalid;
    }
    P.points = ix.points; P.stride = (uint32_t)ix.stride; P.graph = ix.graph; P.Rp = ix.Rp; P.n = ix.n;
    P.d = ix.d; P.start = qa.start; P.L = Lq; P.k = qa.k; P.cut = qa.cut; P.limit = qa.limit;
    P.degree_limit = qa.degree_limit; P.hbits = hash_bits_for(P.L); P.vcap = 0;
    P.ecap = qa.ev_cap; P.query_mode = 1; P.keep_visited = 0; P.err = ix.err;
    P.screen = ix.screen; P.sstride = ix.sstride; P.snorm = ix.snorm;
    P.fgroup_lg = ix.fgroup_lg; P.norms = ix.norms;
    load_vec(S.qv, qa.queries + q * qa.qstride, qb);
    __syncwarp();
    SearchOut o;
    bool keyed = false;  // the frontier is warp_query_search's
    if (lay.nf && !__shfl_sync(0xffffffffu, *(volatile uint32_t*)qa.repeats, 0)) {
      const uint32_t self = qa.skip_self ? (uint32_t)q : DD_NONE;
      if (FPL == 4)
        keyed = lay.nf == 64 ? warp_query_search<DT, MT, 2, CPL>(P, S, self, &o)
                             : warp_query_search<DT, MT, 4, CPL>(P, S, self, &o);
      else
        keyed = warp_query_search<DT, MT, 8, CPL>(P, S, self, &o);
      __syncwarp();
      // rows with repeated ids: the other queries of the call go straight there
      if (!keyed && lane == 0) *(volatile uint32_t*)qa.repeats = 1u;
    }
    if (!keyed) o = warp_beam_search<DT, MT, FPL, CPL>(P, S, qa.skip_self ? q : (uint64_t)-1);
    for (uint32_t j = lane; j < qa.k; j += 32) {
      bool v = j < o.fr_n;
      uint32_t id = DD_NONE;
      float d = INFINITY;
      if (v && keyed) {
        const unsigned long long key = ((const unsigned long long*)S.fr_id)[j];
        id = (uint32_t)key >> 1;
        d = order_dist<MT>((uint32_t)(key >> 32));
      } else if (v) {
        id = S.fr_id[j] & ~DD_VBIT;
        d = S.fr_d[j];
      }
      qa.ids[q * qa.k + j] = id;
      qa.dists[q * qa.k + j] = d;
    }
    if (lane == 0) {
      if (qa.visited) qa.visited[q] = o.vis_n;
      if (qa.cmps) qa.cmps[q] = o.cmps;
    }
    __syncwarp();
  }
  // an overlapped class ends after the one before it, so that what follows on
  // the stream finds both done
  cudaGridDependencySynchronize();
}

__global__ void k_bin_queries(const uint32_t* Ls, uint64_t nq, uint32_t k, uint32_t Lvalid,
                              uint32_t* items, uint32_t* counts) {
  for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nq;
       q += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t L = Ls[q];
    if (L == 0 || L > Lvalid || L < k) L = Lvalid;
    const int c = query_class(L);
    items[(uint64_t)c * nq + atomicAdd(&counts[c], 1u)] = (uint32_t)q;
  }
}

void launch_bin_queries(const uint32_t* Ls, uint64_t nq, uint32_t k, uint32_t Lvalid,
                        uint32_t* items, uint32_t* counts, cudaStream_t st) {
  const int grid = (int)std::min<uint64_t>((nq + 255) / 256, 1024);
  k_bin_queries<<<grid, 256, 0, st>>>(Ls, nq, k, Lvalid, items, counts);
}

template <int DT, int MT>
__global__ void __launch_bounds__(32) k_beam(IndexView ix, BeamArgs ba, WarpLayout lay) {
  extern __shared__ uint4 smem_raw[];
  const uint32_t lane = lane_id();
  const SearchSmem S = carve_query((uint8_t*)smem_raw, lay);
  const uint32_t qb = r16((uint64_t)ix.d * ElemSize<DT>::v);
  for (uint64_t q = blockIdx.x; q < ba.nq; q += gridDim.x) {
    SearchParams P;
    P.points = ix.points; P.stride = (uint32_t)ix.stride; P.graph = ix.graph; P.Rp = ix.Rp; P.n = ix.n;
    P.d = ix.d; P.start = ba.start; P.L = ba.L; P.k = ba.k; P.cut = ba.cut; P.limit = ba.limit;
    P.degree_limit = ba.degree_limit; P.hbits = lay.hbits; P.vcap = lay.vcap; P.ecap = lay.vcap;
    P.query_mode = ba.k > 0; P.keep_visited = 1; P.err = ix.err;
    P.screen = nullptr; P.sstride = 0; P.snorm = nullptr; P.fgroup_lg = 0; P.norms = nullptr;  // the plain form
    load_vec(S.qv, ba.queries + q * ba.qstride, qb);
    __syncwarp();
    SearchOut o = warp_beam_search<DT, MT, 16, 4>(P, S, (uint64_t)ba.self_ids[q]);
    warp_sort_pairs(S.vis_id, S.vis_d, o.vis_n);
    for (uint32_t j = lane; j < o.fr_n; j += 32) {
      ba.fr_ids[q * ba.L + j] = S.fr_id[j] & ~DD_VBIT;
      ba.fr_d[q * ba.L + j] = S.fr_d[j];
    }
    for (uint32_t j = lane; j < o.vis_n; j += 32) {
      ba.vis_ids[q * ba.vcap + j] = S.vis_id[j];
      ba.vis_d[q * ba.vcap + j] = S.vis_d[j];
    }
    if (lane == 0) {
      ba.fr_n[q] = o.fr_n;
      ba.vis_n[q] = o.vis_n;
      ba.cmps[q] = o.cmps;
    }
    __syncwarp();
  }
}

LaunchPlan plan_query(const IndexView& ix, const WarpLayout& lay, uint32_t Lmax) {
  LaunchPlan p{1, 1};
#define CALL4(DT, MT, F, C) p = plan_warp_kernel(k_query<DT, MT, F, C>, lay.total);
#define CALL(DT, MT) DD_DISPATCH_FC(Lmax, ix.Rp, DT, MT, CALL4)
  DD_DISPATCH_DM(ix.dtype, ix.metric, CALL);
#undef CALL
#undef CALL4
  return p;
}

// overlap: the launch may start once every CTA of the k_query launch before it on
// the stream has started (nothing it reads comes from there: the class lists were
// complete when that one began, and each has its own scratch).  A class's last
// searches leave most of the GPU idle, and a call of mixed widths had one such
// tail per class.  Measured on B200, 10,000 queries of L = 10 to 200 mixed, classes
// one after another against overlapped: 10M x 128 uint8 4.89 -> 3.67 ms, 1M 3.57 ->
// 2.64, 100k x 64 f32 3.11 -> 2.32; calls of one width the same.  Forked streams
// overlap the classes a little more (2.43 and 2.14 ms), but a narrow class may
// then start first and take the places of the widest: calls of L = 200 alone on
// 10M took 7.3 or 11.5 ms instead of 7.5.
void launch_query(const IndexView& ix, const QueryArgs& qa, const WarpLayout& lay, int wpc,
                  int grid, bool overlap, cudaStream_t st) {
  size_t sm = (size_t)lay.total * wpc;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(wpc * 32);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = overlap ? 1 : 0;
#define CALL4(DT, MT, F, C)                                                          \
  set_smem(k_query<DT, MT, F, C>, sm);                                               \
  cudaLaunchKernelEx(&cfg, k_query<DT, MT, F, C>, ix, qa, lay);
#define CALL(DT, MT) DD_DISPATCH_FC(qa.Lmax, ix.Rp, DT, MT, CALL4)
  DD_DISPATCH_DM(ix.dtype, ix.metric, CALL);
#undef CALL
#undef CALL4
}

void launch_beam(const IndexView& ix, const BeamArgs& ba, const WarpLayout& lay, int grid,
                 cudaStream_t st) {
  size_t sm = lay.total;
#define CALL(DT, MT)                                                   \
  set_smem(k_beam<DT, MT>, sm);                                        \
  k_beam<DT, MT><<<grid, 32, sm, st>>>(ix, ba, lay);
  DD_DISPATCH_DM(ix.dtype, ix.metric, CALL);
#undef CALL
}

}  // namespace ddk
