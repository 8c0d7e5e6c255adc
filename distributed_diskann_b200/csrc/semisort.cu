// Stable radix sort of the round's (target, key) pairs and segment heads
// (see semisort.cuh).
#include "dd_common.cuh"
#include "kernels.cuh"
#include "semisort.cuh"

#include <algorithm>

namespace ddk {

uint64_t semisort_hist_words(uint64_t E) { return 256ull * ((E + kRadixTile - 1) / kRadixTile); }

// ---- generic exclusive scan of a[0, N) in place; N from *n_dev when given
__global__ void k_gscan1(const uint32_t* a, uint64_t n_host, const uint32_t* n_dev,
                         uint32_t* block_sums) {
  __shared__ uint32_t sh[32];
  const uint64_t N = n_dev ? *n_dev : n_host;
  const uint64_t chunk = (N + gridDim.x - 1) / gridDim.x;
  const uint64_t lo = blockIdx.x * chunk, hi = min(N, lo + chunk);
  uint32_t s = 0;
  for (uint64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) s += a[i];
  uint32_t tot;
  cta_scan_excl(s, &tot, sh);
  if (threadIdx.x == 0) block_sums[blockIdx.x] = tot;
}

__global__ void k_gscan2(uint32_t* block_sums, int nb, uint32_t* total_out) {
  __shared__ uint32_t sh[32];
  uint32_t v = threadIdx.x < (uint32_t)nb ? block_sums[threadIdx.x] : 0;
  uint32_t tot;
  uint32_t ex = cta_scan_excl(v, &tot, sh);
  if (threadIdx.x < (uint32_t)nb) block_sums[threadIdx.x] = ex;
  if (threadIdx.x == 0 && total_out) *total_out = tot;
}

__global__ void k_gscan3(uint32_t* a, uint64_t n_host, const uint32_t* n_dev,
                         const uint32_t* block_sums) {
  __shared__ uint32_t sh[32];
  const uint64_t N = n_dev ? *n_dev : n_host;
  const uint64_t chunk = (N + gridDim.x - 1) / gridDim.x;
  const uint64_t lo = blockIdx.x * chunk, hi = min(N, lo + chunk);
  uint32_t run = block_sums[blockIdx.x];
  for (uint64_t base = lo; base < hi; base += blockDim.x) {
    uint64_t i = base + threadIdx.x;
    uint32_t v = i < hi ? a[i] : 0;
    uint32_t tot;
    uint32_t ex = cta_scan_excl(v, &tot, sh);
    if (i < hi) a[i] = run + ex;
    run += tot;
  }
}

// the same by one CTA, for arrays of a few thousand words
__global__ void __launch_bounds__(1024) k_gscan_small(uint32_t* a, uint32_t n, uint32_t* total_out) {
  __shared__ uint32_t sh[32];
  uint32_t run = 0;
  for (uint32_t base = 0; base < n; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < n ? a[i] : 0u;
    uint32_t tot;
    const uint32_t ex = cta_scan_excl(v, &tot, sh);
    if (i < n) a[i] = run + ex;
    run += tot;
  }
  if (threadIdx.x == 0 && total_out) *total_out = run;
}

// Rounds of up to kSmallPairs pairs (2% rounds of small sets, the first rounds
// of every build): one-CTA scans and one kernel for the segment heads, 7
// launches instead of 20 for two radix passes.  10k x 20 f32 in 2% rounds (6400
// pairs): 64 us of sort a round before, 35 now.  Above, one CTA's walk over the
// pairs takes longer than the launches it saves.
constexpr uint64_t kSmallPairs = 8192;

// returns the number of launches
static uint32_t gscan(uint32_t* a, uint64_t n_host, const uint32_t* n_dev, uint32_t* block_sums,
                      uint32_t* total_out, cudaStream_t st) {
  if (!n_dev && n_host <= kSmallPairs) {
    k_gscan_small<<<1, 1024, 0, st>>>(a, (uint32_t)n_host, total_out);
    return 1;
  }
  k_gscan1<<<kScanBlocks, 256, 0, st>>>(a, n_host, n_dev, block_sums);
  k_gscan2<<<1, kScanBlocks, 0, st>>>(block_sums, kScanBlocks, total_out);
  k_gscan3<<<kScanBlocks, 256, 0, st>>>(a, n_host, n_dev, block_sums);
  return 3;
}

// ---- radix passes; the first pass reads new_out directly (key = index) and
// drops empty slots
// a slot of new_out the first pass keeps: filled, and owned by this rank
__device__ __forceinline__ bool owned_pair(uint32_t t, uint32_t world, uint32_t rank) {
  return t != DD_NONE && (world == 1 || t % world == rank);
}

__global__ void __launch_bounds__(kRadixThreads) k_radix_hist(const uint32_t* t_in,
                                                              const uint32_t* counters, uint64_t E,
                                                              int first, int shift, uint32_t G,
                                                              uint32_t* hist, uint32_t world,
                                                              uint32_t rank) {
  __shared__ uint32_t h[256];
  const uint32_t tid = threadIdx.x;
  h[tid] = 0;
  __syncthreads();
  const uint64_t len = first ? E : counters[0];
  const uint64_t base = (uint64_t)blockIdx.x * kRadixTile;
  for (uint32_t it = 0; it < kRadixItems; it++) {
    uint64_t i = base + (uint64_t)it * kRadixThreads + tid;
    if (i < len) {
      uint32_t t = t_in[i];
      if (!first || owned_pair(t, world, rank)) atomicAdd(&h[(t >> shift) & 255u], 1u);
    }
  }
  __syncthreads();
  hist[(uint64_t)tid * G + blockIdx.x] = h[tid];
}

// Stable scatter of a tile.  Each warp ranks its 512 consecutive pairs against
// digit counters of its own (32 pairs at a time, equal digits grouped with
// __match_any_sync); one pass over the eight warps' counters turns them into
// places in the tile, the pairs are put in that order in shared memory, and
// each digit's run (16 pairs of a full tile) goes out side by side.  A handful
// of block barriers a tile (one per 256 pairs before, and every pair written on
// its own: 14.6 us for a single tile, and 11.2 ms in a 4M x 128 uint8 build).
__global__ void __launch_bounds__(kRadixThreads) k_radix_scatter(
    const uint32_t* t_in, const uint32_t* v_in, const uint32_t* counters, uint64_t E, int first,
    int shift, uint32_t G, const uint32_t* hist, uint32_t* t_out, uint32_t* v_out,
    uint32_t world, uint32_t rank) {
  constexpr uint32_t W = kRadixThreads / 32;
  constexpr uint32_t FULL = 0xffffffffu;
  __shared__ uint32_t wcnt[W][256], delta[256], sh[32];
  __shared__ uint32_t st[kRadixTile], sv[kRadixTile];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (uint32_t d = tid; d < W * 256; d += kRadixThreads) (&wcnt[0][0])[d] = 0;
  const uint64_t len = first ? E : counters[0];
  const uint64_t base = (uint64_t)blockIdx.x * kRadixTile + warp * (32 * kRadixItems) + lane;
  uint32_t lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  uint32_t t[kRadixItems], place[kRadixItems];
#pragma unroll
  for (uint32_t it = 0; it < kRadixItems; it++) {
    const uint64_t i = base + 32 * it;
    t[it] = i < len ? t_in[i] : DD_NONE;
    if (first && !owned_pair(t[it], world, rank)) t[it] = DD_NONE;
  }
  __syncthreads();
#pragma unroll
  for (uint32_t it = 0; it < kRadixItems; it++) {
    const bool valid = t[it] != DD_NONE;
    const uint32_t dig = (t[it] >> shift) & 255u;
    const uint32_t m = __match_any_sync(FULL, valid ? dig : (0x100u | lane));
    uint32_t at = 0;
    if (valid) at = wcnt[warp][dig];
    place[it] = at + __popc(m & lt);
    __syncwarp();
    if (valid && (m & lt) == 0) wcnt[warp][dig] = at + __popc(m);
    __syncwarp();
  }
  __syncthreads();
  uint32_t total;
  {
    uint32_t mine = 0;  // pairs of digit `tid`
#pragma unroll
    for (uint32_t w = 0; w < W; w++) mine += wcnt[w][tid];
    uint32_t run = cta_scan_excl(mine, &total, sh);
    delta[tid] = hist[(uint64_t)tid * G + blockIdx.x] - run;
#pragma unroll
    for (uint32_t w = 0; w < W; w++) {
      const uint32_t c = wcnt[w][tid];
      wcnt[w][tid] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (uint32_t it = 0; it < kRadixItems; it++) {
    if (t[it] != DD_NONE) {
      const uint64_t i = base + 32 * it;
      const uint32_t pos = wcnt[warp][(t[it] >> shift) & 255u] + place[it];
      st[pos] = t[it];
      sv[pos] = first ? (uint32_t)i : v_in[i];
    }
  }
  __syncthreads();
  for (uint32_t j = tid; j < total; j += kRadixThreads) {
    const uint32_t x = st[j], pos = delta[(x >> shift) & 255u] + j;
    t_out[pos] = x;
    v_out[pos] = sv[j];
  }
}

// ---- segment heads: flags, scan, scatter
__global__ void k_head_flags(const uint32_t* t, const uint32_t* counters, uint64_t E,
                             uint32_t* flags) {
  const uint64_t V = counters[0];
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < V;
       i += (uint64_t)gridDim.x * blockDim.x)
    flags[i] = (i == 0 || t[i] != t[i - 1]) ? 1u : 0u;
}

__global__ void k_head_scatter(const uint32_t* t, const uint32_t* counters, const uint32_t* pos,
                               uint32_t* heads) {
  const uint64_t V = counters[0];
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < V;
       i += (uint64_t)gridDim.x * blockDim.x)
    if (i == 0 || t[i] != t[i - 1]) heads[pos[i]] = (uint32_t)i;
}

// flags, scan and heads by one CTA (rounds of up to kSmallPairs pairs)
__global__ void __launch_bounds__(1024) k_heads_small(const uint32_t* t, uint32_t* counters,
                                                      uint32_t* heads) {
  __shared__ uint32_t sh[32];
  const uint32_t V = counters[0];
  uint32_t run = 0;
  for (uint32_t base = 0; base < V; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    const bool head = i < V && (i == 0 || t[i] != t[i - 1]);
    uint32_t tot;
    const uint32_t ex = cta_scan_excl(head ? 1u : 0u, &tot, sh);
    if (head) heads[run + ex] = i;
    run += tot;
  }
  if (threadIdx.x == 0) counters[1] = run;
}

// Measured on B200, whole sort of a build: 4M x 128 uint8 16.5 -> 11.5 ms, 1M x
// 100 int8 in 2% rounds 7.4 -> 6.1 ms, 10k x 20 f32 in 2% rounds 3.7 -> 2.0 ms.
int launch_semisort(const uint32_t* new_out, uint64_t E, uint64_t n, SemisortScratch& s,
                    cudaStream_t st) {
  const uint32_t G = (uint32_t)((E + kRadixTile - 1) / kRadixTile);
  int bits = 1;
  while (bits < 32 && ((uint64_t)1 << bits) < n) bits++;
  const int passes = (bits + 7) / 8;
  const uint32_t* tin = new_out;
  const uint32_t* vin = nullptr;
  int cur = 0;
  for (int p = 0; p < passes; p++) {
    const int first = p == 0;
    k_radix_hist<<<G, kRadixThreads, 0, st>>>(tin, s.counters, E, first, 8 * p, G, s.hist,
                                              s.world, s.rank);
    s.launches += 2 + gscan(s.hist, 256ull * G, nullptr, s.block_sums, first ? &s.counters[0] : nullptr, st);
    k_radix_scatter<<<G, kRadixThreads, 0, st>>>(tin, vin, s.counters, E, first, 8 * p, G, s.hist,
                                                 s.t[cur], s.v[cur], s.world, s.rank);
    tin = s.t[cur];
    vin = s.v[cur];
    cur ^= 1;
  }
  const int res = cur ^ 1;
  if (E <= kSmallPairs) {
    k_heads_small<<<1, 1024, 0, st>>>(s.t[res], s.counters, s.heads);
    s.launches++;
    return res;
  }
  const int g = (int)std::min<uint64_t>((E + 255) / 256, 4096);
  k_head_flags<<<g, 256, 0, st>>>(s.t[res], s.counters, E, s.flags);
  s.launches += 2 + gscan(s.flags, 0, &s.counters[0], s.block_sums, &s.counters[1], st);
  k_head_scatter<<<g, 256, 0, st>>>(s.t[res], s.counters, s.flags, s.heads);
  return res;
}

}  // namespace ddk
