// Graph-format and row-exchange kernels of the B200 Vamana hot path.
//
//   k_to_ref_rows / k_from_ref_rows : device rows <-> the reference's
//                     [deg, nbr...] rows (include/utils/graph.h:126-128)
#include <cstdio>

#include <cuda_bf16.h>

#include "dd_common.cuh"
#include "kernel_util.cuh"
#include "kernels.cuh"
#include "prune_core.cuh"
#include "search_core.cuh"
#include "sort_emul.cuh"

namespace ddk {

// ============================================================ sharded build exchange
// The targets whose rows the reverse-edge step of this rank changed (the
// segment heads of the grouped pairs) and their new rows, for the other ranks.
__global__ void k_export_rows(const uint32_t* graph, uint32_t Rp, const uint32_t* st,
                              const uint32_t* heads, const uint32_t* counters, uint64_t cap,
                              uint32_t* ids_out, uint32_t* rows_out) {
  const uint32_t T = counters[1];
  const uint32_t lane = lane_id();
  for (uint64_t k = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < T && k < cap;
       k += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint32_t t = st[heads[k]];
    if (lane == 0) ids_out[k] = t;
    for (uint32_t j = lane; j < Rp; j += 32) rows_out[k * Rp + j] = graph[(uint64_t)t * Rp + j];
  }
}

// rows received from the other ranks; ids are checked against n
__global__ void k_set_rows(uint32_t* graph, uint64_t n, uint32_t Rp, const uint32_t* ids,
                           const uint32_t* rows, uint64_t count, uint32_t* err) {
  const uint32_t lane = lane_id();
  for (uint64_t k = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < count;
       k += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint32_t t = ids[k];
    if (t >= n) {
      if (lane == 0) dd_set_error(err, DD_EBAD_ID);
      continue;
    }
    for (uint32_t j = lane; j < Rp; j += 32) {
      uint32_t a = rows[k * Rp + j];
      if (a != DD_NONE && a >= n) {
        dd_set_error(err, DD_EBAD_ID);
        a = DD_NONE;
      }
      graph[(uint64_t)t * Rp + j] = a;
    }
  }
}

void launch_export_rows(const IndexView& ix, const uint32_t* st, const uint32_t* heads,
                        const uint32_t* counters, uint64_t cap, uint32_t* ids_out,
                        uint32_t* rows_out, cudaStream_t stream) {
  k_export_rows<<<1184, 256, 0, stream>>>(ix.graph, ix.Rp, st, heads, counters, cap, ids_out,
                                          rows_out);
}

void launch_set_rows(const IndexView& ix, const uint32_t* ids, const uint32_t* rows,
                     uint64_t count, cudaStream_t stream) {
  if (!count) return;
  const int grid = (int)std::min<uint64_t>((count * 32 + 255) / 256, 65536);
  k_set_rows<<<grid, 256, 0, stream>>>(ix.graph, ix.n, ix.Rp, ids, rows, count, ix.err);
}

// ============================================================ graph formats
__global__ void k_to_ref_rows(const uint32_t* graph, uint64_t n, uint32_t R, uint32_t Rp,
                              uint32_t* out) {
  const uint32_t lane = lane_id();
  for (uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n;
       v += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint32_t* row = graph + v * Rp;
    uint32_t* o = out + v * (uint64_t)(R + 1);
    uint32_t deg = 0;
    for (uint32_t base = 0; base < R; base += 32) {
      uint32_t j = base + lane;
      uint32_t a = j < R ? row[j] : DD_NONE;
      deg += __popc(__ballot_sync(0xffffffffu, a != DD_NONE));
      if (j < R) o[1 + j] = a == DD_NONE ? 0u : a;
    }
    if (lane == 0) o[0] = deg;
  }
}

__global__ void k_from_ref_rows(uint32_t* graph, uint64_t n, uint32_t R, uint32_t Rp,
                                const uint32_t* in, uint32_t* err) {
  const uint32_t lane = lane_id();
  for (uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n;
       v += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint32_t* r = in + v * (uint64_t)(R + 1);
    uint32_t deg = r[0];
    if (deg > R) {
      if (lane == 0) dd_set_error(err, DD_EDEGREE);
      deg = R;
    }
    for (uint32_t j = lane; j < Rp; j += 32) {
      uint32_t a = j < deg ? r[1 + j] : DD_NONE;
      if (a != DD_NONE && a >= n) {
        dd_set_error(err, DD_EBAD_ID);
        a = DD_NONE;
      }
      graph[v * Rp + j] = a;
    }
  }
}

void launch_to_ref_rows(const IndexView& ix, uint32_t* out, cudaStream_t st) {
  int grid = (int)std::min<uint64_t>((ix.n * 32 + 255) / 256, 65536);
  k_to_ref_rows<<<grid, 256, 0, st>>>(ix.graph, ix.n, ix.R, ix.Rp, out);
}

void launch_from_ref_rows(const IndexView& ix, const uint32_t* in, cudaStream_t st) {
  int grid = (int)std::min<uint64_t>((ix.n * 32 + 255) / 256, 65536);
  k_from_ref_rows<<<grid, 256, 0, st>>>(ix.graph, ix.n, ix.R, ix.Rp, in, ix.err);
}

// ============================================================ BF16 row copies
// One warp per row: each lane converts 8 values (two float4 of the FP32 row)
// into one 16-byte word of BF16 values; values at or beyond d become zeros.
// The squared norm of the BF16 row is summed in FP32 (its rounding is far
// inside the screen's 1% slack on the bound term it enters).
__global__ void __launch_bounds__(256) k_screen_rows(const uint8_t* points, uint64_t stride,
                                                     uint64_t n, uint32_t d, uint8_t* screen,
                                                     uint64_t sstride, float* snorm) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nw = (d + 7) >> 3;
  const uint64_t nwarps = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t i = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n;
       i += nwarps) {
    const float* row = (const float*)(points + i * stride);
    uint4* out = (uint4*)(screen + i * sstride);
    float nrm = 0.f;
    for (uint32_t w = lane; w < nw; w += 32) {
      uint32_t h[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t e = 8 * w + 2 * j;
        const float x0 = e < d ? __ldg(row + e) : 0.f;
        const float x1 = e + 1 < d ? __ldg(row + e + 1) : 0.f;
        const __nv_bfloat16 b0 = __float2bfloat16_rn(x0), b1 = __float2bfloat16_rn(x1);
        const float f0 = __bfloat162float(b0), f1 = __bfloat162float(b1);
        nrm = fmaf(f0, f0, nrm);
        nrm = fmaf(f1, f1, nrm);
        h[j] = (uint32_t)__bfloat16_as_ushort(b0) | ((uint32_t)__bfloat16_as_ushort(b1) << 16);
      }
      out[w] = make_uint4(h[0], h[1], h[2], h[3]);
    }
    for (uint32_t w = nw + lane; w < sstride / 16; w += 32) out[w] = make_uint4(0, 0, 0, 0);
    for (int o = 16; o; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    if (lane == 0) snorm[i] = nrm;
  }
}

void launch_screen_rows(const IndexView& ix, uint8_t* screen, uint64_t sstride, float* snorm,
                        cudaStream_t st) {
  const int grid = (int)std::min<uint64_t>((ix.n + 7) / 8, 148 * 16);
  k_screen_rows<<<grid, 256, 0, st>>>(ix.points, ix.stride, ix.n, ix.d, screen, sstride, snorm);
}

}  // namespace ddk
