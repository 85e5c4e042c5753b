// mrmg_serving.cu -- the serving batcher's input gather: the device reads
// every planner instance's request arrays straight from host memory (where
// the device reads pageable host memory coherently, as GB300 does over its
// host link) into the step's device buffers, so a step needs no host-side
// packing pass and no staging copy.
#include <cstdint>

#include "mrmg_internal.cuh"

namespace mrmg {
namespace {

// one source array of the step (table row, 32 bytes)
struct GatherEntry {
  const void* src;      // host address of a C-contiguous array
  long long rows;       // rows of D floats (kinds 0-2) or int64 step counts (kind 3)
  long long dst_row;    // first destination row within its region
  int kind;             // 0 configurations, 1 edge starts, 2 edge ends, 3 edge step counts
  int pad;
};

// table: int64 {n_src, n_configs, n_edges, 0}, then n_src GatherEntry rows.
//
// Copies what the sources hold of the step's rows [lo, hi) (rows of q1, q2 and N:
// the configurations' region, then the edges') and sets those rows' step counts
// of configurations (3) and unused slots (2).  A persistent grid: each CTA clips
// the table's entries to the rows in shared memory and its warps take 2 KB pieces
// of them in turn, four 16-byte loads in flight per lane.  Bound: the host link.
// With a CTA per SM the loads in flight (2.5 MB) still cover its latency, and the
// edge scan of rows gathered before runs beside it on the same SMs.  280 MB on its
// own: 1.45 ms (190 GB/s), as with a CTA per source and 1/64 of its rows.
constexpr int kGatherThreads = 256, kGatherSpans = 512;
constexpr int kPieceWords = 512;   // 32-bit words per piece

struct GatherSpan {
  const uint32_t* src;
  uint32_t *d1, *d2;       // d2: a configuration is the edge q -> q (else null)
  long long words;
};

__global__ void __launch_bounds__(kGatherThreads) serving_gather_kernel(const long long* __restrict__ table, int max_src,
                                                                        int D, long long ccap, long long ecap,
                                                                        long long lo, long long hi, float* q1,
                                                                        float* q2, long long* N, int* err) {
  __shared__ GatherSpan s_span[kGatherSpans];
  __shared__ int s_piece[kGatherSpans + 1];   // pieces of the spans before
  const long long n_src = table[0], nc = table[1], ne = table[2];
  const int tid = threadIdx.x, lane = tid & 31;
  const bool first = blockIdx.x == 0;
  if (nc > ccap || ne > ecap || n_src > max_src || nc < 0 || ne < 0 || n_src < 0) {
    if (first && tid == 0) atomicOr(err, E_BAD_INPUT);
  } else {
    for (long long i = lo + (long long)blockIdx.x * blockDim.x + tid; i < hi; i += (long long)gridDim.x * blockDim.x)
      if (i < ccap) N[i] = i < nc ? 3 : 2;
      else if (i >= ccap + ne) N[i] = 2;
  }
  const long long entries = n_src < max_src ? n_src : max_src;
  for (long long e0 = 0; e0 < entries; e0 += kGatherSpans) {
    const int m = (int)(entries - e0 < kGatherSpans ? entries - e0 : kGatherSpans);
    for (int i = tid; i < m; i += kGatherThreads) {
      const GatherEntry e = ((const GatherEntry*)(table + 4))[e0 + i];
      const long long cap = e.kind == 0 ? ccap : ecap;
      GatherSpan sp{nullptr, nullptr, nullptr, 0};
      if (e.rows > 0) {
        if (e.kind < 0 || e.kind > 3 || e.dst_row < 0 || e.dst_row + e.rows > cap || !e.src) {
          if (first) atomicOr(err, E_BAD_INPUT);
        } else {
          const long long row = (e.kind == 0 ? 0 : ccap) + e.dst_row;   // the entry's first row of the step
          const long long a = lo > row ? lo - row : 0, b = hi - row < e.rows ? hi - row : e.rows;
          if (a < b) {
            const int w = e.kind == 3 ? 2 : D;
            sp.src = (const uint32_t*)e.src + a * w;
            sp.d1 = e.kind == 3 ? (uint32_t*)(N + row + a) : (uint32_t*)(e.kind == 2 ? q2 : q1) + (row + a) * D;
            if (e.kind == 0) sp.d2 = (uint32_t*)q2 + (row + a) * D;
            sp.words = (b - a) * w;
          }
        }
      }
      s_span[i] = sp;
    }
    __syncthreads();
    if (tid < 32) {
      int at = 0;
      for (int i = 0; i < m; i += 32) {
        const int p = i + lane < m ? (int)((s_span[i + lane].words + kPieceWords - 1) / kPieceWords) : 0;
        int incl = p;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(MRMG_FULL, incl, o);
          if (lane >= o) incl += y;
        }
        if (i + lane < m) s_piece[i + lane] = at + incl - p;
        at += __shfl_sync(MRMG_FULL, incl, 31);
      }
      if (lane == 0) s_piece[m] = at;
    }
    __syncthreads();
    const int pieces = s_piece[m], warps = (int)gridDim.x * (kGatherThreads / 32);
    for (int p = (int)blockIdx.x * (kGatherThreads / 32) + (tid >> 5); p < pieces; p += warps) {
      int k = 0, top = m - 1;   // the last span whose pieces start at or before p
      while (k < top) {
        const int mid = (k + top + 1) >> 1;
        if (s_piece[mid] <= p) k = mid;
        else top = mid - 1;
      }
      const GatherSpan sp = s_span[k];
      const long long off = (long long)(p - s_piece[k]) * kPieceWords;
      const int n = (int)(sp.words - off < kPieceWords ? sp.words - off : kPieceWords);
      const uint32_t* src = sp.src + off;
      uint32_t* d1 = sp.d1 + off;
      uint32_t* d2 = sp.d2 ? sp.d2 + off : nullptr;
      if (n == kPieceWords && (((uintptr_t)src | (uintptr_t)d1 | (uintptr_t)d2) & 15) == 0) {
        uint4 v[kPieceWords / 128];
#pragma unroll
        for (int i = 0; i < kPieceWords / 128; i++) v[i] = ((const uint4*)src)[i * 32 + lane];
#pragma unroll
        for (int i = 0; i < kPieceWords / 128; i++) {
          ((uint4*)d1)[i * 32 + lane] = v[i];
          if (d2) ((uint4*)d2)[i * 32 + lane] = v[i];
        }
      } else {
#pragma unroll 4
        for (int i = lane; i < n; i += 32) {
          const uint32_t v = src[i];
          d1[i] = v;
          if (d2) d2[i] = v;
        }
      }
    }
    __syncthreads();   // the next entries reuse the spans
  }
}

}  // namespace

cudaError_t serving_gather(const void* table, int max_src, int D, long long ccap, long long ecap, long long lo,
                           long long hi, float* q1, float* q2, long long* N, int* err, int num_sms, cudaStream_t st) {
  serving_gather_kernel<<<num_sms, kGatherThreads, 0, st>>>((const long long*)table, max_src, D, ccap, ecap, lo, hi, q1,
                                                            q2, N, err);
  return cudaGetLastError();
}

}  // namespace mrmg
