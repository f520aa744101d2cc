// Routing tables of a mixture-of-experts layer from its routing map, without the host knowing any count: the rows of the dispatched
// activation ordered by expert and, inside an expert, by token.
//   count   tokens routed to e
//   place   rows of e start at the sum of the counts before e: idx[r] = token, row_prob[r] = probs[token, e]
//   scatter (backward) dprobs[idx[r], e] = g[r], zero elsewhere
// A block per expert walks its column of the map.  Bound by launches (the map is T x E bytes); it stands in for two transposes, two
// masked selections with a device -> host count each, and a copy of the counts to the host and back, which left the GPU idle while
// the host caught up after every one of them (64 experts, 4096 tokens, top 6: 6365 -> 6102 us a layer pass).
#include "msb_common.cuh"
using namespace msb;

namespace {
constexpr int RT = 1024;               // threads = tokens per step

__global__ void __launch_bounds__(RT) route_count_kernel(const uint8_t* __restrict__ map, long long* __restrict__ counts, long long T, int E) {
  __shared__ int warp_n[RT / 32];
  const int e = blockIdx.x, lane = threadIdx.x & 31;
  int n = 0;
  for (long long t = threadIdx.x; t < T; t += RT) n += map[t * E + e] != 0;
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0) warp_n[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x < 32) {
    n = __reduce_add_sync(0xffffffffu, warp_n[threadIdx.x]);
    if (threadIdx.x == 0) counts[e] = n;
  }
}

// first row of expert e, in every thread
__device__ __forceinline__ long long first_row(const long long* counts, int e, long long* sh) {
  if (threadIdx.x < 32) {
    long long s = 0;
    for (int i = threadIdx.x; i < e; i += 32) s += counts[i];
#pragma unroll
    for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (threadIdx.x == 0) *sh = s;
  }
  __syncthreads();
  return *sh;
}

// counts[e]: found[e], cut where the caller's rows end, so that what reads the rows by these counts stays inside them; a map whose entries
// are not as many as the caller said leaves a code in the status word.
template <typename T>
__global__ void __launch_bounds__(RT) route_place_kernel(const uint8_t* __restrict__ map, const T* __restrict__ probs, const long long* __restrict__ found,
                                                         long long* __restrict__ counts, long long* __restrict__ idx, T* __restrict__ row_prob,
                                                         long long tokens, int E, long long rows, unsigned int* status) {
  __shared__ long long base_sh;
  __shared__ int warp_n[RT / 32];
  const int e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long base = first_row(found, e, &base_sh);
  if (threadIdx.x == 0) {
    const long long end = base + found[e];
    counts[e] = max(min(end, rows) - base, 0ll);
    if (e == E - 1 && end != rows) atomicCAS(status, 0u, 0x702u);
  }
  for (long long t0 = 0; t0 < tokens; t0 += RT) {
    const long long t = t0 + threadIdx.x;
    const bool on = t < tokens && map[t * E + e] != 0;
    const unsigned int votes = __ballot_sync(0xffffffffu, on);
    __syncthreads();
    if (lane == 0) warp_n[warp] = __popc(votes);
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < RT / 32; ++w) { const int n = warp_n[w]; before += w < warp ? n : 0; all += n; }
    if (on) {
      const long long r = base + before + __popc(votes & ((1u << lane) - 1u));
      if (r < rows) {                                  // a map with more entries than the caller has rows for loses the last ones
        idx[r] = t;
        row_prob[r] = probs[t * E + e];
      }
    }
    base += all;
  }
}

template <typename T>
__global__ void route_scatter_kernel(const T* __restrict__ g, const long long* __restrict__ idx, const long long* __restrict__ counts,
                                     T* __restrict__ dprobs, int E, long long rows) {
  __shared__ long long base_sh;
  const int e = blockIdx.x;
  const long long base = first_row(counts, e, &base_sh), end = min(base + counts[e], rows);
  for (long long r = base + threadIdx.x; r < end; r += blockDim.x) dprobs[idx[r] * E + e] = g[r];
}
}  // namespace

// map [tokens, E] bytes, probs [tokens, E]; counts [E], idx [rows], row_prob [rows]; found: scratch [E].  rows: the number of non-zero bytes
// of the map.
MSB_API int msb_moe_route(const void* map, const void* probs, long long* found, long long* counts, long long* idx, void* row_prob, long long tokens,
                          int E, long long rows, int dtype, unsigned int* status, cudaStream_t s) {
  MSB_REQUIRE(E > 0 && tokens > 0 && rows >= 0, "moe_route: bad shape tokens=%lld E=%d rows=%lld", tokens, E, rows);
  MSB_REQUIRE(status != nullptr, "moe_route: status word is required");
  route_count_kernel<<<E, RT, 0, s>>>((const uint8_t*)map, found, tokens, E);
  MSB_CHECK_LAUNCH("moe_route_count");
  MSB_DISPATCH_FLOAT(dtype, T, route_place_kernel<T><<<E, RT, 0, s>>>((const uint8_t*)map, (const T*)probs, found, counts, idx, (T*)row_prob, tokens, E, rows, status));
  MSB_CHECK_LAUNCH("moe_route_place");
  return 0;
}
// dprobs [tokens, E] is cleared first.
MSB_API int msb_moe_route_bwd(const void* g, const long long* idx, const long long* counts, void* dprobs, long long tokens, int E, long long rows,
                              int dtype, cudaStream_t s) {
  const size_t esz = dtype == MSB_F32 ? 4 : 2;
  cudaError_t e = cudaMemsetAsync(dprobs, 0, (size_t)tokens * E * esz, s);
  if (e != cudaSuccess) { msb_set_error("moe_route_bwd: %s", cudaGetErrorString(e)); return 1; }
  MSB_DISPATCH_FLOAT(dtype, T, route_scatter_kernel<T><<<E, 256, 0, s>>>((const T*)g, idx, counts, (T*)dprobs, E, rows));
  MSB_CHECK_LAUNCH("moe_route_bwd");
  return 0;
}
