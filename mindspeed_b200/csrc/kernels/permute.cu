// MoE token permutation: row gather and (optionally weighted) row scatter-add with fp32 accumulation.
// The scatter-add runs as a gather: every source row enters its output row's table of eight slots, or a list behind it, then a block
// per output row sums them in registers (slots in ascending order, so that up to eight the order in which threads run does not
// show) and writes the result once.  Bound by the read of the source rows.  (As fp32 atomics into a zeroed buffer that
// was rounded afterwards, 24576 rows of 4096 took 180 us beside 25 us for the passes around it.)
// reference semantics: npu_moe_token_permute / npu_moe_token_unpermute
// (mindspeed/ops/csrc/cann/npu_moe_token_permute.cpp, npu_moe_token_unpermute.cpp).
#include "msb_common.cuh"
using namespace msb;

namespace {
template <typename T>
__global__ void gather_rows_kernel(const T* __restrict__ x, const long long* __restrict__ idx, T* __restrict__ out,
                                   long long n, int cols) {
  const int vec = (cols % 8 == 0) ? cols / 8 : 0;
  for (long long r = blockIdx.x; r < n; r += gridDim.x) {
    const T* src = x + idx[r] * (long long)cols;
    T* dst = out + r * (long long)cols;
    if (vec) {
      for (int v = threadIdx.x; v < vec; v += blockDim.x) { Vec8<T> t; t.load(src + v * 8); t.store(dst + v * 8); }
    } else {
      for (int c = threadIdx.x; c < cols; c += blockDim.x) dst[c] = src[c];
    }
  }
}
constexpr int SLOTS = 8;               // source rows of an output row that are found without walking a list (a token's experts)
constexpr int CHAIN = 64;              // list entries taken at a time (and put in ascending order)

// scratch of one call, long long each: count [rows] | head of the overflow list [rows] | slots [rows, 8] | next [n]
struct Chains {
  long long *count, *head, *slot, *next;
  __host__ __device__ Chains(long long* p, long long rows) : count(p), head(p + rows), slot(p + 2 * rows), next(p + (2 + SLOTS) * rows) {}
};

__global__ void chain_rows_kernel(const long long* __restrict__ idx, Chains c, long long n) {
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (long long)gridDim.x * blockDim.x) {
    const long long o = idx[r], pos = (long long)atomicAdd(reinterpret_cast<unsigned long long*>(c.count + o), 1ull);
    if (pos < SLOTS) c.slot[o * SLOTS + pos] = r;
    else c.next[r] = (long long)atomicExch(reinterpret_cast<unsigned long long*>(c.head + o), (unsigned long long)r);
  }
}

// weight (optional): one factor per source row
template <typename T>
__global__ void sum_chains_kernel(const T* __restrict__ src, const float* __restrict__ weight, Chains ch, T* __restrict__ out, long long rows,
                                  int cols, int vec) {
  __shared__ long long list[CHAIN];
  __shared__ int count;
  for (long long o = blockIdx.x; o < rows; o += gridDim.x) {
    T* dst = out + (size_t)o * cols;
    const long long n = ch.count[o];
    // columns in chunks of 8 per thread; rows with more source rows than a list holds take several rounds per chunk
    for (int c0 = 0; c0 < cols; c0 += (int)blockDim.x * 8) {
      const int c = c0 + (int)threadIdx.x * 8;
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      long long at = n > SLOTS ? ch.head[o] : -1;      // overflow that is still to come
      bool first = true;
      do {
        __syncthreads();
        if (first) {                                   // the slots, every one ranked by its own thread
          const int k = (int)(n < SLOTS ? n : SLOTS);
          if ((int)threadIdx.x < k) {
            const long long mine = ch.slot[o * SLOTS + threadIdx.x];
            int rank = 0;
            for (int i = 0; i < k; ++i) rank += ch.slot[o * SLOTS + i] < mine ? 1 : 0;
            list[rank] = mine;
          }
          if (threadIdx.x == 0) count = k;
        } else if (threadIdx.x == 0) {
          int k = 0;
          for (long long w = at; k < CHAIN && w >= 0; ++k, w = ch.next[w]) {
            int j = k;
            for (; j > 0 && list[j - 1] > w; --j) list[j] = list[j - 1];
            list[j] = w;
          }
          count = k;
        }
        __syncthreads();
        const int k = count;
        if (!first) {                                  // everyone moves on to what the next round takes
          if (k == CHAIN) { for (int i = 0; i < CHAIN; ++i) at = ch.next[at]; }
          else at = -1;
        }
        first = false;
#pragma unroll 4
        for (int i = 0; i < k; ++i) {
          const long long r = list[i];
          const float w = weight ? weight[r] : 1.f;
          const T* s = src + (size_t)r * cols;
          if (vec) {
            if (c < cols) {
              Vec8<T> t;
              float f[8];
              t.load(s + c);
              t.to_float(f);
#pragma unroll
              for (int j = 0; j < 8; ++j) acc[j] = fmaf(f[j], w, acc[j]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) if (c + j < cols) acc[j] = fmaf(to_f(s[c + j]), w, acc[j]);
          }
        }
      } while (at >= 0);
      if (vec) {
        if (c < cols) { Vec8<T> t; t.from_float(acc); t.store(dst + c); }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) if (c + j < cols) dst[c + j] = from_f<T>(acc[j]);
      }
    }
  }
}
// out[idx[r]] += src[r] in fp32, for tables that are far larger than the rows that touch them (gradient of an embedding into its
// accumulator): no dense gradient is formed, cleared, widened and added.  Rows may repeat often, so the sums are atomics, four
// columns each: 8192 rows of 4096 add in 74 us; forming, widening and adding the dense gradient of a 32000-row table took 1.1 ms.  Rows
// with a negative index are not read: under a vocabulary split most ids belong to other ranks, and their zeros added to one row would
// queue at its addresses.
template <typename T>
__global__ void add_rows_kernel(const T* __restrict__ src, const long long* __restrict__ idx, float* __restrict__ out, long long n, int cols, int vec) {
  for (long long r = blockIdx.x; r < n; r += gridDim.x) {
    const long long o = idx[r];
    if (o < 0) continue;
    const T* s = src + r * (long long)cols;
    float* d = out + o * (long long)cols;
    if (vec) {
      for (int c = threadIdx.x * 8; c < cols; c += blockDim.x * 8) {
        Vec8<T> t;
        float f[8];
        t.load(s + c);
        t.to_float(f);
        atomicAdd(reinterpret_cast<float4*>(d + c), make_float4(f[0], f[1], f[2], f[3]));
        atomicAdd(reinterpret_cast<float4*>(d + c + 4), make_float4(f[4], f[5], f[6], f[7]));
      }
    } else {
      for (int c = threadIdx.x; c < cols; c += blockDim.x) atomicAdd(d + c, to_f(s[c]));
    }
  }
}
}  // namespace

MSB_API int msb_gather_rows(const void* x, const long long* idx, void* out, long long n, int cols, int dtype, cudaStream_t s) {
  if (n == 0) return 0;
  int grid = (int)(n < (long long)msb::num_sms() * 16 ? n : (long long)msb::num_sms() * 16);
  MSB_DISPATCH_FLOAT(dtype, T, gather_rows_kernel<T><<<grid, 256, 0, s>>>((const T*)x, idx, (T*)out, n, cols));
  MSB_CHECK_LAUNCH("gather_rows");
  return 0;
}
// out [rows, cols] = for every source row r < n: out[idx[r]] += src[r] * (weight ? weight[r] : 1), summed in fp32; rows that no
// source row names become zero.  chain: int64 scratch [10 rows + n].
MSB_API int msb_scatter_add_rows(const void* src, const long long* idx, const float* weight, void* out, long long* chain, long long n, long long rows,
                                 int cols, int dtype, cudaStream_t s) {
  if (rows == 0 || cols == 0) return 0;
  const Chains ch(chain, rows);
  cudaError_t e = cudaMemsetAsync(ch.count, 0, (size_t)rows * sizeof(long long), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(ch.head, 0xff, (size_t)rows * sizeof(long long), s);
  if (e != cudaSuccess) { msb_set_error("scatter_add_rows: %s", cudaGetErrorString(e)); return 1; }
  if (n > 0) {
    const int cgrid = (int)(((n + 255) / 256) < (long long)msb::num_sms() * 8 ? (n + 255) / 256 : (long long)msb::num_sms() * 8);
    chain_rows_kernel<<<cgrid, 256, 0, s>>>(idx, ch, n);
    MSB_CHECK_LAUNCH("chain_rows");
  }
  const int vec = (cols % 8 == 0 && reinterpret_cast<uintptr_t>(src) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0) ? 1 : 0;
  const int threads = cols >= 4096 ? 512 : cols >= 2048 ? 256 : 128;
  const int grid = (int)(rows < (long long)msb::num_sms() * 32 ? rows : (long long)msb::num_sms() * 32);
  MSB_DISPATCH_FLOAT(dtype, T, sum_chains_kernel<T><<<grid, threads, 0, s>>>((const T*)src, weight, ch, (T*)out, rows, cols, vec));
  MSB_CHECK_LAUNCH("scatter_add_rows");
  return 0;
}
// out [rows, cols] fp32: out[idx[r]] += src[r] for r < n with idx[r] >= 0.
MSB_API int msb_add_rows_f32(const void* src, const long long* idx, float* out, long long n, int cols, int dtype, cudaStream_t s) {
  if (n == 0 || cols == 0) return 0;
  const int vec = (cols % 8 == 0 && (reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(out)) % 16 == 0) ? 1 : 0;
  const int grid = (int)(n < (long long)msb::num_sms() * 16 ? n : (long long)msb::num_sms() * 16);
  MSB_DISPATCH_FLOAT(dtype, T, add_rows_kernel<T><<<grid, 256, 0, s>>>((const T*)src, idx, out, n, cols, vec));
  MSB_CHECK_LAUNCH("add_rows_f32");
  return 0;
}
