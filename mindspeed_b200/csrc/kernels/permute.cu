// MoE token permutation: row gather and (optionally weighted) row scatter-add with fp32 accumulation.
// The scatter-add runs as a gather: every source row enters its output row's table of eight slots, then a block per output row sums
// them in registers (in ascending order, so that up to eight the order in which threads run does not show) and writes the result
// once.  Bound by the read of the source rows.  (As fp32 atomics into a zeroed buffer that was rounded afterwards, 24576 rows of 4096
// took 180 us beside 25 us for the passes around it.)  Source rows behind the slots, which a token of a mixture of experts has not but a
// repeated index has, are listed output row by output row and summed in pieces of 32, a block each; only where an output row has
// several pieces do these meet in atomics.
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
constexpr int SLOTS = 8;               // source rows of an output row that need no list (a token's experts)
constexpr int PIECE = 32;              // source rows behind the slots that a block sums

// Scratch of one call, long long each.  An output row is full when it has more than SLOTS source rows; F = most full rows there can be.
struct Tables {
  long long *count;                    // [rows] source rows of an output row
  long long *ticket, *n_full, *n_task; // blocks that have placed their rows; full rows; pieces.  count and these are cleared first
  long long *full_of;                  // [rows] number of an output row among the full ones
  long long *slot;                     // [rows, SLOTS]
  long long *row, *off, *done;         // [F] of a full row: its output row, where its list starts, pieces that are summed
  long long *pos, *list;               // [n] place of a source row in its output row; the lists behind the slots
  long long *task;                     // [2 (n / PIECE + F)] full row and number of a piece
  static long long most_full(long long n, long long rows) { return rows < n / (SLOTS + 1) ? rows : n / (SLOTS + 1); }
  static long long most_tasks(long long n, long long rows) { return n / PIECE + most_full(n, rows); }
  Tables(long long* p, long long n, long long rows) {
    const long long f = most_full(n, rows);
    auto take = [&p](long long k) { long long* at = p; p += k; return at; };
    count = take(rows); ticket = take(1); n_full = take(1); n_task = take(1);
    full_of = take(rows); slot = take(rows * SLOTS);
    row = take(f); off = take(f); done = take(f);
    pos = take(n); list = take(n); task = take(2 * most_tasks(n, rows));
  }
};
__device__ __forceinline__ long long fetch_add(long long* p, long long v) {
  return (long long)atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v);
}

// Places of the source rows.  Lanes of a warp with the same output row count once together.  The last block to finish deals the lists'
// ranges and the pieces to the full rows.
__global__ void __launch_bounds__(1024) place_rows_kernel(const long long* __restrict__ idx, Tables t, long long n) {
  __shared__ bool last;
  __shared__ unsigned long long next_off, next_task;
  const int lane = threadIdx.x & 31;
  // all lanes of a warp take part in every round
  for (long long r0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); r0 < n; r0 += (long long)gridDim.x * blockDim.x) {
    const long long r = r0 + lane, o = r < n ? idx[r] : -1;
    const unsigned int same = __match_any_sync(0xffffffffu, (unsigned long long)o);
    const int leader = __ffs(same) - 1;
    long long pos = 0;
    if (lane == leader && r < n) pos = fetch_add(t.count + o, __popc(same));
    pos = __shfl_sync(0xffffffffu, pos, leader) + __popc(same & ((1u << lane) - 1u));
    if (r < n) {
      t.pos[r] = pos;
      if (pos < SLOTS) t.slot[o * SLOTS + pos] = r;
      if (pos == SLOTS) {
        const long long f = fetch_add(t.n_full, 1);
        t.full_of[o] = f;
        t.row[f] = o;
      }
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = fetch_add(t.ticket, 1) == (long long)gridDim.x - 1;
    next_off = next_task = 0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const long long full = __ldcg(t.n_full);
  for (long long f0 = threadIdx.x & ~31u; f0 < full; f0 += blockDim.x) {
    const long long f = f0 + lane, rest = f < full ? __ldcg(t.count + __ldcg(t.row + f)) - SLOTS : 0, pieces = (rest + PIECE - 1) / PIECE;
    long long rest_sum = rest, piece_sum = pieces;     // up to and with this lane
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const long long a = __shfl_up_sync(0xffffffffu, rest_sum, d), b = __shfl_up_sync(0xffffffffu, piece_sum, d);
      if (lane >= d) { rest_sum += a; piece_sum += b; }
    }
    long long off = 0, first = 0;
    if (lane == 31) {
      off = (long long)atomicAdd(&next_off, (unsigned long long)rest_sum);
      first = (long long)atomicAdd(&next_task, (unsigned long long)piece_sum);
    }
    off = __shfl_sync(0xffffffffu, off, 31) + rest_sum - rest;
    first = __shfl_sync(0xffffffffu, first, 31) + piece_sum - pieces;
    if (f < full) { t.off[f] = off; t.done[f] = 0; }
    for (long long i = 0; i < pieces; ++i) { t.task[2 * (first + i)] = f; t.task[2 * (first + i) + 1] = i; }
  }
  __syncthreads();
  if (threadIdx.x == 0) *t.n_task = (long long)next_task;
}

template <bool VEC, typename T>
__device__ __forceinline__ void load8(float* f, const T* s, int c, int cols) {
  if (VEC) {
    Vec8<T> v;
    v.load(s + c);
    v.to_float(f);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = c + j < cols ? to_f(s[c + j]) : 0.f;
  }
}
template <bool VEC, typename T>
__device__ __forceinline__ void store8(T* d, const float* f, int c, int cols) {
  if (VEC) {
    Vec8<T> v;
    v.from_float(f);
    v.store(d + c);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) if (c + j < cols) d[c + j] = from_f<T>(f[j]);
  }
}

// The slots of every output row: the result, or, of a full row, the first value of its fp32 sum (acc [F, pitch]).  The first `fill` blocks
// write the lists of the full rows.  weight (optional): one factor per source row
template <typename T, bool VEC>
__global__ void sum_slots_kernel(const T* __restrict__ src, const long long* __restrict__ idx, const float* __restrict__ weight, Tables tb,
                                 T* __restrict__ out, float* __restrict__ acc, long long n, long long rows, int fill, int cols, int pitch) {
  __shared__ long long slots[SLOTS];
  if ((int)blockIdx.x < fill) {
    if (*tb.n_full == 0) return;
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (long long)fill * blockDim.x)
      if (tb.pos[r] >= SLOTS) tb.list[tb.off[tb.full_of[idx[r]]] + tb.pos[r] - SLOTS] = r;
    return;
  }
  for (long long o = (int)blockIdx.x - fill; o < rows; o += (int)gridDim.x - fill) {
    const long long m = tb.count[o];
    const int k = (int)(m < SLOTS ? m : SLOTS);
    __syncthreads();                                   // slots is used again
    if ((int)threadIdx.x < k) {                        // every slot ranked by its own thread
      const long long mine = tb.slot[o * SLOTS + threadIdx.x];
      int rank = 0;
      for (int i = 0; i < k; ++i) rank += tb.slot[o * SLOTS + i] < mine ? 1 : 0;
      slots[rank] = mine;
    }
    __syncthreads();
    for (int c = (int)threadIdx.x * 8; c < cols; c += (int)blockDim.x * 8) {
      float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
      for (int i = 0; i < k; ++i) {
        const long long r = slots[i];
        const float w = weight ? weight[r] : 1.f;
        float f[8];
        load8<VEC>(f, src + (size_t)r * cols, c, cols);
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[j] = fmaf(f[j], w, sum[j]);
      }
      if (m <= SLOTS) {
        store8<VEC>(out + (size_t)o * cols, sum, c, cols);
      } else {
        float4* d = reinterpret_cast<float4*>(acc + (size_t)tb.full_of[o] * pitch + c);
        d[0] = make_float4(sum[0], sum[1], sum[2], sum[3]);
        d[1] = make_float4(sum[4], sum[5], sum[6], sum[7]);
      }
    }
  }
}

// The pieces of the full rows, a block each.  An only piece meets the slots' sum here; several add to it by atomics, and the block that
// adds the last one writes the result.
template <typename T, bool VEC>
__global__ void sum_pieces_kernel(const T* __restrict__ src, const float* __restrict__ weight, Tables tb, T* __restrict__ out, float* __restrict__ acc,
                                  int cols, int pitch) {
  __shared__ long long list[PIECE];
  __shared__ bool last;
  const long long tasks = *tb.n_task;
  for (long long t = blockIdx.x; t < tasks; t += gridDim.x) {
    const long long f = tb.task[2 * t], first = tb.task[2 * t + 1] * PIECE, o = tb.row[f], rest = tb.count[o] - SLOTS;
    const int k = (int)min(rest - first, (long long)PIECE);
    const bool alone = rest <= PIECE;
    __syncthreads();                                   // list and last are used again
    if ((int)threadIdx.x < k) list[threadIdx.x] = tb.list[tb.off[f] + first + threadIdx.x];
    __syncthreads();
    for (int c = (int)threadIdx.x * 8; c < cols; c += (int)blockDim.x * 8) {
      float* d = acc + (size_t)f * pitch + c;
      float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (alone) {
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[j] = d[j];
      }
#pragma unroll 4
      for (int i = 0; i < k; ++i) {
        const long long r = list[i];
        const float w = weight ? weight[r] : 1.f;
        float v[8];
        load8<VEC>(v, src + (size_t)r * cols, c, cols);
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[j] = fmaf(v[j], w, sum[j]);
      }
      if (alone) {
        store8<VEC>(out + (size_t)o * cols, sum, c, cols);
      } else {
        atomicAdd(reinterpret_cast<float4*>(d), make_float4(sum[0], sum[1], sum[2], sum[3]));
        atomicAdd(reinterpret_cast<float4*>(d + 4), make_float4(sum[4], sum[5], sum[6], sum[7]));
      }
    }
    if (alone) continue;
    __threadfence();                                   // this thread's share is in before the piece is counted
    __syncthreads();
    if (threadIdx.x == 0) last = fetch_add(tb.done + f, 1) == (rest + PIECE - 1) / PIECE - 1;
    __syncthreads();
    if (last) {
      __threadfence();
      for (int c = (int)threadIdx.x * 8; c < cols; c += (int)blockDim.x * 8) {
        const float4* d = reinterpret_cast<const float4*>(acc + (size_t)f * pitch + c);
        const float4 a = __ldcg(d), b = __ldcg(d + 1);
        const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        store8<VEC>(out + (size_t)o * cols, v, c, cols);
      }
    }
  }
}

template <typename T, bool VEC>
int launch_scatter_add(const T* src, const long long* idx, const float* weight, T* out, const Tables& tb, float* acc, long long n, long long rows,
                       int cols, cudaStream_t s) {
  const long long sms = msb::num_sms(), tasks = Tables::most_tasks(n, rows);
  const int threads = cols >= 4096 ? 512 : cols >= 2048 ? 256 : 128, pitch = (cols + 7) / 8 * 8;
  if (n > 0) {
    place_rows_kernel<<<(int)min((n + 1023) / 1024, sms * 2), 1024, 0, s>>>(idx, tb, n);
    MSB_CHECK_LAUNCH("place_rows");
  }
  const int fill = n > SLOTS ? (int)min((n + threads - 1) / threads, sms) : 0;
  sum_slots_kernel<T, VEC><<<fill + (int)min(rows, sms * 32), threads, 0, s>>>(src, idx, weight, tb, out, acc, n, rows, fill, cols, pitch);
  MSB_CHECK_LAUNCH("scatter_add_rows");
  if (n > SLOTS) {
    sum_pieces_kernel<T, VEC><<<(int)min(tasks, sms * (1536 / threads)), threads, 0, s>>>(src, weight, tb, out, acc, cols, pitch);
    MSB_CHECK_LAUNCH("scatter_add_pieces");
  }
  return 0;
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
// source row names become zero.  scratch, 16-byte aligned, with F = min(rows, n / 9): fp32 [F, cols rounded up to 8], then
// int64 [10 rows + 3 + 5 F + 2 n + 2 (n / 32)].
MSB_API int msb_scatter_add_rows(const void* src, const long long* idx, const float* weight, void* out, void* scratch, long long n, long long rows,
                                 int cols, int dtype, cudaStream_t s) {
  if (rows == 0 || cols == 0) return 0;
  float* acc = reinterpret_cast<float*>(scratch);
  long long* tables = reinterpret_cast<long long*>(acc + Tables::most_full(n, rows) * ((cols + 7) / 8 * 8));
  const Tables tb(tables, n, rows);
  const cudaError_t e = cudaMemsetAsync(tables, 0, (size_t)(rows + 3) * sizeof(long long), s);
  if (e != cudaSuccess) { msb_set_error("scatter_add_rows: %s", cudaGetErrorString(e)); return 1; }
  const bool vec = cols % 8 == 0 && (reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(out)) % 16 == 0;
  MSB_DISPATCH_FLOAT(dtype, T, {
    return vec ? launch_scatter_add<T, true>((const T*)src, idx, weight, (T*)out, tb, acc, n, rows, cols, s)
               : launch_scatter_add<T, false>((const T*)src, idx, weight, (T*)out, tb, acc, n, rows, cols, s);
  });
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
