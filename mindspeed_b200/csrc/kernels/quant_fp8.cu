// fp8 quantisation of the block-scaled linear layer: one pass over a [rows, cols] matrix writes every form of it that the
// three GEMMs of the layer read.
//
//   row form     q [rows, cols], one scale per row and 128 columns, scales transposed [cols / 128, rows]
//   column form  q [cols, rows_pad] (the transpose), one scale per column and 128 rows, scales transposed [rows_pad / 128, cols];
//                rows_pad = rows rounded up to 128, padding rows count as zeros
//   block form   one scale per 128 x 128 tile: q [rows, cols] with scales [rows / 128, cols / 128] and the transposes of both
// The transposed scale layouts are those that gemm_fp8_sm100.cu reads.  Values are bit for bit those of ops/quant.py: scale =
// max(amax, 1e-30) * (1 / fmax), q = fp8(x / scale) with an IEEE division; a NaN or infinity makes its block's scale NaN or inf.
//
// Bound by memory: 2 bytes read and 1 (row or column) or 2 (both, block) written per bf16 element.  A CTA owns a 128 x 128 tile;
// a thread owns 8 rows x 8 columns of it in registers, so that eight consecutive bytes of a row AND of a column leave one
// thread: row bytes go straight to global memory, column bytes through a shared-memory transpose, both in whole 128-byte lines.
// 4096 x 28672 bf16 (117 M elements, 470 MB): both forms 244 us, block form 178 us, where the PyTorch passes took 2.2 ms each; the IEEE
// divisions keep it from the memory rate (72 us).
// reference: mindspeed/te/pytorch/fp8/recipes/float8_block_scaling_recipe.py:15-26.
#include "msb_common.cuh"
#include <cuda_fp8.h>
using namespace msb;

namespace {
constexpr int QT = 128;                 // tile edge = scale block
enum QForm : int { Q_ROW = 1, Q_COL = 2, Q_BLOCK = 4 };

struct QuantParams {
  const void* x;
  uint8_t* q; float* s;                 // row or block form
  uint8_t* qt; float* st;               // column form, or the transposes of the block form
  int rows, cols, rows_pad;
  float inv_fmax;                       // 1 / largest fp8 value
};

__device__ __forceinline__ uint32_t abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }   // ordered like |v|, NaN on top
__device__ __forceinline__ float scale_of(uint32_t amax_bits, float inv_fmax) {
  const float a = __uint_as_float(amax_bits);
  return __fmul_rn(a < 1e-30f ? 1e-30f : a, inv_fmax);
}
// The quotient rounded to nearest, subnormal operands and results kept.  (The build flushes them to zero, in __fdiv_rn too.  PyTorch does
// not, and under the smallest e5m2 scales, blocks below 1e-28, a subnormal value is not zero in fp8.)
__device__ __forceinline__ float quotient(float v, float s) {
  float q;
  asm("div.rn.f32 %0, %1, %2;" : "=f"(q) : "f"(v), "f"(s));
  return q;
}
template <bool E5M2>
__device__ __forceinline__ uint2 to_fp8x8(const float* v) {
  uint32_t w[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * h], v[4 * h + 1]), __NV_SATFINITE, E5M2 ? __NV_E5M2 : __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * h + 2], v[4 * h + 3]), __NV_SATFINITE, E5M2 ? __NV_E5M2 : __NV_E4M3);
    w[h] = lo | (hi << 16);
  }
  return make_uint2(w[0], w[1]);
}

template <typename T, int FORM, bool E5M2>
__global__ void __launch_bounds__(256) quant_tile_kernel(QuantParams p) {
  __shared__ uint32_t red[8][QT];
  __shared__ float col_scale[QT];
  __shared__ uint32_t part_max[4];
  __shared__ __align__(16) uint8_t tr[FORM == Q_ROW ? 16 : QT * QT];   // transposed tile, see below
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rg = threadIdx.x >> 4, cg = threadIdx.x & 15;              // rows 8 rg .. +7, columns 8 cg .. +7 of the tile
  const int row0 = (int)blockIdx.y * QT + rg * 8, col0 = (int)blockIdx.x * QT + cg * 8;
  const float inv_fmax = p.inv_fmax;
  float v[8][8];
  uint32_t cmax[8] = {0, 0, 0, 0, 0, 0, 0, 0}, rmax[8];
  const T* src = reinterpret_cast<const T*>(p.x) + (size_t)row0 * p.cols + col0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (row0 + i < p.rows) {
      Vec8<T> t;
      t.load(src + (size_t)i * p.cols);
      t.to_float(v[i]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    rmax[i] = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t b = abs_bits(v[i][j]);
      rmax[i] = max(rmax[i], b);
      cmax[j] = max(cmax[j], b);
    }
  }
  float scale_blk = 0.f;
  if (FORM != Q_ROW) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      cmax[j] = max(cmax[j], __shfl_xor_sync(0xffffffffu, cmax[j], 16));
      if (lane < 16) red[warp][cg * 8 + j] = cmax[j];
    }
    __syncthreads();
    if (threadIdx.x < QT) {
      uint32_t m = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) m = max(m, red[w][threadIdx.x]);
      if (FORM == Q_BLOCK) {
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) part_max[warp] = m;
      } else {
        const float s = scale_of(m, inv_fmax);
        col_scale[threadIdx.x] = s;
        p.st[(size_t)blockIdx.y * p.cols + (size_t)blockIdx.x * QT + threadIdx.x] = s;
      }
    }
    __syncthreads();
    if (FORM == Q_BLOCK) {
      const uint32_t m = max(max(part_max[0], part_max[1]), max(part_max[2], part_max[3]));
      scale_blk = scale_of(m, inv_fmax);
      if (threadIdx.x == 0) {
        p.s[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = scale_blk;
        p.st[(size_t)blockIdx.x * gridDim.y + blockIdx.y] = scale_blk;
      }
    }
  }
  if (FORM == Q_BLOCK) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = quotient(v[i][j], scale_blk);
  }
  if (FORM & (Q_ROW | Q_BLOCK)) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float o[8];
      if (FORM & Q_ROW) {
        uint32_t m = rmax[i];                          // the 16 threads of a row are half a warp
#pragma unroll
        for (int d = 1; d < 16; d <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
        const float s = scale_of(m, inv_fmax);
        if (cg == 0 && row0 + i < p.rows) p.s[(size_t)blockIdx.x * p.rows + row0 + i] = s;
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = quotient(v[i][j], s);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = v[i][j];
      }
      if (row0 + i < p.rows) *reinterpret_cast<uint2*>(p.q + (size_t)(row0 + i) * p.cols + col0) = to_fp8x8<E5M2>(o);
    }
  }
  if (FORM & (Q_COL | Q_BLOCK)) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float o[8];
      const float s = (FORM & Q_COL) ? col_scale[cg * 8 + j] : 1.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = (FORM & Q_COL) ? quotient(v[i][j], s) : v[i][j];
      // 8-byte unit rg of column 8 cg + j lies at unit rg ^ cg: the sixteen column groups of a store hit different banks
      *reinterpret_cast<uint2*>(tr + (cg * 8 + j) * QT + ((rg ^ cg) << 3)) = to_fp8x8<E5M2>(o);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = k * 32 + (int)(threadIdx.x >> 3), part = (int)(threadIdx.x & 7), cx = c >> 3;
      uint4 v16 = *reinterpret_cast<const uint4*>(tr + c * QT + ((part ^ (cx >> 1)) << 4));
      if (cx & 1) v16 = make_uint4(v16.z, v16.w, v16.x, v16.y);
      *reinterpret_cast<uint4*>(p.qt + ((size_t)blockIdx.x * QT + c) * p.rows_pad + (size_t)blockIdx.y * QT + part * 16) = v16;
    }
  }
}

template <typename T, int FORM>
int launch_quant(const QuantParams& p, int e5m2, cudaStream_t s) {
  const dim3 grid(p.cols / QT, p.rows_pad / QT);
  if (e5m2) quant_tile_kernel<T, FORM, true><<<grid, 256, 0, s>>>(p);
  else quant_tile_kernel<T, FORM, false><<<grid, 256, 0, s>>>(p);
  MSB_CHECK_LAUNCH("quant_fp8");
  return 0;
}
}  // namespace

// x [rows, cols] contiguous, 16-byte aligned, cols a multiple of 128.  form: 1 row, 2 column, 3 both, 4 block (rows a multiple of
// 128 too).  Unused outputs may be null.  See the top of the file for the layouts; e5m2 0 / 1 selects the fp8 format.
MSB_API int msb_quant_fp8(const void* x, void* q, float* s, void* qt, float* st, int rows, int cols, int form, int e5m2, int dtype,
                          cudaStream_t stream) {
  if (rows == 0) return 0;
  MSB_REQUIRE(rows > 0 && cols > 0 && cols % QT == 0, "quant_fp8: bad shape %d x %d (columns must be a multiple of 128)", rows, cols);
  MSB_REQUIRE(form != Q_BLOCK || rows % QT == 0, "quant_fp8: the block form needs rows=%d to be a multiple of 128", rows);
  MSB_REQUIRE((rows + QT - 1) / QT <= 65535, "quant_fp8: too many rows (%d)", rows);
  QuantParams p;
  p.x = x; p.q = (uint8_t*)q; p.s = s; p.qt = (uint8_t*)qt; p.st = st;
  p.rows = rows; p.cols = cols; p.rows_pad = (rows + QT - 1) / QT * QT;
  p.inv_fmax = e5m2 ? 1.f / 57344.f : 1.f / 448.f;
  switch (form) {
    case Q_ROW: MSB_DISPATCH_FLOAT(dtype, T, return (launch_quant<T, Q_ROW>(p, e5m2, stream))); break;
    case Q_COL: MSB_DISPATCH_FLOAT(dtype, T, return (launch_quant<T, Q_COL>(p, e5m2, stream))); break;
    case Q_ROW | Q_COL: MSB_DISPATCH_FLOAT(dtype, T, return (launch_quant<T, Q_ROW | Q_COL>(p, e5m2, stream))); break;
    case Q_BLOCK: MSB_DISPATCH_FLOAT(dtype, T, return (launch_quant<T, Q_BLOCK>(p, e5m2, stream))); break;
  }
  msb_set_error("quant_fp8: unknown form %d", form);
  return 2;
}
