// Heads of multi-head latent attention: one pass that splits the up-projections, rotates the positional part of the queries and of
// the shared key, and writes q, k and v as the attention kernels read them; and its backward.
//
//   forward   q [T, n, nope + rope], kv [T, n, nope + vd], k_pe [T, rope]  ->  qf [T, n, nope + rope] (last `rope` rotated),
//             kf [T, n, nope + rope] = (k of kv | rotated k_pe, the same for every head), v [T, n, vd]
//   backward  dqf, dkf, dv -> dq, dkv and dk_pe (summed over the heads in fp32, in a fixed order, then rotated back and rounded once)
//
// Bound by memory: every value is read and written once.  A block owns a token, so that k_pe, the angles and the sum over heads
// stay on the SM; 16-byte accesses.  (As slices, concatenations and element-wise rotations in PyTorch the same work made 12
// passes, most of them strided.)  4096 tokens, 32 heads of 128 + 64 / 128, bf16 (250 MB each way, 38 us at the copy rate): 52 us
// forward, 61 backward; about 1000 us as PyTorch operations.
// reference: mindspeed/core/transformer/multi_head_latent_attention/adaptor.py:23-139 (decoupled rotary key shared across heads).
#include "msb_common.cuh"
using namespace msb;

namespace {
struct MlaDims {
  int n, nope, rope, vd;             // heads; widths, multiples of 8 (rope of 16)
  int b;                             // tokens per position
  int interleaved;
};
struct Strided { long long s, b, h; };   // element strides of position, batch and head; the last dimension is contiguous

// (x1, x2): the partner values of eight pairs; rotate-half pairs column j with j + rope / 2, interleaved 2 i with 2 i + 1
__device__ __forceinline__ void rot(float& x1, float& x2, float c1, float s1, float c2, float s2, bool back) {
  const float a = x1, b = x2;
  if (!back) { x1 = a * c1 - b * s1; x2 = b * c2 + a * s2; }
  else { x1 = a * c1 + b * s2; x2 = b * c2 - a * s1; }
}
// Eight pairs starting at pair 8 j of a rotary part held as two vectors of eight values: (columns 8j.., columns rope/2 + 8j..) or,
// interleaved, (columns 16 j .. 16 j + 7, 16 j + 8 .. 16 j + 15)
__device__ __forceinline__ void rot16(float* u, float* w, const float* cos, const float* sin, int j, const MlaDims& d, bool back) {
  if (!d.interleaved) {
    const int a = 8 * j, b = d.rope / 2 + 8 * j;
#pragma unroll
    for (int i = 0; i < 8; ++i) rot(u[i], w[i], cos[a + i], sin[a + i], cos[b + i], sin[b + i], back);
  } else {
    const int a = 16 * j;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      rot(u[2 * i], u[2 * i + 1], cos[a + 2 * i], sin[a + 2 * i], cos[a + 2 * i + 1], sin[a + 2 * i + 1], back);
      rot(w[2 * i], w[2 * i + 1], cos[a + 8 + 2 * i], sin[a + 8 + 2 * i], cos[a + 9 + 2 * i], sin[a + 9 + 2 * i], back);
    }
  }
}
__device__ __forceinline__ int first_col(int j, const MlaDims& d) { return d.interleaved ? 16 * j : 8 * j; }
__device__ __forceinline__ int second_col(int j, const MlaDims& d) { return d.interleaved ? 16 * j + 8 : d.rope / 2 + 8 * j; }

// n rows (heads) of w8 vectors of eight values, from stride ss to stride ds (elements); four loads in flight a thread
template <typename T, int W8>
__device__ __forceinline__ void copy_heads(T* __restrict__ dst, long long ds, const T* __restrict__ src, long long ss, int n, int w8_) {
  const int w8 = W8 ? W8 : w8_, total = n * w8;
  int i = threadIdx.x;
  for (; i + 3 * (int)blockDim.x < total; i += 4 * blockDim.x) {
    Vec8<T> t[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) { const int j = i + k * (int)blockDim.x, h = j / w8; t[k].load(src + h * ss + 8 * (j - h * w8)); }
#pragma unroll
    for (int k = 0; k < 4; ++k) { const int j = i + k * (int)blockDim.x, h = j / w8; t[k].store(dst + h * ds + 8 * (j - h * w8)); }
  }
  for (; i < total; i += blockDim.x) { const int h = i / w8; Vec8<T> t; t.load(src + h * ss + 8 * (i - h * w8)); t.store(dst + h * ds + 8 * (i - h * w8)); }
}
// the rotary part of n heads (src and dst at its first column), p8 groups of eight pairs a head
template <typename T, int P8>
__device__ __forceinline__ void rotate_heads(T* __restrict__ dst, long long ds, const T* __restrict__ src, long long ss, const float* c, const float* s,
                                             const MlaDims& d, bool back) {
  const int p8 = P8 ? P8 : d.rope / 16;
  for (int i = threadIdx.x; i < d.n * p8; i += blockDim.x) {
    const int h = i / p8, j = i - h * p8, a = first_col(j, d), b = second_col(j, d);
    Vec8<T> x, y;
    x.load(src + h * ss + a); y.load(src + h * ss + b);
    float u[8], w[8];
    x.to_float(u); y.to_float(w);
    rot16(u, w, c, s, j, d, back);
    x.from_float(u); y.from_float(w);
    x.store(dst + h * ds + a); y.store(dst + h * ds + b);
  }
}

template <typename T, int N8, int R8, int V8>
__global__ void __launch_bounds__(256) mla_heads_fwd_kernel(const T* __restrict__ q, const T* __restrict__ kv, const T* __restrict__ k_pe,
                                                            Strided sp, const float* __restrict__ cos, const float* __restrict__ sin,
                                                            T* __restrict__ qf, T* __restrict__ kf, T* __restrict__ v, MlaDims d) {
  extern __shared__ float sh[];                        // cos | sin | rotated k_pe
  float *c = sh, *s = sh + d.rope, *pe = sh + 2 * d.rope;
  const long long t = blockIdx.x;
  const long long pos = t / d.b, bi = t - pos * d.b;
  for (int i = threadIdx.x; i < d.rope; i += blockDim.x) {
    c[i] = cos[pos * d.rope + i];
    s[i] = sin[pos * d.rope + i];
  }
  __syncthreads();
  const int pairs8 = d.rope / 16;
  if ((int)threadIdx.x < pairs8) {
    const T* src = k_pe + pos * sp.s + bi * sp.b;
    const int j = threadIdx.x;
    Vec8<T> a, b;
    a.load(src + first_col(j, d)); b.load(src + second_col(j, d));
    float u[8], w[8];
    a.to_float(u); b.to_float(w);
    rot16(u, w, c, s, j, d, false);
#pragma unroll
    for (int i = 0; i < 8; ++i) { pe[first_col(j, d) + i] = u[i]; pe[second_col(j, d) + i] = w[i]; }
  }
  __syncthreads();
  const int qk = d.nope + d.rope, kw = d.nope + d.vd;
  const T *q0 = q + t * d.n * qk, *kv0 = kv + t * d.n * kw;
  T *qf0 = qf + t * d.n * qk, *kf0 = kf + t * d.n * qk, *v0 = v + t * d.n * d.vd;
  copy_heads<T, N8>(qf0, qk, q0, qk, d.n, d.nope / 8);
  copy_heads<T, N8>(kf0, qk, kv0, kw, d.n, d.nope / 8);
  copy_heads<T, V8>(v0, d.vd, kv0 + d.nope, kw, d.n, d.vd / 8);
  rotate_heads<T, R8 / 2>(qf0 + d.nope, qk, q0 + d.nope, qk, c, s, d, false);
  const int r8 = R8 ? R8 : d.rope / 8;
  for (int i = threadIdx.x; i < d.n * r8; i += blockDim.x) {
    const int h = i / r8, k = i - h * r8;
    Vec8<T> x;
    x.from_float(pe + 8 * k);
    x.store(kf0 + h * qk + d.nope + 8 * k);
  }
}

template <typename T, int N8, int R8, int V8>
__global__ void __launch_bounds__(256) mla_heads_bwd_kernel(const T* __restrict__ dqf, Strided sq, const T* __restrict__ dkf, Strided sk,
                                                            const T* __restrict__ dv, Strided sv, const float* __restrict__ cos,
                                                            const float* __restrict__ sin, T* __restrict__ dq, T* __restrict__ dkv,
                                                            T* __restrict__ dk_pe, MlaDims d) {
  extern __shared__ float sh[];                        // cos | sin | sum over heads
  float *c = sh, *s = sh + d.rope, *pe = sh + 2 * d.rope;
  const long long t = blockIdx.x;
  const long long pos = t / d.b, bi = t - pos * d.b;
  for (int i = threadIdx.x; i < d.rope; i += blockDim.x) {
    c[i] = cos[pos * d.rope + i];
    s[i] = sin[pos * d.rope + i];
  }
  const T *dq0 = dqf + pos * sq.s + bi * sq.b, *dk0 = dkf + pos * sk.s + bi * sk.b, *dv0 = dv + pos * sv.s + bi * sv.b;
  __syncthreads();
  const int pairs8 = d.rope / 16, qk = d.nope + d.rope, kw = d.nope + d.vd;
  T *q0 = dq + t * d.n * qk, *kv0 = dkv + t * d.n * kw;
  copy_heads<T, N8>(q0, qk, dq0, sq.h, d.n, d.nope / 8);
  copy_heads<T, N8>(kv0, kw, dk0, sk.h, d.n, d.nope / 8);
  copy_heads<T, V8>(kv0 + d.nope, kw, dv0, sv.h, d.n, d.vd / 8);
  rotate_heads<T, R8 / 2>(q0 + d.nope, qk, dq0 + d.nope, sq.h, c, s, d, true);
  // sum over heads: eight columns a thread, the heads dealt to `parts` threads a column whose sums meet in a fixed order
  const int r8 = d.rope / 8, parts = max(1, min(d.n, (int)blockDim.x / r8));
  for (int i = threadIdx.x; i < r8 * parts; i += blockDim.x) {
    const int part = i / r8, k = i - part * r8;
    float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int h = part; h < d.n; h += parts) {
      Vec8<T> x;
      float f[8];
      x.load(dk0 + h * sk.h + d.nope + 8 * k);
      x.to_float(f);
#pragma unroll
      for (int e = 0; e < 8; ++e) sum[e] += f[e];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) pe[(1 + part) * d.rope + 8 * k + e] = sum[e];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < d.rope; i += blockDim.x) {
    float sum = 0.f;
    for (int part = 0; part < parts; ++part) sum += pe[(1 + part) * d.rope + i];
    pe[i] = sum;
  }
  __syncthreads();
  if ((int)threadIdx.x < pairs8) {
    const int j = threadIdx.x;
    T* dst = dk_pe + t * d.rope;
    float u[8], w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { u[i] = pe[first_col(j, d) + i]; w[i] = pe[second_col(j, d) + i]; }
    rot16(u, w, c, s, j, d, true);
    Vec8<T> x;
    x.from_float(u); x.store(dst + first_col(j, d));
    x.from_float(w); x.store(dst + second_col(j, d));
  }
}

int check_dims(long long tokens, const MlaDims& d) {
  MSB_REQUIRE(d.n > 0 && d.b > 0 && d.nope % 8 == 0 && d.vd % 8 == 0 && d.rope % 16 == 0 && d.rope > 0 && d.rope <= 2048 && d.nope >= 0 && d.vd > 0,
              "mla_heads: bad widths n=%d nope=%d rope=%d v=%d", d.n, d.nope, d.rope, d.vd);
  MSB_REQUIRE(tokens < 0x7fffffffll, "mla_heads: too many tokens (%lld)", tokens);
  return 0;
}
}  // namespace

// q [tokens, n, nope + rope], kv [tokens, n, nope + vd] contiguous; k_pe with element strides (position, batch); tokens = positions * b;
// cos / sin [positions, rope] fp32.  All rows 16-byte aligned.
MSB_API int msb_mla_heads_fwd(const void* q, const void* kv, const void* k_pe, long long pe_s, long long pe_b, const float* cos, const float* sin,
                              void* qf, void* kf, void* v, long long tokens, int b, int n, int nope, int rope, int vd, int interleaved,
                              int dtype, cudaStream_t s) {
  if (tokens == 0) return 0;
  MlaDims d{n, nope, rope, vd, b, interleaved};
  int rc = check_dims(tokens, d); if (rc) return rc;
  Strided sp{pe_s, pe_b, 0};
  const bool common = nope == 128 && rope == 64 && vd == 128;      // widths known at compile time: no divisions, unrolled copies
  MSB_DISPATCH_FLOAT(dtype, T, {
    auto kern = common ? mla_heads_fwd_kernel<T, 16, 8, 16> : mla_heads_fwd_kernel<T, 0, 0, 0>;
    kern<<<(unsigned)tokens, 256, 3 * rope * sizeof(float), s>>>((const T*)q, (const T*)kv, (const T*)k_pe, sp, cos, sin, (T*)qf, (T*)kf, (T*)v, d);
  });
  MSB_CHECK_LAUNCH("mla_heads_fwd");
  return 0;
}
// dqf, dkf [.., nope + rope], dv [.., vd] with element strides (position, batch, head); dq, dkv, dk_pe contiguous.
MSB_API int msb_mla_heads_bwd(const void* dqf, long long q_s, long long q_b, long long q_h, const void* dkf, long long k_s, long long k_b,
                              long long k_h, const void* dv, long long v_s, long long v_b, long long v_h, const float* cos, const float* sin,
                              void* dq, void* dkv, void* dk_pe, long long tokens, int b, int n, int nope, int rope, int vd, int interleaved,
                              int dtype, cudaStream_t s) {
  if (tokens == 0) return 0;
  MlaDims d{n, nope, rope, vd, b, interleaved};
  int rc = check_dims(tokens, d); if (rc) return rc;
  Strided sq{q_s, q_b, q_h}, sk{k_s, k_b, k_h}, sv{v_s, v_b, v_h};
  const bool common = nope == 128 && rope == 64 && vd == 128;
  const int r8 = rope / 8, parts = 256 / r8 < n ? (256 / r8 < 1 ? 1 : 256 / r8) : n;
  const size_t sh = (size_t)(3 + parts) * rope * sizeof(float);
  MSB_DISPATCH_FLOAT(dtype, T, {
    auto kern = common ? mla_heads_bwd_kernel<T, 16, 8, 16> : mla_heads_bwd_kernel<T, 0, 0, 0>;
    kern<<<(unsigned)tokens, 256, sh, s>>>((const T*)dqf, sq, (const T*)dkf, sk, (const T*)dv, sv, cos, sin, (T*)dq, (T*)dkv, (T*)dk_pe, d);
  });
  MSB_CHECK_LAUNCH("mla_heads_bwd");
  return 0;
}
