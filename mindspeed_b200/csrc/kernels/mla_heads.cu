// Heads of multi-head latent attention: one pass that splits the up-projections, rotates the positional part of the queries and of
// the shared key, and writes q, k and v as the attention kernels read them; and its backward.
//
//   forward   q [T, n, nope + rope], kv [T, n, nope + vd], k_pe [T, rope]  ->  qf [T, n, nope + rope] (last `rope` rotated),
//             kf [T, n, nope + rope] = (k of kv | rotated k_pe, the same for every head), v [T, n, vd]
//   backward  dqf, dkf, dv -> dq, dkv and dk_pe (summed over the heads in fp32, in head order, then rotated back and rounded once)
//
// Bound by memory: every value is read and written once.  A block owns a token, so that k_pe, the angles and the sum over heads
// stay on the SM; 16-byte accesses.  (As slices, concatenations and element-wise rotations in PyTorch the same work made 12
// passes, most of them strided.)
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

template <typename T>
__device__ __forceinline__ void copy8(T* dst, const T* src) { Vec8<T> t; t.load(src); t.store(dst); }

template <typename T>
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
  // items of a head, 8 columns each: q nope | q pairs (16 columns) | k nope | k rotary | v
  const int i0 = d.nope / 8, i1 = i0 + pairs8, i2 = i1 + d.nope / 8, i3 = i2 + d.rope / 8, per = i3 + d.vd / 8;
  for (int i = threadIdx.x; i < d.n * per; i += blockDim.x) {
    const int h = i / per, k = i - h * per;
    if (k < i0) {
      copy8(qf0 + h * qk + 8 * k, q0 + h * qk + 8 * k);
    } else if (k < i1) {
      const int j = k - i0, a = d.nope + first_col(j, d), b = d.nope + second_col(j, d);
      Vec8<T> x, y;
      x.load(q0 + h * qk + a); y.load(q0 + h * qk + b);
      float u[8], w[8];
      x.to_float(u); y.to_float(w);
      rot16(u, w, c, s, j, d, false);
      x.from_float(u); y.from_float(w);
      x.store(qf0 + h * qk + a); y.store(qf0 + h * qk + b);
    } else if (k < i2) {
      copy8(kf0 + h * qk + 8 * (k - i1), kv0 + h * kw + 8 * (k - i1));
    } else if (k < i3) {
      Vec8<T> x;
      x.from_float(pe + 8 * (k - i2));
      x.store(kf0 + h * qk + d.nope + 8 * (k - i2));
    } else {
      copy8(v0 + h * d.vd + 8 * (k - i3), kv0 + h * kw + d.nope + 8 * (k - i3));
    }
  }
}

template <typename T>
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
  const int i0 = d.nope / 8, i1 = i0 + pairs8, i2 = i1 + d.nope / 8, per = i2 + d.vd / 8;
  for (int i = threadIdx.x; i < d.n * per; i += blockDim.x) {
    const int h = i / per, k = i - h * per;
    if (k < i0) {
      copy8(q0 + h * qk + 8 * k, dq0 + h * sq.h + 8 * k);
    } else if (k < i1) {
      const int j = k - i0, a = d.nope + first_col(j, d), b = d.nope + second_col(j, d);
      Vec8<T> x, y;
      x.load(dq0 + h * sq.h + a); y.load(dq0 + h * sq.h + b);
      float u[8], w[8];
      x.to_float(u); y.to_float(w);
      rot16(u, w, c, s, j, d, true);
      x.from_float(u); y.from_float(w);
      x.store(q0 + h * qk + a); y.store(q0 + h * qk + b);
    } else if (k < i2) {
      copy8(kv0 + h * kw + 8 * (k - i1), dk0 + h * sk.h + 8 * (k - i1));
    } else {
      copy8(kv0 + h * kw + d.nope + 8 * (k - i2), dv0 + h * sv.h + 8 * (k - i2));
    }
  }
  for (int i = threadIdx.x; i < d.rope; i += blockDim.x) {             // a column per thread, heads in order
    float sum = 0.f;
#pragma unroll 8
    for (int h = 0; h < d.n; ++h) sum += to_f(dk0[h * sk.h + d.nope + i]);
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
  MSB_DISPATCH_FLOAT(dtype, T, mla_heads_fwd_kernel<T><<<(unsigned)tokens, 256, 3 * rope * sizeof(float), s>>>((const T*)q, (const T*)kv, (const T*)k_pe,
                     sp, cos, sin, (T*)qf, (T*)kf, (T*)v, d));
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
  MSB_DISPATCH_FLOAT(dtype, T, mla_heads_bwd_kernel<T><<<(unsigned)tokens, 256, 3 * rope * sizeof(float), s>>>((const T*)dqf, sq, (const T*)dkf, sk,
                     (const T*)dv, sv, cos, sin, (T*)dq, (T*)dkv, (T*)dk_pe, d));
  MSB_CHECK_LAUNCH("mla_heads_bwd");
  return 0;
}
