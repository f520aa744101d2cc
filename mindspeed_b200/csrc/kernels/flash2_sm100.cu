// Flash attention forward for sm_100a, two query tiles per CTA: while the softmax warps of one tile work, the tensor core
// runs the other tile's MMAs.  head_dim 128, bf16, causal or full, GQA, query offset (for chunked / ring use).
//
// One CTA owns 256 query rows (two tiles of 128) of one (batch, head) and walks the key/value tiles of 128 keys.
//   TMEM (512 columns)  S0 | S1 | O0 | O1, 128 fp32 columns each.  The probabilities P_t overwrite the first 64 columns of
//                       S_t as packed bf16 and feed the P V MMA as its A operand straight from tensor memory.
//   warp 8              TMA producer: Q0 and Q1 once, K_j and V_j into separate 2-stage rings
//   warp 9              MMA issuer (one thread):  S_t = Q_t K_j^T,  O_t += P_t V_j.  Issue order
//                       S0 S1 | PV0 S0' | PV1 S1' | ...   so tile t's softmax overlaps the other tile's MMAs
//   warps 0-3 / 4-7     softmax of tile 0 / tile 1, one thread per query row: row maximum (four chains of three-input maxima), exp2,
//                       row sum, P -> TMEM.  They hold a whole score row per thread (setmaxnreg).
//                       O stays in tensor memory; it is rescaled only when the running maximum grew by more than 2^8
//                       since the last rescale (the stale maximum is used for P meanwhile, which stays within range),
//                       so most key tiles never touch O.
// The issuing thread is what bounds it, a softmax warp waits a third of the time: a barrier costs it 75 to 150 cycles, done or
// not.  One commit frees K and V, the scores' commit stands for P V as well, descriptors are one addition each.  s = 8192, 32 / 8
// heads, causal: 573 us at first, 521 with the softmax above, 487 with the heaviest tiles first, 468 with this issue (474 with the row
// sum in the order of the keys).
// Epilogue: O / l -> bf16 -> shared memory (the tile's Q buffer) -> TMA store; LSE (natural log) to global memory.
// reference semantics: torch_npu.npu_fusion_attention returning softmax max/sum
// (mindspeed/core/transformer/flash_attention/flash_attention/adaptor.py:21-85, mindspeed/ops/fusion_attention_v2.py:22-114).
#include "msb_common.cuh"
#include "msb_sm100.cuh"

using namespace msb;
using namespace msb::sm100;

namespace {
constexpr int FB = 128;                   // rows per Q tile, keys per KV tile
constexpr int FD = 128;                   // head dim
constexpr int TILE_BYTES = FB * FD * 2;   // 32 KB
constexpr int HALF_BYTES = FB * 128;      // one 64-wide column block: 128 rows x 128 B
constexpr float RESCALE_THRESHOLD = 8.f;  // log2 units

struct Fwd2Params {
  CUtensorMap tmQ;                 // dims {d, head of the group, group, batch, seq}: the heads of a packed QKV activation are not evenly spaced
  CUtensorMap tmK, tmV, tmO;       // dims {d, head, batch, seq}
  float* lse;                      // [b, nq, sq]
  __nv_bfloat16* O;                // [sq, b, nq, d] (direct stores for rows without any visible key)
  int sq, sk, b, nq, nkv;
  int causal;
  int q_offset;                    // key index visible to query row r is <= r + q_offset
  int group;                       // (batch, head) pairs whose CTAs are numbered together
  float scale_log2;                // softmax_scale * log2(e)
  unsigned int* status;
};

struct Fwd2Smem {
  static constexpr int Q_OFF = 0;                          // 2 tiles
  static constexpr int K_OFF = 2 * TILE_BYTES;             // 2 stages
  static constexpr int V_OFF = K_OFF + 2 * TILE_BYTES;     // 2 stages
  static constexpr int BAR_OFF = V_OFF + 2 * TILE_BYTES;   // 192 KB
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

__device__ __forceinline__ void named_bar(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const void* tmap, uint32_t bar, int x, int y, int z, int v, int w) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(v), "r"(w)
      : "memory");
}
__device__ __forceinline__ void tma_store_4d(const void* tmap, uint32_t src, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tmap)),
               "r"(src), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}

// maximum of three (one instruction on sm_100)
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

constexpr int FWD_THREADS = 12 * 32;

__global__ void __launch_bounds__(FWD_THREADS, 1) flash_fwd2_sm100_kernel(const __grid_constant__ Fwd2Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar = base + Fwd2Smem::BAR_OFF;
  const uint32_t q_full = bar;
  auto k_full = [&](int s) { return bar + 8u * (1 + s); };
  auto v_full = [&](int s) { return bar + 8u * (3 + s); };
  auto s_full = [&](int t) { return bar + 8u * (5 + t); };
  auto p_full = [&](int t) { return bar + 8u * (7 + t); };
  auto kv_free = [&](int s) { return bar + 8u * (9 + s); };
  const uint32_t o_done = bar + 8u * 11, tmem_slot = bar + 8u * 12;
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(base_ptr + Fwd2Smem::BAR_OFF + 8 * 12);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // (batch, head) pairs in groups of p.group; inside a group the query tiles that see most keys first and the heads fastest, so that
  // the last CTAs to start are short ones of several heads
  const int n_m = (p.sq + 2 * FB - 1) / (2 * FB), bh_all = p.b * p.nq;
  const int grp = (int)(blockIdx.x / (unsigned)(p.group * n_m)), first_bh = grp * p.group, in_grp = min(bh_all - first_bh, p.group);
  const int rank = (int)(blockIdx.x - (unsigned)(grp * p.group * n_m));
  const int m_rank = rank / in_grp, bh = first_bh + (rank - m_rank * in_grp);
  const int m_blk = p.causal ? n_m - 1 - m_rank : m_rank;
  const int batch = bh / p.nq, head = bh - batch * p.nq;
  const int kv_head = head / (p.nq / p.nkv);
  const int q0 = m_blk * 2 * FB;
  const int n_all = (p.sk + FB - 1) / FB;
  int n_t[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    int n = n_all;
    const int first = q0 + t * FB;
    if (first >= p.sq) n = 0;
    else if (p.causal) {
      const int last_key = min(first + FB - 1, p.sq - 1) + p.q_offset;    // last key any row of this tile may see
      n = last_key < 0 ? 0 : min(n, last_key / FB + 1);
    }
    n_t[t] = n;
  }
  const int n_max = max(n_t[0], n_t[1]);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < 2; ++s) { mbar_init(k_full(s), 1); mbar_init(v_full(s), 1); }
    for (int t = 0; t < 2; ++t) { mbar_init(s_full(t), 1); mbar_init(p_full(t), 4); }
    mbar_init(kv_free(0), 1); mbar_init(kv_free(1), 1); mbar_init(o_done, 1);
    mbar_fence_init();
  }
  if (warp == 9) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  constexpr uint32_t tmem_base = 0;          // all 512 columns are ours
  if (*tmem_slot_ptr != tmem_base && threadIdx.x == 0) atomicCAS(p.status, 0u, 0x301u);

  // registers of the launch: 384 x 168 = 64512; the two softmax warpgroups hold a whole score row per thread
  if (warp >= 8) {       // warps 10 and 11 only complete the warpgroup that gives registers away
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    if (warp == 8) {
      // ===================== TMA producer =====================
      if (lane == 0 && n_max > 0) {
        mbar_arrive_expect_tx(q_full, 2 * TILE_BYTES);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const uint32_t qs = base + Fwd2Smem::Q_OFF + t * TILE_BYTES;
          tma_load_5d(qs, &p.tmQ, q_full, 0, head - kv_head * (p.nq / p.nkv), kv_head, batch, q0 + t * FB);
          tma_load_5d(qs + HALF_BYTES, &p.tmQ, q_full, 64, head - kv_head * (p.nq / p.nkv), kv_head, batch, q0 + t * FB);
        }
        auto load = [&](uint32_t dst, const CUtensorMap* tm, uint32_t full, int j) {
          mbar_arrive_expect_tx(full, TILE_BYTES);
          tma_load_4d(dst, tm, full, 0, kv_head, batch, j * FB);
          tma_load_4d(dst + HALF_BYTES, tm, full, 64, kv_head, batch, j * FB);
        };
        auto load_k = [&](int j) { if (j < n_max) load(base + Fwd2Smem::K_OFF + (j & 1) * TILE_BYTES, &p.tmK, k_full(j & 1), j); };
        auto load_v = [&](int j) { if (j < n_max) load(base + Fwd2Smem::V_OFF + (j & 1) * TILE_BYTES, &p.tmV, v_full(j & 1), j); };
        load_k(0); load_v(0); load_k(1); load_v(1);
        // kv_free(c & 1): the scores of key tile c and P V of tile c - 1 are done, so K_c and V_c-1 may be overwritten.  Two barriers in
        // turn: the one after next needs tiles that are only loaded here, so no phase can pass unseen.
        for (int c = 0; c + 1 < n_max; ++c) {
          if (!mbar_wait(kv_free(c & 1), (uint32_t)((c >> 1) & 1), p.status, 0x310u)) break;
          if (c > 0) load_v(c + 1);
          load_k(c + 2);
        }
      }
    } else if (warp == 9) {
      // ===================== MMA issuer =====================
      if (lane == 0 && n_max > 0) {
        constexpr uint32_t idesc_qk = make_idesc_f16(128, 128, 1, 0, 0);
        constexpr uint32_t idesc_pv = make_idesc_f16(128, 128, 1, 0, 1);
        // descriptors of tile 0 / stage 0; an address grows by 16-byte units in the low word
        const uint64_t qd = make_smem_desc(base + Fwd2Smem::Q_OFF, 0, 1024), kd = make_smem_desc(base + Fwd2Smem::K_OFF, 0, 1024);
        const uint64_t vd = make_smem_desc(base + Fwd2Smem::V_OFF, HALF_BYTES, 1024);
        auto wait = [&](uint32_t b, uint32_t parity, unsigned int code) {
          const bool ok = mbar_wait(b, parity, p.status, code);
          tc_fence_after();
          return ok;
        };
        auto issue_s = [&](int t, int j) {
          const uint64_t q0d = qd + (uint64_t)(t * (TILE_BYTES >> 4)), k0d = kd + (uint64_t)((j & 1) * (TILE_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < FD / 16; ++k) {
            const uint64_t off = (uint64_t)(((k >> 2) * HALF_BYTES + (k & 3) * 32) >> 4);
            umma_f16(tmem_base + (uint32_t)(t * 128), q0d + off, k0d + off, idesc_qk, k ? 1u : 0u);
          }
          umma_commit(s_full(t));       // completes after everything issued before: P V of the last key tile is in O as well
        };
        auto issue_pv = [&](int t, int j) {
          const uint64_t v0d = vd + (uint64_t)((j & 1) * (TILE_BYTES >> 4));
          const uint32_t tP = tmem_base + (uint32_t)(t * 128), tO = tmem_base + 256u + (uint32_t)(t * 128);
#pragma unroll
          for (int k = 0; k < FB / 16; ++k)      // MN-major: 16 keys = 2048 B; 16 bf16 of P = 8 columns
            umma_f16_ts(tO, tP + (uint32_t)(k * 8), v0d + (uint64_t)(k * (16 * 128 >> 4)), idesc_pv, (j | k) ? 1u : 0u);
        };
        bool ok = wait(q_full, 0, 0x320u);
        if (ok) ok = wait(k_full(0), 0, 0x321u);
        if (ok) {
          if (n_t[0] > 0) issue_s(0, 0);
          if (n_t[1] > 0) issue_s(1, 0);
          umma_commit(kv_free(0));
        }
        for (int j = 0; j < n_max && ok; ++j) {
          const uint32_t ph = (uint32_t)((j >> 1) & 1), jp = (uint32_t)(j & 1);
          if (!(ok = wait(v_full(j & 1), ph, 0x322u))) break;
          if (j + 1 < n_max && !(ok = wait(k_full((j + 1) & 1), (uint32_t)(((j + 1) >> 1) & 1), 0x324u))) break;
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (j < n_t[t]) {
              if (!(ok = wait(p_full(t), jp, 0x323u))) break;
              issue_pv(t, j);
            }
            if (j + 1 < n_t[t]) issue_s(t, j + 1);
          }
          if (!ok) break;
          umma_commit(kv_free((j + 1) & 1));
        }
        if (ok) umma_commit(o_done);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");     // 256 x 208 + 128 x 80 = 63488
    // ===================== softmax (warps 0-3: tile 0, warps 4-7: tile 1) =====================
    const int t = warp >> 2;
    const int q = warp & 3;
    const int row = q * 32 + lane;                 // row inside the tile == TMEM lane
    const int q_idx = q0 + t * FB + row;
    const uint32_t lane_addr = ((uint32_t)(q * 32) << 16);
    const uint32_t tS = tmem_base + (uint32_t)(t * 128) + lane_addr;
    const uint32_t tO = tmem_base + 256u + (uint32_t)(t * 128) + lane_addr;
    const int n_kv = n_t[t];
    float m_used = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < n_kv && ok; ++j) {
      const uint32_t jp = (uint32_t)(j & 1);
      if (!mbar_wait(s_full(t), jp, p.status, 0x330u)) { ok = false; break; }
      tc_fence_after();
      const int key0 = j * FB;
      const int limit = p.causal ? (q_idx + p.q_offset - key0) : FB;    // keys [0, limit] of this tile are visible to this row
      const int vis = min(limit, p.sk - 1 - key0);
      const bool need_mask = vis < FB - 1;
      // the whole score row into registers (four loads in flight, one wait), masked where needed
      uint32_t sv[FB];
#pragma unroll
      for (int c = 0; c < FB; c += 32) tmem_ld_32x32(tS + (uint32_t)c, sv + c);
      tmem_ld_wait();
      if (__any_sync(0xffffffffu, need_mask)) {
#pragma unroll
        for (int i = 0; i < FB; ++i)
          if (i > vis) sv[i] = 0xff800000u;              // -inf
      }
      // four independent chains of three-input maxima: one chain of 128 would cost its latency 128 times
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < FB; i += 8)
#pragma unroll
        for (int e = 0; e < 4; ++e) mx[e] = max3(mx[e], __uint_as_float(sv[i + 2 * e]), __uint_as_float(sv[i + 2 * e + 1]));
      const float m_tile = fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]);
      const float m_tile2 = m_tile * p.scale_log2;
      // rescale O only when the maximum has grown a lot (decision per warp: the TMEM accesses are warp-wide)
      const bool grow = m_tile2 > m_used + RESCALE_THRESHOLD || (m_used == -INFINITY && m_tile2 > -INFINITY);
      if (__any_sync(0xffffffffu, grow)) {
        const float m_new = fmaxf(m_used, m_tile2);
        const float alpha = (m_used == -INFINITY) ? 0.f : exp2f(m_used - m_new);
        if (j > 0) {                             // the scores' commit covered P V of tile j - 1, which is in O
#pragma unroll 1
          for (int c = 0; c < FD; c += 32) {
            uint32_t r[32];
            tmem_ld_32x32(tO + (uint32_t)c, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
            tmem_st_32x32(tO + (uint32_t)c, r);
          }
          tmem_st_wait();
        }
        l_run *= alpha;
        m_used = m_new;
      }
      const float m_ref = (m_used == -INFINITY) ? 0.f : m_used;
      // probabilities -> packed bf16 over the first 64 columns of S, row sum (masked scores are -inf -> 0)
      const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2), nref2 = pack_f32x2(-m_ref, -m_ref);
      // The row sum takes the keys in order, pair after pair: the log-sum-exp's last bits, and with them bf16 roundings of the output, show
      // the order.  (Four interleaved chains of packed additions: 463 us instead of 474 at s = 8192, 32 / 8 heads, causal.  Summed
      // after P is handed over: no difference.)
      float l_tile = 0.f;
#pragma unroll
      for (int c = 0; c < FB; c += 32) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float pa, pb;
          unpack_f32x2(fma_f32x2(pack_u32x2(sv[c + 2 * i], sv[c + 2 * i + 1]), scale2, nref2), pa, pb);
          pa = exp2f(pa);
          pb = exp2f(pb);
          l_tile += pa + pb;
          pk[i] = pack_bf16(pa, pb);
        }
        tmem_st_32x16(tS + (uint32_t)(c >> 1), pk);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full(t));       // one arrival per warp: 128 on one barrier would serialise
      l_run += l_tile;
    }
    // ---- epilogue of this tile ----
    if (n_kv > 0) {
      if (ok) ok = mbar_wait(o_done, 0, p.status, 0x332u);
      tc_fence_after();
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      uint8_t* o_row = base_ptr + Fwd2Smem::Q_OFF + t * TILE_BYTES + row * 128;   // the tile's Q buffer: no MMA reads it any more
      if (ok) {
#pragma unroll 1
        for (int c = 0; c < FD; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32(tO + (uint32_t)c, r);
          tmem_ld_wait();
          uint8_t* blk = o_row + (c >> 6) * HALF_BYTES;
          const int chunk0 = (c & 63) >> 3;
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            uint32_t pk[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[8 * ch + 2 * e]) * inv, __uint_as_float(r[8 * ch + 2 * e + 1]) * inv);
              pk[e] = *reinterpret_cast<uint32_t*>(&h);
            }
            *reinterpret_cast<uint4*>(blk + (((chunk0 + ch) ^ (row & 7)) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          }
        }
        if (q_idx < p.sq)
          p.lse[((size_t)batch * p.nq + head) * p.sq + q_idx] =
              (l_run > 0.f) ? m_used * 0.6931471805599453f + __logf(l_run) : -INFINITY;
      }
      fence_proxy_async_smem();
      named_bar(1 + t, 128);
      if (ok && q == 0 && lane == 0) {     // one thread: both 64-column halves of the tile (rows past sq are clipped)
        const uint32_t os = base + Fwd2Smem::Q_OFF + t * TILE_BYTES;
        tma_store_4d(&p.tmO, os, 0, head, batch, q0 + t * FB);
        tma_store_4d(&p.tmO, os + HALF_BYTES, 64, head, batch, q0 + t * FB);
        tma_store_commit();
        tma_store_wait<0>();
      }
    } else if (q_idx < p.sq) {
      // no key is visible to any row of this tile: zero output, -inf LSE
      __nv_bfloat16* orow = p.O + (((size_t)q_idx * p.b + batch) * p.nq + head) * FD;
      for (int c = 0; c < FD; c += 8) *reinterpret_cast<uint4*>(orow + c) = make_uint4(0, 0, 0, 0);
      p.lse[((size_t)batch * p.nq + head) * p.sq + q_idx] = -INFINITY;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

int make_map4(CUtensorMap* tm, const void* base, int seq, int heads, int b, long long ss, long long sb, long long sh) {
  uint64_t dims[4] = {(uint64_t)FD, (uint64_t)heads, (uint64_t)b, (uint64_t)seq};
  uint64_t str[3] = {(uint64_t)sh * 2, (uint64_t)sb * 2, (uint64_t)ss * 2};
  uint32_t box[4] = {64, 1, 1, (uint32_t)FB};
  return make_tmap_nd(tm, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 4, dims, str, box);
}
// queries: groups of `rep` heads, strides between heads of a group (sh) and between groups (gs)
int make_map_q(CUtensorMap* tm, const void* base, int seq, int rep, int groups, int b, long long ss, long long sb, long long gs, long long sh) {
  uint64_t dims[5] = {(uint64_t)FD, (uint64_t)rep, (uint64_t)groups, (uint64_t)b, (uint64_t)seq};
  uint64_t str[4] = {(uint64_t)sh * 2, (uint64_t)gs * 2, (uint64_t)sb * 2, (uint64_t)ss * 2};
  uint32_t box[5] = {64, 1, 1, 1, (uint32_t)FB};
  return make_tmap_nd(tm, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 5, dims, str, box);
}
}  // namespace

// q [sq, b, nkv, nq / nkv, 128] with element strides (seq, batch, group, head), k / v [sk, b, nkv, 128] with (seq, batch, head), bf16, last
// dim contiguous;
// o [sq, b, nq, 128] contiguous; lse [b, nq, sq] fp32 (natural log of the scaled scores' softmax denominator).
MSB_API int msb_flash_fwd2(const void* q, const void* k, const void* v, void* o, float* lse, int sq, int sk, int b, int nq, int nkv,
                           long long q_ss, long long q_sb, long long q_gs, long long q_sh, long long k_ss, long long k_sb, long long k_sh,
                           long long v_ss, long long v_sb, long long v_sh, int causal, int q_offset, float scale,
                           unsigned int* status, cudaStream_t s) {
  MSB_REQUIRE(sq > 0 && sk > 0 && nq % nkv == 0, "flash_fwd2: bad shape sq=%d sk=%d nq=%d nkv=%d", sq, sk, nq, nkv);
  MSB_REQUIRE(status != nullptr, "flash_fwd2: status word is required");
  Fwd2Params p;
  memset(&p, 0, sizeof(p));
  int rc = make_map_q(&p.tmQ, q, sq, nq / nkv, nkv, b, q_ss, q_sb, q_gs, q_sh); if (rc) return rc;
  rc = make_map4(&p.tmK, k, sk, nkv, b, k_ss, k_sb, k_sh); if (rc) return rc;
  rc = make_map4(&p.tmV, v, sk, nkv, b, v_ss, v_sb, v_sh); if (rc) return rc;
  rc = make_map4(&p.tmO, o, sq, nq, b, (long long)b * nq * FD, (long long)nq * FD, FD); if (rc) return rc;
  p.O = (__nv_bfloat16*)o; p.lse = lse;
  p.sq = sq; p.sk = sk; p.b = b; p.nq = nq; p.nkv = nkv; p.causal = causal; p.q_offset = q_offset;
  p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
  static std::atomic<unsigned long long> stated{0};
  if (int bad = msb::allow_smem((const void*)flash_fwd2_sm100_kernel, Fwd2Smem::TOTAL, "flash_fwd2", stated)) return bad;
  // A group is as many heads as have their K and V in half of L2 (48 MB): every CTA that runs at a time then streams from L2, and the
  // group is wide enough that its shortest CTAs end the launch.  s = 4096, 32 / 8 heads, one head after the other: an SM was busy for
  // three quarters of the launch.
  const int rep = nq / nkv, n_m = (sq + 2 * FB - 1) / (2 * FB);
  const long long kv_heads = (48ll << 20) / ((long long)sk * FD * 4), bh = (long long)b * nq;
  const long long ctas = bh * n_m;
  MSB_REQUIRE(ctas <= 0x7fffffffll, "flash_fwd2: grid too large (%lld)", ctas);
  const long long want = (kv_heads < 1 ? 1 : kv_heads) * rep;
  p.group = (int)(want < bh ? want : bh);
  dim3 grid((unsigned)ctas);
  flash_fwd2_sm100_kernel<<<grid, FWD_THREADS, Fwd2Smem::TOTAL, s>>>(p);
  MSB_CHECK_LAUNCH("flash_fwd2_sm100");
  return 0;
}

// =====================================================================================================================
// Flash attention backward for sm_100a.  head_dim 128, bf16, causal or full, GQA, query offset.
//
// One CTA owns a tile of 128 keys of one (batch, KV head) and walks every query tile of every query head of that KV head
// that can see it.  All five products of an iteration run on tcgen05 in the transposed formulation (keys on the TMEM lanes):
//     S^T  = K Q^T          A = K  (smem, K-major)      B = Q  (smem, K-major)
//     dP^T = V dO^T         A = V  (smem, K-major)      B = dO (smem, K-major)
//     dV  += P^T dO         A = P^T  (TMEM, packed bf16 over the scores)        B = dO (smem, MN-major)
//     dK  += dS^T Q         A = dS^T (TMEM, packed bf16 over dP^T)              B = Q  (smem, MN-major)
//     dQ   = dS K           A = dS^T as written to smem [keys, q] = dS MN-major B = K  (smem, MN-major)
// TMEM (512 columns): S^T | dP^T, then dQ | dV | dK.  A warp packs the 64 score columns it has read over the first half of those same
// columns, so the two halves of a row need no agreement.
// Issue order:  S(0) dP(0) | dV(i) S(i+1) dK(i) dQ(i) dP(i+1) | ...   While the compute warps turn S(i+1) into P, the tensor core runs
// dK and dQ of tile i; while they turn dP(i+1) into dS, it runs dV(i+1) and S(i+2).  Only the read-out of dQ(i), whose columns
// dP(i+1) takes, is not covered.
//   warp 0        TMA producer: K, V once; Q_i with its statistics into a 2-stage ring, dO_i into one stage (its last reader, dV(i),
//                 comes 1500 cycles of MMA before dP(i+1) needs the next)
//   warp 1        MMA issuer (one thread)
//   warps 2-9     warp w: key rows 32 (w mod 4) .. +31 and query columns 0-63 (w < 6) or 64-127:
//                 P^T = exp2(S^T scale log2e - LSE log2e), dS^T = P^T (dP^T - delta), two lanes of arithmetic per instruction, the
//                 statistics of a column by broadcast reads of shared memory
//   warps 10-13   dQ: tensor memory -> softmax scale -> staging -> TMA reduce-add into the fp32 dQ
// Bound: shared memory moves 480 KiB per 128 x 128 tile (operand reads 256, TMA writes of operands 64, dS 32, dQ staging in and out 128),
// 3840 cycles at 128 B a cycle, beside 2560 cycles of MMA.  Measured at s = 8192, 32 / 8 heads, causal: 2173 us with one tile in flight and four
// compute warps, 1251 us so, 1201 with dQ's columns handed back before its first quarter is sent.
// reference semantics: the attention grad op of the reference, mindspeed/ops/csrc/cann/fusion_attention_v2.cpp:431-439.
// =====================================================================================================================
namespace {

struct BwdParams {
  CUtensorMap tmQ;                  // bf16, dims {d, head of the group, group, batch, seq}
  CUtensorMap tmK, tmV, tmdO;       // bf16, dims {d, head, batch, seq}
  CUtensorMap tmdQ;                 // fp32 [sq, b, nq, d], dims {d, head, batch, seq}, box {32, 1, 1, 32}
  CUtensorMap tmdK, tmdV;           // [sk, b, nkv, d] outputs: bf16 stores, or fp32 reduce-add targets (box {32,1,1,32}) when split_heads
  const float* nlse2;               // [b, nq, sq_pad] -LSE * log2(e) (-inf where no key is visible / padding)
  const float* ndelta;              // [b, nq, sq_pad] -rowsum(dO * O)
  int sq, sk, b, nq, nkv, sq_pad;
  int causal, q_offset;
  float scale, scale_log2;
  int split_heads;                  // 1: one CTA per (key tile, QUERY head); dK / dV partial sums are added into fp32 buffers
  unsigned int* status;
};

struct BwdSmem {
  static constexpr int Q_OFF = 0;                          // 2 stages
  static constexpr int DO_OFF = 2 * TILE_BYTES;            // 1 stage: dO_i is last read well before dO_i+1 is first needed
  static constexpr int K_OFF = 3 * TILE_BYTES;
  static constexpr int V_OFF = 4 * TILE_BYTES;
  static constexpr int DS_OFF = 5 * TILE_BYTES;            // dS^T [keys, q] bf16
  static constexpr int DQ_OFF = 6 * TILE_BYTES;            // dQ staging: 8 KB (two 32 x 32 fp32 boxes) per drain warp
  static constexpr int STAT_OFF = 7 * TILE_BYTES;          // 2 stages of 128 x -LSE log2e and 128 x -delta
  static constexpr int STAT_BYTES = 2 * FB * 4;
  static constexpr int BAR_OFF = STAT_OFF + 2 * STAT_BYTES;
  static constexpr int TOTAL = BAR_OFF + 256;              // the base is 1024-byte aligned by declaration: no slack
  static_assert(TOTAL <= 232448, "exceeds the 227 KB of shared memory a CTA may use");
};

__device__ __forceinline__ void bulk_g2s_bar(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_4d(const void* tmap, uint32_t src, int x, int y, int z, int w) {
  asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tmap)),
               "r"(src), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}

// Statistics of the backward: ndelta[b, h, r] = -sum_d dO * O; nlse2 = -LSE * log2(e), with -inf for rows without a visible key and for the
// padding to whole tiles.  Also clears the fp32 accumulators that the main kernel adds into (`zero4` vectors of four).  Bound by the
// read of O and dO and the write of the zeros: 16 lanes per row, 16 bytes a lane.
__global__ void __launch_bounds__(256) flash_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout, long long do_ss,
                                                             long long do_sb, long long do_sh, const float* __restrict__ lse,
                                                             float* __restrict__ nlse2, float* __restrict__ ndelta, int sq, int b, int nq, int sq_pad,
                                                             float4* __restrict__ zero, long long zero4) {
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, threads = (long long)gridDim.x * blockDim.x;
  for (long long i = tid; i < zero4; i += threads) zero[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int l16 = threadIdx.x & 15;
  // row numbers run with the sequence slowest, as O and dO lie in memory; every lane of a warp makes the same number of rounds
  const long long total = (long long)sq_pad * b * nq;
  for (long long w0 = (tid >> 5) * 2; w0 < total; w0 += (threads >> 5) * 2) {
    const long long w = w0 + ((threadIdx.x >> 4) & 1);
    const int h = (int)(w % nq), bb = (int)((w / nq) % b);
    const long long row = w / ((long long)nq * b);
    const bool live = w < total && row < sq;
    float acc = 0.f;
    if (live) {
      const uint4 ov = *reinterpret_cast<const uint4*>(o + w * FD + l16 * 8);
      const uint4 dv = *reinterpret_cast<const uint4*>(dout + row * do_ss + bb * do_sb + h * do_sh + l16 * 8);
      const __nv_bfloat162* oh = reinterpret_cast<const __nv_bfloat162*>(&ov);
      const __nv_bfloat162* dh = reinterpret_cast<const __nv_bfloat162*>(&dv);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = __bfloat1622float2(oh[i]), c = __bfloat1622float2(dh[i]);
        acc += a.x * c.x + a.y * c.y;
      }
    }
#pragma unroll
    for (int d = 8; d; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    if (l16 == 0 && w < total) {
      const float l = live ? lse[((size_t)bb * nq + h) * sq + row] : -INFINITY;
      const size_t at = ((size_t)bb * nq + h) * sq_pad + row;
      ndelta[at] = -acc;
      nlse2[at] = (l == -INFINITY) ? -INFINITY : l * -1.4426950408889634f;
    }
  }
}

// fp32 sums -> bf16 gradients at their place: dQ always, dK and dV when query heads added into fp32 buffers.  16 lanes per 128-wide row.
struct FinishSeg {
  const float* src;                 // [rows, 128]
  __nv_bfloat16* dst;
  long long ss, sb, gs, sh;         // element strides of dst
  int b, groups, per;               // row = ((seq * b + batch) * groups + group) * per + head of the group
  long long rows;
};
struct FinishParams { FinishSeg seg[3]; };
__global__ void __launch_bounds__(256) flash_bwd_finish_kernel(const __grid_constant__ FinishParams p) {
  const int l16 = threadIdx.x & 15;
  const long long r1 = p.seg[0].rows, r2 = r1 + p.seg[1].rows, all = r2 + p.seg[2].rows;
  for (long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 4; r < all; r += ((long long)gridDim.x * blockDim.x) >> 4) {
    const FinishSeg& g = p.seg[r < r1 ? 0 : r < r2 ? 1 : 2];
    const long long w = r - (r < r1 ? 0 : r < r2 ? r1 : r2);
    const float4* src = reinterpret_cast<const float4*>(g.src + w * FD) + 2 * l16;
    const float4 x = src[0], y = src[1];
    const int h = (int)(w % g.per);
    long long t = w / g.per;
    const int gr = (int)(t % g.groups);
    t /= g.groups;
    __nv_bfloat16* dst = g.dst + (t / g.b) * g.ss + (t % g.b) * g.sb + gr * g.gs + h * g.sh + l16 * 8;
    *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w), pack_bf16(y.x, y.y), pack_bf16(y.z, y.w));
  }
}

constexpr int BWD_THREADS = 14 * 32;

__global__ void __launch_bounds__(BWD_THREADS, 1) flash_bwd_sm100_kernel(const __grid_constant__ BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_1k[];
  uint8_t* base_ptr = smem_1k;
  const uint32_t base = smem_u32(smem_1k);
  if (base & 1023u) {                        // the swizzled tiles need it; never seen, and an error rather than wrong results
    if (threadIdx.x == 0) atomicCAS(p.status, 0u, 0x401u);
    return;
  }
  const uint32_t bar = base + BwdSmem::BAR_OFF;
  const uint32_t kv_full = bar;
  auto q_full = [&](int s) { return bar + 8u * (1 + s); };
  auto q_empty = [&](int s) { return bar + 8u * (3 + s); };
  const uint32_t do_full = bar + 8u * 5, do_empty = bar + 8u * 6, st_full = bar + 8u * 7, dpt_full = bar + 8u * 8,
                 pt_ready = bar + 8u * 9, ds_ready = bar + 8u * 10, dq_full = bar + 8u * 11, dq_drained = bar + 8u * 12,
                 acc_done = bar + 8u * 13, tmem_slot = bar + 8u * 14;
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(base_ptr + BwdSmem::BAR_OFF + 8 * 14);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // key tiles that many query tiles see (early ones, when causal) first, over all heads: the last CTAs to start are the shortest
  const int heads = p.split_heads ? p.nq : p.nkv, head_id = (int)(blockIdx.x % (unsigned)heads), j = (int)(blockIdx.x / (unsigned)heads);
  // without the split a CTA walks all query heads of its KV head; with it (few KV heads: too few CTAs otherwise) one each
  const int rep_all = p.nq / p.nkv;
  const int g = p.split_heads ? head_id / rep_all : head_id, batch = blockIdx.z;
  const int head0 = p.split_heads ? head_id : g * rep_all;
  const int rep = p.split_heads ? 1 : rep_all;
  const int key0 = j * FB;
  const int n_q = (p.sq + FB - 1) / FB;
  int i_start = 0;
  if (p.causal) {
    const int first_q = key0 - p.q_offset;                 // first query row that sees key0
    i_start = first_q <= 0 ? 0 : first_q / FB;
  }
  const int n_i = max(n_q - i_start, 0);
  const int n_it = n_i * rep;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < 2; ++s) { mbar_init(q_full(s), 1); mbar_init(q_empty(s), 1); }
    mbar_init(do_full, 1); mbar_init(do_empty, 1);
    mbar_init(st_full, 1); mbar_init(dpt_full, 1); mbar_init(pt_ready, 8); mbar_init(ds_ready, 8);
    mbar_init(dq_full, 1); mbar_init(dq_drained, 4); mbar_init(acc_done, 1);
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  const uint32_t tST = tmem_base, tDPT = tmem_base + 128u, tDV = tmem_base + 256u, tDK = tmem_base + 384u;

  if (warp == 0) {
    // ===================== TMA producer =====================
    if (lane == 0 && n_it > 0) {
      mbar_arrive_expect_tx(kv_full, 2 * TILE_BYTES);
      tma_load_4d(base + BwdSmem::K_OFF, &p.tmK, kv_full, 0, g, batch, key0);
      tma_load_4d(base + BwdSmem::K_OFF + HALF_BYTES, &p.tmK, kv_full, 64, g, batch, key0);
      tma_load_4d(base + BwdSmem::V_OFF, &p.tmV, kv_full, 0, g, batch, key0);
      tma_load_4d(base + BwdSmem::V_OFF + HALF_BYTES, &p.tmV, kv_full, 64, g, batch, key0);
      const uint32_t ds = base + BwdSmem::DO_OFF;
      int head = head0, i = i_start;
      for (int it = 0; it < n_it; ++it) {
        const int s = it & 1;
        if (!mbar_wait(q_empty(s), (uint32_t)((it >> 1) & 1) ^ 1u, p.status, 0x410u)) break;
        mbar_arrive_expect_tx(q_full(s), TILE_BYTES + BwdSmem::STAT_BYTES);
        const uint32_t qs = base + BwdSmem::Q_OFF + s * TILE_BYTES, ss = base + BwdSmem::STAT_OFF + s * BwdSmem::STAT_BYTES;
        const size_t stat = ((size_t)batch * p.nq + head) * p.sq_pad + (size_t)i * FB;
        tma_load_5d(qs, &p.tmQ, q_full(s), 0, head - g * rep_all, g, batch, i * FB);
        tma_load_5d(qs + HALF_BYTES, &p.tmQ, q_full(s), 64, head - g * rep_all, g, batch, i * FB);
        bulk_g2s_bar(ss, p.nlse2 + stat, FB * 4, q_full(s));
        bulk_g2s_bar(ss + FB * 4, p.ndelta + stat, FB * 4, q_full(s));
        if (!mbar_wait(do_empty, (uint32_t)(it & 1) ^ 1u, p.status, 0x411u)) break;
        mbar_arrive_expect_tx(do_full, TILE_BYTES);
        tma_load_4d(ds, &p.tmdO, do_full, 0, head, batch, i * FB);
        tma_load_4d(ds + HALF_BYTES, &p.tmdO, do_full, 64, head, batch, i * FB);
        if (++i == n_q) { i = i_start; ++head; }
      }
    }
  } else if (warp == 1) {
    // ===================== MMA issuer =====================
    if (lane == 0 && n_it > 0) {
      constexpr uint32_t idesc_kk = make_idesc_f16(128, 128, 1, 0, 0);     // both operands K-major
      constexpr uint32_t idesc_tn = make_idesc_f16(128, 128, 1, 0, 1);     // A from TMEM, B MN-major
      constexpr uint32_t idesc_dq = make_idesc_f16(128, 128, 1, 1, 1);     // A and B MN-major
      const uint32_t ks = base + BwdSmem::K_OFF, vs = base + BwdSmem::V_OFF, dss = base + BwdSmem::DS_OFF, dos = base + BwdSmem::DO_OFF;
      auto issue_s = [&](int it) {                // S^T = K Q_it^T
        const uint32_t qs = base + BwdSmem::Q_OFF + (it & 1) * TILE_BYTES;
#pragma unroll
        for (int k = 0; k < FD / 16; ++k) {
          const uint32_t off = (uint32_t)((k >> 2) * HALF_BYTES + (k & 3) * 32);
          umma_f16(tST, make_smem_desc(ks + off, 0, 1024), make_smem_desc(qs + off, 0, 1024), idesc_kk, k ? 1u : 0u);
        }
        umma_commit(st_full);
      };
      auto issue_dp = [&]() {                     // dP^T = V dO^T
#pragma unroll
        for (int k = 0; k < FD / 16; ++k) {
          const uint32_t off = (uint32_t)((k >> 2) * HALF_BYTES + (k & 3) * 32);
          umma_f16(tDPT, make_smem_desc(vs + off, 0, 1024), make_smem_desc(dos + off, 0, 1024), idesc_kk, k ? 1u : 0u);
        }
        umma_commit(dpt_full);
      };
      // column of the packed A operand (P^T or dS^T) that k-step k reads: each half of the query columns keeps its own place
      auto a_col = [](int k) { return (uint32_t)((k >> 2) * 64 + (k & 3) * 8); };
      bool ok = mbar_wait(kv_full, 0, p.status, 0x420u);
      if (ok) ok = mbar_wait(q_full(0), 0, p.status, 0x421u);
      if (ok) { tc_fence_after(); issue_s(0); ok = mbar_wait(do_full, 0, p.status, 0x422u); }
      if (ok) { tc_fence_after(); issue_dp(); }
      for (int it = 0; it < n_it && ok; ++it) {
        const int s = it & 1;
        const uint32_t ip = (uint32_t)(it & 1);
        const uint32_t qs = base + BwdSmem::Q_OFF + s * TILE_BYTES;
        if (!mbar_wait(pt_ready, ip, p.status, 0x423u)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < FB / 16; ++k)      // dV += P^T dO: reduction over the 128 query rows, 16 per MMA
          umma_f16_ts(tDV, tST + a_col(k), make_smem_desc(dos + (uint32_t)(k * 16 * 128), HALF_BYTES, 1024), idesc_tn, (it | k) ? 1u : 0u);
        umma_commit(do_empty);
        if (it + 1 < n_it) {                   // the next scores overwrite P^T, which the MMAs above read before (same issuer: in order)
          if (!mbar_wait(q_full(s ^ 1), (uint32_t)(((it + 1) >> 1) & 1), p.status, 0x421u)) { ok = false; break; }
          tc_fence_after();
          issue_s(it + 1);
        }
        if (!mbar_wait(ds_ready, ip, p.status, 0x424u)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < FB / 16; ++k)      // dK += dS^T Q
          umma_f16_ts(tDK, tDPT + a_col(k), make_smem_desc(qs + (uint32_t)(k * 16 * 128), HALF_BYTES, 1024), idesc_tn, (it | k) ? 1u : 0u);
        umma_commit(q_empty(s));
#pragma unroll
        for (int k = 0; k < FB / 16; ++k)      // dQ = dS K, over dP^T / dS^T in tensor memory (read by the MMAs above)
          umma_f16(tDPT, make_smem_desc(dss + (uint32_t)(k * 16 * 128), HALF_BYTES, 1024),
                   make_smem_desc(ks + (uint32_t)(k * 16 * 128), HALF_BYTES, 1024), idesc_dq, k ? 1u : 0u);
        umma_commit(dq_full);
        if (it + 1 < n_it) {
          if (!mbar_wait(do_full, ip ^ 1u, p.status, 0x422u)) { ok = false; break; }
          if (!mbar_wait(dq_drained, ip, p.status, 0x425u)) { ok = false; break; }
          tc_fence_after();
          issue_dp();
        }
      }
      if (ok) umma_commit(acc_done);
    }
  } else {
    const int q = warp & 3;
    const int row = q * 32 + lane;                     // TMEM lane: key row inside the tile (query row when draining dQ)
    const uint32_t lane_addr = ((uint32_t)(q * 32) << 16);
    const int ch = (warp - 2) >> 2;                    // 0, 1: compute warps of query columns 64 ch .. 64 ch + 63;  2: drain warps
    bool ok = true;
    if (ch < 2) {
      // ===================== warps 2..9: P^T and dS^T, one thread per key row and 64 query columns =====================
      const int key = key0 + row;
      const uint32_t tS = tST + lane_addr + (uint32_t)(ch * 64), tP = tDPT + lane_addr + (uint32_t)(ch * 64);
      uint8_t* ds_row = base_ptr + BwdSmem::DS_OFF + ch * HALF_BYTES + row * 128;
      const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
      int i = i_start;
      for (int it = 0; it < n_it && ok; ++it) {
        const uint32_t ip = (uint32_t)(it & 1);
        // -LSE log2e and -delta of the 64 query columns: broadcast reads of shared memory, two columns per 64-bit word
        const ulonglong2* nl = reinterpret_cast<const ulonglong2*>(base_ptr + BwdSmem::STAT_OFF + (it & 1) * BwdSmem::STAT_BYTES) + ch * 16;
        const ulonglong2* nd = nl + FB / 4;
        // keys of this tile visible to query row r: key <= r + q_offset (causal), key < sk
        // <=> column c of this warp's 64 is visible to this thread's key iff c >= first_c
        const int first_c = (key >= p.sk) ? FB : (p.causal ? key - p.q_offset - i * FB - ch * 64 : 0);
        if (++i == n_q) i = i_start;
        uint32_t pp[32];                               // P^T of this row, packed bf16 pairs (kept for dS^T)
        if (!mbar_wait(q_full(it & 1), (uint32_t)((it >> 1) & 1), p.status, 0x433u)) { ok = false; break; }   // the statistics
        if (!mbar_wait(st_full, ip, p.status, 0x430u)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t r[64];
          tmem_ld_32x32(tS, r);
          tmem_ld_32x32(tS + 32u, r + 32);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const ulonglong2 l = nl[c];
            float a, b;
            unpack_f32x2(fma_f32x2(pack_u32x2(r[4 * c], r[4 * c + 1]), scale2, l.x), a, b);
            pp[2 * c] = pack_bf16(exp2f(a), exp2f(b));
            unpack_f32x2(fma_f32x2(pack_u32x2(r[4 * c + 2], r[4 * c + 3]), scale2, l.y), a, b);
            pp[2 * c + 1] = pack_bf16(exp2f(a), exp2f(b));
          }
        }
        if (__any_sync(0xffffffffu, first_c > 0)) {    // tiles on the diagonal or past the last key
#pragma unroll
          for (int c = 0; c < 32; ++c) pp[c] &= (2 * c < first_c ? 0u : 0xffffu) | (2 * c + 1 < first_c ? 0u : 0xffff0000u);
        }
        tmem_st_32x32(tS, pp);                         // over score columns that this warp alone has read
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(pt_ready);
        // ---- dS^T = P^T (dP^T - delta) ----
        if (!mbar_wait(dpt_full, ip, p.status, 0x431u)) { ok = false; break; }     // implies that dQ of the last tile has read dS
        tc_fence_after();
        {
          uint32_t r[64];
          tmem_ld_32x32(tP, r);
          tmem_ld_32x32(tP + 32u, r + 32);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const ulonglong2 d = nd[c];
            float a, b;
            uint64_t t = add_f32x2(pack_u32x2(r[4 * c], r[4 * c + 1]), d.x);
            unpack_f32x2(mul_f32x2(t, pack_u32x2(pp[2 * c] << 16, pp[2 * c] & 0xffff0000u)), a, b);
            pp[2 * c] = pack_bf16(a, b);
            t = add_f32x2(pack_u32x2(r[4 * c + 2], r[4 * c + 3]), d.y);
            unpack_f32x2(mul_f32x2(t, pack_u32x2(pp[2 * c + 1] << 16, pp[2 * c + 1] & 0xffff0000u)), a, b);
            pp[2 * c + 1] = pack_bf16(a, b);
          }
        }
        tmem_st_32x32(tP, pp);
        // shared-memory copy for the dQ MMA: row = key, 64 query columns = 8 chunks of 16 bytes, 128-byte swizzle
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(ds_row + ((c ^ (row & 7)) << 4)) = make_uint4(pp[4 * c], pp[4 * c + 1], pp[4 * c + 2], pp[4 * c + 3]);
        tmem_st_wait();
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_ready);
      }
    } else {
      // ===================== warps 10..13: dQ (lanes = query rows) -> scale -> staging -> TMA reduce-add into the fp32 dQ =====================
      const uint32_t st_addr = base + BwdSmem::DQ_OFF + (uint32_t)(q * 8192);
      uint8_t* st_ptr = base_ptr + BwdSmem::DQ_OFF + q * 8192 + lane * 128;
      int head = head0, i = i_start;
      for (int it = 0; it < n_it; ++it) {
        if (!mbar_wait(dq_full, (uint32_t)(it & 1), p.status, 0x432u)) { ok = false; break; }
        tc_fence_after();
        uint32_t r[3][32];                               // d columns 32k .. 32k+31 of this lane's query row; the last 32 reuse r[0]
        const uint32_t tQ = tDPT + lane_addr;
        const int qr = i * FB + q * 32;                  // first query row of this warp's block
        auto put = [&](const uint32_t* v, int c) {       // 32 columns -> 4 KB slot c & 1
          if (lane == 0) tma_store_wait_read<1>();       // the reduce-add before the last one has read this slot
          __syncwarp();
          uint8_t* srow = st_ptr + (c & 1) * 4096;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            *reinterpret_cast<float4*>(srow + ((k ^ (lane & 7)) << 4)) =
                make_float4(__uint_as_float(v[4 * k]) * p.scale, __uint_as_float(v[4 * k + 1]) * p.scale,
                            __uint_as_float(v[4 * k + 2]) * p.scale, __uint_as_float(v[4 * k + 3]) * p.scale);
        };
        auto send = [&](int c) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (qr < p.sq) tma_reduce_add_4d(&p.tmdQ, st_addr + (uint32_t)((c & 1) * 4096), c * 32, head, batch, qr);
            tma_store_commit();
          }
        };
        // three quarters fit the registers; the first leaves for shared memory at once (its slot has long been read), the last takes
        // its place, and dQ's columns are free
        tmem_ld_32x32(tQ, r[0]);
        tmem_ld_32x32(tQ + 32u, r[1]);
        tmem_ld_32x32(tQ + 64u, r[2]);
        tmem_ld_wait();
        put(r[0], 0);
        tmem_ld_32x32(tQ + 96u, r[0]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(dq_drained);          // the MMA thread may overwrite dQ with the next dP^T
        send(0);
        put(r[1], 1);
        send(1);
        put(r[2], 2);
        send(2);
        put(r[0], 3);
        send(3);
        if (++i == n_q) { i = i_start; ++head; }
      }
      if (lane == 0) tma_store_wait<0>();
    }
    // ---- dK, dV of this key tile: TMEM -> bf16 -> shared memory (the Q stage buffers) -> TMA store; compute warps only ----
    if (n_it == 0) {
      // no query sees this tile: its gradients are zero (with the split the fp32 buffers are)
      if (!p.split_heads && ch < 2) {
        uint4* z = reinterpret_cast<uint4*>(base_ptr + BwdSmem::Q_OFF);
        for (int c = (int)threadIdx.x - 64; c < TILE_BYTES / 16; c += 256) z[c] = make_uint4(0, 0, 0, 0);
        fence_proxy_async_smem();
        named_bar(2, 256);
        if (warp == 2 && lane == 0) {
          for (int x = 0; x < 2; ++x) {
            tma_store_4d(&p.tmdV, base + BwdSmem::Q_OFF, 64 * x, g, batch, key0);
            tma_store_4d(&p.tmdK, base + BwdSmem::Q_OFF, 64 * x, g, batch, key0);
          }
          tma_store_commit();
          tma_store_wait<0>();
        }
      }
    } else if (ch < 2) {
      if (ok) ok = mbar_wait(acc_done, 0, p.status, 0x434u);
      tc_fence_after();
      if (p.split_heads) {
        // partial sums of one query head: fp32 through this warp's own 8 KB of staging, two [32 x 32] boxes per tensor
        const uint32_t st_addr = base + BwdSmem::Q_OFF + (uint32_t)((warp - 2) * 8192);
        uint8_t* st_ptr = base_ptr + BwdSmem::Q_OFF + (warp - 2) * 8192;
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {
          const uint32_t tA = (which == 0 ? tDV : tDK) + lane_addr + (uint32_t)(ch * 64);
          const float mul = which == 0 ? 1.f : p.scale;
          if (which == 1) { if (lane == 0) tma_store_wait_read<0>(); __syncwarp(); }
#pragma unroll
          for (int b2 = 0; b2 < 2; ++b2) {
            uint32_t r[32];
            tmem_ld_32x32(tA + (uint32_t)(b2 * 32), r);
            tmem_ld_wait();
            uint8_t* srow = st_ptr + b2 * 4096 + lane * 128;
#pragma unroll
            for (int cchunk = 0; cchunk < 8; ++cchunk)
              *reinterpret_cast<float4*>(srow + ((cchunk ^ (lane & 7)) << 4)) =
                  make_float4(__uint_as_float(r[4 * cchunk]) * mul, __uint_as_float(r[4 * cchunk + 1]) * mul,
                              __uint_as_float(r[4 * cchunk + 2]) * mul, __uint_as_float(r[4 * cchunk + 3]) * mul);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (ok && lane == 0 && key0 + q * 32 < p.sk) {
            const CUtensorMap* tm = which == 0 ? &p.tmdV : &p.tmdK;
            tma_reduce_add_4d(tm, st_addr, ch * 64, g, batch, key0 + q * 32);
            tma_reduce_add_4d(tm, st_addr + 4096u, ch * 64 + 32, g, batch, key0 + q * 32);
            tma_store_commit();
          }
        }
        if (lane == 0) tma_store_wait<0>();
      } else {
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {          // 0: dV (no scale), 1: dK (softmax scale)
        const uint32_t tA = (which == 0 ? tDV : tDK) + lane_addr + (uint32_t)(ch * 64);
        const float mul = which == 0 ? 1.f : p.scale;
        uint8_t* srow = base_ptr + BwdSmem::Q_OFF + which * TILE_BYTES + ch * HALF_BYTES + row * 128;
#pragma unroll 1
        for (int c = 0; c < 64; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32(tA + (uint32_t)c, r);
          tmem_ld_wait();
#pragma unroll
          for (int cchunk = 0; cchunk < 4; ++cchunk) {
            uint32_t pk[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(r[8 * cchunk + 2 * e]) * mul, __uint_as_float(r[8 * cchunk + 2 * e + 1]) * mul);
              pk[e] = *reinterpret_cast<uint32_t*>(&hh);
            }
            *reinterpret_cast<uint4*>(srow + ((((c >> 3) + cchunk) ^ (row & 7)) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          }
        }
      }
      fence_proxy_async_smem();
      named_bar(2, 256);
      if (ok && warp == 2 && lane == 0) {
        tma_store_4d(&p.tmdV, base + BwdSmem::Q_OFF, 0, g, batch, key0);
        tma_store_4d(&p.tmdV, base + BwdSmem::Q_OFF + HALF_BYTES, 64, g, batch, key0);
        tma_store_4d(&p.tmdK, base + BwdSmem::Q_OFF + TILE_BYTES, 0, g, batch, key0);
        tma_store_4d(&p.tmdK, base + BwdSmem::Q_OFF + TILE_BYTES + HALF_BYTES, 64, g, batch, key0);
        tma_store_commit();
      }
      if (lane == 0) tma_store_wait<0>();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}
}  // namespace

// Gradients of flash attention.  q / k / v strided like the forward's inputs, dout [sq, b, nq, 128] with strides (seq, batch, head), o
// [sq, b, nq, 128] contiguous, lse [b, nq, sq].  dq / dk / dv: bf16, strides as q / k / v, last dim contiguous, every row written.
// acc: fp32 scratch, sq * b * nq * 128 elements for dQ, and with split_heads 2 * sk * b * nkv * 128 more for dK and dV; nlse2 / ndelta:
// fp32 scratch [b, nq, ceil(sq / 128) * 128] each.  All 16-byte aligned.
// split_heads = 1: one CTA per query head, which add their dK / dV in fp32 (use when ceil(sk / 128) * nkv * b is well below twice the SM
// count); 0: one CTA per KV head, dK / dV written once.
MSB_API int msb_flash_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse, float* acc,
                          void* dq, void* dk, void* dv, float* nlse2, float* ndelta, int split_heads, int sq, int sk, int b, int nq, int nkv,
                          long long q_ss, long long q_sb, long long q_gs, long long q_sh, long long k_ss, long long k_sb, long long k_sh,
                          long long v_ss, long long v_sb, long long v_sh, long long do_ss, long long do_sb, long long do_sh,
                          long long dq_ss, long long dq_sb, long long dq_gs, long long dq_sh, long long dk_ss, long long dk_sb, long long dk_sh,
                          long long dv_ss, long long dv_sb, long long dv_sh, int causal, int q_offset, float scale, unsigned int* status,
                          cudaStream_t s) {
  MSB_REQUIRE(sq > 0 && sk > 0 && nq % nkv == 0, "flash_bwd: bad shape sq=%d sk=%d nq=%d nkv=%d", sq, sk, nq, nkv);
  MSB_REQUIRE(status != nullptr, "flash_bwd: status word is required");
  const int sq_pad = (sq + FB - 1) / FB * FB;
  const long long q_rows = (long long)sq * b * nq, k_rows = (long long)sk * b * nkv;
  float *dk32 = acc + q_rows * FD, *dv32 = dk32 + k_rows * FD;
  {
    const long long pairs = ((long long)b * nq * sq_pad + 1) / 2, blocks = (pairs + 7) / 8, most = (long long)msb::num_sms() * 32;
    flash_bwd_prep_kernel<<<(unsigned)(blocks < most ? blocks : most), 256, 0, s>>>(
        (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, do_ss, do_sb, do_sh, lse, nlse2, ndelta, sq, b, nq, sq_pad, (float4*)acc,
        (q_rows + (split_heads ? 2 * k_rows : 0)) * (FD / 4));
    MSB_CHECK_LAUNCH("flash_bwd_prep");
  }
  BwdParams p;
  memset(&p, 0, sizeof(p));
  int rc = make_map_q(&p.tmQ, q, sq, nq / nkv, nkv, b, q_ss, q_sb, q_gs, q_sh); if (rc) return rc;
  rc = make_map4(&p.tmK, k, sk, nkv, b, k_ss, k_sb, k_sh); if (rc) return rc;
  rc = make_map4(&p.tmV, v, sk, nkv, b, v_ss, v_sb, v_sh); if (rc) return rc;
  rc = make_map4(&p.tmdO, dout, sq, nq, b, do_ss, do_sb, do_sh); if (rc) return rc;
  auto map32 = [&](CUtensorMap* tm, float* base, int seq, int heads) {       // contiguous fp32, boxes of 32 rows x 32 columns
    uint64_t dims[4] = {(uint64_t)FD, (uint64_t)heads, (uint64_t)b, (uint64_t)seq};
    uint64_t str[3] = {(uint64_t)FD * 4, (uint64_t)heads * FD * 4, (uint64_t)b * heads * FD * 4};
    uint32_t box[4] = {32, 1, 1, 32};
    return make_tmap_nd(tm, base, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, 4, dims, str, box);
  };
  if (!split_heads) {
    rc = make_map4(&p.tmdK, dk, sk, nkv, b, dk_ss, dk_sb, dk_sh); if (rc) return rc;
    rc = make_map4(&p.tmdV, dv, sk, nkv, b, dv_ss, dv_sb, dv_sh); if (rc) return rc;
  } else {
    rc = map32(&p.tmdK, dk32, sk, nkv); if (rc) return rc;
    rc = map32(&p.tmdV, dv32, sk, nkv); if (rc) return rc;
  }
  rc = map32(&p.tmdQ, acc, sq, nq); if (rc) return rc;
  p.split_heads = split_heads ? 1 : 0;
  p.nlse2 = nlse2; p.ndelta = ndelta;
  p.sq = sq; p.sk = sk; p.b = b; p.nq = nq; p.nkv = nkv; p.sq_pad = sq_pad; p.causal = causal; p.q_offset = q_offset;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
  static std::atomic<unsigned long long> stated{0};
  if (int bad = msb::allow_smem((const void*)flash_bwd_sm100_kernel, BwdSmem::TOTAL, "flash_bwd", stated)) return bad;
  const long long ctas = (long long)(split_heads ? nq : nkv) * ((sk + FB - 1) / FB);
  MSB_REQUIRE(ctas <= 0x7fffffffll, "flash_bwd: grid too large (%lld)", ctas);
  dim3 grid((unsigned)ctas, 1, b);
  flash_bwd_sm100_kernel<<<grid, BWD_THREADS, BwdSmem::TOTAL, s>>>(p);
  MSB_CHECK_LAUNCH("flash_bwd_sm100");
  FinishParams fp;
  FinishSeg* sg = fp.seg;
  sg[0] = FinishSeg{acc, (__nv_bfloat16*)dq, dq_ss, dq_sb, dq_gs, dq_sh, b, nkv, nq / nkv, q_rows};
  sg[1] = FinishSeg{dk32, (__nv_bfloat16*)dk, dk_ss, dk_sb, dk_sh, 0, b, nkv, 1, split_heads ? k_rows : 0};
  sg[2] = FinishSeg{dv32, (__nv_bfloat16*)dv, dv_ss, dv_sb, dv_sh, 0, b, nkv, 1, split_heads ? k_rows : 0};
  const long long fin = (sg[0].rows + sg[1].rows + sg[2].rows + 15) / 16, most = (long long)msb::num_sms() * 16;
  flash_bwd_finish_kernel<<<(unsigned)(fin < most ? fin : most), 256, 0, s>>>(fp);
  MSB_CHECK_LAUNCH("flash_bwd_finish");
  return 0;
}
