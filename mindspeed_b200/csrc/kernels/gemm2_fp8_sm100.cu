// Block-scaled fp8 GEMM on CTA pairs (tcgen05 cta_group::2, kind::f8f6f4): the plain (not grouped) form of gemm_fp8_sm100.cu for
// outputs of enough 256 x 256 tiles, same operands, scales and promotion:
//   D[m, n] = sum over k-blocks kb of  sA[m, kb] * sB[., kb] * ( A_q[m, 128 kb ..] . B_q[n, 128 kb ..] ),  k-blocks in order, fp32 FMAs.
//
// What bounds it: per k-block an SM's share of the 256 x 256 x 128 product takes 512 cycles of the tensor core, its operands 256
// cycles of shared-memory reads and 256 of TMA writes, and the promotion issues 64 two-lane FMAs (128 with row-wise scales of B) in
// each of 8 warps.  The 128 x 128 single-CTA tile needs twice the shared-memory traffic per product.  Scales of A come from global
// memory four k-blocks ahead, each slot in its own register; the accumulator is handed back by an arrival of CTA scope, because one
// of cluster scope waits for those loads (2300 cycles a k-block instead of 1100).  Row-wise scales of B come by TMA and are read as
// broadcasts.  4096 x 28672 x 4096: block form 809 -> 461 us, weight gradient (row-wise) 2691 -> 769 us.
//
// CTA = 12 warps: 0-7 promotion and epilogue (TMEM lane quarter warp & 3, column half warp >> 2: 128 fp32 accumulators per thread),
// 8 TMA producer, 9 MMA issuer (leader CTA), 10-11 idle (they complete the warpgroup that gives registers away).  Two 256-column
// accumulators in tensor memory: one k-block is promoted while the next is computed.  fp32 -> bf16 / fp32 tiles leave through
// 128-byte-swizzled staging and TMA stores (reduce-adds for the accumulating form).
#include "msb_common.cuh"
#include "msb_sm100.cuh"

using namespace msb;
using namespace msb::sm100;

namespace {
constexpr int PM = 128;                          // rows per CTA (256 per pair)
constexpr int PN = 256;                          // columns per pair
constexpr int PK = 128;                          // k-block, fp8 elements = bytes
constexpr int PSTAGES = 5;
constexpr int PA_BYTES = PM * PK, PB_BYTES = (PN / 2) * PK, P_STAGE = PA_BYTES + PB_BYTES;
constexpr int PSC = 4;                           // ring of B's row-wise scales, 256 floats a slot
constexpr int P_EPI_OFF = PSTAGES * P_STAGE;     // 8 warps x 4 KB
constexpr int P_SC_OFF = P_EPI_OFF + 8 * 4096;
constexpr int P_BAR_OFF = P_SC_OFF + PSC * PN * 4;
constexpr int P_SMEM = P_BAR_OFF + 256 + 1024;
static_assert(P_SMEM <= 232448, "exceeds the 227 KB of shared memory a CTA may use");
constexpr int P_THREADS = 12 * 32;

enum PEpi : int { PEPI_BF16 = 0, PEPI_F32 = 1, PEPI_F32_ACC = 2 };

struct Fp8PairParams {
  CUtensorMap tmA, tmB, tmD;
  const float* sA;            // [K/128, M]
  const float* sB;            // block: [N/128, K/128]   row: [K/128, N]
  int M, N, K;
  int fmt_a, fmt_b;
  unsigned int* status;
};

__device__ __forceinline__ void umma_f8f6f4_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}

template <int EPI, bool B_ROWWISE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P_THREADS, 1) gemm2_fp8_kernel(const __grid_constant__ Fp8PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + P_BAR_OFF;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (PSTAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * PSTAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * PSTAGES + 2 + a); };
  auto sfull_bar = [&](int a) { return bar_base + 8u * (2 * PSTAGES + 4 + a); };
  auto sempty_bar = [&](int a) { return bar_base + 8u * (2 * PSTAGES + 4 + PSC + a); };
  const uint32_t tmem_slot = bar_base + 8u * (2 * PSTAGES + 4 + 2 * PSC);
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(base_ptr + (tmem_slot - smem_base));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int num_m = (p.M + 2 * PM - 1) / (2 * PM), num_n = (p.N + PN - 1) / PN;
  const int num_tiles = num_m * num_n, num_kb = p.K / PK;
  // m fastest inside groups of 8 m-tiles: pairs running together share A and B tiles in L2
  auto tile_mn = [&](int t, int& m, int& n) {
    const int per_group = 8 * num_n, g = t / per_group, first = g * 8, gsz = min(num_m - first, 8), r = t - g * per_group;
    m = first + r % gsz;
    n = r / gsz;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < PSTAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), 16); }
    for (int a = 0; a < PSC; ++a) { mbar_init(sfull_bar(a), 1); mbar_init(sempty_bar(a), 8); }
    mbar_fence_init();
  }
  if (warp == 9) { tmem_alloc_pair(tmem_slot, 512u); tmem_relinquish_pair(); }
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  bool alive = true;

  // registers of the launch: 384 x 168 = 64512
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 8) {
      // ===================== TMA producer (both CTAs) =====================
      if (lane == 0) {
        int stage = 0, slot = 0;
        uint32_t phase = 0, sphase = 0;
        for (int t = pair; t < num_tiles && alive; t += npairs) {
          int m_blk, n_blk;
          tile_mn(t, m_blk, n_blk);
          const int m0 = m_blk * 2 * PM + (int)cta * PM, n0 = n_blk * PN;
          for (int kb = 0; kb < num_kb; ++kb) {
            if (!mbar_wait(empty_bar(stage), phase ^ 1u, p.status, 0x510u)) { alive = false; break; }
            const uint32_t sa = smem_base + stage * P_STAGE;
            if (cta == 0) mbar_arrive_expect_tx(full_bar(stage), 2 * P_STAGE);
            const uint32_t lead_full = mapa_u32(full_bar(stage), 0);
            tma_load_2d_pair(sa, &p.tmA, lead_full, kb * PK, m0);
            tma_load_2d_pair(sa + PA_BYTES, &p.tmB, lead_full, kb * PK, n0 + (int)cta * (PN / 2));
            if (B_ROWWISE) {
              if (!mbar_wait(sempty_bar(slot), sphase ^ 1u, p.status, 0x511u)) { alive = false; break; }
              const uint32_t bytes = (uint32_t)min(PN, p.N - n0) * 4u;
              mbar_arrive_expect_tx(sfull_bar(slot), bytes);
              bulk_g2s(smem_base + P_SC_OFF + slot * (PN * 4), p.sB + (size_t)kb * p.N + n0, bytes, sfull_bar(slot));
              if (++slot == PSC) { slot = 0; sphase ^= 1u; }
            }
            if (++stage == PSTAGES) { stage = 0; phase ^= 1u; }
          }
        }
        for (int i = 0; i < PSTAGES && alive; ++i) {       // the other CTA's MMAs have read every stage before this CTA leaves
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, p.status, 0x512u)) { alive = false; break; }
          if (++stage == PSTAGES) { stage = 0; phase ^= 1u; }
        }
      }
    } else if (warp == 9) {
      // ===================== MMA issuer (leader CTA): one accumulator per k-block =====================
      if (lane == 0 && cta == 0) {
        const uint32_t idesc = make_idesc_f8(2 * PM, PN, p.fmt_a, p.fmt_b);
        int stage = 0, acc = 0;
        uint32_t phase = 0, acc_phase = 0;
        for (int t = pair; t < num_tiles && alive; t += npairs) {
          for (int kb = 0; kb < num_kb; ++kb) {
            if (!mbar_wait(tempty_bar(acc), acc_phase ^ 1u, p.status, 0x520u)) { alive = false; break; }
            if (!mbar_wait(full_bar(stage), phase, p.status, 0x521u)) { alive = false; break; }
            tc_fence_after();
            const uint32_t sa = smem_base + stage * P_STAGE, sb = sa + PA_BYTES;
#pragma unroll
            for (int k = 0; k < PK / 32; ++k)
              umma_f8f6f4_pair(tmem_base + (uint32_t)(acc * PN), make_smem_desc(sa + k * 32, 0, 1024), make_smem_desc(sb + k * 32, 0, 1024),
                               idesc, k != 0 ? 1u : 0u);
            umma_commit_pair(empty_bar(stage), 3);
            umma_commit_pair(tfull_bar(acc), 3);
            if (++stage == PSTAGES) { stage = 0; phase ^= 1u; }
            if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
          }
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");       // 256 x 224 + 128 x 56 = 64512
    // ===================== promotion + epilogue =====================
    const int q = warp & 3, half = warp >> 2;
    const uint32_t lead_tempty[2] = {mapa_u32(tempty_bar(0), 0), mapa_u32(tempty_bar(1), 0)};
    uint8_t* stg = base_ptr + P_EPI_OFF + warp * 4096 + lane * 128;
    const uint32_t stg_addr = smem_base + P_EPI_OFF + (uint32_t)warp * 4096u;
    int acc = 0, slot = 0;
    uint32_t acc_phase = 0, sphase = 0;
    for (int t = pair; t < num_tiles && alive; t += npairs) {
      int m_blk, n_blk;
      tile_mn(t, m_blk, n_blk);
      const int row0 = m_blk * 2 * PM + (int)cta * PM + q * 32, row = row0 + lane;
      const int c0 = n_blk * PN + half * 128;
      const bool row_ok = row < p.M, col_ok = c0 < p.N;
      uint64_t accum[64];                                        // 128 columns of one row, two per word
#pragma unroll
      for (int c = 0; c < 64; ++c) accum[c] = 0ull;
      const float* sa_col = p.sA + row;
      const float* sb_blk = p.sB + (size_t)(c0 / 128) * num_kb;
      // scales are fetched AHEAD k-blocks before they are used: a load from L2 takes longer than a k-block
      constexpr int AHEAD = 4;
      auto scale_a = [&](int kb) { return row_ok && kb < num_kb ? __ldg(sa_col + (size_t)kb * p.M) : 0.f; };
      auto scale_b = [&](int kb) { return !B_ROWWISE && col_ok && kb < num_kb ? __ldg(sb_blk + kb) : 0.f; };
      float sa[AHEAD], sb[AHEAD];
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) { sa[i] = scale_a(i); sb[i] = scale_b(i); }
      for (int kb0 = 0; kb0 < num_kb && alive; kb0 += AHEAD) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {                         // a slot keeps its register: moving it would wait for the load
          const int kb = kb0 + u;
          if (kb >= num_kb) break;
          const float s = B_ROWWISE ? sa[u] : sa[u] * sb[u];
          const uint64_t s2 = pack_f32x2(s, s);
          sa[u] = scale_a(kb + AHEAD);
          sb[u] = scale_b(kb + AHEAD);
          if (B_ROWWISE && !mbar_wait(sfull_bar(slot), sphase, p.status, 0x531u)) { alive = false; break; }
          if (!mbar_wait(tfull_bar(acc), acc_phase, p.status, 0x530u)) { alive = false; break; }
          tc_fence_after();
          const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * PN + half * 128);
          const uint32_t sb_row = smem_base + P_SC_OFF + (uint32_t)(slot * (PN * 4) + half * 512);
          uint32_t r[2][16];                                       // the next 16 columns load while 16 are folded in
          tmem_ld_32x16(t_row, r[0]);
#pragma unroll
          for (int ch = 0; ch < 8; ++ch) {
            tmem_ld_wait();
            if (ch < 7) {
              tmem_ld_32x16(t_row + (uint32_t)(16 * (ch + 1)), r[(ch + 1) & 1]);
            } else {                                               // all of the accumulator is in registers
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive_remote(lead_tempty[acc]);
            }
            const uint32_t* v = r[ch & 1];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint64_t f0 = s2, f1 = s2;
              if (B_ROWWISE) {
                // broadcast: four columns' scales (volatile: hoisted loads cost registers that the accumulators need)
                asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(f0), "=l"(f1) : "r"(sb_row + (uint32_t)((ch * 4 + j) * 16)));
                f0 = mul_f32x2(s2, f0);
                f1 = mul_f32x2(s2, f1);
              }
              accum[ch * 8 + 2 * j] = fma_f32x2(f0, pack_u32x2(v[4 * j], v[4 * j + 1]), accum[ch * 8 + 2 * j]);
              accum[ch * 8 + 2 * j + 1] = fma_f32x2(f1, pack_u32x2(v[4 * j + 2], v[4 * j + 3]), accum[ch * 8 + 2 * j + 1]);
            }
          }
          if (B_ROWWISE) {
            __syncwarp();
            if (lane == 0) mbar_arrive(sempty_bar(slot));
            if (++slot == PSC) { slot = 0; sphase ^= 1u; }
          }
          if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
        }
      }
      if (!alive) break;
      constexpr int CW = EPI == PEPI_BF16 ? 64 : 32;             // columns per 128-byte staging row
#pragma unroll
      for (int ch = 0; ch < 128 / CW; ++ch) {
        if (lane == 0) tma_store_wait_read<0>();
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float lo, hi;
            if (EPI == PEPI_BF16) {
              unpack_f32x2(accum[ch * 32 + 4 * j + e], lo, hi);
              o[e] = pack_bf16(lo, hi);
            } else {
              unpack_f32x2(accum[ch * 16 + 2 * j + (e >> 1)], lo, hi);
              o[e] = __float_as_uint((e & 1) ? hi : lo);
            }
          }
          *reinterpret_cast<uint4*>(stg + ((j ^ (lane & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && row0 < p.M && c0 + ch * CW < p.N) {
          if (EPI == PEPI_F32_ACC) tma_reduce_add_2d(&p.tmD, stg_addr, c0 + ch * CW, row0);
          else tma_store_2d(&p.tmD, stg_addr, c0 + ch * CW, row0);
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncwarp();
  cluster_sync_all();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512u);
  }
}

template <int EPI, bool B_ROWWISE>
int launch_pair(const Fp8PairParams& p, int pairs, cudaStream_t s) {
  auto kern = gemm2_fp8_kernel<EPI, B_ROWWISE>;
  static std::atomic<unsigned long long> stated{0};
  if (int bad = msb::allow_smem((const void*)kern, P_SMEM, "gemm2_fp8", stated)) return bad;
  kern<<<2 * pairs, P_THREADS, P_SMEM, s>>>(p);
  MSB_CHECK_LAUNCH("gemm2_fp8");
  return 0;
}
}  // namespace

namespace msb {
// The pair kernel's share of msb_gemm_fp8_blockscaled (arguments as there, one weight matrix).
int gemm2_fp8_blockscaled(const void* A, const float* sA_t, const void* B, const float* sB, void* D, int M, int N, int K, int b_scale_rowwise,
                          int fmt_a, int fmt_b, int epilogue, long long ldd, unsigned int* status, cudaStream_t s) {
  Fp8PairParams p;
  memset(&p, 0, sizeof(p));
  int rc = make_tmap_2d(&p.tmA, A, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)M, (uint64_t)K, (uint64_t)K, PM, PK);
  if (rc) return rc;
  rc = make_tmap_2d(&p.tmB, B, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, (uint64_t)N, (uint64_t)K, (uint64_t)K, PN / 2, PK);
  if (rc) return rc;
  if (epilogue == PEPI_BF16) rc = make_tmap_2d(&p.tmD, D, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)M, (uint64_t)N, (uint64_t)ldd, 32, 64);
  else rc = make_tmap_2d(&p.tmD, D, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)M, (uint64_t)N, (uint64_t)ldd, 32, 32);
  if (rc) return rc;
  p.sA = sA_t; p.sB = sB; p.M = M; p.N = N; p.K = K; p.fmt_a = fmt_a; p.fmt_b = fmt_b; p.status = status;
  const int tiles = ((M + 2 * PM - 1) / (2 * PM)) * ((N + PN - 1) / PN);
  const int pairs = tiles < num_sms() / 2 ? tiles : num_sms() / 2;
  switch (epilogue * 2 + (b_scale_rowwise ? 1 : 0)) {
    case 0: return launch_pair<PEPI_BF16, false>(p, pairs, s);
    case 1: return launch_pair<PEPI_BF16, true>(p, pairs, s);
    case 2: return launch_pair<PEPI_F32, false>(p, pairs, s);
    case 3: return launch_pair<PEPI_F32, true>(p, pairs, s);
    case 4: return launch_pair<PEPI_F32_ACC, false>(p, pairs, s);
    default: return launch_pair<PEPI_F32_ACC, true>(p, pairs, s);
  }
}
}  // namespace msb
