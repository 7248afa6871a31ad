// Flash-style multi-head attention for sm_100a on tcgen05 tensor cores (causal and non-causal, head
// dimension 64 or 128, bf16, fp32 softmax statistics).
//
// Forward: one CTA per (batch, head, block of 128 queries).  Q stays in shared memory; K/V blocks of 128
// keys stream through a two-stage TMA ring.  Per key block:  S = Q·Kᵀ is a tcgen05.mma into TMEM; the 128
// softmax threads — one query row each, so row max / row sum need no shuffles — read S with tcgen05.ld,
// write P = exp2(scale·S − m) as bf16 into shared memory in the 128-byte-swizzled K-major layout, and the
// second tcgen05.mma computes P·V into TMEM with V consumed in place as an MN-major operand (keys are its K
// dimension, so no transposed copy of V exists).  The running output lives in registers:
// O ← O·exp2(m_old − m_new) + P·V.  The log-sum-exp per row is stored for the backward pass.
//
// Backward: one CTA per (batch, head, block of 128 keys) walks the query blocks that attend to it and, per
// block, issues five tcgen05 GEMMs: S = Q·Kᵀ and dP = dO·Vᵀ into TMEM, then — from P = exp2(scale·S − lse) and
// dS = P∘(dP − δ) in shared memory — dV += Pᵀ·dO, dK += dSᵀ·Q (accumulating in TMEM across query blocks; P and dS
// are read as MN-major A operands, i.e. transposed for free) and dQ_block = dS·K, which is added into an fp32 dQ
// buffer with vector reductions.  δ = rowsum(dO∘O) comes from a small pre-pass kernel.
//
// Q/K/V/O/dO are addressed as (B, T, H, D) views with arbitrary batch / row / head strides (the fused QKV
// projection output is used in place).  All mbarrier waits are bounded.
//
// Takes the place of the reference's attention kernels: flash-attention forward with log-sum-exp output, the
// dO·O pre-pass and the backward producing dQ, dK, dV (reference:
// kernel_gen/kernel_gen/kernels/flash_attention_codegen/compile.py:280-330, kernels/flash_attention_fwd.py:36-266,
// kernels/flash_attention_bwd.py:6-313; selected in src/passes/mha_attention_pass.cpp).  The reference supports
// head dimension 128 only; 64 is added here.
#include "tc05.cuh"

namespace {

using namespace tc05;

constexpr int BQ = 128;   // queries per tile (TMEM lanes)
constexpr int BKV = 128;  // keys per block
enum { ATT_ERR_TIMEOUT = 501 };

struct AttnParams {
  int B, T, H, D;
  int causal;
  float scale_log2;  // softmax scale * log2(e)
  float scale;
  elem_t* out;         // (B, T, H, D) contiguous
  float* lse;        // (B, H, T), natural-log units of the scaled scores
  int* status;
};

__device__ __forceinline__ void tma_load_attn(void* dst, const CUtensorMap* map, uint64_t* bar, int d0, int h, int t,
                                              int b) {
  tma_load_4d(dst, map, bar, d0, h, t, b);
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Arrival of a whole warp (one per warp: 32 arrivals on one barrier would be served one after the other): every lane
// has fenced its own accesses before.
__device__ __forceinline__ void warp_arrive(uint64_t* bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

// Address of element (row, col8 = 8-element group index) in a [rows x 64]-bf16 panel with 128-byte swizzle.
__device__ __forceinline__ uint32_t swz(int row, int chunk) { return row * 128 + ((chunk ^ (row & 7)) << 4); }

// -------------------------------------------------------------------------------------------------
// forward
// -------------------------------------------------------------------------------------------------
// KV_STAGES = 2 prefetches the next K/V block inside the CTA; KV_STAGES = 1 halves the K/V footprint so that two
// CTAs share an SM and overlap each other's softmax and tensor-core phases instead (used for D = 64).
template <int D, int KV_STAGES>
__global__ void __launch_bounds__(160, KV_STAGES == 1 ? 2 : 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const AttnParams p) {
  constexpr int DP = D / 64;                 // 64-wide panels per row
  constexpr int kQBytes = BQ * D * 2;
  constexpr int kKVBytes = BKV * D * 2;
  constexpr int kPBytes = BQ * BKV * 2;
  constexpr uint32_t kTmemCols = 256;        // S: [0,128)  PV: [128, 128 + D)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + kQBytes;                // KV_STAGES stages
  uint8_t* sV = sK + KV_STAGES * kKVBytes;   // KV_STAGES stages
  uint8_t* sP = sV + KV_STAGES * kKVBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sP + kPBytes);
  uint64_t* q_full = bars;                   // 1
  uint64_t* kv_full = bars + 1;              // 2
  uint64_t* kv_empty = bars + 3;             // 2
  uint64_t* s_full = bars + 5;
  uint64_t* p_ready = bars + 6;
  uint64_t* pv_full = bars + 7;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qb = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int q0 = qb * BQ;
  const int nkb = p.causal ? min((p.T + BKV - 1) / BKV, qb + 1) : (p.T + BKV - 1) / BKV;

  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    mbar_init(q_full, 1);
    for (int s = 0; s < 2; ++s) { mbar_init(&kv_full[s], 1); mbar_init(&kv_empty[s], 1); }
    mbar_init(s_full, 1);
    mbar_init(p_ready, 128);
    mbar_init(pv_full, 1);
    mbar_fence_init();
  }
  if (warp == 0) { tmem_alloc(tmem_slot, kTmemCols); tmem_relinquish(); }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_s = tmem, tmem_pv = tmem + 128;

  if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      // Q once; first K/V block
      mbar_expect_tx(q_full, kQBytes);
#pragma unroll
      for (int j = 0; j < DP; ++j) tma_load_attn(sQ + j * BQ * 128, &map_q, q_full, j * 64, h, q0, b);
      auto load_kv = [&](int kb) {
        const int s = kb % KV_STAGES;
        mbar_expect_tx(&kv_full[s], 2 * kKVBytes);
#pragma unroll
        for (int j = 0; j < DP; ++j) {
          tma_load_attn(sK + s * kKVBytes + j * BKV * 128, &map_k, &kv_full[s], j * 64, h, kb * BKV, b);
          tma_load_attn(sV + s * kKVBytes + j * BKV * 128, &map_v, &kv_full[s], j * 64, h, kb * BKV, b);
        }
      };
      load_kv(0);
      const uint32_t idesc_s = make_idesc_f16kind(128, BKV, false, false);
      const uint32_t idesc_pv = make_idesc_f16kind(128, D, false, true);   // B = V is MN-major
      ok = mbar_wait(q_full, 0);
      for (int kb = 0; kb < nkb && ok; ++kb) {
        const int s = kb % KV_STAGES;
        if (KV_STAGES == 2 && kb + 1 < nkb) {   // prefetch the next block into the other stage once it is free
          if (kb >= 1 && !mbar_wait(&kv_empty[s ^ 1], ((kb - 1) >> 1) & 1)) { ok = false; break; }
          load_kv(kb + 1);
        }
        if (KV_STAGES == 1 && kb >= 1) {        // single stage: reload once the previous block's P·V has read it
          if (!mbar_wait(&kv_empty[0], (kb - 1) & 1)) { ok = false; break; }
          load_kv(kb);
        }
        if (!mbar_wait(&kv_full[s], (kb / KV_STAGES) & 1)) { ok = false; break; }
        fence_after_sync();
        const uint32_t q_addr = smem_u32(sQ), k_addr = smem_u32(sK + s * kKVBytes), v_addr = smem_u32(sV + s * kKVBytes);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {   // K-major operands: panel k/4, 32 bytes per step inside the panel
          const uint64_t da = make_smem_desc_sw128(q_addr + (k / 4) * BQ * 128 + (k % 4) * 32, 16, 1024);
          const uint64_t db = make_smem_desc_sw128(k_addr + (k / 4) * BKV * 128 + (k % 4) * 32, 16, 1024);
          mma_f16_ss(tmem_s, da, db, idesc_s, k != 0);
        }
        mma_commit(s_full);
        if (!mbar_wait(p_ready, kb & 1)) { ok = false; break; }
        fence_after_sync();
        const uint32_t p_addr = smem_u32(sP);
#pragma unroll
        for (int k = 0; k < BKV / 16; ++k) {
          // A = P, K-major over keys: two 64-key panels.  B = V, MN-major: 16 key rows per step = 2048 bytes;
          // 64-wide D panels are BKV*128 bytes apart (leading-dimension offset).
          const uint64_t da = make_smem_desc_sw128(p_addr + (k / 4) * BQ * 128 + (k % 4) * 32, 16, 1024);
          const uint64_t db = make_smem_desc_sw128(v_addr + k * 16 * 128, BKV * 128, 1024);
          mma_f16_ss(tmem_pv, da, db, idesc_pv, k != 0);
        }
        mma_commit(pv_full);
        mma_commit(&kv_empty[s]);
      }
      if (!ok) atomicExch(p.status, ATT_ERR_TIMEOUT);
    }
  } else {
    // ---------------------------------------------------------------- softmax / output threads
    const int lane_group = warp & 3;
    const int row = lane_group * 32 + lane;          // query row within the tile == TMEM lane
    const int t_q = q0 + row;
    const uint32_t lane_addr = uint32_t(lane_group * 32) << 16;
    float m = -INFINITY, l = 0.0f;
    float o[D];
#pragma unroll
    for (int d = 0; d < D; ++d) o[d] = 0.0f;
    bool ok = true;
    for (int kb = 0; kb < nkb; ++kb) {
      if (!mbar_wait(s_full, kb & 1)) { ok = false; break; }
      fence_after_sync();
      const int k0 = kb * BKV;
      const bool need_mask = (p.causal && kb == qb) || (k0 + BKV > p.T);
      // pass 1: row maximum
      float mx = m;
#pragma unroll 1
      for (int c0 = 0; c0 < BKV; c0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_s + lane_addr + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          float sv = __uint_as_float(r[j]);
          if (need_mask) {
            const int tk = k0 + c0 + j;
            if (tk >= p.T || (p.causal && tk > t_q)) sv = -INFINITY;
          }
          mx = fmaxf(mx, sv);
        }
      }
      const float m_new = mx;
      const float m_use = (m_new == -INFINITY) ? 0.0f : m_new;   // fully masked row: keep exponents finite
      const float alpha = fast_exp2((m - m_use) * p.scale_log2);     // m = -inf on the first block -> 0
      float rs = 0.0f;
      // pass 2: P = exp2(scale*(S - m)) -> bf16 -> swizzled shared memory
#pragma unroll 1
      for (int c0 = 0; c0 < BKV; c0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_s + lane_addr + c0, r);
        tmem_ld_wait();
        float pv[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          float sv = __uint_as_float(r[j]);
          if (need_mask) {
            const int tk = k0 + c0 + j;
            if (tk >= p.T || (p.causal && tk > t_q)) sv = -INFINITY;
          }
          pv[j] = fast_exp2((sv - m_use) * p.scale_log2);
        }
#pragma unroll
        for (int j8 = 0; j8 < 4; ++j8) {
          __align__(16) elem2_t hh[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            hh[q] = ff2e2(pv[j8 * 8 + 2 * q], pv[j8 * 8 + 2 * q + 1]);
            const float2 back = e22ff(hh[q]);   // sum what the tensor core will actually see
            rs += back.x + back.y;
          }
          const int chunk = (c0 >> 3) + j8;                  // 16-byte chunk index within the 128-key row
          uint8_t* dst = sP + (chunk >> 3) * BQ * 128 + swz(row, chunk & 7);
          *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(hh);
        }
      }
      l = l * alpha + rs;
      m = m_new;
      fence_proxy_async();
      fence_before_sync();
      mbar_arrive(p_ready);
      // accumulate P·V
      if (!mbar_wait(pv_full, kb & 1)) { ok = false; break; }
      fence_after_sync();
#pragma unroll
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_pv + lane_addr + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) o[c0 + j] = o[c0 + j] * alpha + __uint_as_float(r[j]);
      }
      fence_before_sync();
    }
    if (ok && t_q < p.T) {
      const float inv = l > 0.0f ? 1.0f / l : 0.0f;
      elem_t* dst = p.out + (((long long)b * p.T + t_q) * p.H + h) * D;
#pragma unroll
      for (int d = 0; d < D; d += 8) {
        __align__(16) elem2_t hh[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) hh[q] = ff2e2(o[d + 2 * q] * inv, o[d + 2 * q + 1] * inv);
        *reinterpret_cast<uint4*>(dst + d) = *reinterpret_cast<uint4*>(hh);
      }
      if (p.lse != nullptr)
        p.lse[((long long)b * p.H + h) * p.T + t_q] = (l > 0.0f) ? m * p.scale + logf(l) : -INFINITY;
    }
    if (!ok && lane == 0) atomicExch(p.status, ATT_ERR_TIMEOUT);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) { fence_after_sync(); tmem_dealloc(tmem, kTmemCols); }
}

// -------------------------------------------------------------------------------------------------
// forward, two query tiles per CTA
// -------------------------------------------------------------------------------------------------
// Same arithmetic as attn_fwd_kernel, organised for more softmax throughput per SM: a CTA owns 256 consecutive
// queries of one head as two 128-row tiles, each with its own group of four softmax warps, its own S and P·V
// accumulators in TMEM (S_A, S_B, O_A, O_B = 256 + 2·D columns) and its own P buffer in shared memory; K and V
// blocks (one stage each, loaded as soon as the MMAs that read the previous block have completed) are shared by
// both tiles.  One elected thread issues all TMA loads and all MMAs in an order in which no tile ever waits for
// the other: while one group is busy with its softmax, the tensor core works for the other one.  The output
// accumulators stay in tensor memory for the whole key loop (every P·V product adds to them); the softmax threads
// rescale them there only when a row's reference maximum moves (see below), so a group goes from one block's softmax
// straight to the next while its P·V product is still running.
// A group's scores are read from TMEM once and masked in a pass of their own; with masks inside the loops and two reads
// the kernel took 123 us at B8 T1024 H16 D64 causal (now 65) and 56 us at B16 T480 H8 D128 (now 36).
template <int D>
__global__ void __launch_bounds__(288, 1)
attn_fwd2_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                 const __grid_constant__ CUtensorMap map_v, const AttnParams p) {
  constexpr int DP = D / 64;
  constexpr int kQBytes = BQ * D * 2;      // one query tile
  constexpr int kKVBytes = BKV * D * 2;
  constexpr int kPBytes = BQ * BKV * 2;
  constexpr uint32_t kTmemCols = 512;      // S_A [0,128) S_B [128,256) O_A [256,256+D) O_B [256+D,256+2D)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                      // two tiles
  uint8_t* sK = sQ + 2 * kQBytes;
  uint8_t* sV = sK + kKVBytes;
  uint8_t* sP = sV + kKVBytes;             // two tiles
  uint64_t* bars = reinterpret_cast<uint64_t*>(sP + 2 * kPBytes);
  uint64_t* q_full = bars;                 // 1
  uint64_t* k_full = bars + 1;
  uint64_t* k_empty = bars + 2;
  uint64_t* v_full = bars + 3;
  uint64_t* v_empty = bars + 4;
  uint64_t* s_full = bars + 5;             // [2]
  uint64_t* p_ready = bars + 7;            // [2]
  uint64_t* pv_full = bars + 9;            // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // causal: the tiles with the most key blocks are scheduled first
  const int qb2 = p.causal ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
  const int h = blockIdx.y, b = blockIdx.z;
  const int q0 = qb2 * 2 * BQ;
  const int nkb_all = (p.T + BKV - 1) / BKV;
  // key blocks each tile attends to (a tile that starts beyond the sequence has none)
  int nkb_tile[2];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const int qb = qb2 * 2 + g;
    nkb_tile[g] = (q0 + g * BQ >= p.T) ? 0 : (p.causal ? min(nkb_all, qb + 1) : nkb_all);
  }
  const int nkb = max(nkb_tile[0], nkb_tile[1]);

  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    mbar_init(q_full, 1);
    mbar_init(k_full, 1);
    mbar_init(k_empty, 1);
    mbar_init(v_full, 1);
    mbar_init(v_empty, 1);
    for (int g = 0; g < 2; ++g) {
      mbar_init(&s_full[g], 1);
      mbar_init(&p_ready[g], 4);
      mbar_init(&pv_full[g], 1);
    }
    mbar_fence_init();
  }
  if (warp == 0) { tmem_alloc(tmem_slot, kTmemCols); tmem_relinquish(); }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      mbar_expect_tx(q_full, 2 * kQBytes);
#pragma unroll
      for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int j = 0; j < DP; ++j)   // rows beyond the sequence are filled with zeros by TMA
          tma_load_attn(sQ + g * kQBytes + j * BQ * 128, &map_q, q_full, j * 64, h, q0 + g * BQ, b);
      auto load_k = [&](int kb) {
        mbar_expect_tx(k_full, kKVBytes);
#pragma unroll
        for (int j = 0; j < DP; ++j) tma_load_attn(sK + j * BKV * 128, &map_k, k_full, j * 64, h, kb * BKV, b);
      };
      auto load_v = [&](int kb) {
        mbar_expect_tx(v_full, kKVBytes);
#pragma unroll
        for (int j = 0; j < DP; ++j) tma_load_attn(sV + j * BKV * 128, &map_v, v_full, j * 64, h, kb * BKV, b);
      };
      const uint32_t idesc_s = make_idesc_f16kind(128, BKV, false, false);
      const uint32_t idesc_pv = make_idesc_f16kind(128, D, false, true);   // B = V is MN-major
      const uint32_t k_addr = smem_u32(sK), v_addr = smem_u32(sV);
      auto issue_s = [&](int g) {      // S_g = Q_g · Kᵀ
        const uint32_t q_addr = smem_u32(sQ + g * kQBytes);
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint64_t da = make_smem_desc_sw128(q_addr + (k / 4) * BQ * 128 + (k % 4) * 32, 16, 1024);
          const uint64_t db = make_smem_desc_sw128(k_addr + (k / 4) * BKV * 128 + (k % 4) * 32, 16, 1024);
          mma_f16_ss(tmem + g * 128, da, db, idesc_s, k != 0);
        }
        mma_commit(&s_full[g]);
      };
      auto issue_pv = [&](int g, bool first) {     // O_g (+)= P_g · V: accumulated over the key blocks in tensor memory
        const uint32_t p_addr = smem_u32(sP + g * kPBytes);
#pragma unroll
        for (int k = 0; k < BKV / 16; ++k) {
          const uint64_t da = make_smem_desc_sw128(p_addr + (k / 4) * BQ * 128 + (k % 4) * 32, 16, 1024);
          const uint64_t db = make_smem_desc_sw128(v_addr + k * 16 * 128, BKV * 128, 1024);
          mma_f16_ss(tmem + 256 + g * D, da, db, idesc_pv, !first || k != 0);
        }
        mma_commit(&pv_full[g]);
      };
      if (nkb > 0) {
        load_k(0);
        load_v(0);
        ok = mbar_wait(q_full, 0) && mbar_wait(k_full, 0);
        if (ok) {
          fence_after_sync();
          if (0 < nkb_tile[0]) issue_s(0);
          if (0 < nkb_tile[1]) issue_s(1);
          mma_commit(k_empty);
        }
      }
      for (int kb = 0; kb < nkb && ok; ++kb) {
        const uint32_t ph = kb & 1;
        const bool more = kb + 1 < nkb;
        if (more) {                          // K block kb has been read by both S MMAs: fetch the next one
          if (!mbar_wait(k_empty, ph)) { ok = false; break; }
          load_k(kb + 1);
        }
        if (!mbar_wait(v_full, ph)) { ok = false; break; }
        if (kb < nkb_tile[0]) {
          if (!mbar_wait(&p_ready[0], ph)) { ok = false; break; }
          fence_after_sync();
          issue_pv(0, kb == 0);
        }
        if (more) {
          if (!mbar_wait(k_full, ph ^ 1)) { ok = false; break; }
          fence_after_sync();
          if (kb + 1 < nkb_tile[0]) issue_s(0);   // S_A was consumed before p_ready[0] arrived
        }
        if (kb < nkb_tile[1]) {
          if (!mbar_wait(&p_ready[1], ph)) { ok = false; break; }
          fence_after_sync();
          issue_pv(1, kb == 0);
        }
        mma_commit(v_empty);
        if (more) {
          if (kb + 1 < nkb_tile[1]) issue_s(1);
          mma_commit(k_empty);
          if (!mbar_wait(v_empty, ph)) { ok = false; break; }   // both P·V MMAs of this block have read V
          load_v(kb + 1);
        }
      }
      if (!ok) atomicExch(p.status, ATT_ERR_TIMEOUT);
    }
  } else {
    // ---------------------------------------------------------------- softmax / output threads of one tile
    const int g = (warp - 1) >> 2;                   // tile of this warp group
    const int lane_group = warp & 3;                 // TMEM lane quarter this warp may access
    const int row = lane_group * 32 + lane;
    const int qb = qb2 * 2 + g;
    const int t_q = q0 + g * BQ + row;
    const uint32_t lane_addr = uint32_t(lane_group * 32) << 16;
    const uint32_t tmem_s = tmem + g * 128, tmem_pv = tmem + 256 + g * D;
    uint8_t* sPg = sP + g * kPBytes;
    const int my_nkb = nkb_tile[g];
    // m is the reference of the exponentials accumulated so far: p = 2^((s - m) * scale_log2).  It follows the running
    // row maximum lazily — only when the maximum has moved by more than 2^8 past it — so that the output accumulator,
    // which lives in tensor memory and is added to by every P·V product, has to be rescaled on a few blocks only
    // (values of p stay below 2^8, far inside bf16 range; the final division by the row sum uses the same reference).
    float m = -INFINITY, l = 0.0f;
    bool ok = true;
    for (int kb = 0; kb < my_nkb; ++kb) {
      if (!mbar_wait(&s_full[g], kb & 1)) { ok = false; break; }
      fence_after_sync();
      const int k0 = kb * BKV;
      // keys of this block that the row sees: [0, vis)
      int vis = BKV;
      if ((p.causal && kb == qb) || (k0 + BKV > p.T)) vis = min(BKV, (p.causal ? min(p.T, t_q + 1) : p.T) - k0);
      // The row's scores, read from tensor memory once (registers for all 128).  Masking is a pass of its own that
      // only the last blocks of a row take: as a condition inside the loops below it cost every block four
      // instructions per score.
      uint32_t r[BKV];
#pragma unroll
      for (int c0 = 0; c0 < BKV; c0 += 32) tmem_ld_32x32(tmem_s + lane_addr + c0, *reinterpret_cast<uint32_t(*)[32]>(r + c0));
      tmem_ld_wait();
      if (vis < BKV) {
#pragma unroll
        for (int j = 0; j < BKV; ++j)
          if (j >= vis) r[j] = 0xff800000u;      // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < BKV; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], __uint_as_float(r[j]));
      const float m_blk = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      const bool grow = (m_blk - m) * p.scale_log2 > 8.0f;      // true on the first block (m = -inf) of any visible key
      float alpha = 1.0f;
      if (grow) {
        alpha = (m == -INFINITY) ? 0.0f : fast_exp2((m - m_blk) * p.scale_log2);
        m = m_blk;
      }
      const float m_use = (m == -INFINITY) ? 0.0f : m;
      if (kb > 0 && __any_sync(0xffffffffu, grow)) {
        // Some row of this warp moved its reference: scale the accumulated output rows in tensor memory.  The P·V
        // product of the previous block has completed (S of this block was issued after it); the wait makes that
        // ordering explicit and returns at once.
        if (!mbar_wait(&pv_full[g], (kb - 1) & 1)) { ok = false; break; }
        fence_after_sync();
        const float2 a2 = make_float2(alpha, alpha);
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t ro[32];
          tmem_ld_32x32(tmem_pv + lane_addr + c0, ro);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            const float2 v = __fmul2_rn(make_float2(__uint_as_float(ro[j]), __uint_as_float(ro[j + 1])), a2);
            ro[j] = __float_as_uint(v.x);
            ro[j + 1] = __float_as_uint(v.y);
          }
          tmem_st_32x32(tmem_pv + lane_addr + c0, ro);
        }
        tmem_st_wait();
      }
      // p = 2^(s * scale_log2 - m * scale_log2): one packed multiply-add per pair, then the exponential; the row sum
      // is taken over the fp32 values (pairs, packed adds)
      const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
      const float nm = -m_use * p.scale_log2;
      const float2 nm2 = make_float2(nm, nm);
      float2 rs2 = make_float2(0.0f, 0.0f), rs2b = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int chunk = 0; chunk < BKV / 8; ++chunk) {
        __align__(16) elem2_t hh[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int j = chunk * 8 + 2 * q;
          const float2 e = __ffma2_rn(make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), sc2, nm2);
          const float2 pe = make_float2(fast_exp2(e.x), fast_exp2(e.y));
          if (q & 1) rs2b = __fadd2_rn(rs2b, pe); else rs2 = __fadd2_rn(rs2, pe);
          hh[q] = f22e2(pe);
        }
        *reinterpret_cast<uint4*>(sPg + (chunk >> 3) * BQ * 128 + swz(row, chunk & 7)) = *reinterpret_cast<uint4*>(hh);
      }
      l = l * alpha + ((rs2.x + rs2.y) + (rs2b.x + rs2b.y));
      fence_proxy_async();
      fence_before_sync();
      warp_arrive(&p_ready[g]);
    }
    if (ok && my_nkb > 0) {
      // the last P·V product completes the output rows in tensor memory: divide by the row sum and store
      if (!mbar_wait(&pv_full[g], (my_nkb - 1) & 1)) ok = false;
      fence_after_sync();
      if (ok) {
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
        const float2 inv2 = make_float2(inv, inv);
        elem_t* dst = p.out + (((long long)b * p.T + t_q) * p.H + h) * D;
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t r[32];
          tmem_ld_32x32(tmem_pv + lane_addr + c0, r);
          tmem_ld_wait();
          if (t_q < p.T) {
#pragma unroll
            for (int d = 0; d < 32; d += 8) {
              __align__(16) elem2_t hh[4];
#pragma unroll
              for (int q = 0; q < 4; ++q)
                hh[q] = f22e2(__fmul2_rn(
                    make_float2(__uint_as_float(r[d + 2 * q]), __uint_as_float(r[d + 2 * q + 1])), inv2));
              *reinterpret_cast<uint4*>(dst + c0 + d) = *reinterpret_cast<uint4*>(hh);
            }
          }
        }
        if (t_q < p.T && p.lse != nullptr)
          p.lse[((long long)b * p.H + h) * p.T + t_q] = (l > 0.0f) ? m * p.scale + logf(l) : -INFINITY;
      }
      fence_before_sync();
    }
    if (!ok && lane == 0) atomicExch(p.status, ATT_ERR_TIMEOUT);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) { fence_after_sync(); tmem_dealloc(tmem, kTmemCols); }
}

// -------------------------------------------------------------------------------------------------
// backward pre-pass: delta[b,h,t] = sum_d dO*O.  D / 8 lanes per row, 16-byte loads: DRAM-bound (the two tensors are
// read once).  28 us -> 9 us at B8 T1024 H16 D64 (a warp per row with 4-byte loads before).
// -------------------------------------------------------------------------------------------------
template <int D>
__global__ void attn_delta_kernel(const elem_t* __restrict__ o, const elem_t* __restrict__ d_o, float* __restrict__ delta,
                                  int B, int T, int H, long long do_sb, long long do_st, long long do_sh) {
  constexpr int kLanes = D / 8;
  const long long idx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;   // (b, t, h) row
  const int part = threadIdx.x % kLanes;
  const bool on = idx < (long long)B * T * H;
  float s = 0.0f;
  const int hh = (int)(idx % H);
  const long long bt = idx / H;
  const int t = (int)(bt % T), b = (int)(bt / T);
  if (on) {
    const uint4 ov = *reinterpret_cast<const uint4*>(o + idx * D + part * 8);
    const uint4 gv = *reinterpret_cast<const uint4*>(d_o + b * do_sb + t * do_st + hh * do_sh + part * 8);
    const elem2_t* oe = reinterpret_cast<const elem2_t*>(&ov);
    const elem2_t* ge = reinterpret_cast<const elem2_t*>(&gv);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = e22ff(oe[i]), y = e22ff(ge[i]);
      s += x.x * y.x + x.y * y.y;
    }
  }
#pragma unroll
  for (int off = kLanes / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  if (on && part == 0) delta[((long long)b * H + hh) * T + t] = s;
}

// The fp32 sums of dQ are kept by (batch, head, query block) as [D / 4 pieces][rows][4]: the threads that add to them
// own one row each, and in this order a warp's 16-byte reductions cover 512 consecutive bytes.  In row order they touch
// 32 different lines per instruction, which kept the load/store unit busy for 2700 (D = 64) and 5700 cycles per block
// and delayed every shared-memory store behind it.  A block has 128 rows, the last one of a sequence what is left: the
// scratch, its zero fill and this pass are as large as dQ also where a sequence is a few tokens.  This kernel turns a
// block into 16-bit rows of a strided view.
// WHOLE, here and in the main kernel: T is a multiple of 128, so every block has 128 rows and the pitch of the pieces is a
// constant.  Backward at B8 T1024 H16 D64 causal 135.8 us, 137.3 with the pitch at run time; B64 T200 H16 D64, ragged,
// 154.8 (160.1 with all blocks rounded up), B512 T24 H8 D128 233.6 (291.1).
template <int D, bool WHOLE>
__global__ void __launch_bounds__(256) attn_dq_store_kernel(const float4* __restrict__ src, elem_t* __restrict__ dst, int T, int H,
                                                            int nqb, long long sb, long long st, long long sh) {
  constexpr int kLd = D + 8;   // 16-byte pieces of 8 rows on different banks
  __shared__ __align__(16) elem_t tile[128 * kLd];
  const int qb = blockIdx.x % nqb, rows = WHOLE ? 128 : min(128, T - qb * 128);
  const long long bh = blockIdx.x / nqb;
  const float4* in = src + (WHOLE ? (long long)blockIdx.x * 128 : bh * T + qb * 128) * (D / 4);
  auto put = [&](const float4& v, int row, int piece) {
    __align__(8) elem2_t e[2] = {ff2e2(v.x, v.y), ff2e2(v.z, v.w)};
    *reinterpret_cast<uint2*>(tile + row * kLd + piece * 4) = *reinterpret_cast<uint2*>(e);
  };
  if constexpr (WHOLE) {
#pragma unroll
    for (int i = threadIdx.x; i < 128 * D / 4; i += 256) put(in[i], i % 128, i / 128);
  } else if (threadIdx.x % 128 < rows) {
    const int row = threadIdx.x % 128;
#pragma unroll
    for (int piece = threadIdx.x / 128; piece < D / 4; piece += 2) put(in[piece * rows + row], row, piece);
  }
  __syncthreads();
  elem_t* out = dst + bh / H * sb + bh % H * sh;
#pragma unroll
  for (int i = threadIdx.x; i < 128 * D / 8; i += 256) {
    const int row = i / (D / 8), d = i % (D / 8) * 8, t = qb * 128 + row;
    if (row < rows) *reinterpret_cast<uint4*>(out + t * st + d) = *reinterpret_cast<const uint4*>(tile + row * kLd + d);
  }
}

// -------------------------------------------------------------------------------------------------
// backward main kernel
// -------------------------------------------------------------------------------------------------
// One CTA per (batch, head, 128 keys) walks the query blocks.  The five products of a block and the point-wise work
// between them form a cycle; what bounds the kernel is how much of that cycle overlaps.  Roles:
//   warp 21     TMA: K, V once; Q two blocks deep; dO two blocks deep (D = 64) or one (D = 128: shared memory is full)
//   warp 20     MMA issue, in the order  S(i+1), dV(i)  once P(i) is stored, then  dP(i+1), dQ(i), dK(i)  (D = 64) or
//               dQ(i), dK(i), dP(i+1)  (D = 128, where dQ borrows dP's columns) once dS(i) is stored: while the tensor
//               core works on block i, the point-wise warps already have S(i+1)
//   warps 4-19  point-wise: P = exp2(scale·S − lse) -> shared memory, then dS = P∘(dP − δ)·scale -> shared memory; four
//               threads per query row, 32 keys each, and the row statistics fetched one block ahead
//   warps 0-3   drain dQ from tensor memory into the fp32 sums (16-byte reductions), off everybody else's path
// Every barrier that a role waits on can complete its next phase only after that role has gone on (Q and dO have one
// "free" barrier per stage for this reason), so a wait by phase parity cannot miss a phase.
// Tensor memory: S 128 | dP 128 | dV D | dK D | (D = 64) dQ 64 columns.
//
// Before, one group of four warps did load, products, point-wise work and drain in turn: at B8 T1024 H16 D64 causal
// 291 us, now 108 us; at B16 T480 H8 D128 197 us, now 82 us.
struct AttnBwdParams {
  int B, T, H;
  int causal;
  float scale_log2, scale;
  const float* lse;    // (B, H, T)
  const float* delta;  // (B, H, T)
  float4* dq;          // (B, H, query block, D / 4, rows) fp32, zero-initialised; accumulated with reductions
  elem_t* dk;          // (B, T, H, D) views with strides g_sb, g_st, g_sh
  elem_t* dv;
  long long g_sb, g_st, g_sh;
  int* status;
};

constexpr int kBwdWarps = 22, kBwdThreads = kBwdWarps * 32;

template <int D>
constexpr int kBwdDoStages = D == 64 ? 2 : 1;
template <int D>
constexpr int kBwdPBuffers = D == 64 ? 2 : 1;
template <int D>
constexpr int bwd_smem_bytes() { return (4 + kBwdDoStages<D>) * 128 * D * 2 + (1 + kBwdPBuffers<D>) * 128 * 128 * 2 + 256 + 1024; }

template <int D, bool WHOLE>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                const AttnBwdParams p) {
  constexpr int DP = D / 64;
  constexpr int kTile = 128 * D * 2;           // a 128-row x D operand tile
  constexpr int kSq = 128 * 128 * 2;           // P / dS tiles
  constexpr int kDoStages = kBwdDoStages<D>;
  constexpr int kPBuffers = kBwdPBuffers<D>;
  constexpr bool kOwnDq = D == 64;             // dQ has tensor-memory columns of its own
  constexpr uint32_t kTmemCols = 512;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + kTile;
  uint8_t* sQ = sV + kTile;                    // two stages
  uint8_t* sDO = sQ + 2 * kTile;               // kDoStages stages
  uint8_t* sP = sDO + kDoStages * kTile;
  uint8_t* sDS = sP + kPBuffers * kSq;         // P: kPBuffers buffers
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDS + kSq);
  uint64_t* kv_full = bars;
  uint64_t* q_full = bars + 1;      // [2]
  uint64_t* do_full = bars + 3;     // [2]
  uint64_t* q_free = bars + 5;      // [2] dK(i) has read the stage
  uint64_t* do_free = bars + 7;     // [2] dV(i) has read the stage
  uint64_t* s_full = bars + 9;      // S(i) in tensor memory
  uint64_t* dp_full = bars + 10;    // dP(i) in tensor memory
  uint64_t* p_ready = bars + 11;    // P(i) stored, S(i) read (16 warps)
  uint64_t* ds_ready = bars + 12;   // dS(i) stored, dP(i) read (16 warps)
  uint64_t* dv_done = bars + 13;    // [2] dV(i) has read the P buffer
  uint64_t* dq_full = bars + 15;    // dQ(i) in tensor memory
  uint64_t* dq_read = bars + 16;    // dQ(i) drained (4 warps)
  uint64_t* dk_done = bars + 17;    // dQ(i) and dK(i) have read dS; all products so far are complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // causal: the key blocks with the most query blocks first, over all heads
  const int kb = p.causal ? blockIdx.z : blockIdx.x;
  const int h = p.causal ? blockIdx.x : blockIdx.y;
  const int b = p.causal ? blockIdx.y : blockIdx.z;
  const int k0 = kb * BKV;
  const int qb0 = p.causal ? kb : 0;
  const int nqb = (p.T + BQ - 1) / BQ, n = nqb - qb0;     // query blocks; at least one of them ours

  if (threadIdx.x == 0) {
    prefetch_tensormap(&map_q); prefetch_tensormap(&map_k); prefetch_tensormap(&map_v); prefetch_tensormap(&map_do);
    for (int i = 0; i < 18; ++i) mbar_init(&bars[i], i == 11 || i == 12 ? 16 : i == 16 ? 4 : 1);
    mbar_fence_init();
  }
  if (warp == 20) { tmem_alloc(tmem_slot, kTmemCols); tmem_relinquish(); }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tm_s = tmem, tm_dp = tmem + 128, tm_dv = tmem + 256, tm_dk = tmem + 256 + D;
  const uint32_t tm_dq = kOwnDq ? tmem + 256 + 2 * D : tm_dp;

  if (warp == 21) {
    if (elect_one()) {
      bool ok = true;
      auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int t) {
#pragma unroll
        for (int j = 0; j < DP; ++j) tma_load_attn(dst + j * 128 * 128, map, bar, j * 64, h, t, b);
      };
      auto load_q = [&](int i) {
        if (i >= 2 && !mbar_wait(&q_free[i & 1], ((i >> 1) - 1) & 1)) { ok = false; return; }
        mbar_expect_tx(&q_full[i & 1], kTile);
        load(sQ + (i & 1) * kTile, &map_q, &q_full[i & 1], (qb0 + i) * BQ);
      };
      auto load_do = [&](int i) {
        const int s = i % kDoStages;
        if (i >= kDoStages && !mbar_wait(&do_free[s], (i / kDoStages - 1) & 1)) { ok = false; return; }
        mbar_expect_tx(&do_full[s], kTile);
        load(sDO + s * kTile, &map_do, &do_full[s], (qb0 + i) * BQ);
      };
      mbar_expect_tx(kv_full, 2 * kTile);
      load(sK, &map_k, kv_full, k0);
      load_q(0);
      load(sV, &map_v, kv_full, k0);
      load_do(0);
      if (n > 1) load_q(1);
      for (int i = 1; i < n && ok; ++i) {
        load_do(i);
        if (ok && i + 1 < n) load_q(i + 1);
      }
      if (!ok) atomicExch(p.status, ATT_ERR_TIMEOUT);
    }
  } else if (warp == 20) {
    if (elect_one()) {
      bool ok = true;
      const uint32_t id_s = make_idesc_f16kind(128, 128, false, false);   // S = Q Kᵀ, dP = dO Vᵀ
      const uint32_t id_t = make_idesc_f16kind(128, D, true, true);       // dV = Pᵀ dO, dK = dSᵀ Q (A, B MN-major)
      const uint32_t id_q = make_idesc_f16kind(128, D, false, true);      // dQ = dS K (B MN-major)
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aP = smem_u32(sP), aDS = smem_u32(sDS);
      auto scores = [&](uint32_t d, uint32_t a, uint32_t bb) {            // both operands K-major over D
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k / 4) * 128 * 128 + (k % 4) * 32;
          mma_f16_ss(d, make_smem_desc_sw128(a + off, 16, 1024), make_smem_desc_sw128(bb + off, 16, 1024), id_s, k != 0);
        }
      };
      auto transposed = [&](uint32_t d, uint32_t a, uint32_t bb, bool first) {
        // K dimension = queries, 16 rows per step.  A (P or dS) is [query rows][keys]: as an MN-major operand its M =
        // keys; two 64-key panels, LBO = panel
#pragma unroll
        for (int k = 0; k < 128 / 16; ++k)
          mma_f16_ss(d, make_smem_desc_sw128(a + k * 16 * 128, 128 * 128, 1024),
                     make_smem_desc_sw128(bb + k * 16 * 128, 128 * 128, 1024), id_t, !first || k != 0);
      };
      auto issue_s = [&](int i) {
        if (!mbar_wait(&q_full[i & 1], (i >> 1) & 1)) { ok = false; return; }
        fence_after_sync();
        scores(tm_s, smem_u32(sQ + (i & 1) * kTile), aK);
        mma_commit(s_full);
      };
      auto issue_dp = [&](int i) {
        if (!mbar_wait(&do_full[i % kDoStages], (i / kDoStages) & 1)) { ok = false; return; }
        fence_after_sync();
        scores(tm_dp, smem_u32(sDO + (i % kDoStages) * kTile), aV);
        mma_commit(dp_full);
      };
      ok = mbar_wait(kv_full, 0);
      if (ok) issue_s(0);
      if (ok) issue_dp(0);
      for (int i = 0; i < n && ok; ++i) {
        if (!mbar_wait(p_ready, i & 1)) { ok = false; break; }
        fence_after_sync();
        if (i + 1 < n) issue_s(i + 1);
        if (!ok) break;
        transposed(tm_dv, aP + (i % kPBuffers) * kSq, smem_u32(sDO + (i % kDoStages) * kTile), i == 0);
        mma_commit(&dv_done[i % kPBuffers]);
        mma_commit(&do_free[i % kDoStages]);
        if (!mbar_wait(ds_ready, i & 1)) { ok = false; break; }
        fence_after_sync();
        if (kOwnDq) {
          if (i + 1 < n) issue_dp(i + 1);
          if (!ok || (i > 0 && !mbar_wait(dq_read, (i - 1) & 1))) { ok = false; break; }
          fence_after_sync();
        }
#pragma unroll
        for (int k = 0; k < 128 / 16; ++k) {   // dQ = dS (K-major over keys) · K (MN-major: key rows, D contiguous)
          const uint64_t a_ds = make_smem_desc_sw128(aDS + (k / 4) * 128 * 128 + (k % 4) * 32, 16, 1024);
          const uint64_t b_k = make_smem_desc_sw128(aK + k * 16 * 128, 128 * 128, 1024);
          mma_f16_ss(tm_dq, a_ds, b_k, id_q, k != 0);
        }
        mma_commit(dq_full);
        transposed(tm_dk, aDS, smem_u32(sQ + (i & 1) * kTile), i == 0);
        mma_commit(dk_done);
        mma_commit(&q_free[i & 1]);
        if (!kOwnDq && i + 1 < n) {
          if (!mbar_wait(dq_read, i & 1)) { ok = false; break; }
          fence_after_sync();
          issue_dp(i + 1);
        }
      }
      if (!ok) atomicExch(p.status, ATT_ERR_TIMEOUT);
    }
  } else if (warp >= 4) {
    // ---------------------------------------------------------------- point-wise: one query row, 32 keys per thread
    const int lane_group = warp & 3, part = (warp - 4) >> 2;
    const int row = lane_group * 32 + lane;
    const uint32_t lane_addr = uint32_t(lane_group * 32) << 16;
    const long long stat0 = ((long long)b * p.H + h) * p.T;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    uint8_t* pRow = sP + (part >> 1) * 128 * 128;      // the 64-key panel
    uint8_t* dsRow = sDS + (part >> 1) * 128 * 128;
    const int chunk0 = (part & 1) * 4;                 // first 16-byte piece of the panel row
    bool ok = true;
    float lse_next = 0.0f, dl_next = 0.0f;             // statistics of the next block: fetched one block ahead
    if (qb0 * BQ + row < p.T) {
      lse_next = p.lse[stat0 + qb0 * BQ + row];
      dl_next = p.delta[stat0 + qb0 * BQ + row];
    }
    for (int i = 0; i < n; ++i) {
      const int t_q = (qb0 + i) * BQ + row;
      const bool row_ok = t_q < p.T;
      const float lse = lse_next, dl = dl_next;
      if (t_q + BQ < p.T) {
        lse_next = p.lse[stat0 + t_q + BQ];
        dl_next = p.delta[stat0 + t_q + BQ];
      }
      const float nl = -lse * 1.4426950408889634f;
      const float2 nl2 = make_float2(nl, nl);
      // keys of this thread that the row sees: [0, vis)
      int vis = 32;
      if ((p.causal && i == 0) || (k0 + BKV > p.T) || !row_ok) {
        const int lim = !row_ok ? 0 : (p.causal ? min(p.T, t_q + 1) : p.T);
        vis = min(32, max(0, lim - (k0 + part * 32)));
      }
      if (!mbar_wait(s_full, i & 1)) { ok = false; break; }
      fence_after_sync();
      uint32_t r[32];
      float pr[32];
      tmem_ld_32x32(tm_s + lane_addr + part * 32, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        const float2 e = __ffma2_rn(make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), sc2, nl2);
        pr[j] = fast_exp2(e.x);
        pr[j + 1] = fast_exp2(e.y);
      }
      if (vis < 32) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j >= vis) pr[j] = 0.0f;
      }
      // dV(i - kPBuffers) has read the buffer
      if (i >= kPBuffers && !mbar_wait(&dv_done[i % kPBuffers], (i / kPBuffers - 1) & 1)) { ok = false; break; }
#pragma unroll
      for (int j8 = 0; j8 < 4; ++j8) {
        __align__(16) elem2_t hp[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) hp[q] = ff2e2(pr[j8 * 8 + 2 * q], pr[j8 * 8 + 2 * q + 1]);
        *reinterpret_cast<uint4*>(pRow + (i % kPBuffers) * kSq + swz(row, chunk0 + j8)) = *reinterpret_cast<uint4*>(hp);
      }
      fence_proxy_async();
      fence_before_sync();
      warp_arrive(p_ready);
      if (!mbar_wait(dp_full, i & 1)) { ok = false; break; }
      fence_after_sync();
      tmem_ld_32x32(tm_dp + lane_addr + part * 32, r);
      tmem_ld_wait();
      if (i > 0 && !mbar_wait(dk_done, (i - 1) & 1)) { ok = false; break; }   // dQ(i-1), dK(i-1) have read dS
#pragma unroll
      for (int j8 = 0; j8 < 4; ++j8) {
        __align__(16) elem2_t hd[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int j = j8 * 8 + 2 * q;
          hd[q] = ff2e2(pr[j] * (__uint_as_float(r[j]) - dl) * p.scale, pr[j + 1] * (__uint_as_float(r[j + 1]) - dl) * p.scale);
        }
        *reinterpret_cast<uint4*>(dsRow + swz(row, chunk0 + j8)) = *reinterpret_cast<uint4*>(hd);
      }
      fence_proxy_async();
      fence_before_sync();
      warp_arrive(ds_ready);
    }
    // dV (parts 0, 1) and dK (parts 2, 3) of this key block, half of the columns each
    if (ok && mbar_wait(dk_done, (n - 1) & 1)) {
      fence_after_sync();
      const int t_k = k0 + row;
      elem_t* dst = (part < 2 ? p.dv : p.dk) + (long long)b * p.g_sb + (long long)t_k * p.g_st + (long long)h * p.g_sh;
      const uint32_t src = part < 2 ? tm_dv : tm_dk;
#pragma unroll 1
      for (int c0 = (part & 1) * (D / 2); c0 < ((part & 1) + 1) * (D / 2); c0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32(src + lane_addr + c0, r);
        tmem_ld_wait();
        if (t_k < p.T) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            __align__(16) elem2_t hh[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              hh[q] = ff2e2(__uint_as_float(r[j + 2 * q]), __uint_as_float(r[j + 2 * q + 1]));
            *reinterpret_cast<uint4*>(dst + c0 + j) = *reinterpret_cast<uint4*>(hh);
          }
        }
      }
    } else {
      ok = false;
    }
    if (!ok && lane == 0) atomicExch(p.status, ATT_ERR_TIMEOUT);
  } else {
    // ---------------------------------------------------------------- dQ drain: one query row per thread
    const int row = warp * 32 + lane;
    const uint32_t lane_addr = uint32_t(warp * 32) << 16;
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      const int t_q = (qb0 + i) * BQ + row, rows = WHOLE ? 128 : min(BQ, p.T - (qb0 + i) * BQ);
      float4* dst = WHOLE ? p.dq + (((long long)b * p.H + h) * nqb + qb0 + i) * (D / 4) * 128 + row
                          : p.dq + (((long long)b * p.H + h) * p.T + (qb0 + i) * BQ) * (D / 4) + row;
      if (!mbar_wait(dq_full, i & 1)) { ok = false; break; }
      fence_after_sync();
#pragma unroll 1
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tm_dq + lane_addr + c0, r);
        tmem_ld_wait();
        if (c0 + 32 == D) {      // all of dQ(i) has been read: the columns may be written again
          fence_before_sync();
          warp_arrive(dq_read);
        }
        if (t_q < p.T) {
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            atomicAdd(dst + (c0 + j) / 4 * rows,
                      make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                                  __uint_as_float(r[j + 3])));
        }
      }
    }
    if (!ok && lane == 0) atomicExch(p.status, ATT_ERR_TIMEOUT);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 20) { fence_after_sync(); tmem_dealloc(tmem, kTmemCols); }
}

// -------------------------------------------------------------------------------------------------
// host
// -------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

// (B, T, H, D) view with element strides sb, st, sh (inner stride 1); box = 64 x 1 x 128 x 1.
int encode_bthd(CUtensorMap* map, const void* base, int B, int T, int H, int D, long long sb, long long st,
                long long sh) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return 4;
  {  // the driver entry point needs a context current on this thread (see gemm_tcgen05.h)
    static thread_local int bound = -1;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev != bound) {
      cudaSetDevice(dev);
      bound = dev;
    }
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (sb * 2) % 16 || (st * 2) % 16 || (sh * 2) % 16) return 2;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)T, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)sh * 2, (cuuint64_t)st * 2, (cuuint64_t)sb * 2};
  cuuint32_t box[4] = {64, 1, 128, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(map, ELEM_TMAP, 4, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 3;
}

template <typename K>
int set_smem(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess ? 0 : 5;
}

}  // namespace

extern "C" {

// q/k/v: (B, T, H, D) views, strides in elements (batch, time, head); out: contiguous (B, T, H, D); lse: (B, H, T).
int fbam_attn_fwd(const void* q, const void* k, const void* v, long long sb, long long st, long long sh, void* out,
                  float* lse, int B, int T, int H, int D, int causal, float scale, int* status, void* stream) {
  if ((D != 64 && D != 128) || B < 1 || T < 1 || H < 1) return 1;
  CUtensorMap mq, mk, mv;
  int e;
  if ((e = encode_bthd(&mq, q, B, T, H, D, sb, st, sh))) return e;
  if ((e = encode_bthd(&mk, k, B, T, H, D, sb, st, sh))) return e;
  if ((e = encode_bthd(&mv, v, B, T, H, D, sb, st, sh))) return e;
  AttnParams p{B, T, H, D, causal, scale * 1.4426950408889634f, scale, (elem_t*)out, lse, status};
  dim3 grid((T + BQ - 1) / BQ, H, B);
  const int stages = D == 64 ? 1 : 2;
  const int smem = BQ * D * 2 + 2 * stages * BKV * D * 2 + BQ * BKV * 2 + 256 + 1024;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (D == 64) {
    if (set_smem(attn_fwd_kernel<64, 1>, smem)) return 5;
    attn_fwd_kernel<64, 1><<<grid, 160, smem, s>>>(mq, mk, mv, p);
  } else {
    if (set_smem(attn_fwd_kernel<128, 2>, smem)) return 5;
    attn_fwd_kernel<128, 2><<<grid, 160, smem, s>>>(mq, mk, mv, p);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 5;
}

// Variant of fbam_attn_fwd with two query tiles per CTA (attn_fwd2_kernel); same arguments and results.
int fbam_attn_fwd2(const void* q, const void* k, const void* v, long long sb, long long st, long long sh, void* out,
                   float* lse, int B, int T, int H, int D, int causal, float scale, int* status, void* stream) {
  if ((D != 64 && D != 128) || B < 1 || T < 1 || H < 1) return 1;
  CUtensorMap mq, mk, mv;
  int e;
  if ((e = encode_bthd(&mq, q, B, T, H, D, sb, st, sh))) return e;
  if ((e = encode_bthd(&mk, k, B, T, H, D, sb, st, sh))) return e;
  if ((e = encode_bthd(&mv, v, B, T, H, D, sb, st, sh))) return e;
  AttnParams p{B, T, H, D, causal, scale * 1.4426950408889634f, scale, (elem_t*)out, lse, status};
  dim3 grid((T + 2 * BQ - 1) / (2 * BQ), H, B);
  const int smem = 2 * BQ * D * 2 + 2 * BKV * D * 2 + 2 * BQ * BKV * 2 + 256 + 1024;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (D == 64) {
    if (set_smem(attn_fwd2_kernel<64>, smem)) return 5;
    attn_fwd2_kernel<64><<<grid, 288, smem, s>>>(mq, mk, mv, p);
  } else {
    if (set_smem(attn_fwd2_kernel<128>, smem)) return 5;
    attn_fwd2_kernel<128><<<grid, 288, smem, s>>>(mq, mk, mv, p);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 5;
}

// d_o: (B, T, H, D) view with its own strides; o: contiguous forward output; dq32: fp32 scratch for the sums of dQ,
// B * T * H * D values; dq/dk/dv: 16-bit (B, T, H, D) views that share the strides g_*; delta: (B, H, T) scratch.
int fbam_attn_bwd(const void* q, const void* k, const void* v, long long sb, long long st, long long sh, const void* o,
                  const void* d_o, long long do_sb, long long do_st, long long do_sh, const float* lse, float* delta,
                  float* dq32, void* dq, void* dk, void* dv, long long g_sb, long long g_st, long long g_sh, int B, int T,
                  int H, int D, int causal, float scale, int* status, void* stream) {
  if ((D != 64 && D != 128) || B < 1 || T < 1 || H < 1) return 1;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap mq, mk, mv, mdo;
  int e;
  if ((e = encode_bthd(&mq, q, B, T, H, D, sb, st, sh))) return e;
  if ((e = encode_bthd(&mk, k, B, T, H, D, sb, st, sh))) return e;
  if ((e = encode_bthd(&mv, v, B, T, H, D, sb, st, sh))) return e;
  if ((e = encode_bthd(&mdo, d_o, B, T, H, D, do_sb, do_st, do_sh))) return e;
  const uintptr_t outs = (uintptr_t)dq | (uintptr_t)dk | (uintptr_t)dv | (uintptr_t)o | (uintptr_t)dq32;
  if ((outs & 15) || g_sb % 8 || g_st % 8 || g_sh % 8) return 2;
  const long long rows = (long long)B * T * H, pieces = rows * (D / 8);
  const unsigned nkb = (T + BKV - 1) / BKV;      // also the query blocks
  if ((long long)B * H * nkb > 0x7fffffffll) return 1;
  if (cudaMemsetAsync(dq32, 0, (size_t)rows * D * sizeof(float), s) != cudaSuccess) return 5;
  const unsigned blocks = (unsigned)((pieces + 255) / 256);
  if (D == 64)
    attn_delta_kernel<64><<<blocks, 256, 0, s>>>((const elem_t*)o, (const elem_t*)d_o, delta, B, T, H, do_sb, do_st, do_sh);
  else
    attn_delta_kernel<128><<<blocks, 256, 0, s>>>((const elem_t*)o, (const elem_t*)d_o, delta, B, T, H, do_sb, do_st, do_sh);
  AttnBwdParams p{B, T, H, causal, scale * 1.4426950408889634f, scale, lse, delta, reinterpret_cast<float4*>(dq32), (elem_t*)dk, (elem_t*)dv,
                  g_sb, g_st, g_sh, status};
  const dim3 grid = causal ? dim3(H, B, nkb) : dim3(nkb, H, B);
  const bool whole = T % BQ == 0;
  auto kernel = D == 64 ? (whole ? attn_bwd_kernel<64, true> : attn_bwd_kernel<64, false>)
                        : (whole ? attn_bwd_kernel<128, true> : attn_bwd_kernel<128, false>);
  const int smem = D == 64 ? bwd_smem_bytes<64>() : bwd_smem_bytes<128>();
  if (set_smem(kernel, smem)) return 5;
  kernel<<<grid, kBwdThreads, smem, s>>>(mq, mk, mv, mdo, p);
  const unsigned tiles = (unsigned)B * H * nkb;
  auto store = D == 64 ? (whole ? attn_dq_store_kernel<64, true> : attn_dq_store_kernel<64, false>)
                       : (whole ? attn_dq_store_kernel<128, true> : attn_dq_store_kernel<128, false>);
  store<<<tiles, 256, 0, s>>>((const float4*)dq32, (elem_t*)dq, T, H, nkb, g_sb, g_st, g_sh);
  return cudaGetLastError() == cudaSuccess ? 0 : 5;
}

}  // extern "C"
