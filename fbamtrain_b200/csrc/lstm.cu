// Persistent recurrent LSTM kernels.
//
// The input projection X·W_ihᵀ for the whole sequence is one large tensor-core GEMM done elsewhere; what
// remains per time step is a (batch) x H · H x 4H product plus the gate arithmetic — far too small to launch as
// kernels 1024 times.  These kernels run the whole sequence in one cooperative launch, with W_hh resident on chip as
// mma.sync A fragments (registers; half in shared memory for H > 1024).  Batch rows are the 8-wide N of
// mma.sync.m16n8k16 (tcgen05 tiles start at M = 64 rows per CTA and would be mostly padding for this shape).
//
// What bounds a step is a chain of latencies, not bandwidth or arithmetic: publish the new vector, see the vectors of
// all other CTAs, multiply, reduce over warps, gate functions.  Hence:
//
//  * The exchanged vector is its own flag.  Forward: y[t] is both the output and the vector the next step reads;
//    backward: dGates[t].  The buffer is filled with 0xFF bytes beforehand and a reader polls the words it needs until
//    none of them is 0xFFFFFFFF (a 16-bit NaN pattern the conversions never produce; the writer maps it away all the
//    same).  Every word has exactly one writer and is written once, so no fence, counter or barrier is needed: one
//    store to L2 and one load from it per step.  A counter barrier with separate data took three L2 round trips.
//  * A warp owns a K slice and reads only that slice of the vector, straight into its MMA fragments (the 32 columns of
//    a K block are dealt to the lanes 8 at a time, with the weights permuted alike, so that a fragment is one 16-byte
//    load): no staging in shared memory, and a warp starts when its own slice has arrived.
//  * One block-wide barrier per step (partial sums over the K slices; two buffers take turns).  A quad of lanes owns
//    one (unit, batch row), one lane per gate, and exchanges the gates by shuffles.
//  * More than 8 batch rows are groups of 8 that have nothing to do with one another: they go to different CTAs while
//    the machine has room, then take turns inside a CTA.  A turn is a whole step of its group: poll, products, barrier
//    and publication of one group are over before the next one is looked at, so two turns cost about twice one.
//
// Forward: CTA j owns U = 8 or 16 hidden units (4U gate rows of W_hh).  The buffer of gate pre-activations is
// overwritten in place with the activated gates, which is exactly what the backward pass needs.
// Backward (BPTT): a cluster of four CTAs owns 4U units; CTA r of the cluster holds the columns of gate r of W_hhᵀ,
// reads gate r of dGates[t] only (a quarter of what a CTA without partners would have to read), and sends its partial
// sums of dh_{t-1} through distributed shared memory to the CTA that owns the unit.
//
// Measured on a B200, bf16, us per step over 1024 steps, with a grid-wide counter barrier, staged vectors and no clusters
// -> in this form:
//   H 1024, batch 8:  forward 2.93 -> 1.88, backward 5.08 -> 2.06
//   H 2048, batch 4:  forward 4.18 -> 3.32, backward 6.24 -> 3.75
//   H  256, batch 8:  forward 2.30 -> 1.03, backward 2.59 -> 1.66
//   H 1024, batch 32 (two groups, two turns): forward 3.49, backward 6.30
//   H 2048, batch 32 (one group, four turns): forward 12.9, backward 16.2
// A wider form of the cluster for the forward pass too (each CTA a quarter of h, partial sums through distributed
// shared memory) was 2.24 us at H = 1024: the cluster barrier costs more than the fewer polls give.
//
// The reference runs the recurrence as one GEMM launch plus a point-wise cell kernel per time step (reference:
// kernel_gen/kernel_gen/kernels/lstm_cell.py:6-144, kernels/lstm_cell_bwd.py:6-273 for the cell arithmetic and the
// recompute / backward point-wise kernels; tensorlib/src/streaming_lstm.cpp and streaming_lstm_bwd.cpp for the loop
// around them); gate order i, f, g, o, fp32 gates and cell state as there (tanh is tanhf here; the reference
// writes it as 2·sigmoid(2x) - 1, the same function).
#include "elem16.cuh"
#include <cuda_runtime.h>
#include <stdint.h>

namespace {

constexpr unsigned kSpinLimit = 1u << 22;  // polls of at least an L2 round trip each: seconds
constexpr uint32_t kEmpty = 0xffffffffu;   // a word of the exchange buffer that has not been written yet
constexpr int kCluster = 4;                // CTAs of a backward cluster: one per gate
constexpr int kLaunchRows = 32;            // batch rows of one launch
enum { LSTM_ERR_EXCHANGE_TIMEOUT = 201 };

__device__ __forceinline__ uint4 ld_relaxed_v4(const elem_t* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_relaxed_u16(const elem_t* p) {
  uint16_t v;
  asm volatile("ld.relaxed.gpu.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u32(elem_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed_u16(elem_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u16 [%0], %1;" ::"l"(p), "h"((uint16_t)v) : "memory");
}

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32." ELEM_PTX "." ELEM_PTX ".f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + __expf(-x)); }

// 8 consecutive elements of a weight row (4-byte loads: the weights need no more than 4-byte alignment).
__device__ __forceinline__ uint4 load_row8(const elem_t* p, bool on) {
  uint4 v = make_uint4(0, 0, 0, 0);
  if (on) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
    v = make_uint4(w[0], w[1], w[2], w[3]);
  }
  return v;
}

// The K slice of a warp: K blocks kb = warp + WARPS·j (32 columns each); lane q of a quad owns columns 8q..8q+7 of a
// block.  The two k-steps of a block use elements (0,1 | 2,3) and (4,5 | 6,7) of those for the two K halves of the
// MMA, in the weights and in the vector alike, so the order of the sum is all that changes.
// The first RB blocks of a warp have their weights in registers, the remaining SB in shared memory.
template <int WARPS, int TILES, int RB, int SB>
struct Weights {
  uint4 lo[RB][TILES], hi[RB][TILES];

  template <typename RowPtr>  // row(tile, r): pointer to row r of an MMA tile, or nullptr
  __device__ __forceinline__ void load(RowPtr row, int H, uint4* wsm) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int j = 0; j < RB + SB; ++j)
#pragma unroll
      for (int tile = 0; tile < TILES; ++tile) {
        const int k = (warp + WARPS * j) * 32 + q * 8;
        const elem_t *p = row(tile, g), *p8 = row(tile, g + 8);
        const uint4 a = load_row8(p + k, p != nullptr && k < H), b = load_row8(p8 + k, p8 != nullptr && k < H);
        if (j < RB) {
          lo[j < RB ? j : 0][tile] = a;
          hi[j < RB ? j : 0][tile] = b;
        } else {  // read back by the same thread only: no barrier
          wsm[(((j - RB) * TILES + tile) * 2) * (WARPS * 32) + threadIdx.x] = a;
          wsm[(((j - RB) * TILES + tile) * 2 + 1) * (WARPS * 32) + threadIdx.x] = b;
        }
      }
  }

  __device__ __forceinline__ void multiply(float (&acc)[TILES][4], const uint4 (&v)[RB + SB], const uint4* wsm) const {
    float odd[TILES][4];  // second accumulator: halves the chain of dependent MMAs
#pragma unroll
    for (int tile = 0; tile < TILES; ++tile)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[tile][i] = odd[tile][i] = 0.0f;
#pragma unroll
    for (int j = 0; j < RB + SB; ++j)
#pragma unroll
      for (int tile = 0; tile < TILES; ++tile) {
        uint4 a, b;
        if (j < RB) {
          a = lo[j < RB ? j : 0][tile];
          b = hi[j < RB ? j : 0][tile];
        } else {
          a = wsm[(((j - RB) * TILES + tile) * 2) * (WARPS * 32) + threadIdx.x];
          b = wsm[(((j - RB) * TILES + tile) * 2 + 1) * (WARPS * 32) + threadIdx.x];
        }
        mma_16816(acc[tile], a.x, b.x, a.y, b.y, v[j].x, v[j].y);
        mma_16816(TILES > 2 ? acc[tile] : odd[tile], a.z, b.z, a.w, b.w, v[j].z, v[j].w);
      }
    if (TILES <= 2) {
#pragma unroll
      for (int tile = 0; tile < TILES; ++tile)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[tile][i] += odd[tile][i];
    }
  }
};

__device__ __forceinline__ bool written(const uint4& v) {
  return v.x != kEmpty && v.y != kEmpty && v.z != kEmpty && v.w != kEmpty;
}

// Waits until the lane's columns of the vector at `p` (row start + 8q) have been written and returns them; false when
// the wait ran out.  `vec`: 16-byte aligned rows; otherwise element by element.  KEEP: a round loads only what was not
// ready in the round before.  The forward pass needs that: every CTA polls the whole vector, and the polls themselves
// delay the stores they wait for (H = 1024, 128 CTAs: 2.89 us per step without, 2.33 with it).  In the backward pass a
// CTA polls a quarter, and the plain form is the faster one (2.06 against 2.12 us).
template <int WARPS, bool KEEP, int NB>
__device__ __forceinline__ bool poll_vector(uint4 (&v)[NB], const elem_t* p, bool row_ok, int H, int vec) {
  const int warp = threadIdx.x >> 5, q = threadIdx.x & 3;
  for (unsigned spins = 0;; ++spins) {
    bool ready = true;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const int kb = (warp + WARPS * j) * 32;
      if (!KEEP || spins == 0) v[j] = make_uint4(0, 0, 0, 0);
      if (row_ok && kb + q * 8 < H) {
        if (vec) {
          if (!KEEP || spins == 0 || !written(v[j])) v[j] = ld_relaxed_v4(p + kb);
        } else {
          uint32_t e[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            e[i] = ld_relaxed_u16(p + kb + i);
            ready = ready && e[i] != 0xffffu;
          }
          v[j] = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < NB; ++j)
      ready = ready && written(v[j]);
    if (__all_sync(0xffffffffu, ready)) return true;
    if (spins > kSpinLimit) return false;
  }
}

// Publishes the values of two neighbouring units (lanes 4 apart; `writer` lanes hold the even one) as one word.
__device__ __forceinline__ void publish_pair(elem_t* p, float value, bool even_unit, bool on, int vec) {
  const elem_t e = f2e(value);
  uint32_t bits = *reinterpret_cast<const uint16_t*>(&e);
  if (bits == 0xffffu) bits = 0x7fffu;  // NaN stays NaN
  const uint32_t other = __shfl_xor_sync(0xffffffffu, bits, 4);
  if (!on) return;
  if (!vec) {
    st_relaxed_u16(p, bits);
  } else if (even_unit) {
    st_relaxed_u32(p, bits | other << 16);
  }
}

// -------------------------------------------------------------------------------------------------
// forward
// -------------------------------------------------------------------------------------------------
// U = 8·UT units per CTA, 8·UT warps, H <= 32·8·UT·(RB + SB), P groups of 8 batch rows per CTA.
template <int UT, int SB>
constexpr size_t fwd_smem() {
  return (size_t)SB * 2 * UT * 2 * (256 * UT) * 16 + (size_t)2 * (8 * UT) * 8 * (32 * UT + 4) * sizeof(float);
}

template <int UT, int RB, int SB, int P>
__global__ void __launch_bounds__(256 * UT, 1)
lstm_fwd_kernel(float* __restrict__ gates, const elem_t* __restrict__ whh, const float* __restrict__ h0,
                const float* __restrict__ c0, elem_t* y, float* __restrict__ c_all, int* status, int T, int B, int H,
                int per_sample, int b0, int groups, int vec) {
  constexpr int kWarps = 8 * UT, kTiles = 2 * UT, kLd = 32 * UT + 4;  // row pitch: conflict-free both ways
  extern __shared__ uint4 dyn_smem[];
  uint4* wsm = dyn_smem;
  float* part = reinterpret_cast<float*>(dyn_smem + SB * kTiles * 2 * kWarps * 32);  // [2][warp][8 batch][kLd]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  const int unit_ctas = H / (8 * UT);
  const int unit0 = (blockIdx.x % unit_ctas) * 8 * UT, grp = blockIdx.x / unit_ctas;

  // MMA tile = (unit group of 8) * 2 + {i|f, g|o}; rows 0-7 the first gate, 8-15 the second
  Weights<kWarps, kTiles, RB, SB> w;
  w.load([&](int tile, int r) { return whh + ((long long)((tile & 1) * 2 + (r >> 3)) * H + unit0 + (tile >> 1) * 8 + (r & 7)) * H; },
         H, wsm);

  // this thread's gate value: batch row ob of a group, unit `unit`, gate q (a quad of lanes owns one unit and row)
  const int ob = warp / UT, unit = unit0 + (warp % UT) * 8 + g;
  const int prow = (warp % UT) * 32 + q * 8 + g;  // its row among the CTA's gate rows
  float c[P], xg[P];
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const int row = b0 + 8 * (p * groups + grp) + ob;
    c[p] = xg[p] = 0.0f;
    if (row < B) {
      // initial state: one learned vector broadcast over the batch, or (per_sample) a (B, H) state carried over
      c[p] = c0[per_sample ? (long long)row * H + unit : unit];
      xg[p] = gates[(long long)row * 4 * H + (long long)q * H + unit];
    }
  }

  int par = 0;
  for (int t = 0; t < T; ++t) {
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int row0 = b0 + 8 * (p * groups + grp);
      if (row0 >= B) continue;  // the same for the whole block
      uint4 v[RB + SB];
      int bad = 0;
      {
        const int row = row0 + g;  // the MMA's batch column of this lane
        if (t > 0) {
          bad = !poll_vector<kWarps, true>(v, y + ((long long)(t - 1) * B + row) * H + q * 8, row < B, H, vec);
        } else {
#pragma unroll
          for (int j = 0; j < RB + SB; ++j) {
            const int k = (warp + kWarps * j) * 32 + q * 8;
            elem2_t e[4] = {ff2e2(0, 0), ff2e2(0, 0), ff2e2(0, 0), ff2e2(0, 0)};
            if (row < B && k < H) {
              const float* hp = h0 + (per_sample ? (long long)row * H : 0) + k;
#pragma unroll
              for (int i = 0; i < 4; ++i) e[i] = ff2e2(hp[2 * i], hp[2 * i + 1]);
            }
            const uint32_t* eb = reinterpret_cast<const uint32_t*>(e);
            v[j] = make_uint4(eb[0], eb[1], eb[2], eb[3]);
          }
        }
      }
      float acc[kTiles][4];
      w.multiply(acc, v, wsm);
      float* pp = part + (par * kWarps + warp) * 8 * kLd;
#pragma unroll
      for (int tile = 0; tile < kTiles; ++tile) {
        pp[(2 * q) * kLd + tile * 16 + g] = acc[tile][0];
        pp[(2 * q + 1) * kLd + tile * 16 + g] = acc[tile][1];
        pp[(2 * q) * kLd + tile * 16 + g + 8] = acc[tile][2];
        pp[(2 * q + 1) * kLd + tile * 16 + g + 8] = acc[tile][3];
      }
      if (__syncthreads_or(bad)) {  // a wait ran out: the whole block leaves at the same step
        if (threadIdx.x == 0) atomicExch(status, LSTM_ERR_EXCHANGE_TIMEOUT);
        return;
      }
      float s0 = 0.0f, s1 = 0.0f;
      const float* ps = part + (par * kWarps * 8 + ob) * kLd + prow;
#pragma unroll
      for (int i = 0; i < kWarps; i += 2) {
        s0 += ps[i * 8 * kLd];
        s1 += ps[(i + 1) * 8 * kLd];
      }
      par ^= 1;  // the next barrier separates these reads from the writes of the step after the next
      const float pre = (s0 + s1) + xg[p];
      const float a = q == 2 ? tanhf(pre) : sigmoid_f(pre);
      const float ig = __shfl_sync(0xffffffffu, a, lane & ~3), fg = __shfl_sync(0xffffffffu, a, (lane & ~3) + 1);
      const float gg = __shfl_sync(0xffffffffu, a, (lane & ~3) + 2), og = __shfl_sync(0xffffffffu, a, (lane & ~3) + 3);
      c[p] = fg * c[p] + ig * gg;
      const float h = og * tanhf(c[p]);
      const int row = row0 + ob;
      const long long at = (long long)t * B + row;
      publish_pair(y + at * H + unit, h, (g & 1) == 0, row < B && q == 0, vec);
      if (row < B) {
        gates[at * 4 * H + (long long)q * H + unit] = a;
        if (q == 0) c_all[at * H + unit] = c[p];
        if (t + 1 < T) xg[p] = gates[(at + B) * 4 * H + (long long)q * H + unit];  // needed after the next exchange
      }
    }
  }
}

// -------------------------------------------------------------------------------------------------
// backward
// -------------------------------------------------------------------------------------------------
// [2][source rank][warp][8·UT units][8 batch] floats; the pitch of a source keeps the four lanes of a quad, which
// read from the four sources, on different banks.
template <int UT>
__host__ __device__ constexpr int bwd_src_pitch() { return 8 * UT * UT * 64 + 2; }
template <int UT, int SB>
constexpr size_t bwd_smem() {
  return (size_t)SB * 2 * UT * 2 * (256 * UT) * 16 + (size_t)2 * kCluster * bwd_src_pitch<UT>() * sizeof(float) + 16;
}

__device__ __forceinline__ uint32_t map_to_rank(const void* p, int rank) {
  uint32_t local = (uint32_t)__cvta_generic_to_shared(p), remote;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  return remote;
}
__device__ __forceinline__ void st_cluster_v2(uint32_t addr, float a, float b) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1,%2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void st_cluster_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int UT, int RB, int SB, int P>
__global__ void __launch_bounds__(256 * UT, 1)
lstm_bwd_kernel(const float* __restrict__ gates, const float* __restrict__ c_all, const float* __restrict__ c0,
                const elem_t* __restrict__ dy, const elem_t* __restrict__ whh_t, elem_t* dgates, float* __restrict__ dh0,
                float* __restrict__ dc0, const float* __restrict__ dh_last, const float* __restrict__ dc_last,
                int* status, int T, int B, int H, int per_sample, int b0, int groups, int vec) {
  constexpr int kWarps = 8 * UT, kTiles = 2 * UT, kSrc = bwd_src_pitch<UT>();
  extern __shared__ uint4 dyn_smem[];
  uint4* wsm = dyn_smem;
  float* inbox = reinterpret_cast<float*>(dyn_smem + SB * kTiles * 2 * kWarps * 32);
  uint32_t* gave_up = reinterpret_cast<uint32_t*>(inbox + 2 * kCluster * kSrc);  // [2]: a wait of the cluster ran out
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  const int rank = blockIdx.x % kCluster, K = 4 * H;
  const int unit_clusters = (H + kCluster * 8 * UT - 1) / (kCluster * 8 * UT);
  const int cluster = blockIdx.x / kCluster;
  const int cunit0 = (cluster % unit_clusters) * kCluster * 8 * UT, grp = cluster / unit_clusters;
  if (threadIdx.x < 2) gave_up[threadIdx.x] = 0;

  // rows: the cluster's 32·UT units in order; columns: gate `rank`
  Weights<kWarps, kTiles, RB, SB> w;
  w.load([&](int tile, int r) {
    const int u = cunit0 + tile * 16 + r;
    return u < H ? whh_t + (long long)u * K + (long long)rank * H : nullptr;
  }, H, wsm);
  uint32_t box[kCluster], flag[kCluster];
#pragma unroll
  for (int r = 0; r < kCluster; ++r) {
    box[r] = map_to_rank(inbox + rank * kSrc + warp * UT * 64 + g * 8 + 2 * q, r);
    flag[r] = map_to_rank(gave_up, r);
  }

  // this thread's value: batch row ob of a group, unit `unit`, gate q (a quad of lanes owns one unit and row)
  const int ob = warp / UT, ug = warp % UT, unit = cunit0 + rank * 8 * UT + ug * 8 + g;
  float dc[P] = {}, n_a[P] = {}, n_ct[P] = {}, n_cp[P] = {}, n_dy[P] = {};

  auto fetch = [&](int p, int t, int row, float ct) {  // point-wise inputs of step t
    const long long at = (long long)t * B + row;
    n_a[p] = gates[at * K + (long long)q * H + unit];
    n_ct[p] = ct;
    n_cp[p] = t > 0 ? c_all[(at - B) * H + unit] : c0[per_sample ? (long long)row * H + unit : unit];
    n_dy[p] = e2f(dy[at * H + unit]);
  };
  // gate gradients of step t from dh, published as dGates[t]
  auto pointwise = [&](int p, int t, int row, float dh_in) {
    const float a = n_a[p];
    const float ig = __shfl_sync(0xffffffffu, a, lane & ~3), fg = __shfl_sync(0xffffffffu, a, (lane & ~3) + 1);
    const float gg = __shfl_sync(0xffffffffu, a, (lane & ~3) + 2), og = __shfl_sync(0xffffffffu, a, (lane & ~3) + 3);
    const float dh = n_dy[p] + dh_in;
    const float tc = tanhf(n_ct[p]);
    const float dcv = dh * og * (1.0f - tc * tc) + dc[p];
    float d = dcv * gg * ig * (1.0f - ig);
    if (q == 1) d = dcv * n_cp[p] * fg * (1.0f - fg);
    if (q == 2) d = dcv * ig * (1.0f - gg * gg);
    if (q == 3) d = dh * tc * og * (1.0f - og);
    dc[p] = dcv * fg;
    const bool on = row < B && unit < H;
    publish_pair(dgates + ((long long)t * B + row) * K + (long long)q * H + unit, d, (g & 1) == 0, on, vec);
    if (on && t > 0) fetch(p, t - 1, row, n_cp[p]);
  };

  cluster_barrier();  // the partners' shared memory exists and their flags are clear
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const int row = b0 + 8 * (p * groups + grp) + ob;
    const bool on = row < B && unit < H;
    float dh = 0.0f;
    if (on) {
      if (dh_last != nullptr) dh = dh_last[(long long)row * H + unit];
      if (dc_last != nullptr) dc[p] = dc_last[(long long)row * H + unit];
      fetch(p, T - 1, row, c_all[((long long)(T - 1) * B + row) * H + unit]);
    }
    pointwise(p, T - 1, row, dh);
  }

  int par = 0;
  for (int t = T - 1; t >= 0; --t) {
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int row0 = b0 + 8 * (p * groups + grp);
      if (row0 >= B) continue;  // the same for the whole cluster
      // partial dh_{t-1}[b, unit] = sum over the columns of gate `rank` of dGates[t][b, k] * W_hh[k, unit]
      uint4 v[RB + SB];
      if (!poll_vector<kWarps, false>(v, dgates + ((long long)t * B + row0 + g) * K + (long long)rank * H + q * 8, row0 + g < B, H, vec)) {
#pragma unroll
        for (int r = 0; r < kCluster; ++r) st_cluster_u32(flag[r] + par * 4, 1);
      }
      float acc[kTiles][4];
      w.multiply(acc, v, wsm);
#pragma unroll
      for (int half = 0; half < 2 * kTiles; ++half) {  // 8 units each: the ones of rank half / UT, group half % UT
        const uint32_t at = box[half / UT] + (par * kCluster * kSrc + (half % UT) * 64) * 4;
        st_cluster_v2(at, acc[half >> 1][(half & 1) * 2], acc[half >> 1][(half & 1) * 2 + 1]);
      }
      cluster_barrier();
      if (reinterpret_cast<volatile uint32_t*>(gave_up)[par]) {  // written before the barrier, for all four alike
        if (threadIdx.x == 0) atomicExch(status, LSTM_ERR_EXCHANGE_TIMEOUT);
        return;
      }
      float s0 = 0.0f, s1 = 0.0f;
      const float* ps = inbox + (par * kCluster + q) * kSrc + ug * 64 + g * 8 + ob;
#pragma unroll
      for (int i = 0; i < kWarps; i += 2) {
        s0 += ps[i * UT * 64];
        s1 += ps[(i + 1) * UT * 64];
      }
      par ^= 1;  // the next barrier separates these reads from the writes of the step after the next
      float dh = s0 + s1;
      dh += __shfl_xor_sync(0xffffffffu, dh, 1);
      dh += __shfl_xor_sync(0xffffffffu, dh, 2);
      const int row = row0 + ob;
      if (t > 0) {
        pointwise(p, t - 1, row, dh);
      } else if (row < B && unit < H && q == 0) {
        dh0[(long long)row * H + unit] = dh;
        dc0[(long long)row * H + unit] = dc[p];
      }
    }
  }
}

// -------------------------------------------------------------------------------------------------
// launch
// -------------------------------------------------------------------------------------------------
// All blocks of a grid wait for one another: cooperative launches, which the driver refuses when they do not fit.
template <typename K>
int coop_launch(K kernel, int grid, int threads, int cluster, void** args, size_t smem, cudaStream_t stream) {
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return 5;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelExC(&cfg, (const void*)kernel, args);
  if (e == cudaSuccess) return 0;
  cudaGetLastError();
  return e == cudaErrorCooperativeLaunchTooLarge ? 1 : 5;
}

// How a launch covers `rows` (<= 32) batch rows at hidden size H.
// 16 units per CTA (half the CTAs of a group of 8 rows, so half the pollers, and the machine holds two groups at
// H = 1024, four at 512) against 8 units (less work in each CTA), 8 rows:
//   H = 1024 forward   1.88 us per step with 16 units, 2.33 with 8: fewer pollers of each line win;
//   H = 1024 backward  2.85 us with 16 units, 2.06 with 8: polls are a quarter already, the smaller share wins;
//   H <= 512           8 units while there is one group; more groups fit beside one another with 16 (H > 256).
// Above 1024 the weights need 16 units per CTA on all SMs.  What does not fit side by side takes turns.
struct Shape {
  bool wide;   // 16 units per CTA instead of 8
  int groups;  // groups of 8 rows on different CTAs
  int turns;   // groups of 8 rows per CTA (1, 2 or 4)
};
Shape lstm_shape(int rows, int H, bool forward) {
  const int sub = (rows + 7) / 8;
  Shape s;
  s.wide = H > 1024 || (H > 256 && sub > 1) || (H > 512 && forward);
  const int fit = H <= 512 ? 4 : H <= 1024 ? 2 : 1;
  s.groups = sub < fit ? sub : fit;
  const int turns = (sub + s.groups - 1) / s.groups;
  s.turns = turns > 2 ? 4 : turns;
  return s;
}

// SIDE: 0 forward, 1 backward.
template <int SIDE, int UT, int RB, int SB, int P>
int launch_one(int H, int groups, void** args, cudaStream_t s) {
  if constexpr (SIDE == 0)
    return coop_launch(lstm_fwd_kernel<UT, RB, SB, P>, H / (8 * UT) * groups, 256 * UT, 1, args, fwd_smem<UT, SB>(), s);
  else
    return coop_launch(lstm_bwd_kernel<UT, RB, SB, P>, (H + kCluster * 8 * UT - 1) / (kCluster * 8 * UT) * kCluster * groups,
                       256 * UT, kCluster, args, bwd_smem<UT, SB>(), s);
}

template <int SIDE>
int launch_shape(const Shape& sh, int H, void** args, cudaStream_t s) {
  if (!sh.wide) {
    if (H <= 256) return launch_one<SIDE, 1, 1, 0, 1>(H, sh.groups, args, s);
    if (H <= 512) return launch_one<SIDE, 1, 2, 0, 1>(H, sh.groups, args, s);
    if constexpr (SIDE == 1) return launch_one<SIDE, 1, 4, 0, 1>(H, sh.groups, args, s);
  }
  if (H <= 512) return launch_one<SIDE, 2, 1, 0, 1>(H, sh.groups, args, s);
  if (H <= 1024) {
    if (sh.turns == 1) return launch_one<SIDE, 2, 2, 0, 1>(H, sh.groups, args, s);
    return launch_one<SIDE, 2, 2, 0, 2>(H, sh.groups, args, s);
  }
  if (sh.turns == 1) return launch_one<SIDE, 2, 2, 2, 1>(H, sh.groups, args, s);
  if (sh.turns == 2) return launch_one<SIDE, 2, 2, 2, 2>(H, sh.groups, args, s);
  return launch_one<SIDE, 2, 2, 2, 4>(H, sh.groups, args, s);
}

}  // namespace

extern "C" {

// Largest hidden size the persistent kernels accept.
int fbam_lstm_persistent_max_hidden() { return 2048; }

// gates: (T, B, 4H) fp32, pre-activations incl. bias on entry, activated gates on exit.
// hbuf and counter: ignored, may be null (y itself is what the CTAs exchange; the arguments stay for callers of the C
// interface).  whh: 4-byte aligned.
int fbam_lstm_fwd_ex(float* gates, const void* whh, const float* h0, const float* c0, void* y, float* c_all,
                     void* hbuf, unsigned* counter, int* status, int T, int B, int H, int per_sample, void* stream) {
  (void)hbuf;
  (void)counter;
  if (B < 1 || H < 16 || H % 16 != 0 || H > 2048 || T < 1) return 1;
  if (reinterpret_cast<uintptr_t>(whh) % 4 != 0) return 2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const size_t exchanged = (size_t)(T - 1) * B * H * sizeof(elem_t);  // nobody reads the last step's y
  if (exchanged != 0 && cudaMemsetAsync(y, 0xff, exchanged, s) != cudaSuccess) return 5;
  int vec = reinterpret_cast<uintptr_t>(y) % 16 == 0;
  for (int b0 = 0; b0 < B; b0 += kLaunchRows) {
    Shape sh = lstm_shape(B - b0 < kLaunchRows ? B - b0 : kLaunchRows, H, true);
    void* args[] = {&gates, &whh, &h0, &c0, &y, &c_all, &status, &T, &B, &H, &per_sample, &b0, &sh.groups, &vec};
    const int rc = launch_shape<0>(sh, H, args, s);
    if (rc != 0) return rc;
  }
  return 0;
}

// h0 / c0 are (H) vectors broadcast over the batch.
int fbam_lstm_fwd(float* gates, const void* whh, const float* h0, const float* c0, void* y, float* c_all,
                  void* hbuf, unsigned* counter, int* status, int T, int B, int H, void* stream) {
  return fbam_lstm_fwd_ex(gates, whh, h0, c0, y, c_all, hbuf, counter, status, T, B, H, 0, stream);
}

// whh_t: (H, 4H) bf16 = W_hh transposed, 4-byte aligned.  counter: ignored, may be null.  dgates: (T, B, 4H) bf16 out.  dh0/dc0: (B, H) fp32 out.
int fbam_lstm_bwd_ex(const float* gates, const float* c_all, const float* c0, const void* dy, const void* whh_t,
                     void* dgates, float* dh0, float* dc0, const float* dh_last, const float* dc_last,
                     unsigned* counter, int* status, int T, int B, int H, int per_sample, void* stream) {
  (void)counter;
  if (B < 1 || H < 16 || H % 16 != 0 || H > 2048 || T < 1) return 1;
  if (reinterpret_cast<uintptr_t>(whh_t) % 4 != 0) return 2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(dgates, 0xff, (size_t)T * B * 4 * H * sizeof(elem_t), s) != cudaSuccess) return 5;
  int vec = reinterpret_cast<uintptr_t>(dgates) % 16 == 0;
  for (int b0 = 0; b0 < B; b0 += kLaunchRows) {
    Shape sh = lstm_shape(B - b0 < kLaunchRows ? B - b0 : kLaunchRows, H, false);
    void* args[] = {&gates, &c_all, &c0, &dy, &whh_t, &dgates, &dh0, &dc0, &dh_last, &dc_last, &status,
                    &T, &B, &H, &per_sample, &b0, &sh.groups, &vec};
    const int rc = launch_shape<1>(sh, H, args, s);
    if (rc != 0) return rc;
  }
  return 0;
}

int fbam_lstm_bwd(const float* gates, const float* c_all, const float* c0, const void* dy, const void* whh_t,
                  void* dgates, float* dh0, float* dc0, const float* dh_last, const float* dc_last, unsigned* counter,
                  int* status, int T, int B, int H, void* stream) {
  return fbam_lstm_bwd_ex(gates, c_all, c0, dy, whh_t, dgates, dh0, dc0, dh_last, dc_last, counter, status, T, B, H, 0,
                          stream);
}

}  // extern "C"

// -------------------------------------------------------------------------------------------------
// Forward entry point that takes no scratch from the caller and allocates none (see lstm_noalloc.h for who needs it
// and the contract).
// -------------------------------------------------------------------------------------------------
#include "lstm_noalloc.h"

extern "C" {

int fbam_lstm_fwd_noalloc_max_hidden(void) { return FBAM_LSTM_NOALLOC_MAX_HIDDEN; }

const char* fbam_lstm_fwd_noalloc_strerror(int code) {
  switch (code) {
    case 0: return "ok";
    case 1: return "unsupported shape: need 1 <= B <= 8, H a multiple of 16, T >= 1";
    case 2: return "recurrent weight not 4-byte aligned";
    case 5: return "kernel launch failed";
    case FBAM_LSTM_NOALLOC_ERR_TOO_LARGE:
      return "hidden size exceeds FBAM_LSTM_NOALLOC_MAX_HIDDEN (1024): use fbam_lstm_fwd instead";
    default: return "unknown error";
  }
}

int fbam_lstm_fwd_noalloc(float* gates, const void* whh, const float* h0, const float* c0, void* y, float* c_all,
                          int* status, int T, int B, int H, void* stream) {
  if (H > FBAM_LSTM_NOALLOC_MAX_HIDDEN) return FBAM_LSTM_NOALLOC_ERR_TOO_LARGE;
  if (B < 1 || B > 8 || H < 16 || H % 16 != 0 || T < 1) return 1;
  return fbam_lstm_fwd_ex(gates, whh, h0, c0, y, c_all, nullptr, nullptr, status, T, B, H, 0, stream);
}

}  // extern "C"
