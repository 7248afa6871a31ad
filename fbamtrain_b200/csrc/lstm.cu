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
//  * Polls start when the vector can be there and not before (`hold`): polls of lines that are being written delay the
//    stores they wait for.  Reading 16 KB that nobody writes takes every CTA of a full machine 540 to 680 cycles, whether
//    they read the same lines or not; copies of the vector for different readers only cost more stores.
//  * All groups of 8 batch rows of a CTA go through a step together: the chain of latencies is paid once, not once per
//    group.  Groups go to different CTAs while the machine has room.
//
// Forward: CTA j owns 8·UT hidden units (32·UT gate rows of W_hh).  A quad of lanes owns one (unit, batch row), one lane
// per gate, and exchanges the gates by shuffles.  The buffer of gate pre-activations is overwritten in place with the
// activated gates, which is exactly what the backward pass needs.
// Backward (BPTT): a cluster of four CTAs owns 32·UT units; CTA r of the cluster holds the columns of gate r of W_hhᵀ,
// reads gate r of dGates[t] only (a quarter of what a CTA without partners would have to read), adds its warps' partial
// sums of dh_{t-1} and sends them to the CTA that owns the unit: st.async on an mbarrier there, 267 cycles one way, where
// an idle cluster barrier takes 400 and one behind the stores of unsummed partials took about 1000.  One thread owns one
// (unit, batch row) with its four gates, and what does not depend on dh is computed while the sums are on their way.
//
// Measured on a B200, bf16, us per step over 1024 steps, before (polls at once, IEEE gate functions, groups of rows in turn, cluster
// barrier) -> in this form:
//   H 1024, batch 8:    forward 1.82 -> 1.52, backward 2.06 -> 1.75
//   H 2048, batch 4:    forward 3.09 -> 2.50, backward 3.72 -> 2.71
//   H  256, batch 8:    forward 1.02 -> 0.94, backward 1.65 -> 1.27
//   H  512, batch 32:   forward 1.97 -> 1.47, backward 2.76 -> 1.72
//   H 1024, batch 32:   forward 3.43 -> 2.79, backward 6.22 -> 2.99
//   H 2048, batch 32:   forward 12.9 -> 11.4, backward 16.1 -> 9.8
// (At H = 1024 a forward cluster that divides K, with partial sums sent as in the backward pass, takes 1.75 us at batch 8,
// 1.50 without: its second hop costs more than the smaller share of the vector gives.)
//
// The reference runs the recurrence as one GEMM launch plus a point-wise cell kernel per time step (reference:
// kernel_gen/kernel_gen/kernels/lstm_cell.py:6-144, kernels/lstm_cell_bwd.py:6-273 for the cell arithmetic and the
// recompute / backward point-wise kernels; tensorlib/src/streaming_lstm.cpp and streaming_lstm_bwd.cpp for the loop
// around them); gate order i, f, g, o, fp32 gates and cell state as there.
#include "elem16.cuh"
#include <cuda_runtime.h>
#include <stdint.h>

namespace {

constexpr unsigned kSpinLimit = 1u << 22;  // polls of at least an L2 round trip each: seconds
constexpr unsigned kTestLimit = 1u << 26;  // tests of a barrier in shared memory, some tens of cycles each: seconds
constexpr uint32_t kEmpty = 0xffffffffu;   // a word of the exchange buffer that has not been written yet
constexpr int kCluster = 4;                // CTAs of a cluster
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

// -------------------------------------------------------------------------------------------------
// gate functions
// -------------------------------------------------------------------------------------------------
// One path through the hardware's 2^x and 1/x for both functions, no branch: sigmoid(x) = 1 / (1 + e^-x), tanh(|x|) =
// 1 - 2 / (1 + e^2|x|), and x + x³·p(x²) where that would cancel (p: a fit of the least largest relative error; with these
// coefficients 4.8e-9 on |x| < 0.9).  Errors against 64 bits, relative, largest | rms, of 1 / (1 + __expf(-x)) and tanhf
// -> of these:
//   sigmoid  [-8, 8] 5.0e-7 | 9.7e-8 -> 2.2e-7 | 4.1e-8   [-1, 1] 1.6e-7 | 4.4e-8 -> 1.7e-7 | 3.5e-8
//   tanh     [-8, 8] 1.9e-7 | 2.6e-8 -> 1.1e-7 | 2.0e-8   [-1, 1] 2.0e-7 | 5.6e-8 -> 1.1e-7 | 2.8e-8
// (2 / (1 + e^-2x) - 1 instead is off by up to 3.7e-7 where x is around 1: the rounding of a value near one counts twice.)
// us per forward step with an IEEE division | uncorrected | as here: H = 1024, 8 rows 1.56 | 1.52 | 1.54, 32 rows 2.86 |
// 2.74 | 2.80, H = 2048, 8 rows 2.98 | 2.81 | 2.84; with tanhf too, which a quad goes through after the sigmoids, the
// gates of a step take 743 cycles instead of some 350.
__device__ __forceinline__ float ex2_f(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_f(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// 1 / (1 + 2^(k·x)) for k = ±log2 e or twice that, as the nearest float.  Three roundings are made good where the result is
// a normal number: that of the exponent, by its error-free product (Dekker; k·x = hi + lo, and what k lacks) and 2^lo = 1 +
// lo·ln 2; that of the sum, by the part of the smaller addend that it dropped (Dekker's fast two-sum); that of the
// reciprocal, by one step of Newton's iteration.
__device__ __forceinline__ float logistic(float x, float k) {
  const float hi = k * x;
  const bool normal = fabsf(hi) < 100.0f;  // false for infinities and NaN, which the plain terms carry through
  const float e0 = ex2_f(hi), lo = fmaf(hi, 1.335e-8f, fmaf(k, x, -hi));
  const float e = normal ? fmaf(e0, lo * 0.69314718f, e0) : e0;
  const float d = 1.0f + e, r = rcp_f(d), dropped = fminf(e, 1.0f) - (d - fmaxf(e, 1.0f));
  return normal ? fmaf(r, fmaf(-dropped, r, fmaf(-d, r, 1.0f)), r) : r;
}
// tanh(x), given 1 / (1 + e^2|x|).
__device__ __forceinline__ float tanh_from(float x, float r) {
  const float s = x * x;
  float p = fmaf(-0.0004554584447760135f, s, 0.0025826634373515844f);
  p = fmaf(p, s, -0.008264538832008839f);
  p = fmaf(p, s, 0.021663539111614227f);
  p = fmaf(p, s, -0.053929299116134644f);
  p = fmaf(p, s, 0.13332977890968323f);
  p = fmaf(p, s, -0.33333322405815125f);
  float near = fmaf(x * s, p, x);
  asm volatile("" : "+f"(near));  // computed by all lanes: as a branch it cost 0.1 us a step
  return fabsf(x) < 0.9f ? near : copysignf(fmaf(-2.0f, r, 1.0f), x);
}
__device__ __forceinline__ float tanh_f(float x) { return tanh_from(x, rcp_f(1.0f + ex2_f(2.88539008f * fabsf(x)))); }

// -------------------------------------------------------------------------------------------------
// cluster
// -------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t map_to_rank(const void* p, int rank) {
  uint32_t remote;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_address(p)), "r"(rank));
  return remote;
}
// Stores that count towards the transaction bytes of the receiver's barrier.
__device__ __forceinline__ void st_async_v4(uint32_t at, const float (&v)[4], uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1,%2,%3,%4}, [%5];" ::"r"(at), "f"(v[0]),
               "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(smem_address(bar)) : "memory");
}
// Opens the barrier's phase for `bytes`; what has arrived before this counts.
__device__ __forceinline__ void bar_expect(uint64_t* bar, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_address(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_wait(uint64_t* bar, int parity) {  // false: the wait ran out
  const uint32_t at = smem_address(bar);
  for (unsigned spins = 0; spins < kTestLimit; ++spins) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
        : "=r"(done) : "r"(at), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The last thing a CTA does: its shared memory stays until its partners have stopped sending.  After a wait that ran out
// some of their stores may still be on the way when all have arrived here, hence the pause (the stores take well under a
// microsecond).
__device__ __forceinline__ void leave(bool failed, int* status) {
  if (failed && threadIdx.x == 0) atomicExch(status, LSTM_ERR_EXCHANGE_TIMEOUT);
  cluster_barrier();
  if (failed) {
    const long long t0 = clock64();
    while (clock64() - t0 < 40000) {
    }
  }
}

// -------------------------------------------------------------------------------------------------
// weights
// -------------------------------------------------------------------------------------------------
// 8 consecutive elements of a weight row (4-byte loads: the weights need no more than 4-byte alignment).
__device__ __forceinline__ uint4 load_row8(const elem_t* p, bool on) {
  uint4 v = make_uint4(0, 0, 0, 0);
  if (on) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
    v = make_uint4(w[0], w[1], w[2], w[3]);
  }
  return v;
}

// A warp's MMA tiles (16 rows) times its K blocks (32 columns).  Lane q of a quad owns columns 8q..8q+7 of a block, so
// that a fragment of the vector is one 16-byte piece.  The two k-steps of a block use elements (0,1 | 2,3) and
// (4,5 | 6,7) of those for the two K halves of the MMA, in the weights and in the vector alike, so the order of the sum
// is all that changes.
// The first RB blocks of a warp have their weights in registers, the remaining SB in shared memory.
template <int THREADS, int TILES, int RB, int SB>
struct Weights {
  uint4 lo[RB][TILES], hi[RB][TILES];

  // row(tile, r): pointer to row r of an MMA tile, or nullptr; col(j): first column of block j, or one past the end
  template <typename RowPtr, typename Col>
  __device__ __forceinline__ void load(RowPtr row, Col col, int end, uint4* wsm) {
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int j = 0; j < RB + SB; ++j)
#pragma unroll
      for (int tile = 0; tile < TILES; ++tile) {
        const int k = col(j) + q * 8;
        const elem_t *p = row(tile, g), *p8 = row(tile, g + 8);
        const uint4 a = load_row8(p + k, p != nullptr && k < end), b = load_row8(p8 + k, p8 != nullptr && k < end);
        if (j < RB) {
          lo[j < RB ? j : 0][tile] = a;
          hi[j < RB ? j : 0][tile] = b;
        } else {  // read back by the same thread only: no barrier
          wsm[(((j - RB) * TILES + tile) * 2) * THREADS + threadIdx.x] = a;
          wsm[(((j - RB) * TILES + tile) * 2 + 1) * THREADS + threadIdx.x] = b;
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
        get(j, tile, a, b, wsm);
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

  __device__ __forceinline__ void get(int j, int tile, uint4& a, uint4& b, const uint4* wsm) const {
    if (j < RB) {
      a = lo[j < RB ? j : 0][tile];
      b = hi[j < RB ? j : 0][tile];
    } else {
      a = wsm[(((j - RB) * TILES + tile) * 2) * THREADS + threadIdx.x];
      b = wsm[(((j - RB) * TILES + tile) * 2 + 1) * THREADS + threadIdx.x];
    }
  }
};

// -------------------------------------------------------------------------------------------------
// exchange
// -------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool written(const uint4& v) {
  return v.x != kEmpty && v.y != kEmpty && v.z != kEmpty && v.w != kEmpty;
}

// Loads the lane's N pieces of 8 elements again and again until every one that is `on` has been written (piece i at
// p + i·stride; what is not on reads as zeros); false when the wait ran out.  `vec`: 16-byte aligned pieces; otherwise
// element by element.  KEEP: a round loads only what was not ready in the round before.
template <bool KEEP, int N>
__device__ __forceinline__ bool poll(uint4 (&v)[N], const elem_t* p, long long stride, const bool (&on)[N], int vec) {
  for (unsigned spins = 0;; ++spins) {
    bool ready = true;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (!KEEP || spins == 0) v[i] = make_uint4(0, 0, 0, 0);
      if (!on[i]) continue;
      if (vec) {
        if (!KEEP || spins == 0 || !written(v[i])) v[i] = ld_relaxed_v4(p + i * stride);
      } else {
        uint32_t e[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          e[k] = ld_relaxed_u16(p + i * stride + k);
          ready = ready && e[k] != 0xffffu;
        }
        v[i] = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) ready = ready && written(v[i]);
    if (__all_sync(0xffffffffu, ready)) return true;
    if (spins > kSpinLimit) return false;
  }
}

// The 16 bits under which a value is published.
__device__ __forceinline__ uint32_t publish_bits(float value) {
  const elem_t e = f2e(value);
  const uint32_t bits = *reinterpret_cast<const uint16_t*>(&e);
  return bits == 0xffffu ? 0x7fffu : bits;  // NaN stays NaN
}

// The lines a CTA writes `kAhead` steps later come back into L2 meanwhile: over long sequences the other streams have
// pushed out the 0xFF bytes, and polls and partial writes would wait for DRAM.  H = 1024, batch 8, 1024 steps: forward
// 1.54 -> 1.49, backward 1.90 -> 1.74 us a step; nothing up to H = 512; 1 % slower above 1024, where it is left out.
constexpr int kAhead = 8;
// The step whose lines are fetched when step `published` of T has been, going up (forward) or down (backward); -1: past the
// last one.  The buffers end there, and what lies behind is another tensor's memory or nobody's.
__host__ __device__ constexpr int step_ahead(int published, int T, bool down) {
  return down ? (published >= kAhead ? published - kAhead : -1) : (published + kAhead < T ? published + kAhead : -1);
}
__device__ __forceinline__ void prefetch_l2(const elem_t* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ long long clock_now() {
  long long c;
  asm volatile("mov.u64 %0, %%clock64;" : "=l"(c)::"memory");
  return c;
}
// Waits until `cycles` after `since`.  A vector cannot be there before about 900 cycles after its publication (one store to
// L2 and one load from it), and polls of a line that is being written hold the writer up.  us per step of the forward pass
// at H = 1024, batch 8, with waits of 0, 200, 300 .. 600 cycles: 2.19 2.12 1.71 1.54 1.54 1.58.
__device__ __forceinline__ void hold(long long since, int cycles) {
  while (clock_now() - since < cycles) {
  }
}


// -------------------------------------------------------------------------------------------------
// forward
// -------------------------------------------------------------------------------------------------
// 8·UT warps, 8·UT units per CTA; warp w multiplies K blocks w + 8·UT·j with all 32·UT gate rows of the CTA;
// H <= 256·UT·(RB + SB); P groups of 8 batch rows per CTA go through a step together, TURNS times in turn.
template <int UT, int SB, int P>
constexpr size_t fwd_smem() {
  return (size_t)SB * 2 * UT * 2 * (256 * UT) * 16 + (size_t)2 * P * (8 * UT) * 8 * (32 * UT + 4) * sizeof(float);
}

template <int UT, int RB, int SB, int P, int TURNS>
__global__ void __launch_bounds__(256 * UT, 1)
lstm_fwd_kernel(float* __restrict__ gates, const elem_t* __restrict__ whh, const float* __restrict__ h0,
                const float* __restrict__ c0, elem_t* y, float* __restrict__ c_all, int* status, int T, int B, int H,
                int per_sample, int b0, int groups, int vec, int wait) {
  constexpr int kWarps = 8 * UT, kThreads = 32 * kWarps, kTiles = 2 * UT, kBlocks = RB + SB;
  constexpr int kLd = 32 * UT + 4;  // row pitch of the partial sums: conflict-free both ways
  extern __shared__ uint4 dyn_smem[];
  uint4* wsm = dyn_smem;
  float* part = reinterpret_cast<float*>(dyn_smem + SB * kTiles * 2 * kThreads);  // [2][P][warp][8 batch][kLd]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int unit_ctas = H / (8 * UT);
  const int unit0 = (blockIdx.x % unit_ctas) * 8 * UT, grp = blockIdx.x / unit_ctas;
  const int row_base = b0 + 8 * grp, row_step = 8 * groups;  // first row of group p: row_base + p·row_step

  // MMA tile = (unit group of 8) * 2 + {i|f, g|o}; rows 0-7 the first gate, 8-15 the second
  Weights<kThreads, kTiles, RB, SB> w;
  w.load([&](int tile, int r) { return whh + ((long long)((tile & 1) * 2 + (r >> 3)) * H + unit0 + (tile >> 1) * 8 + (r & 7)) * H; },
         [&](int j) { return (warp + kWarps * j) * 32; }, H, wsm);

  // this quad's cells: batch row ob of each group, unit `unit`; a lane has gate q
  const int ob = warp / UT, unit = unit0 + (warp % UT) * 8 + g;
  const int prow = (warp % UT) * 32 + q * 8 + g;  // its row among the CTA's gate rows
  const float act_scale = q == 2 ? 2.88539008f : -1.44269504f;
  const bool writes = q == 0 && (!vec || (g & 1) == 0);
  const long long step = (long long)B * H;
  // Element of y and c_all at the step at hand, group 0 (the lane's gate lies at 4·at + gate_at), and what the lane polls.
  // With weights in shared memory too there is no register to spare and both come from t each time (2.44 against 2.58 us a
  // step with running addresses at H = 2048, batch 4); the other forms are up to 8 % faster with running addresses.
  long long at = (long long)(row_base + ob) * H + unit;
  const int gate_at = q * H - 3 * unit;
  const elem_t* src = y + (long long)(row_base + g) * H + warp * 32 + q * 8;
  float c_of[TURNS][P], xg_of[TURNS][P];
#pragma unroll
  for (int i = 0; i < TURNS * P; ++i) {
    const int row = row_base + i * row_step + ob;
    float &c = c_of[i / P][i % P], &xg = xg_of[i / P][i % P];
    c = xg = 0.0f;
    if (row < B) {
      // initial state: one learned vector broadcast over the batch, or (per_sample) a (B, H) state carried over
      c = c0[per_sample ? (long long)row * H + unit : unit];
      xg = gates[((long long)row * 4 + q) * H + unit];
    }
  }

  bool bad = false;
  long long published = clock_now();
  // One step of P groups from batch row `base` on.
  auto advance = [&](int t, int base, int par, float (&c)[P], float (&xg)[P]) {
    if (t > 0 && TURNS == 1) hold(published, wait);  // another group's turn is longer than any wait
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int row0 = base + p * row_step;
      if (row0 >= B) continue;  // the same for the whole block
      uint4 v[kBlocks];
      bool on[kBlocks];
#pragma unroll
      for (int j = 0; j < kBlocks; ++j) on[j] = row0 + g < B && (warp + kWarps * j) * 32 + q * 8 < H;
      if (t > 0) {
        const elem_t* from = SB > 0 ? y + ((long long)(t - 1) * B + row0 + g) * H + warp * 32 + q * 8 : src + p * row_step * H;
        bad = !poll<true>(v, from, kWarps * 32, on, vec) || bad;
      } else {
#pragma unroll
        for (int j = 0; j < kBlocks; ++j) {
          elem2_t e[4] = {ff2e2(0, 0), ff2e2(0, 0), ff2e2(0, 0), ff2e2(0, 0)};
          if (on[j]) {
            const float* hp = h0 + (per_sample ? (long long)(row0 + g) * H : 0) + (warp + kWarps * j) * 32 + q * 8;
#pragma unroll
            for (int i = 0; i < 4; ++i) e[i] = ff2e2(hp[2 * i], hp[2 * i + 1]);
          }
          const uint32_t* eb = reinterpret_cast<const uint32_t*>(e);
          v[j] = make_uint4(eb[0], eb[1], eb[2], eb[3]);
        }
      }
      float acc[kTiles][4];
      w.multiply(acc, v, wsm);
      float* pp = part + ((par * P + p) * kWarps + warp) * 8 * kLd + g;
#pragma unroll
      for (int tile = 0; tile < kTiles; ++tile) {
        pp[(2 * q) * kLd + tile * 16] = acc[tile][0];
        pp[(2 * q + 1) * kLd + tile * 16] = acc[tile][1];
        pp[(2 * q) * kLd + tile * 16 + 8] = acc[tile][2];
        pp[(2 * q + 1) * kLd + tile * 16 + 8] = acc[tile][3];
      }
    }
    if (__syncthreads_or(bad)) return false;  // a wait ran out: the whole block leaves at the same step
    float a[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      float s0 = 0.0f, s1 = 0.0f;
      const float* ps = part + ((par * P + p) * kWarps * 8 + ob) * kLd + prow;
#pragma unroll
      for (int k = 0; k < kWarps; k += 2) {
        s0 += ps[k * 8 * kLd];
        s1 += ps[(k + 1) * 8 * kLd];
      }
      a[p] = (s0 + s1) + xg[p];
    }
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const float pre = a[p], s = logistic(q == 2 ? fabsf(pre) : pre, act_scale);
      a[p] = q == 2 ? tanh_from(pre, s) : s;
      const float ig = __shfl_sync(0xffffffffu, a[p], lane & ~3), fg = __shfl_sync(0xffffffffu, a[p], (lane & ~3) + 1);
      const float gg = __shfl_sync(0xffffffffu, a[p], (lane & ~3) + 2), og = __shfl_sync(0xffffffffu, a[p], (lane & ~3) + 3);
      c[p] = fg * c[p] + ig * gg;
      const uint32_t bits = publish_bits(og * tanh_f(c[p])), other = __shfl_xor_sync(0xffffffffu, bits, 4);
      const int row = base + p * row_step + ob;
      if (writes && row < B) {
        elem_t* yp = SB > 0 ? y + ((long long)t * B + row) * H + unit : y + at + p * row_step * H;
        if (vec)
          st_relaxed_u32(yp, bits | other << 16);
        else
          st_relaxed_u16(yp, bits);
      }
    }
    published = clock_now();
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int row = base + p * row_step + ob;
      if (row < B) {
        const long long from_t = (long long)t * B + row;
        const long long cell = SB > 0 ? from_t * H + unit : at + p * row_step * H;
        const long long gate = SB > 0 ? (from_t * 4 + q) * H + unit : 4 * cell + gate_at;
        gates[gate] = a[p];
        if (q == 0) c_all[cell] = c[p];
        if (t + 1 < T) xg[p] = gates[gate + 4 * step];  // needed after the next exchange
        if (SB == 0 && writes && step_ahead(t, T, false) >= 0) prefetch_l2(y + cell + kAhead * step);
      }
    }
    if (SB == 0) {
      at += step;
      if (t > 0) src += step;
    }
    return true;
  };
  int turns = 0;
  for (int t = 0; t < T; ++t) {
#pragma unroll
    for (int i = 0; i < TURNS; ++i) {
      const int base = row_base + i * P * row_step;
      if (TURNS > 1 && base >= B) continue;  // the same for the whole block
      // two buffers of partial sums take turns: a barrier lies between the reads of one and its next writes
      if (!advance(t, base, TURNS == 1 ? t & 1 : turns++ & 1, c_of[i], xg_of[i])) {
        if (threadIdx.x == 0) atomicExch(status, LSTM_ERR_EXCHANGE_TIMEOUT);
        return;
      }
    }
  }
}

// -------------------------------------------------------------------------------------------------
// backward
// -------------------------------------------------------------------------------------------------
// Warp w multiplies K blocks w + 8·UT·j of gate `rank` with the rows of all 32·UT units of the cluster.
// H <= 256·UT·(RB + SB); P groups of 8 batch rows per CTA.
//
// The gate gradients belong to cells: 8·UT units x 8 batch rows x P groups of a CTA, one thread each, 8·UT neighbouring
// lanes on one batch row.  H is a multiple of 16, so a CTA's units are all there or none of them is.
struct Cell {
  int p, unit, row;  // group; unit and row within the CTA
};
template <int UT>
__device__ __forceinline__ Cell my_cell() {
  const int rest = threadIdx.x % (64 * UT);
  return {(int)threadIdx.x / (64 * UT), rest % (8 * UT), rest / (8 * UT)};
}

template <int UT, int SB, int P>
constexpr size_t bwd_smem() {
  return (size_t)SB * 2 * UT * 2 * (256 * UT) * 16 + ((size_t)2 * 8 * UT * 256 * UT + (size_t)2 * kCluster * P * 64 * UT) * sizeof(float) +
         2 * P * 8;
}

template <int UT, int RB, int SB, int P>
__global__ void __launch_bounds__(256 * UT, 1)
lstm_bwd_kernel(const float* __restrict__ gates, const float* __restrict__ c_all, const float* __restrict__ c0,
                const elem_t* __restrict__ dy, const elem_t* __restrict__ whh_t, elem_t* dgates, float* __restrict__ dh0,
                float* __restrict__ dc0, const float* __restrict__ dh_last, const float* __restrict__ dc_last,
                int* status, int T, int B, int H, int per_sample, int b0, int groups, int vec, int wait) {
  constexpr int kThreads = 256 * UT, kWarps = 8 * UT, kTiles = 2 * UT, kBlocks = RB + SB, kUnits = 8 * UT, kBox = 64 * UT;
  extern __shared__ uint4 dyn_smem[];
  uint4* wsm = dyn_smem;
  float* part = reinterpret_cast<float*>(wsm + SB * kTiles * 2 * kThreads);     // [2][warp][32·UT units][8 rows]
  // [2][P][source][8·UT units][8 rows]; two boxes take turns from step to step.  A partner fills a box again two steps
  // later, and by then it has been read: the partner's sums of that step need the dGates that this CTA's cells made of it.
  float* inbox = part + 2 * kWarps * kThreads;
  uint64_t* bars = reinterpret_cast<uint64_t*>(inbox + 2 * kCluster * P * kBox);  // [2][P]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int rank = blockIdx.x % kCluster, K = 4 * H;
  const int unit_clusters = (H + kCluster * kUnits - 1) / (kCluster * kUnits);
  const int cluster = blockIdx.x / kCluster;
  const int cunit0 = (cluster % unit_clusters) * kCluster * kUnits, grp = cluster / unit_clusters;
  const int row_base = b0 + 8 * grp, row_step = 8 * groups;

  // rows: the cluster's 32·UT units in order; columns: gate `rank`
  Weights<kThreads, kTiles, RB, SB> w;
  w.load([&](int tile, int r) {
    const int u = cunit0 + tile * 16 + r;
    return u < H ? whh_t + (long long)u * K + (long long)rank * H : nullptr;
  }, [&](int j) { return (warp + kWarps * j) * 32; }, H, wsm);

  // the sums this thread makes: unit threadIdx / 2 of the cluster, four batch rows of a group; they go out as one 16-byte
  // store (every store costs the receiver's barrier an update: 256 of 4 bytes took 200 cycles longer than 64 of 16)
  const int sum_unit = threadIdx.x >> 1, sum_row = (threadIdx.x & 1) * 4, owner = (sum_unit / kUnits) % kCluster;
  const uint32_t box = map_to_rank(inbox + rank * kBox + threadIdx.x * 4 % kBox, owner), box_bar = map_to_rank(bars, owner);
  const bool sum_on = threadIdx.x < 64 * UT && cunit0 + sum_unit < H;

  const Cell cell = my_cell<UT>();
  const int unit = cunit0 + rank * kUnits + cell.unit, row = row_base + cell.p * row_step + cell.row;
  const bool live = cell.p < P && row < B && unit < H;
  const bool warp_live = __any_sync(0xffffffffu, live);
  const bool writes = live && (!vec || (lane & 1) == 0);
  const bool opens = live && threadIdx.x % (64 * UT) == 0;  // opens the phases of its group's barriers
  const int expected = kCluster * kUnits * ((min(8, B - (row_base + cell.p * row_step)) + 3) / 4) * 16;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * P; ++i) bar_init(bars + i);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (opens) {
    bar_expect(bars + cell.p, expected);
    bar_expect(bars + P + cell.p, expected);
  }

  const long long t_step = (long long)B * H;
  const float* gp = gates + ((long long)(T - 1) * B + row) * K + unit;    // point-wise inputs of the step at hand
  const float* cp = c_all + ((long long)(T - 1) * B + row) * H + unit;
  const elem_t* dyp = dy + ((long long)(T - 1) * B + row) * H + unit;
  elem_t* dgp = dgates + ((long long)(T - 1) * B + row) * K + unit;
  float dc = 0.0f, gate[4] = {}, ct = 0.0f, c_prev = 0.0f;  // ct, c_prev: cell state of the step at hand and of the one before
  uint16_t dy_bits = 0;
  auto fetch = [&](int t) {  // moves on to step t, whose cell state is the c_prev of the step before
#pragma unroll
    for (int i = 0; i < 4; ++i) gate[i] = gp[(long long)i * H];
    c_prev = *(t > 0 ? cp - t_step : c0 + (per_sample ? (long long)row * H + unit : unit));
    dy_bits = *reinterpret_cast<const uint16_t*>(dyp);
    gp -= 4 * t_step;
    cp -= t_step;
    dyp -= t_step;
  };
  // What the gate gradients of a step need besides dh: computed while the partial sums are on their way.
  float to_c, to_o, to_i, to_f, to_g;
  auto factors = [&] {
    const float tc = tanh_f(ct);
    to_c = gate[3] * (1.0f - tc * tc);
    to_o = tc * gate[3] * (1.0f - gate[3]);
    to_i = gate[2] * gate[0] * (1.0f - gate[0]);
    to_f = c_prev * gate[1] * (1.0f - gate[1]);
    to_g = gate[0] * (1.0f - gate[2] * gate[2]);
  };
  // gate gradients from dh, published as dGates of the step at hand
  auto pointwise = [&](float dh_in) {
    // the move keeps the conversion here: next to its load it would wait for that load, in front of the next exchange
    uint16_t now;
    asm volatile("mov.u16 %0, %1;" : "=h"(now) : "h"(dy_bits));
    const float dh = e2f(*reinterpret_cast<const elem_t*>(&now)) + dh_in;
    const float dcv = dh * to_c + dc;
    uint32_t bits[4] = {publish_bits(dcv * to_i), publish_bits(dcv * to_f), publish_bits(dcv * to_g), publish_bits(dh * to_o)};
    if (vec) {
#pragma unroll
      for (int i = 0; i < 4; ++i) bits[i] |= __shfl_xor_sync(0xffffffffu, bits[i], 1) << 16;
      if (writes)
#pragma unroll
        for (int i = 0; i < 4; ++i) st_relaxed_u32(dgp + i * H, bits[i]);
    } else if (writes) {
#pragma unroll
      for (int i = 0; i < 4; ++i) st_relaxed_u16(dgp + i * H, bits[i]);
    }
    dc = dcv * gate[1];
    ct = c_prev;
    dgp -= 4 * t_step;
  };

  if (warp_live) {
    float dh = 0.0f;
    if (live) {
      if (dh_last != nullptr) dh = dh_last[(long long)row * H + unit];
      if (dc_last != nullptr) dc = dc_last[(long long)row * H + unit];
      ct = *cp;
      fetch(T - 1);
    }
    factors();
    pointwise(dh);
    if (live && T > 1) fetch(T - 2);
  }
  const elem_t* src = dgates + ((long long)(T - 1) * B + row_base + g) * K + (long long)rank * H + warp * 32 + q * 8;
  bool cols[kBlocks];
#pragma unroll
  for (int j = 0; j < kBlocks; ++j) cols[j] = (warp + kWarps * j) * 32 + q * 8 < H;

  cluster_barrier();  // the partners' barriers exist
  bool bad = false, failed = false;
  int buf = 0;
  long long published = clock_now();
  for (int t = T - 1; t >= 0 && !failed; --t) {
    const int n = T - 1 - t, par = n & 1;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int row0 = row_base + p * row_step;
      if (row0 >= B || failed) continue;  // the same for the whole cluster, and for the whole block
      // partial dh_{t-1}[b, unit] = sum over the columns of gate `rank` of dGates[t][b, k] * W_hh[k, unit]
      uint4 v[kBlocks];
      bool on[kBlocks];
#pragma unroll
      for (int j = 0; j < kBlocks; ++j) on[j] = cols[j] && row0 + g < B;
      if (p == 0) hold(published, wait);
      bad = !poll<false>(v, src + (long long)p * row_step * K, kWarps * 32, on, vec) || bad;
      float acc[kTiles][4];
      w.multiply(acc, v, wsm);
      float* pp = part + (buf * kWarps + warp) * kThreads + g * 8 + 2 * q;
#pragma unroll
      for (int tile = 0; tile < kTiles; ++tile) {
        *reinterpret_cast<float2*>(pp + tile * 128) = make_float2(acc[tile][0], acc[tile][1]);
        *reinterpret_cast<float2*>(pp + tile * 128 + 64) = make_float2(acc[tile][2], acc[tile][3]);
      }
      if (__syncthreads_or(bad)) {  // a wait ran out: the whole block leaves at the same step
        failed = true;
        continue;
      }
      if (sum_on && row0 + sum_row < B) {
        float s[4] = {}, s1[4] = {};
        const float4* ps = reinterpret_cast<const float4*>(part + buf * kWarps * kThreads) + threadIdx.x;
#pragma unroll
        for (int i = 0; i < kWarps; i += 2) {
          const float4 a = ps[i * (kThreads / 4)], b = ps[(i + 1) * (kThreads / 4)];
          const float even[4] = {a.x, a.y, a.z, a.w}, odd[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            s[r] += even[r];
            s1[r] += odd[r];
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] += s1[i];
        st_async_v4(box + ((par * P + p) * kCluster * kBox) * 4, s, box_bar + (par * P + p) * 8);
      }
      buf ^= 1;  // the next barrier separates these reads from the writes after the next ones
    }
    src -= 4 * t_step;
    if (warp_live && !failed) {
      if (t > 0) factors();
      if (!bar_wait(bars + par * P + (cell.p < P ? cell.p : 0), (n >> 1) & 1)) bad = true;
      if (opens) bar_expect(bars + par * P + cell.p, expected);
      float dh = 0.0f;
      if (live) {
        const float* in = inbox + (par * P + cell.p) * kCluster * kBox + cell.unit * 8 + cell.row;
        dh = (in[0] + in[kBox]) + (in[2 * kBox] + in[3 * kBox]);
      }
      if (t > 0) {
        pointwise(dh);
      } else if (live) {
        dh0[(long long)row * H + unit] = dh;
        dc0[(long long)row * H + unit] = dc;
      }
    }
    if (t > 0 && !failed) {
      __syncthreads();  // no warp polls before the CTA has published
      published = clock_now();
      if (live && t > 1) fetch(t - 2);
      const int ahead = step_ahead(t - 1, T, true);  // t - 1 has just been published, and dgp has moved on to t - 2
      if (SB == 0 && writes && ahead >= 0) {
        const elem_t* to = dgp - 4 * (t - 2 - ahead) * t_step;
#pragma unroll
        for (int i = 0; i < 4; ++i) prefetch_l2(to + i * H);
      }
    }
  }
  leave(__syncthreads_or(failed || bad), status);
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

// How a launch covers `rows` (at most 32) batch rows at hidden size H.  us per step, forward | backward:
//   H <= 512, to 16 rows    8 units per CTA: H = 512, 8 rows 1.19 | 1.41; with 16 units 1.47 | 1.57
//   H <= 512, 17 to 32      16 units, so that four groups fit beside one another: H = 512, 32 rows 1.45 | 1.84; with 8 units
//                           and two groups per CTA 2.07 | 2.60
//   H <= 1024, to 8 rows    8 units: 8 rows 1.49 | 1.74; with 16 units 1.65 | 2.15
//   H <= 1024, more         16 units, two groups beside one another, up to two in a CTA: 16 rows 1.75 | 1.91, 32 rows
//                           2.73 | 3.06; with 8 units 2.40 | 2.97 and 4.9 | 5.1
//   above                   16 units on all SMs, groups in a CTA: H = 2048, 8 rows 2.78 | 3.00, 32 rows - | 9.8.  In the
//                           forward pass they take turns: the weights leave no shared memory for their partial sums.
struct Shape {
  bool wide;   // 16 units per CTA instead of 8
  int groups;  // groups of 8 rows on different CTAs
  int shared;  // groups of 8 rows per CTA
  int wait;    // cycles from a CTA's publication to its first poll
};
Shape lstm_shape(int rows, int H, int T, bool forward) {
  const int sub = (rows + 7) / 8;
  Shape s;
  s.wide = H > 1024 || (H > 512 ? sub > 1 : H > 256 && sub > 2);
  const int fit = H <= 256 || (H <= 512 && s.wide) ? 4 : H <= 512 || (H <= 1024 && s.wide) ? 2 : 1;
  s.groups = sub < fit ? sub : fit;
  s.shared = (sub + s.groups - 1) / s.groups;
  // Lowest time per step over waits of 0, 100 .. 1400 cycles; flat around it, except in the backward pass at H = 1024:
  // 8 rows 2.23 us with 400, 1.74 with 800; 3 rows 1.78 and 1.95.
  // Four groups at H <= 512 publish earlier while what a launch reads and writes (22 bytes a unit, row and step) stays in L2:
  // us per step with 250 | 450 cycles, H = 512, 24 rows, 256 steps (69 MB) 1.32 | 1.42, 32 rows (92 MB) 1.67 | 1.44.
  const bool in_l2 = 22ll * rows * H * T < 80000000;
  if (forward)
    s.wait = H <= 256 ? 150 : H <= 512 ? (!s.wide ? 300 : in_l2 ? 250 : 450) : s.shared > 1 ? 300 : 450;
  else
    s.wait = H <= 256 ? 150 : H > 512 && H <= 1024 && rows > 3 && !s.wide ? 800 : 400;
  return s;
}
// Batch rows of one launch.  Above H = 1024 a forward step of four groups in turn takes 12.3 us and one of a group alone
// 2.80, but each launch loads the weights (11 us): a launch per group pays from about 30 steps on (16 steps of 32 rows in
// turn 12.3 us a step, 13.8 in four launches; 256 steps 12.7 and 11.4).
int launch_rows(int H, int T, bool forward) { return forward && H > 1024 && T >= 32 ? 8 : 32; }

// SIDE: 0 forward, 1 backward.
template <int SIDE, int UT, int RB, int SB, int P, int TURNS = 1>
int launch_one(int H, int groups, void** args, cudaStream_t s) {
  if constexpr (SIDE == 0)
    return coop_launch(lstm_fwd_kernel<UT, RB, SB, P, TURNS>, H / (8 * UT) * groups, 256 * UT, 1, args, fwd_smem<UT, SB, P>(), s);
  else
    return coop_launch(lstm_bwd_kernel<UT, RB, SB, P>, (H + kCluster * 8 * UT - 1) / (kCluster * 8 * UT) * kCluster * groups,
                       256 * UT, kCluster, args, bwd_smem<UT, SB, P>(), s);
}

template <int SIDE>
int launch_shape(const Shape& sh, int H, void** args, cudaStream_t s) {
  if (H <= 256) return launch_one<SIDE, 1, 1, 0, 1>(H, sh.groups, args, s);
  if (H <= 512) {
    if (!sh.wide) return launch_one<SIDE, 1, 2, 0, 1>(H, sh.groups, args, s);
    return launch_one<SIDE, 2, 1, 0, 1>(H, sh.groups, args, s);
  }
  if (H <= 1024) {
    if (!sh.wide) return launch_one<SIDE, 1, 4, 0, 1>(H, sh.groups, args, s);
    if (sh.shared == 1) return launch_one<SIDE, 2, 2, 0, 1>(H, sh.groups, args, s);
    return launch_one<SIDE, 2, 2, 0, 2>(H, sh.groups, args, s);
  }
  if (sh.shared == 1) return launch_one<SIDE, 2, 2, 2, 1>(H, sh.groups, args, s);
  constexpr int kTurn2 = SIDE == 0 ? 2 : 1, kTurn4 = SIDE == 0 ? 4 : 1;
  if (sh.shared == 2) return launch_one<SIDE, 2, 2, 2, 2 / kTurn2, kTurn2>(H, sh.groups, args, s);
  return launch_one<SIDE, 2, 2, 2, 4 / kTurn4, kTurn4>(H, sh.groups, args, s);
}

}  // namespace

extern "C" {

// Largest hidden size the persistent kernels accept.
int fbam_lstm_persistent_max_hidden() { return 2048; }

// For tests: which step's lines the kernels fetch behind the publication of a step, or -1.
int fbam_lstm_step_ahead(int published, int T, int down) { return step_ahead(published, T, down != 0); }

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
  for (int b0 = 0, most = launch_rows(H, T, true); b0 < B; b0 += most) {
    Shape sh = lstm_shape(B - b0 < most ? B - b0 : most, H, T, true);
    void* args[] = {&gates, &whh, &h0, &c0, &y, &c_all, &status, &T, &B, &H, &per_sample, &b0, &sh.groups, &vec, &sh.wait};
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
  for (int b0 = 0, most = launch_rows(H, T, false); b0 < B; b0 += most) {
    Shape sh = lstm_shape(B - b0 < most ? B - b0 : most, H, T, false);
    void* args[] = {&gates, &c_all, &c0, &dy, &whh_t, &dgates, &dh0, &dc0, &dh_last, &dc_last, &status,
                    &T, &B, &H, &per_sample, &b0, &sh.groups, &vec, &sh.wait};
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
