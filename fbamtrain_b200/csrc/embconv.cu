// Cell embedding fused with the first convolution of the frame head.
//
// The cell embedding is linear in three small tables (code-point rows, position rows, six colour vectors) and a
// convolution without a normalisation in front of it is linear in its input, so the pre-activation of the first
// convolution is a sum of table look-ups:
//
//   Z[n, p, :] = sum_taps T[cp(n, cell(p, tap))][tap][:]            code points:  T[v][tap] = cp_embed[v] . W[:, tap, :]^T
//              + POS[p][:]                                         positions:    the convolution of the position table
//              + sum_taps sum_c (rgb_c / 255) . CC[tap][c][:]      colours:      CC[tap][c] = colour[c] . W[:, tap, :]^T
//
// and its backward needs only three reductions of dZ: by (code point, tap), over the frames, and colour-weighted.
// The (frames x cells x channels) embedding tensor, the data-gradient convolution into it and its scatter into the
// tables are never computed.  What the reference does with build_cell_embeds + conv2d and their backward kernels
// (kernel_gen/kernel_gen/kernels/build_cell_embeds.py:74-134, build_cell_embeds_bwd.py:6-322,
// src/framehead_model.cpp:126-175, 601-731) is covered here by
//
//   fbam_embconv_fwd_colour  Z = POS + table rows + F . CC; Y = GELU(Z), with the colour features
//                            F[n, p, tap*6 + c] = rgb_c(cell(p, tap)) / 255 (bf16, 64 per pixel) made on the way and
//                            kept for the backward, whose colour term is the product F^T . dZ
//   fbam_embconv_features    F alone, and
//   fbam_embconv_fwd         Z += POS + table rows; Y = GELU(Z): the parts of the above, for tests and measurements
//   fbam_embconv_bwd_reduce  S[v][tap][:] += dZ rows by code point and tap;  D[p][:] += dZ summed over frames
//
// A warp owns one output pixel (32 lanes x 8 channels = a 256-channel block; 4 in the backward) and walks a run of
// consecutive frames.  Terminal frames change little from one frame to the next, and both kernels use that without depending on it:
// the forward kernel keeps the sum of the nine table rows and, when a few of the nine code points changed, subtracts
// the old rows and adds the new ones (it rebuilds the sum from scratch when more than four changed and at the start
// of every run, which also bounds the rounding drift); the backward kernel accumulates dZ in registers per tap
// while that tap's code point stays the same and adds the run to S with vector reductions only when it changes.
// Frames that share nothing cost nine row loads (forward) or nine row reductions (backward) per pixel and frame.
#include "elem16.cuh"
#include <cuda_runtime.h>
#include <stdint.h>

#include "gelu_math.cuh"

namespace {


struct EmbConvGeom {
  int rows, cols;        // cells per frame
  int oh, ow;            // output pixels per frame
  int stride, pad, dil;  // 3x3 filter geometry
};

struct alignas(16) Pack8 { elem2_t h[4]; };
// Cell index (row-major within the frame) that output pixel (oy, ox) reads through filter tap `tap`, or -1 when the
// tap falls into the padding.
__device__ __forceinline__ int tap_cell(const EmbConvGeom& g, int oy, int ox, int tap) {
  const int iy = oy * g.stride + (tap / 3) * g.dil - g.pad;
  const int ix = ox * g.stride + (tap % 3) * g.dil - g.pad;
  if (iy < 0 || iy >= g.rows || ix < 0 || ix >= g.cols) return -1;
  return iy * g.cols + ix;
}

// ------------------------------------------------------------------------------------------------
// colour features: one thread per output pixel writes its 128-byte row
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) embconv_features_kernel(const int* __restrict__ cells, elem_t* __restrict__ feat,
                                                               long long frames, EmbConvGeom g) {
  const int p_out = g.oh * g.ow;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= frames * p_out) return;
  const long long n = idx / p_out;
  const int p = (int)(idx % p_out);
  const int oy = p / g.ow, ox = p % g.ow;
  const long long frame_base = n * (long long)(g.rows * g.cols);
  uint32_t w[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) w[i] = 0u;
#pragma unroll
  for (int t = 0; t < 9; ++t) {
    const int cell = tap_cell(g, oy, ox, t);
    if (cell >= 0) {
      const int* cw = cells + (frame_base + cell) * 3;
      const uint32_t fg = (uint32_t)__ldg(cw + 1), bg = (uint32_t)__ldg(cw + 2);
      const float k = 1.0f / 255.0f;
      const elem2_t a = ff2e2(((fg >> 16) & 255) * k, ((fg >> 8) & 255) * k);
      const elem2_t b = ff2e2((fg & 255) * k, ((bg >> 16) & 255) * k);
      const elem2_t c = ff2e2(((bg >> 8) & 255) * k, (bg & 255) * k);
      w[t * 3 + 0] = *reinterpret_cast<const uint32_t*>(&a);
      w[t * 3 + 1] = *reinterpret_cast<const uint32_t*>(&b);
      w[t * 3 + 2] = *reinterpret_cast<const uint32_t*>(&c);
    }
  }
  uint4* dst = reinterpret_cast<uint4*>(feat + idx * 64);
#pragma unroll
  for (int i = 0; i < 8; ++i) dst[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
}

// ------------------------------------------------------------------------------------------------
// forward: Z = [colour term or Z] + POS + sum of table rows, Y = GELU(Z)
// ------------------------------------------------------------------------------------------------
constexpr int kPrefetchBwd = 16;   // frames whose cell words / rows the backward reduction fetches before it uses any
                                   // (8-byte pieces: 128 bytes in flight per lane)

using gelu_math::f2;
using gelu_math::gelu2;

// Eight warps, eight neighbouring pixels, 256 channels; a pass of the loop takes eight frames:
//   1  the nine cells under each of the 64 (pixel, frame) pairs, loaded during the previous pass, become code points
//      and colour features in shared memory;
//   2  each warp lists the table rows by which the sum of its pixel changes from frame to frame, and multiplies the 64
//      feature rows with the colour matrix for 32 of the 256 channels (mma.sync; the matrix waits in shared memory in
//      fragment order, and its columns are permuted so that a lane holds eight neighbouring channels of a row);
//   3  each warp walks the eight frames of its pixel, a lane with eight channels: rows from the list (the next pair
//      of rows is always on its way), plus the colour term, GELU, stores.
// The colour term was a product of its own before (features to memory, a GEMM with K = 64 into Z, Z read back here) and
// the rows were loaded when a change was met, with the warp waiting for each: 1024 frames of 24 x 80 pixels, 256
// channels, took 1195 / 1290 / 1570 / 2630 us with 1 / 5 / 15 / 100 % of the cells changing, 1096 / 1214 without Z kept;
// now 744 / 829 / 1039 / 1774 and 673 / 760.  The 2.2 GB written are 0.34 ms: instructions bound it, 255 a pixel and
// frame at 5 % of the cells changing, at 55 % of the issue rate (256 frames); sixteen warps an SM do as much as twenty-four.
constexpr int kFwdPix = 8;
constexpr int kFwdFrames = 8;
constexpr int kFwdThreads = 32 * kFwdPix;
constexpr int kFwdBlocks = 2;                             // per SM, 128 registers; three with 80 spill: 395 against 385 us
                                                          // for 444 frames of 24 x 80 pixels and 256 channels
constexpr int kFwdRows = kFwdPix * kFwdFrames;            // rows of the colour product
constexpr int kFwdLoads = 3;                              // cells a thread looks at per pass: taps part, part + 4, part + 8
constexpr int kRebuild = 4;                               // more changed taps than this: the sum is built anew
constexpr int kNewPairs = kRebuild + 1;                   // five pairs cover nine rows
constexpr int kMaxPairs = kFwdFrames * kNewPairs + 1;     // one more marks the end

struct FwdSmem {
  uint4 cc[kFwdPix][7][32];                               // 28 KB: B fragments of three K = 16 steps and one K = 8 step
  uint4 term[kFwdRows][32];                               // 32 KB: colour term, 16-bit
  uint4 feat[kFwdRows][8];                                //  8 KB: features, 54 of 64 columns used
  int2 pairs[kFwdPix][kMaxPairs];
  int cp[kFwdPix][kFwdFrames + 1][9];                     // slot 0: the frame before this pass
};

// 16-byte chunks of a feature row are permuted by pixel and frame: the stores of a warp (eight pixels, four frames) and
// the fragment loads (eight frames of a pixel) both spread over the banks.
__device__ __forceinline__ int feat_key(int row) { return (row ^ (row >> 3)) & 7; }
__device__ __forceinline__ int term_chunk(int row, int chunk) { return chunk ^ ((row & 1) << 2); }

__device__ __forceinline__ void mma_k16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float c0, float c1,
                                        float c2, float c3) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32." ELEM_PTX "." ELEM_PTX ".f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%10,%11,%12,%13};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}
__device__ __forceinline__ void mma_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32." ELEM_PTX "." ELEM_PTX ".f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(b0));
}

// three colour bytes of a word as floats: the byte goes into the mantissa of 2^23
__device__ __forceinline__ float byte_of(uint32_t w, uint32_t selector) {
  return __uint_as_float(__byte_perm(w, 0x4b000000u, selector)) - 8388608.0f;
}

template <bool COLOUR>
__global__ void __launch_bounds__(kFwdThreads, kFwdBlocks) embconv_fwd_kernel(const int* __restrict__ cells, const elem_t* __restrict__ table,
                                                             const float* __restrict__ pos, const elem_t* __restrict__ cc,
                                                             elem_t* __restrict__ feat, elem_t* __restrict__ z,
                                                             elem_t* __restrict__ y, long long frames, int vocab, int O,
                                                             EmbConvGeom g, int seg_len, int z_has_input,
                                                             int apply_gelu, int write_z) {
  extern __shared__ __align__(16) char smem_raw[];
  FwdSmem& sm = *reinterpret_cast<FwdSmem*>(smem_raw);
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int p_out = g.oh * g.ow;
  const int groups = (p_out + kFwdPix - 1) / kFwdPix;
  const long long seg = blockIdx.x / groups;
  const int p0 = (int)(blockIdx.x % groups) * kFwdPix, p = p0 + warp;
  const bool walks = p < p_out;
  const int cb = blockIdx.y * 256, co = cb + lane * 8;
  const bool act = walks && co < O;
  const long long f0 = seg * seg_len, f1 = min(frames, f0 + seg_len);
  const long long frame_words = (long long)g.rows * g.cols * 3;

  // the cells that this thread fetches: pixel px of the eight, frame fu of a pass, every fourth tap from `part`
  const int px = tid & 7, fu = (tid >> 3) & 7, part = tid >> 6;
  const int frow = px * kFwdFrames + fu, fkey = feat_key(frow);
  int item_off[kFwdLoads];                                // word of the cell within its frame; -1: padding or no such tap
#pragma unroll
  for (int k = 0; k < kFwdLoads; ++k) {
    const int t = part + 4 * k;
    item_off[k] = -1;
    if (t < 9 && p0 + px < p_out) {
      const int c = tap_cell(g, (p0 + px) / g.ow, (p0 + px) % g.ow, t);
      if (c >= 0) item_off[k] = c * 3;
    }
  }
  const int* cell_ptr = cells + (f0 + fu) * frame_words;
  int raw[kFwdLoads][3];
  auto fetch = [&](int left) {                            // left: frames from the pass on
#pragma unroll
    for (int k = 0; k < kFwdLoads; ++k) {
      raw[k][0] = -1; raw[k][1] = 0; raw[k][2] = 0;
      if (item_off[k] >= 0 && fu < left) {
        raw[k][0] = __ldg(cell_ptr + item_off[k]);
        if (COLOUR) { raw[k][1] = __ldg(cell_ptr + item_off[k] + 1); raw[k][2] = __ldg(cell_ptr + item_off[k] + 2); }
      }
    }
    cell_ptr += kFwdFrames * frame_words;
  };
  fetch((int)min(f1 - f0, (long long)kFwdFrames));
  if (COLOUR && part == 3) {                              // columns 54 to 63 stay zero
#pragma unroll
    for (int w = 27; w < 32; ++w) reinterpret_cast<uint32_t*>(sm.feat[frow])[((w >> 2) ^ fkey) * 4 + (w & 3)] = 0u;
  }

  if (COLOUR) {                                           // colour matrix rows (channels) as B fragments
    const int n = lane >> 2, kq = (lane & 3) * 2;
    const int ch0 = cb + warp * 32 + 8 * (n >> 1) + (n & 1);
    uint32_t w[28];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int ch = ch0 + 2 * j;
      const uint32_t* row = reinterpret_cast<const uint32_t*>(cc + (long long)ch * 64);
#pragma unroll
      for (int h = 0; h < 7; ++h) w[j * 7 + h] = ch < O ? __ldg(row + (h * 8 + kq) / 2) : 0u;
    }
#pragma unroll
    for (int i = 0; i < 7; ++i) sm.cc[warp][i][lane] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  }

  float2 sum[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) sum[j] = f2(0.0f);
  const char* tab = reinterpret_cast<const char*>(table + (act ? co : 0));
  const int row_bytes = O * (int)sizeof(elem_t);
  auto load_row = [&](int row, Pack8& r) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (row >= 0 && act) v = __ldg(reinterpret_cast<const uint4*>(tab + (long long)row * row_bytes));
    r = *reinterpret_cast<Pack8*>(&v);
  };
  const long long z_step = (long long)p_out * O;
  const long long off = (f0 * p_out + p) * O + co;
  elem_t* z_ptr = z + off;                                // not followed when there is no z or y
  elem_t* y_ptr = y + off;

  for (long long fb = f0; fb < f1; fb += kFwdFrames) {
    const int nf = (int)min((long long)kFwdFrames, f1 - fb);
    // 1: cells -> code points and features
#pragma unroll
    for (int k = 0; k < kFwdLoads; ++k) {
      const int t = part + 4 * k;
      if (k < 2 || part == 0) {
        const int c = raw[k][0];
        sm.cp[px][fu + 1][t] = (unsigned)c >= (unsigned)vocab ? -1 : c;         // outside the table contributes nothing
        if (COLOUR) {
          const uint32_t fg = (uint32_t)raw[k][1], bg = (uint32_t)raw[k][2];
          const float s = 1.0f / 255.0f;
          const elem2_t v[3] = {ff2e2(byte_of(fg, 0x7542) * s, byte_of(fg, 0x7541) * s),
                                ff2e2(byte_of(fg, 0x7540) * s, byte_of(bg, 0x7542) * s),
                                ff2e2(byte_of(bg, 0x7541) * s, byte_of(bg, 0x7540) * s)};
          uint32_t* dst = reinterpret_cast<uint32_t*>(sm.feat[frow]);
#pragma unroll
          for (int h = 0; h < 3; ++h) {
            const int w = part * 3 + h;                                         // 32-bit word of the row, less 12 k
            dst[(((w >> 2) + 3 * k) ^ fkey) * 4 + (w & 3)] = *reinterpret_cast<const uint32_t*>(&v[h]);
          }
        }
      }
    }
    __syncthreads();
    // 2a: rows that change this pixel's sum, in pairs: (old, new) of a changed tap, or two taps of a sum built anew
    uint32_t counts = 0;                                                        // pairs per frame, four bits each; kNewPairs: built anew
    if (walks) {
      int npairs = 0;
      const int t = lane & 15, half = lane >> 4;
      const bool tap = t < 9;
      const int* cps = &sm.cp[warp][half][tap ? t : 0];
      int2* pairs = sm.pairs[warp];
#pragma unroll
      for (int r = 0; r < kFwdFrames / 2; ++r) {
        const bool on = tap && 2 * r + half < nf;
        const int c = cps[(2 * r + 1) * 9], o = cps[2 * r * 9];
        unsigned bal = __ballot_sync(full, on && c != o);
        if (r == 0 && fb == f0) bal |= 0x1ffu;                                  // nothing to change yet: built anew
        if (bal != 0) {
          const int c0 = min(__popc(bal & 0xffffu), kNewPairs), c1 = min(__popc(bal >> 16), kNewPairs);
          const unsigned mine = half ? bal >> 16 : bal & 0xffffu;
          int2* slot = pairs + npairs + (half ? c0 : 0);
          if ((half ? c1 : c0) == kNewPairs) {
            const int n = t < 8 ? cps[(2 * r + 1) * 9 + 1] : -1;                // the next tap
            if (on && !(t & 1)) slot[t >> 1] = make_int2(c >= 0 ? c * 9 + t : -1, n >= 0 ? n * 9 + t + 1 : -1);
          } else if ((mine >> t) & 1u) {
            slot[__popc(mine & ((1u << t) - 1u))] = make_int2(o >= 0 ? o * 9 + t : -1, c >= 0 ? c * 9 + t : -1);
          }
          npairs += c0 + c1;
          counts |= (uint32_t)(c0 | (c1 << 4)) << (8 * r);
        }
      }
      if (lane == 0) pairs[npairs] = make_int2(-1, -1);
      __syncwarp();
      if (lane < 9) sm.cp[warp][0][lane] = sm.cp[warp][kFwdFrames][lane];
    }
    if (COLOUR) {
      // features that the backward reads
      if (feat != nullptr && blockIdx.y == 0) {
#pragma unroll
        for (int k = 0; k < kFwdRows * 8 / kFwdThreads; ++k) {
          const int i = tid + k * kFwdThreads;
          const int chunk = i & 7, x = (i >> 3) % kFwdPix, u = (i >> 3) / kFwdPix;
          const int row = x * kFwdFrames + u;
          if (u < nf && p0 + x < p_out)
            reinterpret_cast<uint4*>(feat + ((fb + u) * p_out + p0 + x) * 64)[chunk] = sm.feat[row][chunk ^ feat_key(row)];
        }
      }
      // 2b: colour term of 64 rows, 32 channels a warp
      uint32_t b[28];
#pragma unroll
      for (int i = 0; i < 7; ++i) {
        const uint4 v = sm.cc[warp][i][lane];
        b[4 * i] = v.x; b[4 * i + 1] = v.y; b[4 * i + 2] = v.z; b[4 * i + 3] = v.w;
      }
      const int r = lane & 15, hi = lane >> 4;
#pragma unroll
      for (int mt = 0; mt < kFwdRows / 16; ++mt) {
        float d[4][4];
        const int row = mt * 16 + r;
#pragma unroll
        for (int ks = 0; ks < 3; ++ks) {
          uint32_t a[4];
          const uint32_t addr = (uint32_t)__cvta_generic_to_shared(&sm.feat[row][(2 * ks + hi) ^ feat_key(row)]);
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                       : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(addr) : "memory");
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float c = 0.0f;
            mma_k16(d[j], a, b[j * 7 + 2 * ks], b[j * 7 + 2 * ks + 1], ks == 0 ? c : d[j][0], ks == 0 ? c : d[j][1],
                    ks == 0 ? c : d[j][2], ks == 0 ? c : d[j][3]);
          }
        }
        uint32_t a0, a1;
        const uint32_t addr = (uint32_t)__cvta_generic_to_shared(&sm.feat[row][6 ^ feat_key(row)]);
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(a0), "=r"(a1) : "r"(addr) : "memory");
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_k8(d[j], a0, a1, b[j * 7 + 6]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int orow = mt * 16 + 8 * h + (lane >> 2);
          Pack8 v;
#pragma unroll
          for (int j = 0; j < 4; ++j) v.h[j] = ff2e2(d[j][2 * h], d[j][2 * h + 1]);
          sm.term[orow][term_chunk(orow, warp * 4 + (lane & 3))] = *reinterpret_cast<uint4*>(&v);
        }
      }
    }
    // 3: walk the frames; the next cells and the first pair of rows are on their way meanwhile
    Pack8 ra, rb;
    const int2* pair = sm.pairs[warp];
    auto next_pair = [&]() {
      const int2 pr = *pair++;
      load_row(pr.x, ra);
      load_row(pr.y, rb);
    };
    if (walks) next_pair();
    if (fb + kFwdFrames < f1) fetch((int)min(f1 - fb - kFwdFrames, (long long)kFwdFrames));
    __syncthreads();
    if (!walks) continue;
#pragma unroll 1
    for (int u = 0; u < nf; ++u) {
      const int n = counts & 15u;
      counts >>= 4;
      if (n != 0) {
        const bool anew = n == kNewPairs;
        if (anew) {
#pragma unroll
          for (int j = 0; j < 4; ++j) sum[j] = f2(0.0f);
          if (act && pos != nullptr) {
            const float4* pp = reinterpret_cast<const float4*>(pos + (long long)p * O + co);
            const float4 a = __ldg(pp), b = __ldg(pp + 1);
            sum[0] = make_float2(a.x, a.y); sum[1] = make_float2(a.z, a.w);
            sum[2] = make_float2(b.x, b.y); sum[3] = make_float2(b.z, b.w);
          }
        }
        const float2 sign = f2(anew ? 1.0f : -1.0f);
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
#pragma unroll
          for (int j = 0; j < 4; ++j) sum[j] = __fadd2_rn(__ffma2_rn(sign, e22ff(ra.h[j]), sum[j]), e22ff(rb.h[j]));
          next_pair();
        }
      }
      if (act) {
        Pack8 term;
        if (COLOUR) {
          const int row = warp * kFwdFrames + u;
          *reinterpret_cast<uint4*>(&term) = sm.term[row][term_chunk(row, lane)];
        } else if (z_has_input) {
          term = *reinterpret_cast<const Pack8*>(z_ptr);
        }
        float2 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = COLOUR || z_has_input ? __fadd2_rn(sum[j], e22ff(term.h[j])) : sum[j];
        Pack8 out;
        if (write_z) {
#pragma unroll
          for (int j = 0; j < 4; ++j) out.h[j] = f22e2(v[j]);
          *reinterpret_cast<Pack8*>(z_ptr) = out;
        }
        if (COLOUR || y != nullptr) {
#pragma unroll
          for (int j = 0; j < 4; ++j) out.h[j] = f22e2(COLOUR || apply_gelu ? gelu2(v[j]) : v[j]);
          *reinterpret_cast<Pack8*>(y_ptr) = out;
        }
      }
      z_ptr += z_step;
      y_ptr += z_step;
    }
  }
}

// ------------------------------------------------------------------------------------------------
// backward: S[v][tap][:] += dZ rows whose tap shows code point v;  D[p][:] += sum over frames of dZ[:, p, :]
// ------------------------------------------------------------------------------------------------
// A lane owns 4 channels (a warp covers a 128-channel block).  All nine taps of a pixel accumulate the same dZ
// values and differ only in where their runs begin and end, so the lane keeps ONE running prefix sum of its dZ over
// the frames of the segment and, per tap, the value of that prefix when the tap's current run began: a run's sum is
// the difference of two prefixes, taken when the run ends.  Per frame that is four additions instead of forty; the
// prefix at the end of the segment is the pixel's contribution to D.  (The prefix spans at most one segment, so the
// difference loses at most log2(segment) bits of fp32 — far below the bf16 resolution of dZ.)
struct alignas(8) Pack4 { elem2_t h[2]; };

__device__ __forceinline__ void red_add4(float* dst, float4 v) { atomicAdd(reinterpret_cast<float4*>(dst), v); }

__global__ void __launch_bounds__(256, 3) embconv_bwd_reduce_kernel(const int* __restrict__ cells, const elem_t* __restrict__ dz,
                                                                    float* __restrict__ S, float* __restrict__ D,
                                                                    long long frames, int vocab, int O, EmbConvGeom g,
                                                                    int seg_len, int nseg) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int p_out = g.oh * g.ow;
  const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= (long long)p_out * nseg) return;
  const int seg = (int)(item / p_out), p = (int)(item % p_out);
  const int cell = lane < 9 ? tap_cell(g, p / g.ow, p % g.ow, lane) : -1;
  const int co = blockIdx.y * 128 + lane * 4;
  const bool act = co < O;
  const long long cells_per_frame = (long long)g.rows * g.cols;
  const long long row9 = 9ll * O;
  float2 pre[2] = {f2(0.0f), f2(0.0f)};                     // prefix sum of this lane's dZ over the frames so far
  // per tap: the prefix when its current run began.  Touched only when a run ends, so it lives in shared memory
  // (one 16-byte slot per thread and tap, conflict-free) and the loop over the changed taps is a real loop.
  __shared__ float4 start_sm[9][256];
  float4* start = &start_sm[0][threadIdx.x];
#pragma unroll
  for (int t = 0; t < 9; ++t) start[t * 256] = make_float4(0.f, 0.f, 0.f, 0.f);
  int cur = -1;
  const long long f0 = (long long)seg * seg_len;
  const long long f1 = min(frames, f0 + seg_len);
  const int* cell_ptr = cells + (f0 * cells_per_frame + max(cell, 0)) * 3;
  const elem_t* dz_ptr = dz + (f0 * p_out + p) * O + (act ? co : 0);
  const long long cell_step = cells_per_frame * 3, dz_step = (long long)p_out * O;
  float* s_base = S + (act ? co : 0);
  for (long long fb = f0; fb < f1; fb += kPrefetchBwd) {
    int ncp[kPrefetchBwd];
    Pack4 din[kPrefetchBwd];
#pragma unroll
    for (int u = 0; u < kPrefetchBwd; ++u) {
      ncp[u] = -1;
      if (fb + u < f1) {
        if (cell >= 0) ncp[u] = __ldg(cell_ptr + u * cell_step);
        if (act) din[u] = *reinterpret_cast<const Pack4*>(dz_ptr + u * dz_step);
      }
    }
    cell_ptr += kPrefetchBwd * cell_step;
    dz_ptr += kPrefetchBwd * dz_step;
#pragma unroll
    for (int u = 0; u < kPrefetchBwd; ++u) {
      if (fb + u >= f1) break;
      int nc = ncp[u];
      if ((unsigned)nc >= (unsigned)vocab) nc = -1;
      unsigned changed = __ballot_sync(full, nc != cur) & 0x1ffu;
      while (changed) {
        const int t = __ffs(changed) - 1;
        changed &= changed - 1;
        const int o = __shfl_sync(full, cur, t);
        const float4 st = start[t * 256];
        if (o >= 0 && act)
          red_add4(s_base + o * row9 + t * O, make_float4(pre[0].x - st.x, pre[0].y - st.y, pre[1].x - st.z, pre[1].y - st.w));
        start[t * 256] = make_float4(pre[0].x, pre[0].y, pre[1].x, pre[1].y);
      }
      cur = nc;
      if (act) {
        pre[0] = __fadd2_rn(pre[0], e22ff(din[u].h[0]));
        pre[1] = __fadd2_rn(pre[1], e22ff(din[u].h[1]));
      }
    }
  }
#pragma unroll 1
  for (int t = 0; t < 9; ++t) {
    const int o = __shfl_sync(full, cur, t);
    const float4 st = start[t * 256];
    if (o >= 0 && act)
      red_add4(s_base + o * row9 + t * O, make_float4(pre[0].x - st.x, pre[0].y - st.y, pre[1].x - st.z, pre[1].y - st.w));
  }
  if (act && f1 > f0) red_add4(D + (long long)p * O + co, make_float4(pre[0].x, pre[0].y, pre[1].x, pre[1].y));
}

// ------------------------------------------------------------------------------------------------
// sum of split-K slabs: out[i] = sum_s work[s][i], written as fp32 or bf16
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) slab_reduce_kernel(const float* __restrict__ work, void* __restrict__ out,
                                                          long long n, int slabs, int out_elem) {
  const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i >= n) return;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k = 0; k < slabs; ++k) {
    const float4 v = *reinterpret_cast<const float4*>(work + (long long)k * n + i);
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  if (out_elem) {
    elem2_t* o = reinterpret_cast<elem2_t*>(reinterpret_cast<elem_t*>(out) + i);
    o[0] = ff2e2(s.x, s.y);
    o[1] = ff2e2(s.z, s.w);
  } else {
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + i) = s;
  }
}

bool geom_ok(const EmbConvGeom& g) {
  if (g.rows < 1 || g.cols < 1 || g.oh < 1 || g.ow < 1 || g.stride < 1 || g.dil < 1 || g.pad < 0) return false;
  // the last output pixel's first tap must not start beyond the frame by more than the padding allows
  const int need_h = (g.oh - 1) * g.stride - g.pad, need_w = (g.ow - 1) * g.stride - g.pad;
  return need_h < g.rows && need_w < g.cols;
}

int launch_result() { return cudaGetLastError() == cudaSuccess ? 0 : 5; }

}  // namespace

// Return codes: 0 ok, 1 unsupported shape, 2 misaligned pointer, 5 launch failure.
extern "C" int fbam_embconv_features(const void* cells, void* feat, long long frames, int rows, int cols, int oh, int ow,
                                     int stride, int pad, int dil, void* stream) {
  const EmbConvGeom g{rows, cols, oh, ow, stride, pad, dil};
  if (!geom_ok(g) || frames < 0) return 1;
  if (reinterpret_cast<uintptr_t>(feat) % 16 != 0) return 2;
  const long long total = frames * (long long)(oh * ow);
  if (total == 0) return 0;
  const long long blocks = (total + 255) / 256;
  if (blocks > 0x7fffffffll) return 1;
  embconv_features_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const int*>(cells), reinterpret_cast<elem_t*>(feat), frames, g);
  return launch_result();
}

namespace {
template <bool COLOUR>
int launch_fwd(const void* cells, const void* table, const void* pos, const void* cc, void* feat, void* z, void* y,
               long long frames, int vocab, int O, const EmbConvGeom& g, int seg_len, int z_has_input, int apply_gelu,
               int write_z, void* stream) {
  if (!geom_ok(g) || frames < 0 || vocab < 1 || O < 8 || O % 8 != 0 || seg_len < 1) return 1;
  for (const void* q : {table, pos, cc, (const void*)feat, (const void*)z, (const void*)y})
    if (reinterpret_cast<uintptr_t>(q) % 16 != 0) return 2;
  if (frames == 0) return 0;
  const long long nseg = (frames + seg_len - 1) / seg_len;
  const long long blocks = ((long long)g.oh * g.ow + kFwdPix - 1) / kFwdPix * nseg;
  if (blocks > 0x7fffffffll) return 1;
  auto kernel = embconv_fwd_kernel<COLOUR>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FwdSmem)) != cudaSuccess) return 5;
  kernel<<<dim3((unsigned)blocks, (unsigned)((O + 255) / 256)), kFwdThreads, sizeof(FwdSmem),
           reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const int*>(cells), reinterpret_cast<const elem_t*>(table), reinterpret_cast<const float*>(pos),
      reinterpret_cast<const elem_t*>(cc), reinterpret_cast<elem_t*>(feat), reinterpret_cast<elem_t*>(z),
      reinterpret_cast<elem_t*>(y), frames, vocab, O, g, seg_len, z_has_input, apply_gelu, write_z);
  return launch_result();
}
}  // namespace

// table: bf16 [vocab][9][O]; pos: fp32 [oh*ow][O] or null; z: bf16 [frames][oh*ow][O], read (when z_has_input) and
// overwritten with the pre-activation (left alone without write_z); y: bf16 like z or null, receives GELU(z) (or z itself without apply_gelu).
extern "C" int fbam_embconv_fwd(const void* cells, const void* table, const void* pos, void* z, void* y,
                                long long frames, int vocab, int O, int rows, int cols, int oh, int ow, int stride,
                                int pad, int dil, int seg_len, int z_has_input, int apply_gelu, int write_z, void* stream) {
  return launch_fwd<false>(cells, table, pos, nullptr, nullptr, z, y, frames, vocab, O,
                           EmbConvGeom{rows, cols, oh, ow, stride, pad, dil}, seg_len, z_has_input, apply_gelu, write_z, stream);
}

// The same with the colour term computed on the way: cc: bf16 [O][64], colour matrix (54 columns used, the rest
// ignored); feat: bf16 [frames][oh*ow][64] or null, receives the colour features (what fbam_embconv_features writes);
// z: written only, or null; y: GELU(z).
extern "C" int fbam_embconv_fwd_colour(const void* cells, const void* table, const void* pos, const void* cc, void* feat,
                                       void* z, void* y, long long frames, int vocab, int O, int rows, int cols, int oh,
                                       int ow, int stride, int pad, int dil, void* stream) {
  if (cc == nullptr || y == nullptr) return 1;
  // Runs of 64 frames, or of 16 where that would not give every SM its blocks twice over (256 frames of 12 x 40 pixels:
  // 80 us against 86 with 64 and 123 with 128; 1024 frames of 24 x 80: 836 with 64 and 128, 873 with 32).
  const long long groups = ((long long)oh * ow + kFwdPix - 1) / kFwdPix;
  const int seg_len = groups * ((frames + 63) / 64) >= 2ll * 148 * kFwdBlocks ? 64 : 16;
  return launch_fwd<true>(cells, table, pos, cc, feat, z, y, frames, vocab, O,
                          EmbConvGeom{rows, cols, oh, ow, stride, pad, dil}, seg_len, 0, 1, z != nullptr, stream);
}

// S: fp32 [vocab][9][O] and D: fp32 [oh*ow][O]; both are added to (the caller zeroes them).
extern "C" int fbam_embconv_bwd_reduce(const void* cells, const void* dz, void* S, void* D, long long frames, int vocab,
                                       int O, int rows, int cols, int oh, int ow, int stride, int pad, int dil,
                                       int seg_len, void* stream) {
  const EmbConvGeom g{rows, cols, oh, ow, stride, pad, dil};
  if (!geom_ok(g) || frames < 0 || vocab < 1 || O < 8 || O % 8 != 0 || seg_len < 1) return 1;
  if (reinterpret_cast<uintptr_t>(dz) % 16 != 0 || reinterpret_cast<uintptr_t>(S) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(D) % 16 != 0)
    return 2;
  if (frames == 0) return 0;
  const int nseg = (int)((frames + seg_len - 1) / seg_len);
  const long long items = (long long)oh * ow * nseg;
  const long long blocks = (items + 7) / 8;
  if (blocks > 0x7fffffffll) return 1;
  dim3 grid((unsigned)blocks, (unsigned)((O + 127) / 128));
  embconv_bwd_reduce_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const int*>(cells), reinterpret_cast<const elem_t*>(dz), reinterpret_cast<float*>(S),
      reinterpret_cast<float*>(D), frames, vocab, O, g, seg_len, nseg);
  return launch_result();
}

// out[i] = sum over `slabs` fp32 slabs of n elements each (n a multiple of 4, 16-byte aligned pointers).
extern "C" int fbam_slab_reduce(const void* work, void* out, long long n, int slabs, int out_elem, void* stream) {
  if (n < 0 || n % 4 != 0 || slabs < 1) return 1;
  if (reinterpret_cast<uintptr_t>(work) % 16 != 0 || reinterpret_cast<uintptr_t>(out) % (out_elem ? 8 : 16) != 0) return 2;
  if (n == 0) return 0;
  const long long blocks = (n / 4 + 255) / 256;
  slab_reduce_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float*>(work), out, n, slabs, out_elem);
  return launch_result();
}
