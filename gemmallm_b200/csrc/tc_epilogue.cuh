// Epilogue of one CTA's 128-row x 256-column accumulator tile in the CTA-pair
// grouped GEMM kernel: TMEM -> registers (one row per thread) ->
// bias (+ GeGLU, + dropout in training mode) -> bf16 -> shared-memory staging ->
// global memory in 128-byte runs per row.
#pragma once
#include "common.cuh"
#include "tc_ptx.cuh"
#include "philox.cuh"

namespace moe {
namespace tc {

constexpr int kStgPitch = 144;               // bytes per staged row: 64 bf16 + 16 bytes pad
constexpr int kStgRows = 16;                 // half a warp's rows are staged at a time
constexpr int kStgBytes = kStgRows * kStgPitch;
constexpr int kStg32Pitch = 80;              // the same for 32 columns
constexpr int kStg32Bytes = kStgRows * kStg32Pitch;

// 64 output columns of this thread's row, as 8 x 16 bytes, go through this warp's staging
// area 16 rows at a time and leave as 128-byte runs (8 lanes per row, 4 rows per store
// instruction): an eighth of the memory requests a one-row-per-thread store would make,
// which compete with the TMA loads for the SM's path to L2, and the run length NVLink wants
// for the expert-parallel scatter. dst = this thread's row (nullptr: nothing to store),
// n = first column, Nlimit = number of valid columns of the row. skip: what this lane adds to the pieces it
// stores, in fp32, rounded again (load_skip64), or nullptr.
__device__ __forceinline__ void flush64(const uint4 (&packed)[8], __nv_bfloat16* dst, int n,
                                        int Nlimit, uint8_t* stg, int lane, const uint4 (*skip)[8] = nullptr) {
#pragma unroll
  for (int hr = 0; hr < 2; ++hr) {
    if ((lane >> 4) == hr) {
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<uint4*>(stg + (lane & 15) * kStgPitch + q * 16) = packed[q];
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = i * 4 + (lane >> 3), piece = lane & 7;
      __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(
          __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(dst), hr * 16 + rr));
      const int nn = n + piece * 8;
      if (d != nullptr && nn < Nlimit) {
        uint4 v = *reinterpret_cast<const uint4*>(stg + rr * kStgPitch + piece * 16);
        if (skip != nullptr) {
          const uint4 k = (*skip)[hr * 4 + i];
          uint32_t w[4] = {v.x, v.y, v.z, v.w};
          const uint32_t o[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) w[q] = pack_bf16x2(bf16_lo(w[q]) + bf16_lo(o[q]), bf16_hi(w[q]) + bf16_hi(o[q]));
          v = make_uint4(w[0], w[1], w[2], w[3]);
        }
        *reinterpret_cast<uint4*>(d + nn) = v;
      }
    }
    __syncwarp();
  }
}

// The pieces of a skip connection [rows, pitch] that a lane adds in flush64: rows of this warp from `row` on, `rows` of them
// exist, 64 columns from n on of Nlimit.
__device__ __forceinline__ void load_skip64(uint4 (&k)[8], const __nv_bfloat16* skip, int row, int rows, int pitch, int n,
                                            int Nlimit, int lane) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int rr = i * 4 + (lane >> 3), nn = n + (lane & 7) * 8;
    k[i] = rr < rows && nn < Nlimit ? *reinterpret_cast<const uint4*>(skip + (int64_t)(row + rr) * pitch + nn)
                                    : make_uint4(0u, 0u, 0u, 0u);
  }
}

__device__ __forceinline__ uint4 pack8(const float (&o)[8]) {
  return make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]), pack_bf16x2(o[4], o[5]),
                    pack_bf16x2(o[6], o[7]));
}

//   taddr  : TMEM address of this warp's 32 lanes, column 0 of the accumulator
//   row    : sorted-buffer row this thread owns; row_ok: inside the expert's segment
//   half   : two warps share each TMEM lane quadrant and split the tile's columns
//   GEGLU  : columns [0,128) gate, [128,256) up; 128 outputs per row, 64 per warp
//   plain  : 256 outputs per row, 128 per warp (two passes); bias may be nullptr (none)
//   SCATTER: plain, but the row goes to sc.ret_y[meta >> 24] + (meta & 0xffffff) * Nout
//            (the token owner's buffer, possibly on another GPU)
//   release(): called once the warp has read its part of the accumulator
//   pitch  : elements from one output row to the next, where it is not Nout (0)
//   SKIP   : plain, plus skip[pass], asked for before the accumulator was awaited
template <bool GEGLU, bool SCATTER, bool SKIP = false, typename Release>
__device__ __forceinline__ void store_tile(uint32_t taddr, int row, bool row_ok, int n0, int Nout,
                                           const __nv_bfloat16* __restrict__ bias,
                                           __nv_bfloat16* __restrict__ out, const EpScatter& sc,
                                           uint8_t* stg, int lane, int half, Release release, int pitch = 0,
                                           const uint4 (*skip)[8] = nullptr) {
  constexpr int BN = 256;
  constexpr int kTileN = GEGLU ? BN / 2 : BN;
  constexpr int kPasses = kTileN / 128;        // 64-column passes per warp
  // destination of this thread's row (nullptr: nothing to store)
  __nv_bfloat16* dst = nullptr;
  if (row_ok) {
    if (SCATTER) {
      const int meta = __ldg(&sc.meta[row]);
      dst = static_cast<__nv_bfloat16*>(sc.ret_y[(meta >> 24) & 7]) + (int64_t)(meta & 0xffffff) * Nout;
    } else {
      dst = out + (int64_t)row * (pitch > 0 ? pitch : Nout);
    }
  }
#pragma unroll(SKIP ? kPasses : 1)
  for (int p = 0; p < kPasses; ++p) {
    const int col0 = (half * kPasses + p) * 64;   // first output column of this pass inside the tile
    uint4 packed[8];
#pragma unroll
    for (int hc = 0; hc < 2; ++hc) {              // two 32-column chunks
      const int c = col0 / 32 + hc;
      uint32_t g[32];
      tc_ld32(taddr + c * 32, g);
      if (GEGLU) {
        uint32_t u[32];
        tc_ld32(taddr + BN / 2 + c * 32, u);
        tc_ld_wait();
        if (hc == 1 && p == kPasses - 1) release();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int n = n0 + c * 32 + q * 8;
          float bg[8], bu[8], o[8];
          if (n < Nout) {
            load8_ldg(bias + n, bg);
            load8_ldg(bias + Nout + n, bu);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) bg[i] = bu[i] = 0.f;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float gv = __uint_as_float(g[q * 8 + i]) + bg[i];
            const float uv = __uint_as_float(u[q * 8 + i]) + bu[i];
            o[i] = gelu_tanh_fast(gv) * uv;
          }
          packed[hc * 4 + q] = pack8(o);
        }
      } else {
        tc_ld_wait();
        if (hc == 1 && p == kPasses - 1) release();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int n = n0 + c * 32 + q * 8;
          float b[8], o[8];
          if (bias != nullptr && n < Nout) {
            load8_ldg(bias + n, b);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) b[i] = 0.f;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = __uint_as_float(g[q * 8 + i]) + b[i];
          packed[hc * 4 + q] = pack8(o);
        }
      }
    }
    flush64(packed, dst, n0 + col0, Nout, stg, lane, SKIP ? skip + p : nullptr);
  }
}

// Zeros for `rows` rows x 128 columns of a weight-gradient tile (an expert without rows).
__device__ __forceinline__ void store_zero_tile(__nv_bfloat16* __restrict__ out, int row0, int rows, int Nout, int n,
                                                int lane) {
  for (int i = lane; i < rows * 16; i += 32) {
    const int rr = i >> 4, c = n + (i & 15) * 8;
    if (c < Nout) *reinterpret_cast<uint4*>(out + (int64_t)(row0 + rr) * Nout + c) = make_uint4(0, 0, 0, 0);
  }
}

// 32 columns of a warp's 32 rows (thread = row) as 64-byte runs; base = first row, first column.
__device__ __forceinline__ void flush32(const uint4 (&packed)[4], __nv_bfloat16* base, int64_t pitch, int rows,
                                        int cols, uint8_t* stg, int lane) {
#pragma unroll
  for (int hr = 0; hr < 2; ++hr) {
    if ((lane >> 4) == hr) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<uint4*>(stg + (lane & 15) * kStg32Pitch + q * 16) = packed[q];
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int rr = i * 8 + (lane >> 2), piece = lane & 3;
      if (hr * 16 + rr < rows && piece * 8 < cols)
        *reinterpret_cast<uint4*>(base + (hr * 16 + rr) * pitch + piece * 8) =
            *reinterpret_cast<const uint4*>(stg + rr * kStg32Pitch + piece * 16);
    }
    __syncwarp();
  }
}

// Output boxes of 32 rows x 32 columns of an epilogue warp whose 32 rows all exist: written to the
// warp's buffer (64-byte swizzle: 16-byte piece c of row r lies at c ^ (r / 2 mod 4)) and stored by TMA,
// about a fifth of the instructions of flush32 and no wait for the memory.
constexpr int kBoxBytes = 32 * 64;
struct BoxOut {
  uint8_t* buf;
  __device__ __forceinline__ void put(const uint4 (&packed)[4], const void* tmap, int col, int row, int lane) {
    if (lane == 0) bulk_wait_read<0>();      // the store before this one has read the buffer
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<uint4*>(buf + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4)) = packed[q];
    fence_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_2d(tmap, buf, col, row);
      bulk_commit();
    }
  }
};

// GEGLU pass in training mode (TrainArgs in common.cuh), 16 epilogue warps: this one takes output
// columns [32 part, 32 part + 32) of its 32 rows. h gets its dropout mask (s_mask[row][part], bits drawn by four other
// warps while the products of the tile run, draw_mask), and what the backward pass multiplies dh by is kept, the
// derivatives of h after the gate and the up value, mask and scale included:
//   h = m gelu(g) u,   h_g = m u gelu'(g),   h_u = m gelu(g),   m = scale where the element is kept, else 0
//   with s = 1 / (1 + exp(-2 z)), z = b (g + a g^3):  gelu(g) = g s,
//   gelu'(g) = s + 2 g s (1 - s) b (1 + 3 a g^2)       (0.5 (1 + tanh z) = s)
// (Keeping g and u instead left GELU, its derivative and the mask to the backward epilogue, which had twice the elements
// per product and was bound by them, and rounded g and u before they went through the GELU. 32768 rows, d 1024, f 4096, 8
// experts: that product 385 -> 302 us, now bound by the column sums' shuffles and its boxes' way through shared memory;
// this one 438 -> 443; whole training step 2472 -> 2413. Gradients against 64 bits, 2-norm, 13 sizes of 99 to 16384 tokens with
// dropout 0.1: of x 3.75e-3 to 3.81e-3 -> 3.65e-3 to 3.73e-3, w1 3.44e-3 -> 3.32e-3, b1 3.00e-3 -> 2.87e-3, the router's and
// the down Linear's as before. A dropped element's derivatives are zeros that dh is multiplied by: with dh infinite or NaN
// its gradients are NaN, as autograd's through a product with the mask, where they were 0; with g beyond 1e19 they are 0,
// where they were NaN.)
// PRE, LoRA steps: g, u and the mask are kept all the same, whose rounding such a step repeats (lora_bwd.cu says why).
// start() fetches the biases into this warp's 64 floats of shared memory before the products are awaited.
template <bool PRE>
struct GegluTrain {
  __device__ __forceinline__ static void start(int n0, int Nout, const __nv_bfloat16* __restrict__ bias, float* s_bias,
                                               int lane, int part) {
    const int n = n0 + part * 32 + lane;
    const float bg = n < Nout ? __bfloat162float(__ldg(bias + n)) : 0.f;
    const float bu = n < Nout ? __bfloat162float(__ldg(bias + Nout + n)) : 0.f;
    __syncwarp();
    s_bias[lane] = bg;
    s_bias[32 + lane] = bu;
    __syncwarp();
  }
  template <typename Release>
  __device__ __forceinline__ static void finish(uint32_t taddr, int row_warp, int rows, int n0, int Nout,
                                                __nv_bfloat16* __restrict__ out, const TrainArgs& tr,
                                                const void* tmap_h, const void* tmap_gu, const float* s_bias,
                                                uint32_t keep, BoxOut& box, int lane, int part, Release release) {
    const int n = n0 + part * 32;
    const int cols = Nout - n;
    uint4 ph[4], pg[4], pu[4];
#pragma unroll
    for (int hc = 0; hc < 2; ++hc) {      // 16 columns at a time: fewer registers, more warps
      uint32_t g[16], u[16];
      tc_ld16(taddr + part * 32 + hc * 16, g);
      tc_ld16(taddr + 128 + part * 32 + hc * 16, u);
      tc_ld_wait();
      if (hc == 1) release();
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c = hc * 16 + q * 8;
        float gv[8], uv[8], o[8];
        load8(s_bias + c, gv);
        load8(s_bias + 32 + c, uv);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          gv[i] += __uint_as_float(g[q * 8 + i]);
          uv[i] += __uint_as_float(u[q * 8 + i]);
          if constexpr (PRE) {
            const float hv = gelu_tanh_fast(gv[i]) * uv[i];
            o[i] = (keep >> (c + i)) & 1u ? hv * tr.scale : 0.f;
            continue;
          }
          constexpr float kB = 0.7978845608028654f, kA = 0.044715f, kL = -2.f * 1.4426950408889634f;
          const float x = gv[i], x2 = x * x;
          const float sg = __fdividef(1.f, 1.f + exp2f_fast(x * fmaf(kL * kB * kA, x2, kL * kB)));
          const float gs = x * sg;
          const float dgelu = fmaf(fmaf(-gs, sg, gs), fmaf(6.f * kA * kB, x2, 2.f * kB), sg);
          const bool kept = (keep >> (c + i)) & 1u;
          gv[i] = kept ? uv[i] * dgelu * tr.scale : 0.f;
          const float hu = kept ? gs * tr.scale : 0.f;
          o[i] = kept ? hu * uv[i] : 0.f;
          uv[i] = hu;
        }
        pg[c / 8] = pack8(gv);
        pu[c / 8] = pack8(uv);
        ph[c / 8] = pack8(o);
      }
    }
    if (rows >= 32 && cols >= 32) {
      box.put(ph, tmap_h, n, row_warp, lane);
      box.put(pg, tmap_gu, n, row_warp, lane);
      box.put(pu, tmap_gu, Nout + n, row_warp, lane);
    } else {       // the expert's last rows, or the last columns of an odd width
      if (lane == 0) bulk_wait_read<0>();
      __syncwarp();
      flush32(ph, out + (int64_t)row_warp * Nout + n, Nout, rows, cols, box.buf, lane);
      flush32(pg, tr.gu + (int64_t)row_warp * 2 * Nout + n, 2 * (int64_t)Nout, rows, cols, box.buf, lane);
      flush32(pu, tr.gu + (int64_t)row_warp * 2 * Nout + Nout + n, 2 * (int64_t)Nout, rows, cols, box.buf, lane);
    }
  }
};

// The dropout mask of one row's 128 columns from n0 (bit i of word w: column n0 + 32 w + i, set = kept), to
// shared memory for the epilogue and, where it is kept (PRE), to global memory for the backward pass.
template <bool PRE>
__device__ __forceinline__ void draw_mask(const TrainArgs& tr, int64_t row, bool row_ok, int n0, int Nout,
                                          uint32_t* s_row) {
  const uint32_t pair = tr.pair_of == nullptr ? (uint32_t)row : row_ok ? (uint32_t)__ldg(&tr.pair_of[row]) : 0u;
  uint32_t w[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    uint32_t keep = 0u;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const uint4 r = philox4x32_10((uint32_t)((n0 >> 2) + p * 8 + b), pair, tr.seed_lo, tr.seed_hi);
      keep |= (r.x >= tr.thresh ? 1u : 0u) << (4 * b) | (r.y >= tr.thresh ? 2u : 0u) << (4 * b) |
              (r.z >= tr.thresh ? 4u : 0u) << (4 * b) | (r.w >= tr.thresh ? 8u : 0u) << (4 * b);
    }
    w[p] = keep;
  }
  *reinterpret_cast<uint4*>(s_row) = make_uint4(w[0], w[1], w[2], w[3]);
  if (PRE && row_ok) {
    uint8_t* m = tr.mask + row * (Nout >> 3) + (n0 >> 3);
    if ((Nout & 127) == 0) {
      *reinterpret_cast<uint4*>(m) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
      for (int q = 0; q < 16 && n0 + q * 8 < Nout; ++q) m[q] = (uint8_t)(w[q >> 2] >> ((q & 3) * 8));
    }
  }
}

// Epilogue of dh = dy W2 in the backward pass (model.py:180-183), 16 epilogue warps, one accumulator row per
// thread, back through dropout, product and GELU in place over the derivatives the forward kept (GegluTrain):
//   dg = dh h_g;  du = dh h_u
// LoRA steps (ROUND) form them from the pre-activations and the mask, in one rounding:
//   dhe = dh * mask * scale;  du = dhe * gelu(g);  dg = dhe * u * gelu'(g)
// The tile is worked on in chunks of 64 columns: another warp (gu_warp in the kernel) brings a chunk of the two
// values (two boxes of 128 rows x 64 columns, 128-byte swizzle) to shared memory two chunks ahead, the epilogue
// replaces them by the gradients there, and the boxes are stored again. (With the loads issued by the epilogue
// warps themselves, however far ahead registers allowed, their latency made the kernel 2.3 times as long.)
// This warp takes columns [16 part, 16 part + 16) of the chunk for its 32 rows; it also sums dg and du over the
// rows (the bias gradient of gate_and_up) into s_col[0..15] and s_col[du_off ..].
struct GegluBwd {
  static constexpr int kChunk = 64;
  static constexpr int kBoxBytes = 128 * 128;
  __device__ __forceinline__ static uint32_t mask_bits(const TrainArgs& tr, int64_t row, bool row_ok, int n, int f) {
    if (tr.thresh == 0u) return 0xffffu;
    if (!row_ok || n >= f) return 0u;
    const uint8_t* m = tr.mask + row * (f >> 3) + (n >> 3);
    if ((f & 15) == 0) return *reinterpret_cast<const uint16_t*>(m);
    return n + 8 < f ? (uint32_t)m[0] | (uint32_t)m[1] << 8 : (uint32_t)m[0];
  }
  // v: dh of this row's 16 columns; box: the chunk's gate box in shared memory, the up box behind it.
  // direct: the row's place in gu for a chunk that cannot be stored as boxes, else nullptr; cols: columns that exist;
  // ROUND: dh is rounded to bf16 first, and the sums take the rounded dg and du (lora_bwd.cu says why)
  template <bool ROUND>
  __device__ __forceinline__ static void chunk(uint32_t (&v)[16], uint8_t* box, uint32_t keep, float scale, bool row_ok,
                                               __nv_bfloat16* direct, int f, int cols, float* s_col, int du_off, int quad,
                                               int part, int lane) {
    float dg[16], du[16];
    const int r = quad * 32 + lane;
    if (!ROUND && !row_ok) {      // rows of other experts: nothing of them in the sums
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = 0u;
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      uint4* gp = reinterpret_cast<uint4*>(box + r * 128 + (((part * 2 + j) ^ (r & 7)) << 4));
      uint4* up = gp + kBoxBytes / 16;
      uint4 g4 = *gp, u4 = *up;
      if (!ROUND && !row_ok) g4 = u4 = make_uint4(0, 0, 0, 0);
      const uint32_t gw[4] = {g4.x, g4.y, g4.z, g4.w};
      const uint32_t uw[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int c = j * 8 + i;
        const float x = (i & 1) ? bf16_hi(gw[i >> 1]) : bf16_lo(gw[i >> 1]);
        const float uv = (i & 1) ? bf16_hi(uw[i >> 1]) : bf16_lo(uw[i >> 1]);
        if constexpr (!ROUND) {
          dg[c] = __uint_as_float(v[c]) * x;
          du[c] = __uint_as_float(v[c]) * uv;
        } else {
          constexpr float kB = 0.7978845608028654f, kA = 0.044715f, kL = -2.f * 1.4426950408889634f;
          const float dh = __bfloat162float(__float2bfloat16_rn(__uint_as_float(v[c])));
          const float dv = (keep >> c) & 1u ? dh * scale : 0.f;
          const float x2 = x * x;
          const float s = __fdividef(1.f, 1.f + exp2f_fast(x * fmaf(kL * kB * kA, x2, kL * kB)));
          const float gs = x * s;
          const float dgelu = fmaf(fmaf(-gs, s, gs), fmaf(6.f * kA * kB, x2, 2.f * kB), s);
          du[c] = row_ok ? dv * gs : 0.f;
          dg[c] = row_ok ? dv * uv * dgelu : 0.f;
        }
      }
      const uint4 og = make_uint4(pack_bf16x2(dg[j * 8], dg[j * 8 + 1]), pack_bf16x2(dg[j * 8 + 2], dg[j * 8 + 3]),
                                  pack_bf16x2(dg[j * 8 + 4], dg[j * 8 + 5]), pack_bf16x2(dg[j * 8 + 6], dg[j * 8 + 7]));
      const uint4 ou = make_uint4(pack_bf16x2(du[j * 8], du[j * 8 + 1]), pack_bf16x2(du[j * 8 + 2], du[j * 8 + 3]),
                                  pack_bf16x2(du[j * 8 + 4], du[j * 8 + 5]), pack_bf16x2(du[j * 8 + 6], du[j * 8 + 7]));
      if (ROUND) {
        const uint32_t ogw[4] = {og.x, og.y, og.z, og.w}, ouw[4] = {ou.x, ou.y, ou.z, ou.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          dg[j * 8 + i] = (i & 1) ? bf16_hi(ogw[i >> 1]) : bf16_lo(ogw[i >> 1]);
          du[j * 8 + i] = (i & 1) ? bf16_hi(ouw[i >> 1]) : bf16_lo(ouw[i >> 1]);
        }
      }
      if (direct == nullptr) {
        *gp = og;
        *up = ou;
      } else if (row_ok && j * 8 < cols) {
        *reinterpret_cast<uint4*>(direct + j * 8) = og;
        *reinterpret_cast<uint4*>(direct + f + j * 8) = ou;
      }
    }
    // sums over the 32 lanes, each step keeping half of the 32 values: lane l ends with one of them
    float t[32];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      t[i] = dg[i];
      t[16 + i] = du[i];
    }
    int first = 0;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      const bool upper = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (i < o) {
          const float give = upper ? t[i] : t[o + i];
          const float mine = upper ? t[o + i] : t[i];
          t[i] = mine + __shfl_xor_sync(0xffffffffu, give, o);
        }
      if (upper) first += o;
    }
    s_col[(first & 15) + (first >= 16 ? du_off : 0)] = t[0];
  }
};

}  // namespace tc
}  // namespace moe
