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
// n = first column, Nlimit = number of valid columns of the row.
__device__ __forceinline__ void flush64(const uint4 (&packed)[8], __nv_bfloat16* dst, int n,
                                        int Nlimit, uint8_t* stg, int lane) {
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
      if (d != nullptr && nn < Nlimit)
        *reinterpret_cast<uint4*>(d + nn) =
            *reinterpret_cast<const uint4*>(stg + rr * kStgPitch + piece * 16);
    }
    __syncwarp();
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
template <bool GEGLU, bool SCATTER>
__device__ __forceinline__ void store_tile(uint32_t taddr, int row, bool row_ok, int n0, int Nout,
                                           const __nv_bfloat16* __restrict__ bias,
                                           __nv_bfloat16* __restrict__ out, const EpScatter& sc,
                                           uint8_t* stg, int lane, int half) {
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
      dst = out + (int64_t)row * Nout;
    }
  }
#pragma unroll 1
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
    flush64(packed, dst, n0 + col0, Nout, stg, lane);
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

// GEGLU pass in training mode (TrainArgs in common.cuh), 16 epilogue warps: this one takes output
// columns [32 part, 32 part + 32) of its 32 rows. The gate/up pre-activations are kept for the backward
// pass, h gets its dropout mask, and the mask itself is kept as one bit per element, so that the
// backward pass does not run Philox again.
__device__ __forceinline__ void store_tile_train(uint32_t taddr, int row_warp, int rows, int n0, int Nout,
                                                 const __nv_bfloat16* __restrict__ bias,
                                                 __nv_bfloat16* __restrict__ out, const TrainArgs& tr, uint8_t* stg,
                                                 int lane, int part) {
  const int n = n0 + part * 32;
  const int cols = Nout - n;
  const int64_t row = row_warp + lane;
  const bool row_ok = lane < rows;
  const uint32_t pair = row_ok ? (uint32_t)__ldg(&tr.pair_of[row]) : 0u;
  uint32_t g[32], u[32];
  tc_ld32(taddr + part * 32, g);
  tc_ld32(taddr + 128 + part * 32, u);
  tc_ld_wait();
  uint4 ph[4], pg[4], pu[4];
  uint32_t keep = 0xffffffffu;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float gv[8], uv[8], o[8];
    if (q * 8 < cols) {
      load8_ldg(bias + n + q * 8, gv);
      load8_ldg(bias + Nout + n + q * 8, uv);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) gv[i] = uv[i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      gv[i] += __uint_as_float(g[q * 8 + i]);
      uv[i] += __uint_as_float(u[q * 8 + i]);
      o[i] = gelu_tanh_fast(gv[i]) * uv[i];
    }
    pg[q] = pack8(gv);
    pu[q] = pack8(uv);
    if (tr.thresh != 0u) {
#pragma unroll
      for (int b4 = 0; b4 < 2; ++b4) {
        const uint4 r = philox4x32_10((uint32_t)((n + q * 8) >> 2) + b4, pair, tr.seed_lo, tr.seed_hi);
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool kept = w[i] >= tr.thresh;
          o[b4 * 4 + i] = kept ? o[b4 * 4 + i] * tr.scale : 0.f;
          if (!kept) keep &= ~(1u << (q * 8 + b4 * 4 + i));
        }
      }
    }
    ph[q] = pack8(o);
  }
  if (tr.thresh != 0u && row_ok) {
    uint8_t* m = tr.mask + row * (Nout >> 3) + (n >> 3);
    if ((Nout & 31) == 0) {
      *reinterpret_cast<uint32_t*>(m) = keep;
    } else {
      for (int q = 0; q < 4 && q * 8 < cols; ++q) m[q] = (uint8_t)(keep >> (q * 8));
    }
  }
  flush32(ph, out + (int64_t)row_warp * Nout + n, Nout, rows, cols, stg, lane);
  flush32(pg, tr.gu + (int64_t)row_warp * 2 * Nout + n, 2 * (int64_t)Nout, rows, cols, stg, lane);
  flush32(pu, tr.gu + (int64_t)row_warp * 2 * Nout + Nout + n, 2 * (int64_t)Nout, rows, cols, stg, lane);
}

// Epilogue of dh = dy W2 in the backward pass (model.py:180-183), 16 epilogue warps, this one for 64
// columns of its 32 rows: dh is rounded to bf16 and staged so that a lane owns eight neighbouring columns
// of a row, whose gate/up pre-activations (and mask bits) it reads and whose gradients it writes in 128-byte
// runs of eight lanes:
//   dhe = dh * mask * scale;  du = dhe * gelu(g);  dg = dhe * u * gelu'(g)
//   with s = 1 / (1 + exp(-2 z)), z = b (g + a g^3):  gelu(g) = g s,
//   gelu'(g) = s + 2 g s (1 - s) b (1 + 3 a g^2)       (0.5 (1 + tanh z) = s)
// in place over gu. It also sums dg and du over its rows (the bias gradient of gate_and_up).
struct GegluBwd {
  uint4 g[4], u[4];      // pre-activations of 16 rows: rows i*4 + lane/8, columns 8 (lane % 8) ..
  uint32_t m[4];
  __nv_bfloat16* gp;     // row lane/8, this lane's columns
  const uint8_t* mp;
  int64_t f;
  int rows, lane;
  bool col_ok, masked;
  float scale;

  __device__ __forceinline__ void fetch(int hr) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = hr * 16 + i * 4 + (lane >> 3);
      g[i] = u[i] = make_uint4(0, 0, 0, 0);
      m[i] = 0xffu;
      if (col_ok && rr < rows) {
        const __nv_bfloat16* p = gp + (hr * 16 + i * 4) * 2 * f;
        g[i] = *reinterpret_cast<const uint4*>(p);
        u[i] = *reinterpret_cast<const uint4*>(p + f);
        if (masked) m[i] = mp[(hr * 16 + i * 4) * (f >> 3)];
      }
    }
  }
  __device__ __forceinline__ void start(const TrainArgs& tr, int row_warp, int rows_, int Nout, int n, int lane_) {
    lane = lane_;
    rows = rows_;
    f = Nout;
    scale = tr.scale;
    masked = tr.thresh != 0u;
    const int c = n + (lane & 7) * 8;
    col_ok = c < Nout;
    const int64_t row = row_warp + (lane >> 3);
    gp = tr.gu + row * 2 * f + c;
    mp = tr.mask + row * (f >> 3) + (c >> 3);
    fetch(0);
  }
  // taddr: this warp's 64 columns; s_col: where the column sums go, du's `du_off` floats behind dg's
  template <typename Release>
  __device__ __forceinline__ void finish(uint32_t taddr, uint8_t* stg, float* s_col, int du_off, Release release) {
    uint4 dh[8];
#pragma unroll
    for (int hc = 0; hc < 2; ++hc) {
      uint32_t v[32];
      tc_ld32(taddr + hc * 32, v);
      tc_ld_wait();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = __uint_as_float(v[q * 8 + i]);
        dh[hc * 4 + q] = pack8(o);
      }
    }
    release();
    float cg[8], cu[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) cg[i] = cu[i] = 0.f;
#pragma unroll
    for (int hr = 0; hr < 2; ++hr) {
      if ((lane >> 4) == hr) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<uint4*>(stg + (lane & 15) * kStgPitch + q * 16) = dh[q];
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int rl = i * 4 + (lane >> 3);
        if (col_ok && hr * 16 + rl < rows) {
          const uint4 dv4 = *reinterpret_cast<const uint4*>(stg + rl * kStgPitch + (lane & 7) * 16);
          const uint32_t dw[4] = {dv4.x, dv4.y, dv4.z, dv4.w};
          const uint32_t gw[4] = {g[i].x, g[i].y, g[i].z, g[i].w};
          const uint32_t uw[4] = {u[i].x, u[i].y, u[i].z, u[i].w};
          float dg[8], du[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            float dv = (c & 1) ? bf16_hi(dw[c >> 1]) : bf16_lo(dw[c >> 1]);
            const float x = (c & 1) ? bf16_hi(gw[c >> 1]) : bf16_lo(gw[c >> 1]);
            const float uv = (c & 1) ? bf16_hi(uw[c >> 1]) : bf16_lo(uw[c >> 1]);
            if (masked) dv = ((m[i] >> c) & 1u) ? dv * scale : 0.f;
            constexpr float kB = 0.7978845608028654f, kA = 0.044715f, kL = -2.f * 1.4426950408889634f;
            const float x2 = x * x;
            const float s = __fdividef(1.f, 1.f + exp2f_fast(x * fmaf(kL * kB * kA, x2, kL * kB)));
            const float gs = x * s;
            const float dgelu = fmaf(fmaf(-gs, s, gs), fmaf(6.f * kA * kB, x2, 2.f * kB), s);
            du[c] = dv * gs;
            dg[c] = dv * uv * dgelu;
            cg[c] += dg[c];
            cu[c] += du[c];
          }
          __nv_bfloat16* p = gp + (hr * 16 + i * 4) * 2 * f;
          *reinterpret_cast<uint4*>(p) = pack8(dg);
          *reinterpret_cast<uint4*>(p + f) = pack8(du);
        }
      }
      __syncwarp();
      if (hr == 0) fetch(1);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int o = 8; o <= 16; o <<= 1) {
        cg[i] += __shfl_xor_sync(0xffffffffu, cg[i], o);
        cu[i] += __shfl_xor_sync(0xffffffffu, cu[i], o);
      }
    }
    if (lane < 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        s_col[lane * 8 + i] = cg[i];
        s_col[du_off + lane * 8 + i] = cu[i];
      }
    }
  }
};

}  // namespace tc
}  // namespace moe
