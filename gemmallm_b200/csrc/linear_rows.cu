// Linears of the decoder layer's attention (reference model.py:76, 139 and 150) for the rows of a short sequence or a few:
//   out[t] = in[t] W^T + b, rounded, optionally with the first LayerNorm in front (model.py:297,303) and the skip connection
//   behind (model.py:308), and optionally with a second Linear on the same rows (the fused QKV projection and the head gate).
//
// A block owns 16 rows of W and 16 or 32 tokens. The weights are the 16-row A operand of mma.sync, eight tokens the B operand;
// eight warps share K, chunks of 32 in turn, and their sums are added in warp order. A lane loads 16 bytes of a row of W and
// of a token, the same ones of both, so that the products see K in an order of their own. With the LayerNorm every block
// normalises its tokens itself, as layernorm_rows_kernel does, into shared memory.
//
// What bounds it: latency. The work is 4.4 MB of weights over a chain of loads, and what counts is how few launches there are
// and that each has its first loads under way when the kernel before it ends: weights are asked for before the wait where
// the launch says that nothing in flight writes them. A decoder layer of 37 tokens (d 1024, 16 heads, 8 experts) took 93.4 us
// with six launches around the attention (LayerNorm, three library products, the core, the addition) and takes 69.5 with
// three; one token 84 -> 39.6, 102 tokens 92.6 -> 79.6, 128 tokens 93.9 -> 80.7. Beyond 128 rows the Linears are tiles of
// experts_tc2.cu (kLinear): 64 tokens 81.8 so and 72.3 here, 128 86.9 and 80.7, 140 89.9 and 91.3, 160 91.8 and 94.8. Large
// ones are torch's (attention_own_linears below).
#include "common.cuh"
#include "internal.h"

namespace moe {

namespace {

constexpr int kWarps = 8;
constexpr int kRowsW = 16;
constexpr int kInFlight = 4;        // chunks of 32 of K a warp asks for at a time
constexpr int kRedPitch = kRowsW + 1;

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// elements from one staged token to the next: 64 bytes on in the banks, so that eight lanes of a 16-byte load, two tokens of
// four pieces, meet in none
__host__ __device__ inline int staged_pitch(int K) { return ((K + 63) & ~63) + 32; }

struct Operand {
  const __nv_bfloat16 *W, *b;   // [rows, K], [rows]
  __nv_bfloat16* out;           // [N, rows]
  int rows;
};

// KEEP: 256 KEEP elements of K at most where rows are normalised; 0: they are not
template <int TOK, int KEEP>
__global__ void __launch_bounds__(32 * kWarps)
linear_rows_kernel(const __nv_bfloat16* x, const __nv_bfloat16* gamma, const __nv_bfloat16* beta, float eps,
                   const Operand first, const Operand second, const __nv_bfloat16* skip, int N, int K, int chained) {
  constexpr bool NORM = KEEP > 0;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __nv_bfloat16* sX = reinterpret_cast<__nv_bfloat16*>(smem_raw);       // NORM: [TOK][pitch]; then the warps' sums
  float* red = reinterpret_cast<float*>(smem_raw);                      // [kWarps][TOK][kRedPitch]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int blocks0 = (first.rows + kRowsW - 1) / kRowsW;
  const bool one = (int)blockIdx.x < blocks0;
  const Operand op = one ? first : second;
  const int r0 = ((int)blockIdx.x - (one ? 0 : blocks0)) * kRowsW;
  const int tok0 = (int)blockIdx.y * TOK;
  const int pieces = K >> 3, nchunk = (K + 31) >> 5;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const uint4* wa = reinterpret_cast<const uint4*>(op.W + (int64_t)min(r0 + g, op.rows - 1) * K);
  const uint4* wb = reinterpret_cast<const uint4*>(op.W + (int64_t)min(r0 + g + 8, op.rows - 1) * K);
  uint4 a[kInFlight], b[kInFlight];
  auto load_weights = [&](int c0) {
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) {
      const int p = (c0 + u * kWarps) * 4 + t;
      a[u] = p < pieces ? __ldcg(wa + p) : zero;
      b[u] = p < pieces ? __ldcg(wb + p) : zero;
    }
  };
  if (!chained) pdl_wait();
  load_weights(warp);
  if (chained) pdl_wait();
  pdl_launch_dependents();

  const int pitch = staged_pitch(K);
  if constexpr (NORM) {
    // mean, biased variance around the mean, (x - mean) rstd gamma + beta, rounded: as layernorm_rows_kernel, to the bit
    constexpr int kRows = TOK / kWarps;
    uint4 raw[kRows][KEEP];       // of all the warp's rows at once
#pragma unroll
    for (int rr = 0; rr < kRows; ++rr) {
      const __nv_bfloat16* xr = x + (int64_t)min(tok0 + rr * kWarps + warp, N - 1) * K;
#pragma unroll
      for (int i = 0; i < KEEP; ++i) {
        const int c = lane * 8 + i * 256;
        if (c < K) raw[rr][i] = __ldcg(reinterpret_cast<const uint4*>(xr + c));
      }
    }
#pragma unroll
    for (int rr = 0; rr < kRows; ++rr) {
      const int r = rr * kWarps + warp;
      __nv_bfloat16* o = sX + r * pitch;
      const bool live = tok0 + r < N;
      auto each = [&](auto f) {
#pragma unroll
        for (int i = 0; i < KEEP; ++i) {
          const int c = lane * 8 + i * 256;
          if (c < K) {
            const uint32_t w[4] = {raw[rr][i].x, raw[rr][i].y, raw[rr][i].z, raw[rr][i].w};
            float v[8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              v[2 * q] = bf16_lo(w[q]);
              v[2 * q + 1] = bf16_hi(w[q]);
            }
            f(c, v);
          }
        }
      };
      float sum = 0.f;
      each([&](int, const float (&v)[8]) {
#pragma unroll
        for (int q = 0; q < 8; ++q) sum += v[q];
      });
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
      const float mean = sum / (float)K;
      float sq = 0.f;
      each([&](int, const float (&v)[8]) {
#pragma unroll
        for (int q = 0; q < 8; ++q) sq = fmaf(v[q] - mean, v[q] - mean, sq);
      });
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, s);
      const float rstd = rsqrtf(sq / (float)K + eps);
      each([&](int c, const float (&v)[8]) {
        float gm[8], bt[8], y[8];
        load8(gamma + c, gm);
        load8(beta + c, bt);
#pragma unroll
        for (int q = 0; q < 8; ++q) y[q] = live ? fmaf((v[q] - mean) * rstd, gm[q], bt[q]) : 0.f;
        store8(o + c, y);
      });
      for (int c = K + lane * 8; c < nchunk * 32; c += 256) *reinterpret_cast<uint4*>(o + c) = zero;
    }
    __syncthreads();
  }

  float acc[TOK / 8][4];
#pragma unroll
  for (int j = 0; j < TOK / 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
  for (int c0 = warp; c0 < nchunk; c0 += kWarps * kInFlight) {
    if (c0 != warp) load_weights(c0);
    uint4 v[NORM ? 1 : kInFlight][TOK / 8];
    if constexpr (!NORM) {
#pragma unroll
      for (int u = 0; u < kInFlight; ++u)
#pragma unroll
        for (int j = 0; j < TOK / 8; ++j) {
          const int p = (c0 + u * kWarps) * 4 + t, tok = tok0 + 8 * j + g;
          v[u][j] = p < pieces && tok < N ? __ldcg(reinterpret_cast<const uint4*>(x + (int64_t)tok * K) + p) : zero;
        }
    }
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) {
      const int c = c0 + u * kWarps;
      if (NORM && c >= nchunk) break;
#pragma unroll
      for (int j = 0; j < TOK / 8; ++j) {
        const uint4 xv = NORM ? *reinterpret_cast<const uint4*>(sX + (8 * j + g) * pitch + c * 32 + t * 8) : v[NORM ? 0 : u][j];
        mma16816(acc[j], a[u].x, b[u].x, a[u].y, b[u].y, xv.x, xv.y);
        mma16816(acc[j], a[u].z, b[u].z, a[u].w, b[u].w, xv.z, xv.w);
      }
    }
  }
  if (NORM) __syncthreads();      // the staged tokens have been read
#pragma unroll
  for (int j = 0; j < TOK / 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) red[(warp * TOK + 8 * j + 2 * t + (i & 1)) * kRedPitch + g + (i >> 1) * 8] = acc[j][i];
  __syncthreads();
  for (int i = threadIdx.x; i < TOK * kRowsW / 2; i += 32 * kWarps) {
    const int tok = i / (kRowsW / 2), r = (i % (kRowsW / 2)) * 2;
    if (tok0 + tok >= N || r0 + r >= op.rows) continue;
    float s[2] = {0.f, 0.f};
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      s[0] += red[(w * TOK + tok) * kRedPitch + r];
      s[1] += red[(w * TOK + tok) * kRedPitch + r + 1];
    }
    const bool two = r0 + r + 1 < op.rows;
    s[0] += to_f32(op.b[r0 + r]);
    if (two) s[1] += to_f32(op.b[r0 + r + 1]);
    const int64_t at = (int64_t)(tok0 + tok) * op.rows + r0 + r;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (q == 1 && !two) break;
      __nv_bfloat16 o = __float2bfloat16_rn(s[q]);
      if (skip != nullptr) o = __float2bfloat16_rn(__bfloat162float(o) + __bfloat162float(skip[at + q]));
      op.out[at + q] = o;
    }
  }
}

template <int TOK, int KEEP>
int launch(const void* x, const void* gamma, const void* beta, float eps, const Operand& first, const Operand& second,
           const void* skip, int64_t N, int K, bool chained, cudaStream_t s) {
  size_t smem = (size_t)kWarps * TOK * kRedPitch * sizeof(float);
  if (KEEP > 0 && smem < (size_t)TOK * staged_pitch(K) * 2) smem = (size_t)TOK * staged_pitch(K) * 2;
  static PerDeviceOnce once;
  int rc = ensure_dynamic_smem(once, linear_rows_kernel<TOK, KEEP>, 160 * 1024);
  if (rc) return rc;
  const dim3 grid((unsigned)((first.rows + kRowsW - 1) / kRowsW + (second.rows + kRowsW - 1) / kRowsW),
                  (unsigned)((N + TOK - 1) / TOK));
  auto p = [](const void* q) { return static_cast<const __nv_bfloat16*>(q); };
  MOE_CUDA_CHECK(launch_pdl(linear_rows_kernel<TOK, KEEP>, grid, dim3(32 * kWarps), smem, s, p(x), p(gamma), p(beta), eps,
                            first, second, p(skip), (int)N, K, chained ? 1 : 0));
  return 0;
}
template <int TOK, typename... Args>
int launch_by_norm(bool norm, int K, Args... args) {
  if (!norm) return launch<TOK, 0>(args...);
  return K <= 1024 ? launch<TOK, 4>(args...) : launch<TOK, 8>(args...);
}

}  // namespace

int launch_linear_rows(const void* x, const void* gamma, const void* beta, float eps, const LinearRows& first,
                       const LinearRows& second, const void* skip, int64_t N, int K, bool chained, cudaStream_t s) {
  auto op = [](const LinearRows& l) {
    return Operand{static_cast<const __nv_bfloat16*>(l.W), static_cast<const __nv_bfloat16*>(l.b),
                   static_cast<__nv_bfloat16*>(l.out), l.rows};
  };
  const Operand a = op(first), b = op(second);
  // 16 tokens a block while their blocks are two an SM at most: the chain of a block is the shorter one
  const int64_t blocks = (first.rows + kRowsW - 1) / kRowsW + (second.rows + kRowsW - 1) / kRowsW;
  if (blocks * ((N + 15) / 16) <= 2 * kNumSMs)
    return launch_by_norm<16>(gamma != nullptr, K, x, gamma, beta, eps, a, b, skip, N, K, chained, s);
  return launch_by_norm<32>(gamma != nullptr, K, x, gamma, beta, eps, a, b, skip, N, K, chained, s);
}

// K up to which the rows kernel keeps rows for their LayerNorm
constexpr int kNormMaxK = 2048;

bool attention_normalises_apart(const AttentionArgs& p) {
  return p.norm_weight != nullptr && (p.B * p.S > kLinearRowsMax || p.hidden > kNormMaxK);
}

namespace {
// Rounds of a launch's blocks (two an SM; one where 32 rows of more than 1024 elements wait in shared memory for their
// LayerNorm) times what a block does, 1 for 16 tokens and K 1024.
double rows_cost(int rows, int rows2, int64_t N, int K, bool norm) {
  const int64_t b = (rows + kRowsW - 1) / kRowsW + (rows2 + kRowsW - 1) / kRowsW;
  const int tok = b * ((N + 15) / 16) <= 2 * kNumSMs ? 16 : 32;
  const int at_once = norm && K > 1024 && K <= kNormMaxK && tok == 32 ? kNumSMs : 2 * kNumSMs;
  return (double)(b * ((N + tok - 1) / tok)) / at_once * tok / 16. * K / 1024.;
}
}  // namespace

// Whether the Linears of an attention are launches of this library or torch's. Up to kLinearRowsMax rows a block reads its
// tokens, and its share of W, once for every 16 or 32 of the others': a small product is over before a library's would have
// begun, a large one is not. 336 sizes (hidden 256 to 4096, 4 to 32 heads, 1 to 128 rows) were timed, LayerNorm to skip connection,
// both ways: up to a cost of 3 none is slower than with torch's Linears (2056, 8 heads, 128 rows: 39.5 us both; 1024, 16 heads, one KV
// head, 37 rows 32 -> 16, 128 rows 38 -> 31), beyond it most are (2048, 32 heads, eight KV heads: 17 rows 33 -> 38, 128 rows 44 ->
// 107), the best left out is 1.2 times as fast. Tiles (323 sizes, 129 to 8192 rows): 0.97 to 1.18 times as fast from 4096 rows on; below,
// 0.93 to 1.15 with K of 1024 to 1536 (1024, 16 heads, 512 rows 32 / 32, 2048 39 -> 37; 520, 8 heads, 129 rows 25 -> 28), but with longer K, where
// few tiles leave the chip idle however K is split, 0.81 to 1.15 (2056, 8 heads, 129 rows 32 -> 40; 4096, 32 heads, 640 rows 62 -> 73).
bool attention_own_linears(int64_t N, int hidden, int q_heads, int kv_heads, int head_dim) {
  const int inner = q_heads * head_dim;
  if (N > kLinearRowsMax) return N >= 4096 || (hidden <= 1536 && inner <= 1536);
  return rows_cost(inner + 2 * kv_heads * head_dim, q_heads, N, hidden, true) <= 3. && rows_cost(hidden, 0, N, inner, false) <= 3.;
}

bool attention_supported(const AttentionArgs& p) {
  const int64_t N = p.B * p.S;
  if (N < 1 || N > (int64_t)1 << 28 || p.S > 128 || p.head_dim != 64 || p.kv_heads < 1 || p.q_heads % p.kv_heads != 0 ||
      (p.hidden & 7) != 0 || p.hidden < 8 || !attention_own_linears(N, p.hidden, p.q_heads, p.kv_heads, p.head_dim))
    return false;
  for (const void* q : {p.x, p.wqkv, p.wgate, p.wo, p.norm_weight, p.norm_bias, p.skip})
    if (!aligned16(q)) return false;
  // as tiles the head gate's rows are stored, and biases loaded, 16 bytes at a time
  return N <= kLinearRowsMax || ((p.q_heads & 7) == 0 && aligned16(p.bqkv) && aligned16(p.bgate) && aligned16(p.bo));
}

int attention_layer(const AttentionArgs& p, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t N = p.B * p.S;
  const LinearRows qkv = {p.wqkv, p.bqkv, p.qkv, (p.q_heads + 2 * p.kv_heads) * p.head_dim};
  const LinearRows gate = {p.wgate, p.bgate, p.gate, p.q_heads}, out = {p.wo, p.bo, p.out, p.hidden}, none = {};
  const int inner = p.q_heads * p.head_dim;
  const bool few = N <= kLinearRowsMax;
  const void *x = p.x, *gamma = p.norm_weight;
  int rc = 0;
  if (attention_normalises_apart(p)) {
    rc = launch_layernorm_rows(x, gamma, p.norm_bias, p.eps, N, p.hidden, MOE_B200_BF16, p.xn, nullptr, s);
    if (rc) return rc;
    x = p.xn;
    gamma = nullptr;
  }
  rc = few ? launch_linear_rows(x, gamma, p.norm_bias, p.eps, qkv, gate, nullptr, N, p.hidden, false, s)
           : launch_linear_tiles(x, qkv, gate, nullptr, N, p.hidden, p.status, s);
  if (rc) return rc;
  rc = launch_attention(p.qkv, p.gate, p.pos_emb, p.mask, p.B, p.S, p.q_heads, p.kv_heads, p.head_dim, p.scaler, p.core, true,
                        s);
  if (rc) return rc;
  return few ? launch_linear_rows(p.core, nullptr, nullptr, 0.f, out, none, p.skip, N, inner, true, s)
             : launch_linear_tiles(p.core, out, none, p.skip, N, inner, p.status, s);
}

}  // namespace moe

using namespace moe;

extern "C" int64_t moe_b200_linear_rows_max(void) { return kLinearRowsMax; }

extern "C" int moe_b200_attention_linears(int64_t N, int hidden, int q_heads, int kv_heads, int head_dim) {
  if (N < 1 || N > (int64_t)1 << 28 || hidden < 8 || hidden > 1 << 24 || q_heads < 1 || kv_heads < 1 || head_dim < 1 ||
      (int64_t)(q_heads + 2 * (int64_t)kv_heads) * head_dim > 1 << 24)
    return 0;
  return attention_own_linears(N, hidden, q_heads, kv_heads, head_dim) ? 1 : 0;
}

extern "C" int moe_b200_linear_rows(const void* x, const void* W, const void* b, int rows, const void* W2, const void* b2,
                                    int rows2, int64_t N, int K, void* out, void* out2, int32_t* status, void* stream) {
  if (N < 0 || N > (int64_t)1 << 28) return set_error(MOE_B200_ERR_SHAPE, "N out of range");
  if (K < 8 || (K & 7) || rows < 1 || rows2 < 0) return set_error(MOE_B200_ERR_SHAPE, "K must be a positive multiple of 8, rows positive");
  if (N == 0) return 0;
  if (!x || !W || !b || !out || !status || (rows2 > 0 && (!W2 || !b2 || !out2)))
    return set_error(MOE_B200_ERR_NULL, "NULL argument");
  if (!aligned16(x) || !aligned16(W) || (rows2 > 0 && !aligned16(W2)))
    return set_error(MOE_B200_ERR_ALIGN, "x and the weights must be 16-byte aligned");
  const LinearRows first = {W, b, out, rows}, second = {W2, b2, out2, rows2};
  if (N <= kLinearRowsMax)
    return launch_linear_rows(x, nullptr, nullptr, 0.f, first, second, nullptr, N, K, false, (cudaStream_t)stream);
  if ((rows & 7) || (rows2 & 7)) return set_error(MOE_B200_ERR_SHAPE, "rows must be multiples of 8 at this N");
  if (!aligned16(b) || !aligned16(out) || (rows2 > 0 && (!aligned16(b2) || !aligned16(out2))))
    return set_error(MOE_B200_ERR_ALIGN, "buffers must be 16-byte aligned");
  return launch_linear_tiles(x, first, second, nullptr, N, K, status, (cudaStream_t)stream);
}
