// Core of the reference's Attention.forward (model.py:96-152) between its two Linears, for
// head_dim 64 and contexts up to 128 tokens, in one kernel:
//   split of the fused QKV projection (model.py:104), KV heads shared by groups of query heads
//   (the repeat_interleave of model.py:112-115 becomes "all heads of a group read the same K/V
//   in shared memory"), RoPE on queries and keys from the model's own table (model.py:123-124,
//   table rows [cos | signed sin] of model.py:14-36), scores = q k^T / sqrt(head_dim) + mask
//   (model.py:127-130), softmax (:131), times V (:132), times the sigmoid head gate (:139-142).
// The [B, H, S, S] score tensor of the reference is never written: a block owns one
// (sequence, KV head) or, where sequences are few, a part of that KV head's query heads. It keeps
// the rotated K and transposed V in shared memory, and each warp runs tiles of 16 queries of one
// head through mma.sync m16n8k16 with the probabilities staying in registers between the two
// products. HBM traffic = QKV in, output out; what bounds it is the trips to shared memory and their latency with
// two blocks an SM. Fragments come by ldmatrix (36 loads an item instead of 144), the position table 16 bytes a
// lane, eight lanes to 128 contiguous bytes, the mask 8 bytes a lane (512 sequences of 64 tokens, 16 heads: 95 -> 80 us).
#include "common.cuh"

namespace moe {

namespace {

constexpr int HD = 64;            // head_dim
constexpr int kMaxS = 128;        // context limit of this kernel
constexpr int kWarpsAtt = 8;

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// four 8 x 8 matrices of 16-bit elements; lanes 8 i .. 8 i + 7 give the row addresses of matrix i
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}

// out[i] = x[i] * pe[i] + x[i ^ 1] * pe[HD + i]: the reference's cat(x, swap_pairs(x)) * pos_emb,
// halves added (model.py:50-57); four consecutive elements at a time, pe 16-byte aligned.
__device__ __forceinline__ uint2 rope4(uint2 x, const float* __restrict__ pe) {
  const float4 p = *reinterpret_cast<const float4*>(pe), q = *reinterpret_cast<const float4*>(pe + HD);
  const float x0 = bf16_lo(x.x), x1 = bf16_hi(x.x), x2 = bf16_lo(x.y), x3 = bf16_hi(x.y);
  return make_uint2(pack_bf16x2(x0 * p.x + x1 * q.x, x1 * p.y + x0 * q.y),
                    pack_bf16x2(x2 * p.z + x3 * q.z, x3 * p.w + x2 * q.w));
}

// Shared memory: K [S][72] bf16 (rotated), Vt [64][S+8] bf16, per warp Q [16][72] bf16,
// pos_emb [S][128] f32, mask [S][S + 8] f32 (optional).
template <int S_TILES>   // ceil(S / 16), 1..8
__global__ void __launch_bounds__(kWarpsAtt * 32)
attention_kernel(const __nv_bfloat16* qkv, const __nv_bfloat16* gate, const float* pos_emb, const float* mask, int S, int H,
                 int KV, float scaler, __nv_bfloat16* __restrict__ out) {
  constexpr int SP = S_TILES * 16;        // padded context
  constexpr int KP = HD + 8;              // K / Q row pitch (bf16): conflict-free fragment loads
  constexpr int VP = SP + 8;              // Vt row pitch
  constexpr int MP = SP + 8;              // mask row pitch: rows 8 or 24 words apart modulo the banks
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(smem_raw);           // [SP][KP]
  __nv_bfloat16* sVt = sK + SP * KP;                                        // [HD][VP]
  __nv_bfloat16* sQ = sVt + HD * VP;                                        // [warps][16][KP]
  float* sPE = reinterpret_cast<float*>(sQ + kWarpsAtt * 16 * KP);          // [SP][2*HD]
  float* sM = sPE + SP * 2 * HD;                                            // [SP][MP] when mask

  const int b = blockIdx.x / KV, kvh = blockIdx.x - b * KV;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int row_elems = (H + 2 * KV) * HD;                   // one token's fused QKV row
  const __nv_bfloat16* base = qkv + (size_t)b * S * row_elems;
  const int heads_per_kv = H / KV;

  // ---- stage the table, the mask, rotated K and transposed V ----
  if ((reinterpret_cast<uintptr_t>(pos_emb) & 15) == 0) {
    for (int i = threadIdx.x; i < SP * 2 * HD / 4; i += blockDim.x) {
      const int r = i / (2 * HD / 4);
      reinterpret_cast<float4*>(sPE)[i] =
          r < S ? reinterpret_cast<const float4*>(pos_emb)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else {      // a table that is a view at an odd place
    for (int i = threadIdx.x; i < SP * 2 * HD; i += blockDim.x) sPE[i] = i < S * 2 * HD ? pos_emb[i] : 0.f;
  }
  if (mask != nullptr)
    for (int i = threadIdx.x; i < SP * SP; i += blockDim.x) {
      const int r = i / SP, c = i - r * SP;
      sM[r * MP + c] = (r < S && c < S) ? mask[r * S + c] : (c < S ? 0.f : -INFINITY);
    }
  // (table and mask are older than the kernel in front, which may still run where this one is its dependent; qkv and gate
  // come from it: ordinary loads behind the wait)
  pdl_wait();
  pdl_launch_dependents();
  __nv_bfloat16* myQ = sQ + warp * 16 * KP;
  // A warp's work: (query head, 16-row tile) items, one in kWarpsAtt of the block's. The rows of
  // the next item and its gate values are requested before the products of the current one, so
  // that a warp always has loads in flight. A lane holds elements 4j and 32 + 4j (j = lane & 7,
  // four of each) of four rows.
  const int per_block = (heads_per_kv + (int)gridDim.y - 1) / (int)gridDim.y;
  const int head0 = (int)blockIdx.y * per_block;
  const int items = max(0, min(per_block, heads_per_kv - head0)) * S_TILES;
  const int lc = (lane & 7) * 4;
  const uint2 zero2 = make_uint2(0u, 0u);
  auto fetch = [&](int item, uint2 (&raw)[8], float& ga, float& gb) {
    const int h = kvh * heads_per_kv + head0 + item / S_TILES, mt = item % S_TILES;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int s = mt * 16 + (lane >> 3) + 4 * q;
      const __nv_bfloat16* p = base + (size_t)s * row_elems + h * HD + lc;
      raw[2 * q] = s < S ? __ldcg(reinterpret_cast<const uint2*>(p)) : zero2;
      raw[2 * q + 1] = s < S ? __ldcg(reinterpret_cast<const uint2*>(p + 32)) : zero2;
    }
    const int r0 = mt * 16 + g;
    ga = r0 < S ? __bfloat162float(gate[((size_t)b * S + r0) * H + h]) : 0.f;
    gb = r0 + 8 < S ? __bfloat162float(gate[((size_t)b * S + r0 + 8) * H + h]) : 0.f;
  };
  uint2 raw[8];
  float gate_a = 0.f, gate_b = 0.f;
  if (warp < items) fetch(warp, raw, gate_a, gate_b);
  __syncthreads();
  for (int i = threadIdx.x; i < SP * (HD / 4); i += blockDim.x) {
    const int s = i / (HD / 4), c = (i - s * (HD / 4)) * 4;
    uint2 k4 = make_uint2(0u, 0u), v4 = make_uint2(0u, 0u);
    if (s < S) {
      k4 = __ldcg(reinterpret_cast<const uint2*>(base + (size_t)s * row_elems + (H + kvh) * HD + c));
      v4 = __ldcg(reinterpret_cast<const uint2*>(base + (size_t)s * row_elems + (H + KV + kvh) * HD + c));
      k4 = rope4(k4, sPE + s * 2 * HD + c);
    }
    *reinterpret_cast<uint2*>(sK + s * KP + c) = k4;
    const __nv_bfloat16* v = reinterpret_cast<const __nv_bfloat16*>(&v4);
#pragma unroll
    for (int q = 0; q < 4; ++q) sVt[(c + q) * VP + s] = v[q];
  }
  __syncthreads();

  for (int item = warp; item < items; item += kWarpsAtt) {
    {
      const int h = kvh * heads_per_kv + head0 + item / S_TILES, mt = item % S_TILES;
      // ---- 16 query rows of this head, rotated, into the warp's staging area ----
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int sl = (lane >> 3) + 4 * q;
        const float* pe = sPE + (mt * 16 + sl) * 2 * HD + lc;      // zeros behind the last row
        *reinterpret_cast<uint2*>(myQ + sl * KP + lc) = rope4(raw[2 * q], pe);
        *reinterpret_cast<uint2*>(myQ + sl * KP + lc + 32) = rope4(raw[2 * q + 1], pe + 32);
      }
      const float cur_ga = gate_a, cur_gb = gate_b;
      if (item + kWarpsAtt < items) fetch(item + kWarpsAtt, raw, gate_a, gate_b);
      __syncwarp();
      // ---- scores of 16 query rows against all keys ----
      float sc[2 * S_TILES][4];
#pragma unroll
      for (int n = 0; n < 2 * S_TILES; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[n][i] = 0.f;
#pragma unroll
      for (int kk = 0; kk < HD / 16; ++kk) {
        uint32_t a[4];
        ldmatrix_x4(a, myQ + (lane & 15) * KP + kk * 16 + (lane >> 4) * 8);
#pragma unroll
        for (int n = 0; n < 2 * S_TILES; n += 2) {
          uint32_t kb[4];      // k and k + 8 of keys 8 n .., then of keys 8 n + 8 ..
          ldmatrix_x4(kb, sK + (n * 8 + (lane >> 4) * 8 + (lane & 7)) * KP + kk * 16 + ((lane >> 3) & 1) * 8);
          mma16816(sc[n], a[0], a[1], a[2], a[3], kb[0], kb[1]);
          mma16816(sc[n + 1], a[0], a[1], a[2], a[3], kb[2], kb[3]);
        }
      }
      // ---- scale, mask, softmax over the keys (rows g and g + 8 of the tile) ----
      const int r0 = mt * 16 + g, r1 = r0 + 8;
      float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
      for (int n = 0; n < 2 * S_TILES; ++n) {
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[n][i] *= scaler;
        const int col = n * 8 + 2 * t;
        if (mask != nullptr) {
          const float2 ma = *reinterpret_cast<const float2*>(sM + r0 * MP + col);
          const float2 mb = *reinterpret_cast<const float2*>(sM + r1 * MP + col);
          sc[n][0] += ma.x; sc[n][1] += ma.y;
          sc[n][2] += mb.x; sc[n][3] += mb.y;
        } else {
          if (col >= S) sc[n][0] = sc[n][2] = -INFINITY;
          if (col + 1 >= S) sc[n][1] = sc[n][3] = -INFINITY;
        }
        m0 = fmaxf(m0, fmaxf(sc[n][0], sc[n][1]));
        m1 = fmaxf(m1, fmaxf(sc[n][2], sc[n][3]));
      }
#pragma unroll
      for (int o = 1; o <= 2; o <<= 1) {
        m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, o));
        m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
      }
      float l0 = 0.f, l1 = 0.f;
#pragma unroll
      for (int n = 0; n < 2 * S_TILES; ++n) {
        sc[n][0] = __expf(sc[n][0] - m0); sc[n][1] = __expf(sc[n][1] - m0);
        sc[n][2] = __expf(sc[n][2] - m1); sc[n][3] = __expf(sc[n][3] - m1);
        l0 += sc[n][0] + sc[n][1];
        l1 += sc[n][2] + sc[n][3];
      }
#pragma unroll
      for (int o = 1; o <= 2; o <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, o);
        l1 += __shfl_xor_sync(0xffffffffu, l1, o);
      }
      const float inv0 = 1.f / l0, inv1 = 1.f / l1;
      // ---- probabilities (bf16, straight from the accumulator registers) times V ----
      float o_acc[HD / 8][4];
#pragma unroll
      for (int n = 0; n < HD / 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) o_acc[n][i] = 0.f;
#pragma unroll
      for (int kk = 0; kk < S_TILES; ++kk) {
        const uint32_t a0 = pack_bf16x2(sc[2 * kk][0] * inv0, sc[2 * kk][1] * inv0);
        const uint32_t a1 = pack_bf16x2(sc[2 * kk][2] * inv1, sc[2 * kk][3] * inv1);
        const uint32_t a2 = pack_bf16x2(sc[2 * kk + 1][0] * inv0, sc[2 * kk + 1][1] * inv0);
        const uint32_t a3 = pack_bf16x2(sc[2 * kk + 1][2] * inv1, sc[2 * kk + 1][3] * inv1);
#pragma unroll
        for (int n = 0; n < HD / 8; n += 2) {
          uint32_t vb[4];
          ldmatrix_x4(vb, sVt + (n * 8 + (lane >> 4) * 8 + (lane & 7)) * VP + kk * 16 + ((lane >> 3) & 1) * 8);
          mma16816(o_acc[n], a0, a1, a2, a3, vb[0], vb[1]);
          mma16816(o_acc[n + 1], a0, a1, a2, a3, vb[2], vb[3]);
        }
      }
      // ---- sigmoid head gate (model.py:139-142); the tile leaves through the warp's staging
      // area (free since the score products) as 128-byte runs per row ----
      const float g0 = 1.f / (1.f + __expf(-cur_ga)), g1 = 1.f / (1.f + __expf(-cur_gb));
      __syncwarp();
#pragma unroll
      for (int n = 0; n < HD / 8; ++n) {
        *reinterpret_cast<uint32_t*>(myQ + g * KP + n * 8 + 2 * t) = pack_bf16x2(o_acc[n][0] * g0, o_acc[n][1] * g0);
        *reinterpret_cast<uint32_t*>(myQ + (g + 8) * KP + n * 8 + 2 * t) = pack_bf16x2(o_acc[n][2] * g1, o_acc[n][3] * g1);
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = lane + 32 * q;
        const int sl = i >> 3, c = (i & 7) * 8;
        const int srow = mt * 16 + sl;
        if (srow < S)
          *reinterpret_cast<uint4*>(out + ((size_t)b * S + srow) * H * HD + h * HD + c) =
              *reinterpret_cast<const uint4*>(myQ + sl * KP + c);
      }
    }
  }
}

template <int ST>
int launch_att(const void* qkv, const void* gate, const float* pos_emb, const float* mask, int B, int S,
               int H, int KV, float scaler, void* out, bool chained, cudaStream_t s) {
  constexpr int SP = ST * 16;
  const size_t smem = (size_t)(SP * (HD + 8) + HD * (SP + 8) + kWarpsAtt * 16 * (HD + 8)) * 2 +
                      (size_t)SP * 2 * HD * 4 + (mask != nullptr ? (size_t)SP * (SP + 8) * 4 : 0);
  static PerDeviceOnce once;
  int rc = ensure_dynamic_smem(once, attention_kernel<ST>, 227 * 1024);
  if (rc) return rc;
  if (smem > 227 * 1024) return set_error(MOE_B200_ERR_UNSUPPORTED, "context too long for the shared-memory layout");
  // fewer blocks than fit at once (two an SM): a KV head's query heads over several blocks, down to one
  // head each; every block stages K and V for itself (one sequence of 37 tokens, 16 heads: 22 us on one SM,
  // 8 us on sixteen)
  const int64_t blocks = (int64_t)B * KV, heads = H / KV;
  const int64_t want = blocks < 2 * kNumSMs ? (2 * kNumSMs + blocks - 1) / blocks : 1;
  const dim3 grid((unsigned)blocks, (unsigned)(want < heads ? want : heads));
  const __nv_bfloat16 *q = static_cast<const __nv_bfloat16*>(qkv), *gt = static_cast<const __nv_bfloat16*>(gate);
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
  if (chained) {
    MOE_CUDA_CHECK(launch_pdl(attention_kernel<ST>, grid, dim3(kWarpsAtt * 32), smem, s, q, gt, pos_emb, mask, S, H, KV,
                              scaler, o));
    return 0;
  }
  attention_kernel<ST><<<grid, kWarpsAtt * 32, smem, s>>>(q, gt, pos_emb, mask, S, H, KV, scaler, o);
  MOE_CUDA_CHECK(cudaGetLastError());
  return 0;
}

}  // namespace


int launch_attention(const void* qkv, const void* gate, const float* pos_emb, const float* mask, int64_t B, int S, int q_heads,
                     int kv_heads, int head_dim, float scaler, void* out, bool chained, cudaStream_t s) {
  if (head_dim != HD) return set_error(MOE_B200_ERR_UNSUPPORTED, "head_dim must be 64");
  if (S < 1 || S > kMaxS) return set_error(MOE_B200_ERR_UNSUPPORTED, "context must be in [1,128]");
  if (B < 0 || B > (1 << 24) || q_heads < 1 || kv_heads < 1 || q_heads % kv_heads != 0)
    return set_error(MOE_B200_ERR_SHAPE, "B or head counts out of range");
  if (B == 0) return 0;
  if (!qkv || !gate || !pos_emb || !out) return set_error(MOE_B200_ERR_NULL, "NULL argument");
  if (!aligned16(qkv) || !aligned16(out)) return set_error(MOE_B200_ERR_ALIGN, "buffers must be 16-byte aligned");
  switch ((S + 15) / 16) {
    case 1: return launch_att<1>(qkv, gate, pos_emb, mask, (int)B, S, q_heads, kv_heads, scaler, out, chained, s);
    case 2: return launch_att<2>(qkv, gate, pos_emb, mask, (int)B, S, q_heads, kv_heads, scaler, out, chained, s);
    case 3: return launch_att<3>(qkv, gate, pos_emb, mask, (int)B, S, q_heads, kv_heads, scaler, out, chained, s);
    case 4: return launch_att<4>(qkv, gate, pos_emb, mask, (int)B, S, q_heads, kv_heads, scaler, out, chained, s);
    case 5: return launch_att<5>(qkv, gate, pos_emb, mask, (int)B, S, q_heads, kv_heads, scaler, out, chained, s);
    case 6: return launch_att<6>(qkv, gate, pos_emb, mask, (int)B, S, q_heads, kv_heads, scaler, out, chained, s);
    case 7: return launch_att<7>(qkv, gate, pos_emb, mask, (int)B, S, q_heads, kv_heads, scaler, out, chained, s);
    default: return launch_att<8>(qkv, gate, pos_emb, mask, (int)B, S, q_heads, kv_heads, scaler, out, chained, s);
  }
}

}  // namespace moe

using namespace moe;

extern "C" int moe_b200_attention(const void* qkv, const void* gate, const float* pos_emb,
                                  const float* mask, int64_t B, int S, int q_heads, int kv_heads,
                                  int head_dim, float scaler, void* out, void* stream) {
  return launch_attention(qkv, gate, pos_emb, mask, B, S, q_heads, kv_heads, head_dim, scaler, out, false,
                          (cudaStream_t)stream);
}
