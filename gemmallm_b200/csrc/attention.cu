// Core of the reference's Attention.forward (model.py:96-152) between its two Linears, for
// head_dim 64 and contexts up to 128 tokens, in one kernel:
//   split of the fused QKV projection (model.py:104), KV heads shared by groups of query heads
//   (the repeat_interleave of model.py:112-115 becomes "all heads of a group read the same K/V
//   in shared memory"), RoPE on queries and keys from the model's own table (model.py:123-124,
//   table rows [cos | signed sin] of model.py:14-36), scores = q k^T / sqrt(head_dim) + mask
//   (model.py:127-130), softmax (:131), times V (:132), times the sigmoid head gate (:139-142).
// The [B, H, S, S] score tensor of the reference is never written: a block keeps the rotated K and transposed V of one
// (sequence, KV head) in shared memory, and each warp runs tiles of 16 queries of one
// head through mma.sync m16n8k16 with the probabilities staying in registers between the two
// products. HBM traffic = QKV in, output out; what bounds it is the trips to shared memory and their latency with
// two blocks an SM. Fragments come by ldmatrix (36 loads an item instead of 144), the position table 16 bytes a
// lane, the mask 8 bytes a lane; queries and outputs do not go through shared memory. (Three blocks an SM, which then fit,
// took longer: 110 us in that trace.)
// A block takes an equal share of all rounds of eight tiles, whatever sequence they are of, and stages table and mask once
// (a block a sequence: 512 sequences were 1.7 waves of blocks, and took two). Sequences of 64 tokens, 16 heads, queries and outputs
// through shared memory before: 512 of them 79.7 -> 71.1 us, 100 25.9 -> 20.6 (behind the QKV product, in a trace: 99 -> 89.6 and
// 30 -> 26.6).
#include "common.cuh"

namespace moe {

namespace {

constexpr int HD = 64;            // head_dim
constexpr int kMaxS = 128;        // context limit of this kernel
constexpr int kWarpsAtt = 8;
constexpr int kTablePitch = 2 * HD + 4;      // floats: rows 16 bytes apart modulo the banks

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

// Of every 32 columns a lane of a tile's row has eight neighbouring ones, 16 bytes from memory and to memory: as operands of two
// products its four pairs are the contraction indices 2 t, 2 t + 8 of the first and of the second, as results they are its
// columns of four tiles. K's columns and V's lie in shared memory in that order.
// place of column c of K in its row (a product's indices side by side), and row of column c of V in Vt
__device__ __forceinline__ int k_place(int c) {
  return (c & 32) + ((c >> 2) & 1) * 16 + ((c >> 1) & 1) * 8 + ((c >> 3) & 3) * 2 + (c & 1);
}
__device__ __forceinline__ int v_place(int c) { return (c & 32) + ((c >> 1) & 3) * 8 + ((c >> 3) & 3) * 2 + (c & 1); }

template <int S_TILES>
constexpr int kPerSM = S_TILES <= 6 ? 2 : 1;      // blocks, as registers allow

// Shared memory: K [S][72] bf16 (rotated), Vt [64][S+8] bf16, pos_emb [S][132] f32, mask [S][S + 8] f32 (optional).
template <int S_TILES>   // ceil(S / 16), 1..8
__global__ void __launch_bounds__(kWarpsAtt * 32, kPerSM<S_TILES>)
attention_kernel(const __nv_bfloat16* qkv, const __nv_bfloat16* gate, const float* pos_emb, const float* mask, int S, int H,
                 int KV, float scaler, __nv_bfloat16* __restrict__ out, int share, int extra, int at_once, int each) {
  constexpr int SP = S_TILES * 16;        // padded context
  constexpr int KP = HD + 8;              // K row pitch (bf16): conflict-free fragment loads
  constexpr int VP = SP + 8;              // Vt row pitch
  constexpr int PP = kTablePitch;
  constexpr int MP = SP + 8;              // mask row pitch: rows 8 or 24 words apart modulo the banks
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(smem_raw);           // [SP][KP]
  __nv_bfloat16* sVt = sK + SP * KP;                                        // [HD][VP]
  float* sPE = reinterpret_cast<float*>(sVt + HD * VP);                     // [SP][PP]
  float* sM = sPE + SP * PP;                                                // [SP][MP] when mask

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int row_elems = (H + 2 * KV) * HD;                   // one token's fused QKV row
  const int heads_per_kv = H / KV;

  // ---- stage the table and the mask ----
  if ((reinterpret_cast<uintptr_t>(pos_emb) & 15) == 0) {
    for (int i = threadIdx.x; i < SP * 2 * HD / 4; i += blockDim.x) {
      const int r = i / (2 * HD / 4);
      reinterpret_cast<float4*>(sPE)[i + r * ((PP - 2 * HD) / 4)] =
          r < S ? reinterpret_cast<const float4*>(pos_emb)[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  } else {      // a table that is a view at an odd place
    for (int i = threadIdx.x; i < SP * 2 * HD; i += blockDim.x)
      sPE[i + i / (2 * HD) * (PP - 2 * HD)] = i < S * 2 * HD ? pos_emb[i] : 0.f;
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
  // A warp's work: (query head, 16-row tile) items of a (sequence, KV head), an item of each of the block's rounds. The rows
  // of the next item and its gate values are requested before the products of the current one, so
  // that a warp always has loads in flight. A lane holds eight elements from 8 t and from 32 + 8 t on
  // of rows g and g + 8.
  const int items = heads_per_kv * S_TILES;      // of a (sequence, KV head), in `each` rounds
  const int first = share * (int)blockIdx.x + min((int)blockIdx.x, extra), last = first + share + ((int)blockIdx.x < extra ? 1 : 0);
  const uint2 zero2 = make_uint2(0u, 0u);
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  auto fetch = [&](int unit, int item, uint4 (&raw)[2][2], float& ga, float& gb) {
    const int b = unit / KV, kvh = unit - b * KV;
    const __nv_bfloat16* base = qkv + (size_t)b * S * row_elems;
    const int h = kvh * heads_per_kv + item / S_TILES, mt = item % S_TILES;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int s = mt * 16 + g + 8 * q;
      const __nv_bfloat16* p = base + (size_t)s * row_elems + h * HD + 8 * t;
      raw[q][0] = s < S ? __ldcg(reinterpret_cast<const uint4*>(p)) : zero4;
      raw[q][1] = s < S ? __ldcg(reinterpret_cast<const uint4*>(p + 32)) : zero4;
    }
    const int r0 = mt * 16 + g;
    ga = r0 < S ? __bfloat162float(gate[((size_t)b * S + r0) * H + h]) : 0.f;
    gb = r0 + 8 < S ? __bfloat162float(gate[((size_t)b * S + r0 + 8) * H + h]) : 0.f;
  };
  uint4 raw[2][2];
  float gate_a = 0.f, gate_b = 0.f;
  int unit = first / each, turn = first - unit * each;      // of the round at hand: (sequence, KV head); the how manieth there
  bool staged = false;
  const bool works = warp < at_once;
  if (works && turn * at_once + warp < items) fetch(unit, turn * at_once + warp, raw, gate_a, gate_b);
  for (int round = first; round < last; ++round) {
    const int b = unit / KV, kvh = unit - b * KV;
    if (!staged) {      // rotated K and transposed V
      const __nv_bfloat16* base = qkv + (size_t)b * S * row_elems;
      __syncthreads();      // (the table is there; no warp needs the last ones any more)
      for (int i = threadIdx.x; i < SP * (HD / 4); i += blockDim.x) {
        const int s = i / (HD / 4), c = (i - s * (HD / 4)) * 4;
        uint2 k4 = zero2, v4 = zero2;
        if (s < S) {
          k4 = __ldcg(reinterpret_cast<const uint2*>(base + (size_t)s * row_elems + (H + kvh) * HD + c));
          v4 = __ldcg(reinterpret_cast<const uint2*>(base + (size_t)s * row_elems + (H + KV + kvh) * HD + c));
          k4 = rope4(k4, sPE + s * PP + c);
        }
        *reinterpret_cast<uint32_t*>(sK + s * KP + k_place(c)) = k4.x;
        *reinterpret_cast<uint32_t*>(sK + s * KP + k_place(c + 2)) = k4.y;
        const __nv_bfloat16* v = reinterpret_cast<const __nv_bfloat16*>(&v4);
#pragma unroll
        for (int q = 0; q < 4; ++q) sVt[v_place(c + q) * VP + s] = v[q];
      }
      __syncthreads();
      staged = true;
    }
    const int item = turn * at_once + warp;
    const int next_turn = turn + 1 < each ? turn + 1 : 0, next_unit = next_turn > 0 ? unit : unit + 1;
    const int next_item = next_turn * at_once + warp;
    const bool more = works && round + 1 < last && next_item < items;
    if (works && item < items) {
      const int h = kvh * heads_per_kv + item / S_TILES, mt = item % S_TILES;
      // ---- 16 query rows of this head, rotated ----
      uint32_t qa[HD / 16][4];
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float* pe = sPE + (mt * 16 + g + 8 * q) * PP + 32 * c + 8 * t;      // zeros behind the last row
          const uint2 lo = rope4(make_uint2(raw[q][c].x, raw[q][c].y), pe);
          const uint2 hi = rope4(make_uint2(raw[q][c].z, raw[q][c].w), pe + 4);
          qa[2 * c][q] = lo.x;
          qa[2 * c][2 + q] = lo.y;
          qa[2 * c + 1][q] = hi.x;
          qa[2 * c + 1][2 + q] = hi.y;
        }
      const float cur_ga = gate_a, cur_gb = gate_b;
      if (more) fetch(next_unit, next_item, raw, gate_a, gate_b);
      // ---- scores of 16 query rows against all keys ----
      float sc[2 * S_TILES][4];
#pragma unroll
      for (int n = 0; n < 2 * S_TILES; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[n][i] = 0.f;
#pragma unroll
      for (int kk = 0; kk < HD / 16; ++kk) {
        const uint32_t (&a)[4] = qa[kk];
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
      uint32_t pr[S_TILES][4];
#pragma unroll
      for (int kk = 0; kk < S_TILES; ++kk) {
        pr[kk][0] = pack_bf16x2(sc[2 * kk][0] * inv0, sc[2 * kk][1] * inv0);
        pr[kk][1] = pack_bf16x2(sc[2 * kk][2] * inv1, sc[2 * kk][3] * inv1);
        pr[kk][2] = pack_bf16x2(sc[2 * kk + 1][0] * inv0, sc[2 * kk + 1][1] * inv0);
        pr[kk][3] = pack_bf16x2(sc[2 * kk + 1][2] * inv1, sc[2 * kk + 1][3] * inv1);
      }
      float o_acc[HD / 8][4];
#pragma unroll
      for (int n = 0; n < HD / 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) o_acc[n][i] = 0.f;
#pragma unroll
      for (int kk = 0; kk < S_TILES; ++kk) {
#pragma unroll
        for (int n = 0; n < HD / 8; n += 2) {
          uint32_t vb[4];
          ldmatrix_x4(vb, sVt + (n * 8 + (lane >> 4) * 8 + (lane & 7)) * VP + kk * 16 + ((lane >> 3) & 1) * 8);
          mma16816(o_acc[n], pr[kk][0], pr[kk][1], pr[kk][2], pr[kk][3], vb[0], vb[1]);
          mma16816(o_acc[n + 1], pr[kk][0], pr[kk][1], pr[kk][2], pr[kk][3], vb[2], vb[3]);
        }
      }
      // ---- sigmoid head gate (model.py:139-142); 64 contiguous bytes a row and store ----
      const float g0 = 1.f / (1.f + __expf(-cur_ga)), g1 = 1.f / (1.f + __expf(-cur_gb));
      __nv_bfloat16* to = out + ((size_t)b * S + r0) * H * HD + h * HD + 8 * t;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          lo[j] = pack_bf16x2(o_acc[4 * c + j][0] * g0, o_acc[4 * c + j][1] * g0);
          hi[j] = pack_bf16x2(o_acc[4 * c + j][2] * g1, o_acc[4 * c + j][3] * g1);
        }
        if (r0 < S) *reinterpret_cast<uint4*>(to + 32 * c) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        if (r1 < S) *reinterpret_cast<uint4*>(to + (size_t)8 * H * HD + 32 * c) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      }
    } else if (more) {
      fetch(next_unit, next_item, raw, gate_a, gate_b);
    }
    staged = next_turn > 0;
    unit = next_unit;
    turn = next_turn;
  }
}

template <int ST>
int launch_att(const void* qkv, const void* gate, const float* pos_emb, const float* mask, int B, int S,
               int H, int KV, float scaler, void* out, bool chained, cudaStream_t s) {
  constexpr int SP = ST * 16;
  const size_t smem = (size_t)(SP * (HD + 8) + HD * (SP + 8)) * 2 + (size_t)SP * kTablePitch * 4 +
                      (mask != nullptr ? (size_t)SP * (SP + 8) * 4 : 0);
  static PerDeviceOnce once;
  int rc = ensure_dynamic_smem(once, attention_kernel<ST>, 227 * 1024);
  if (rc) return rc;
  if (smem > 227 * 1024) return set_error(MOE_B200_ERR_UNSUPPORTED, "context too long for the shared-memory layout");
  // rounds of eight items, of fewer where they would leave most SMs without any (one sequence of 37 tokens, 16 heads: 22 us on one
  // SM, 8 us on sixteen)
  const int64_t units = (int64_t)B * KV;
  const int items = H / KV * ST;
  int at_once = kWarpsAtt;
  while (at_once > 2 && units * ((items + at_once - 1) / at_once) * 4 <= kNumSMs) at_once /= 2;
  const int each = (items + at_once - 1) / at_once;
  // (of 81 to 96 tokens two fit without a mask only: 500 sequences of 81, 8 heads, two KV heads 99.5 us with one block an SM, 71.7 with two)
  const int64_t rounds = units * each, most = (int64_t)(2 * (smem + 1024) <= 228 * 1024 ? kPerSM<ST> : 1) * kNumSMs;
  if (rounds >= (int64_t)1 << 31) return set_error(MOE_B200_ERR_SHAPE, "too many sequences");
  const dim3 grid((unsigned)(rounds < most ? rounds : most));
  // (divided here: in the kernel it took 0.5 us)
  const int share = (int)(rounds / grid.x), extra = (int)(rounds - (int64_t)share * grid.x);
  const __nv_bfloat16 *q = static_cast<const __nv_bfloat16*>(qkv), *gt = static_cast<const __nv_bfloat16*>(gate);
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
  if (chained) {
    MOE_CUDA_CHECK(launch_pdl(attention_kernel<ST>, grid, dim3(kWarpsAtt * 32), smem, s, q, gt, pos_emb, mask, S, H, KV,
                              scaler, o, share, extra, at_once, each));
    return 0;
  }
  attention_kernel<ST><<<grid, kWarpsAtt * 32, smem, s>>>(q, gt, pos_emb, mask, S, H, KV, scaler, o, share, extra, at_once, each);
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
