// Router and dispatch of a small call in ONE launch: with at most a few hundred
// tokens the separate router and cooperative dispatch kernels are pure launch
// and barrier latency (13 + 19 us against a few us of work). A few blocks run;
// each one derives the complete routing by itself (the same instructions on the
// same data, so every block gets the same answer and no grid barrier is needed),
// block 0 writes the routing results, and the row copies are split over the blocks.
// Covers reference model.py:206-253 for N <= 512, N*k <= 1024, E <= 32, bf16 (fp32, whose blocks share the work: up to 2048
// tokens):
//   A. logits: 32 warps = (16-token group) x (slice of K); each warp forms its
//      partial x Wg^T with mma.sync m16n8k16 exactly like router_mma_kernel
//      (router.cu), all its loads in flight at once; partials are summed over
//      the K slices in slice order, plus bias. fp32: a thread per (token,
//      expert mod 8, slice of K), eight sums of every eighth element there;
//   B. 8, 16 or 32 lanes per token, lane e = expert e: fp32 softmax, k passes of
//      arg-max ordered by (logit desc, index asc) with shuffle reductions
//      on order-preserving keys, renormalise;
//   C. warp 0: per-slot counts, offsets (scan over E), stable ranks in (token,
//      slot) order; then row copies into the sorted buffer with 16-byte accesses
//      (their loads were issued before B; fp32: also as planes, three bf16 parts of every value, [3][N k][d]);
//   E. block 0: probabilities summed per expert in token order; loss.
#pragma once
#include <cooperative_groups.h>
#include "common.cuh"

namespace moe {

constexpr int kFrontThreads = 1024;
constexpr int kFrontMaxTok = 512;
constexpr int kFrontMaxE = 32;
constexpr int kFrontMaxPairs = 1024;

namespace front_detail {

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                               uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

}  // namespace front_detail

using front_detail::mma_bf16_16816;

// bf16: every block derives the complete routing (fastest up to about a hundred tokens; beyond, front_mid_kernel in
//   front_small.cu).
// fp32 (SPLIT): block b routes tokens per*b .. per*b+per-1 only (at most 16); the blocks then exchange their per-slot
//   expert counts and probability sums through `xch` and meet at a grid barrier (a cooperative launch, as the dispatch kernel's
//   that these calls took before; the launch, not the barrier, costs 2.3 us of a call of 512 tokens, 101.3 us without),
//   and each block places and copies its own rows.
// `smem`: front_small_smem_bytes() of shared memory.
// The partial logits' area also takes the blocks' probability sums (SPLIT, up to 128 blocks) once the logits are summed.
// fp32: behind the rest, kFrontChunk elements of K of 16 tokens and 8 NT experts.
template <int NT>
constexpr int kFrontChunk = NT == 1 ? 512 : 256;
constexpr int kFrontPad = 4;        // floats: rows 16 bytes apart modulo the banks
__host__ __device__ inline size_t front_small_smem_bytes(int NT, int ntok, int E, int k) {
  return sizeof(float) * ((size_t)32 * 16 * 8 * NT + (size_t)ntok * (E + 1)) +
         sizeof(int) * (2 * (size_t)ntok * k + 2 * kMaxTopK * kFrontMaxE + 4 * kFrontMaxE + 1);
}
__host__ __device__ constexpr size_t front_f32_chunk_bytes(int NT) {
  return (size_t)(16 + 8 * NT) * ((NT == 1 ? 512 : 256) + kFrontPad) * sizeof(float) + 16;
}

template <int NT, typename T>  // n-tiles of 8 experts: E <= 8*NT
__device__ __forceinline__ void front_small_body(float* smem,
                 const T* __restrict__ x, const T* Wg, const T* bg, int Ntotal, int d, int E, int k,
                 float* __restrict__ out_logits, int32_t* __restrict__ out_idx,
                 float* __restrict__ out_w, int32_t* __restrict__ cnt_slot,
                 int32_t* __restrict__ offsets, int32_t* __restrict__ row_of,
                 T* __restrict__ perm, __nv_bfloat16* __restrict__ planes, float* __restrict__ psum,
                 float* __restrict__ aux, int* __restrict__ xch, int32_t* __restrict__ status, int per) {
  constexpr int kThreads = kFrontThreads;
  constexpr int kMaxE = kFrontMaxE;
  constexpr bool F32 = sizeof(T) == 4, SPLIT = F32;
  const int blk = (int)blockIdx.x, nblk = (int)gridDim.x;
  constexpr int kPiece = 16 / sizeof(T);                   // elements of a 16-byte piece
  const int ld = E + 1;
  // SPLIT: this block's tokens are "the problem" for the phases A and B below
  const int tok_base = SPLIT ? per * blk : 0;
  const int N = SPLIT ? min(per, Ntotal - tok_base) : Ntotal;
  const bool writer = SPLIT || blk == 0;     // this block writes the per-token results
  if (SPLIT) {
    x += (size_t)tok_base * d;
    if (out_logits != nullptr) out_logits += (size_t)tok_base * E;
    out_idx += (size_t)tok_base * k;
    out_w += (size_t)tok_base * k;
    row_of += (size_t)tok_base * k;
  }
  const int ngroups = (N + 15) >> 4;                       // 16-token groups
  int gp2 = 1;
  while (gp2 < ngroups) gp2 <<= 1;                         // 1, 2, 4 or 8
  // fp32: a warp has four tokens; 1, 2 or 4 of them side by side
  const int tg4 = per <= 4 ? 1 : per <= 8 ? 2 : 4;
  const int nslices = F32 ? 32 / tg4 : 32 / gp2;           // K slices
  const int tok_pitch = F32 ? 4 * tg4 : 16 * gp2;          // tokens of a slice
  float* s_part = smem;                                    // [nslices][tok_pitch][8*NT]
  float* s_logit = s_part + (size_t)nslices * tok_pitch * 8 * NT;   // [N][E+1]
  int* s_idx = reinterpret_cast<int*>(s_logit + (size_t)N * ld);   // [N*k]
  int* s_row = s_idx + N * k;                              // [N*k]
  int* s_cnt = s_row + N * k;                              // [kMaxTopK][kMaxE]
  int* s_off = s_cnt + kMaxTopK * kMaxE;                   // [kMaxE+1]
  int* s_run = s_off + kMaxE + 1;                          // [kMaxE]
  float* s_bias = reinterpret_cast<float*>(s_run + kMaxE); // [kMaxE], then s_base, s_tot (SPLIT)

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  constexpr int ET_C = 8 * NT;
  const int ET = ET_C;
  // (the router's weights and biases may have been written by the kernel before this one: ordinary loads behind the wait,
  // and no __restrict__, which would make them loads of constant data)
  if (tid < E) s_bias[tid] = to_f32(bg[tid]);   // visible after the barrier behind part A

  // ---- A. partial logits -----------------------------------------------------
  if constexpr (F32) {
    // A chunk of K of the block's tokens and of all experts is brought to shared memory, all its loads in flight at once
    // (read where they lie, 16 bytes at a time, they took 9.7 us of this kernel's 17 at d 512; a call of 512
    // tokens 102.5 -> 94.7). Lane = (token
    // of four, expert mod 8), warps also take a slice of K each: its pieces in order, even and odd places apart.
    constexpr int KC = kFrontChunk<NT>, KP = KC + kFrontPad;
    const int tok = (warp % tg4) * 4 + (lane >> 3), e0 = lane & 7, ks = warp / tg4;
    const int n4 = d >> 2, each = (n4 + nslices - 1) / nslices;
    float* s_x = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(smem) + front_small_smem_bytes(NT, per, E, k) + 15) &
                                          ~(uintptr_t)15);          // [16][KP], then [8 NT][KP]
    float* s_w = s_x + 16 * KP;
    // a chunk holds the same part of every slice
    const int step = KC / 4 / nslices;
    float4 acc[2][NT];       // pieces of even and of odd place
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
#pragma unroll
      for (int j = 0; j < NT; ++j) acc[hh][j] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c0 = 0; c0 < each; c0 += step) {
      if (c0 > 0) __syncthreads();
      const int rows = N + min(8 * NT, E);
      for (int i = tid; i < rows * (KC / 4); i += kThreads) {
        const int r = i / (KC / 4), q = i - r * (KC / 4);
        const int slice = q / step, c = slice * each + c0 + (q - slice * step);     // piece of the row
        const bool ok = c0 + (q - slice * step) < each && c < n4;
        const T* src = r < N ? x + (size_t)r * d : Wg + (size_t)(r - N) * d;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared((r < N ? s_x + r * KP : s_w + (r - N) * KP) + q * 4);
        if (ok)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + (size_t)c * 4) : "memory");
      }
      asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      const int n = min(step, min(each - c0, n4 - (ks * each + c0)));
      const float4* xr = reinterpret_cast<const float4*>(s_x + tok * KP) + ks * step;
      const float4* wr = reinterpret_cast<const float4*>(s_w) + ks * step;
#pragma unroll 4
      for (int c = 0; c < n; ++c) {
        const float4 v = xr[c];
        // (a chunk has an even number of pieces of a slice: even places stay even)
        float4 (&s)[NT] = acc[c & 1];
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const float4 w = wr[min(8 * j + e0, E - 1) * (KP / 4) + c];
          s[j].x = fmaf(v.x, w.x, s[j].x);
          s[j].y = fmaf(v.y, w.y, s[j].y);
          s[j].z = fmaf(v.z, w.z, s[j].z);
          s[j].w = fmaf(v.w, w.w, s[j].w);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < NT; ++j)
      s_part[((size_t)ks * tok_pitch + tok) * ET + 8 * j + e0] =
          ((acc[0][j].x + acc[1][j].x) + (acc[0][j].y + acc[1][j].y)) +
          ((acc[0][j].z + acc[1][j].z) + (acc[0][j].w + acc[1][j].w));
  } else {
    const int tg = warp % gp2, ks = warp / gp2;
    if (tg < ngroups) {
      const int tok0 = tg * 16;
      const int row_pieces = d >> 3;
      const int ra = min(tok0 + g, N - 1), rb = min(tok0 + g + 8, N - 1);
      const uint4* xa = reinterpret_cast<const uint4*>(x + (size_t)ra * d);
      const uint4* xb = reinterpret_cast<const uint4*>(x + (size_t)rb * d);
      const uint4* w4 = reinterpret_cast<const uint4*>(Wg);
      const int nchunk = (d + 31) >> 5;
      const uint4 zero = make_uint4(0, 0, 0, 0);
      float acc[NT][4];
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = 0.f;
      for (int c0 = ks; c0 < nchunk; c0 += nslices * 4) {
        uint4 A[4], B[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = c0 + u * nslices;
          const int piece = 4 * c + t;
          const bool ok = c < nchunk && piece < row_pieces;
          // x may be the output of the kernel before this one: through L2, not the read-only path
          A[u] = ok ? __ldcg(xa + piece) : zero;
          B[u] = ok ? __ldcg(xb + piece) : zero;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int c = c0 + u * nslices;
          const int piece = 4 * c + t;
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            const int row = 8 * j + g;
            const uint4 w = (row < E && c < nchunk && piece < row_pieces)
                                ? w4[(size_t)row * row_pieces + piece] : zero;
            mma_bf16_16816(acc[j], A[u].x, B[u].x, A[u].y, B[u].y, w.x, w.y);
            mma_bf16_16816(acc[j], A[u].z, B[u].z, A[u].w, B[u].w, w.z, w.w);
          }
        }
      }
      float* pp = s_part + ((size_t)ks * 16 * gp2 + tok0) * ET;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int e = 8 * j + 2 * t;
        pp[g * ET + e] = acc[j][0];
        pp[g * ET + e + 1] = acc[j][1];
        pp[(g + 8) * ET + e] = acc[j][2];
        pp[(g + 8) * ET + e + 1] = acc[j][3];
      }
    }
  }
  for (int i = tid; i < kMaxTopK * kMaxE; i += kThreads) s_cnt[i] = 0;
  __syncthreads();
  // the first batch of row copies: the loads do not depend on the routing, so they are
  // issued now and wait in registers until the destination rows are known
  const int pieces = d / kPiece;
  const int items = perm != nullptr ? N * pieces : 0;      // nullptr: the next kernel reads x itself
  const uint4* src = reinterpret_cast<const uint4*>(x);
  constexpr int kInFlight = 4;
  const int first_item = (SPLIT ? 0 : blk * kThreads * kInFlight) + tid;
  const int item_stride = (SPLIT ? 1 : nblk) * kThreads * kInFlight;
  // fp32: 2^lg warps (32 over the block's tokens, those rounded up to a power of two) share a token's row, which is stored
  // in five pieces: no division for each
  const int lg = F32 ? min(5, __clz(N - 1) - 27) : 0;
  const int copy_tok = warp >> lg, copy_pc = ((warp & ((1 << lg) - 1)) << 5) + lane, copy_stride = 32 << lg;
  uint4 pre[kInFlight];
#pragma unroll
  for (int u = 0; u < kInFlight; ++u) {
    const int p = copy_pc + u * copy_stride;
    const int i = F32 ? copy_tok * pieces + p : first_item + u * kThreads;
    if (F32 ? copy_tok < N && p < pieces : i < items)
      asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(pre[u].x), "=r"(pre[u].y), "=r"(pre[u].z), "=r"(pre[u].w)
                   : "l"(src + i)
                   : "memory");
  }
  for (int i = tid; i < N * E; i += kThreads) {
    const int tok = i / E, e = i - tok * E;
    float s = 0.f;
    if constexpr (F32) {
      for (int k0 = 0; k0 < nslices; k0 += 8) {
        float q[8];
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) q[ks] = s_part[((size_t)(k0 + ks) * tok_pitch + tok) * ET + e];
        s += ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
      }
    } else {
      for (int ks = 0; ks < nslices; ++ks) s += s_part[((size_t)ks * 16 * gp2 + tok) * ET + e];
    }
    s += s_bias[e];
    s_logit[tok * ld + e] = s;
    if (out_logits != nullptr && writer) out_logits[i] = s;
  }
  __syncthreads();

  // ---- B. softmax, top-k, renormalise: a group of ET lanes per token, lane e = expert e ----
  {
    constexpr int G = ET_C;                 // 8, 16 or 32 lanes
    constexpr int kTokPerWarp = 32 / G;
    const int grp = lane / G, e = lane % G;
    const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (grp * G));
    for (int tok0 = warp * kTokPerWarp; tok0 < N; tok0 += (kThreads / 32) * kTokPerWarp) {
      const int tok = tok0 + grp;
      const bool live = tok < N && e < E;
      float* lg = s_logit + (size_t)min(tok, N - 1) * ld;
      const float v = live ? lg[e] + 0.f : -INFINITY;      // + 0: no negative zero
      // order-preserving map float -> unsigned: the maximum and its first position by integer compares
      const unsigned u = __float_as_uint(v);
      unsigned key = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
      // fp32: as in router_kernel, which takes the larger calls, NaN is never chosen, and slots that are left without an
      // expert have an index out of range; the dispatch reports them and gives them no row
      if (F32 && !(live && v == v)) key = 0u;
      unsigned kmax = key;
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) kmax = max(kmax, __shfl_xor_sync(gmask, kmax, o));
      const float m = __uint_as_float((kmax & 0x80000000u) ? (kmax & 0x7fffffffu) : ~kmax);
      const float p = live ? expf(v - m) : 0.f;
      float sum = p;
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(gmask, sum, o);
      const float inv_sum = __frcp_rn(sum);  // one reciprocal per token, products below: a division
                                             // is a long subroutine, and this code runs once, cold
      if (live) lg[e] = p * inv_sum;        // probabilities, for the loss below
      // k passes of arg-max ordered by (logit descending, index ascending); lane j of the group
      // keeps slot j's result. The loop is kept rolled: this code runs once per launch, from a cold
      // instruction cache, and every extra line of it costs a miss on the path to the next kernel.
      int my_sel = 0;
      float my_val = 0.f;
      float total = 0.f;
#pragma unroll 1
      for (int j = 0; j < k; ++j) {
        unsigned km = key;
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) km = max(km, __shfl_xor_sync(gmask, km, o));
        const unsigned hit = __ballot_sync(gmask, key == km) & gmask;
        const int winner = __ffs(hit) - 1;
        const float bv = __uint_as_float((km & 0x80000000u) ? (km & 0x7fffffffu) : ~km);
        const bool none = F32 && km == 0u;
        const float val = none ? 0.f : expf(bv - m) * inv_sum;
        total += val;
        if (e == j) { my_sel = none ? 0x7fffffff : winner - grp * G; my_val = val; }
        if (lane == winner) key = 0u;     // below every real key
      }
      if (e < k && tok < N) {
        if (writer) {
          out_idx[tok * k + e] = my_sel;
          out_w[tok * k + e] = my_val * __frcp_rn(total);
        }
        s_idx[tok * k + e] = my_sel;
        if (!F32 || my_sel < E) atomicAdd(&s_cnt[e * kMaxE + my_sel], 1);
      }
    }
  }
  __syncthreads();

  // ---- C. counts, offsets, ranks: warp 0 -------------------------------------------
  int* s_base = reinterpret_cast<int*>(s_bias + kMaxE);    // [kMaxE] SPLIT: rows of earlier blocks
  int* s_tot = s_base + kMaxE;                             // [kMaxTopK][kMaxE] SPLIT: grid totals
  if constexpr (SPLIT) {
    const int nb = nblk, b = blk;
    float* xps = reinterpret_cast<float*>(xch + nb * k * E);    // [nb][E] probability sums
    static_assert(32 * 4 >= 128, "128 blocks' sums of 8 NT experts in [nslices][tok_pitch][8 NT]");
    // (a count's blocks side by side, for a warp to add)
    if (tid < k * E) xch[tid * nb + b] = s_cnt[(tid / E) * kMaxE + tid % E];
    if (tid < E) {
      float ps = 0.f;
      for (int tok = 0; tok < N; ++tok) ps += s_logit[tok * ld + tid];
      xps[b * E + tid] = ps;
    }
    for (int i = tid; i < kMaxE + kMaxTopK * kMaxE; i += kThreads) s_base[i] = 0;   // s_base, s_tot
    // the status words are this call's; what a block has to say it says behind the barrier
    if (b == 0 && tid < MOE_B200_STATUS_INTS) status[tid] = 0;
    __threadfence();
    if (nblk > 1) cooperative_groups::this_grid().sync();
    else __syncthreads();
    // totals per (slot, expert) and the rows that earlier blocks put in front of this block's
    for (int je = warp; je < k * E; je += kThreads / 32) {
      unsigned sum = 0;      // both, 16 bits each: 2048 tokens at most
      for (int bb = lane; bb < nb; bb += 32) {
        const unsigned c = (unsigned)__ldcg(&xch[je * nb + bb]);
        sum += c | (bb < b ? c << 16 : 0u);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) {
        const int j = je / E, e = je - j * E;
        s_tot[j * kMaxE + e] = (int)(sum & 0xffffu);
        if (sum >> 16) atomicAdd(&s_base[e], (int)(sum >> 16));
      }
    }
    // the blocks' probability sums, for the loss
    if (b == 0)
      for (int i = tid; i < nb * E; i += kThreads) s_part[i] = __ldcg(&xps[i]);
    __syncthreads();
    // ---- E. the loss (model.py:213-216), beside the ranks: behind the copies it kept the kernels that wait for this one
    // waiting (1173 tokens: 3.3 us) ----
    if (b == 0 && warp == 1) {
      float part = 0.f;
      if (lane < E) {
        float ps = 0.f;
#pragma unroll 8
        for (int bb = 0; bb < nb; ++bb) ps += s_part[bb * E + lane];      // in block order
        psum[lane] = ps;
        part = (ps / (float)Ntotal) * ((float)s_tot[lane] / (float)Ntotal);
      }
      float a = 0.f;
      for (int e = 0; e < E; ++e) a += __shfl_sync(0xffffffffu, part, e);
      if (lane == 0) aux[0] = a / (float)E * (float)(E * E);
    }
  }
  if (warp == 0) {
    int tot = 0;
    if (lane < E) {
      for (int j = 0; j < k; ++j) {
        const int c = SPLIT ? s_tot[j * kMaxE + lane] : s_cnt[j * kMaxE + lane];
        if (blk == 0) cnt_slot[j * E + lane] = c;
        tot += c;
      }
    }
    int incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane < E) {
      s_off[lane] = incl - tot + (SPLIT ? s_base[lane] : 0);   // first row of this block's tokens
      s_run[lane] = 0;
      if (blk == 0) offsets[lane] = incl - tot;
    }
    if (lane == 31) {
      s_off[E] = incl;
      if (blk == 0) offsets[E] = incl;
    }
    __syncwarp();
    const int npair = F32 ? 0 : N * k;
    for (int p0 = 0; p0 < npair; p0 += 32) {
      const int p = p0 + lane;
      const int e = p < npair ? s_idx[p] : -1;
      const bool ok = e >= 0;
      const unsigned grp = __match_any_sync(0xffffffffu, ok ? e : -1 - lane);
      int row = -1;
      if (ok) row = s_off[e] + s_run[e] + __popc(grp & ((1u << lane) - 1u));
      __syncwarp();
      if (ok && (grp >> lane) == 1u) s_run[e] += __popc(grp);
      __syncwarp();
      if (p < npair) {
        s_row[p] = row;
        if (writer) row_of[p] = row;
      }
    }
  }
  __syncthreads();

  if constexpr (F32) {
    // ranks: a warp per expert, 32 pairs at a time; slots without an expert have no row
    const int npair = N * k;
    if (warp < E) {
      int next = s_off[warp];
      for (int p0 = 0; p0 < npair; p0 += 32) {
        const int p = p0 + lane;
        const bool mine = p < npair && s_idx[p] == warp;
        const unsigned hit = __ballot_sync(0xffffffffu, mine);
        if (mine) {
          const int row = next + __popc(hit & ((1u << lane) - 1u));
          s_row[p] = row;
          row_of[p] = row;
        }
        next += __popc(hit);
      }
    }
    for (int p = tid; p < npair; p += kThreads)
      if ((unsigned)s_idx[p] >= (unsigned)E) {
        atomicMax(&status[0], MOE_B200_DEV_BAD_INDEX);
        s_row[p] = -1;
        row_of[p] = -1;
      }
    __syncthreads();
    for (int tok = copy_tok; tok < N; tok += 32 >> lg)
      for (int p0 = copy_pc; p0 < pieces; p0 += copy_stride * kInFlight) {
        uint4 v[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
          const int p = p0 + u * copy_stride;
          if (tok == copy_tok && p0 == copy_pc) v[u] = pre[u];
          else if (p < pieces) v[u] = __ldcg(src + (size_t)tok * pieces + p);
        }
        for (int j = 0; j < k; ++j) {
          const int row = s_row[tok * k + j];
          if (row < 0) continue;
#pragma unroll
          for (int u = 0; u < kInFlight; ++u) {
            const int p = p0 + u * copy_stride;
            if (p >= pieces) break;
            // the rows as they are, and as the three bf16 planes the products read (split once here, not by every tile)
            reinterpret_cast<uint4*>(perm + (size_t)row * d)[p] = v[u];
            uint2 part[3];
            split2(__uint_as_float(v[u].x), __uint_as_float(v[u].y), part[0].x, part[1].x, part[2].x);
            split2(__uint_as_float(v[u].z), __uint_as_float(v[u].w), part[0].y, part[1].y, part[2].y);
#pragma unroll
            for (int q = 0; q < 3; ++q)
              reinterpret_cast<uint2*>(planes + ((size_t)q * Ntotal * k + row) * d)[p] = part[q];
          }
        }
      }
  }

  // ---- D. copy the token rows into the sorted buffer (split over the blocks) -----
  for (int i0 = first_item; !F32 && i0 < items; i0 += item_stride) {
    uint4 v[kInFlight];
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) {
      const int i = i0 + u * kThreads;
      if (i0 == first_item) v[u] = pre[u];
      else if (i < items) v[u] = __ldcg(src + i);
    }
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) {
      const int i = i0 + u * kThreads;
      if (i < items) {
        const int tok = i / pieces, pc = i - tok * pieces;
        for (int j = 0; j < k; ++j) reinterpret_cast<uint4*>(perm + (size_t)s_row[tok * k + j] * d)[pc] = v[u];
      }
    }
  }

  // ---- E. the loss of the form in which every block has all tokens (model.py:213-216) ----
  if (!SPLIT && blk == 0) {
    __syncthreads();       // the partial-logit area is free again: every thread is past the reduction
    // probabilities summed per expert: warp w takes tokens w, w + 32, ...; the 32 partial sums
    // of an expert are then added in warp order
    if (lane < E) {
      float ps = 0.f;
      for (int tok = warp; tok < N; tok += kThreads / 32) ps += s_logit[tok * ld + lane];
      s_part[warp * 32 + lane] = ps;
    }
    __syncthreads();
    if (tid < E) {
      float ps = 0.f;
      for (int w = 0; w < kThreads / 32; ++w) ps += s_part[w * 32 + tid];
      psum[tid] = ps;
      s_part[1024 + tid] = (ps / (float)N) * ((float)s_cnt[tid] / (float)N);
    }
    __syncthreads();
    if (tid == 0) {
      float a = 0.f;
      for (int e = 0; e < E; ++e) a += s_part[1024 + e];
      aux[0] = a / (float)E * (float)(E * E);
    }
  }
}

}  // namespace moe
