// Expert feed-forward in fp32 on the tensor cores: FeedForward.forward (reference model.py:173-190,
// fine_tuning=False, eval), grouped over experts by the row offsets the dispatch kernel wrote:
//   h = gelu_tanh(x W1[:f]^T + b1[:f]) * (x W1[f:]^T + b1[f:])   (model.py:174,180-182)
//   y = h W2^T + b2                                               (model.py:184)
//
// Every fp32 operand of 2^-110 or more is the exact sum of three bf16 values (24 = 8 + 8 + 8 bits of mantissa; the third of
// a smaller one falls under bf16's smallest, and up to 2^-133 is left out), and six of the nine products of parts make up
// the fp32 product to 2^-24 of it: a0 b0, a0 b1, a1 b0, a1 b1, a0 b2, a2 b0 (after Henry, Tang and Heinecke, "Leveraging the
// bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations", ARITH 2019). a0 is cut off, not rounded, so
// that nothing overflows; a1 and a2 are rounded, so that what is left out has either sign. The tensor core adds with
// truncation, which would make long sums drift towards zero: the large products a0 b0 stay in its accumulator for 64 of K
// only and are then added, rounded to nearest, to fp32 registers; the five small ones, 2^-8 of them, are summed apart over
// 256 of K.
//
// Infinities and NaN survive in the first parts only (the others are inf - inf): the large products say what becomes of
// them. Small products that are not finite are therefore left out and noted (an infinity times a value under bf16's
// smallest, 2^-133, so counts as one times zero). Where a sum is finite without them, with operands near the end of fp32's
// range, it is formed again by an fp32 loop over K, which gives what fp32 arithmetic gives. Forming every sum that was not
// finite that way made calls slow that hold infinities: 512 tokens, d 512, f 2048, 8 experts, top-2 took 8500 us with one
// infinite weight and 19800 with an infinity in every token, now 105 and 110; without any 101.3 and now 102.9, for looking.
//
// Tile: 128 weight rows (the GEGLU pass: 64 gate and the 64 up rows of the same features) are the A operand, up to 160
// tokens of one expert the B operand, N = their number rounded up to 16: the pipe's time is in proportion to N from 64
// on (64 clk per K = 16 at N 128, 46 at N 16 to 64), so that an expert's last rows cost what they are. K in
// steps of 32.
//   warp 0       loads fp32 boxes by TMA, three stages ahead
//   warp 1       issues the products (A from tensor memory, B from shared memory)
//   warps 4-19   split, eight on even and eight on odd steps: their row of A into tensor memory (tcgen05.st), tokens of
//                B into three bf16 tiles
//   warps 20-27  add up the products, then bias, GELU and the store
// A cluster of up to eight CTAs shares a tile and splits K where tiles are few; every CTA sends each other one its
// sums of that one's tokens through distributed shared memory, and they are added in rank order.
//
// What bounds it: shared-memory bandwidth (per step of 32 at N 128: 32 KiB in by TMA, 32 read and 24 written by the
// split, 48 read by the products, about 1060 clk of 128 bytes) and the issue slots of the split (600 clk) against 768 clk
// of products; a step takes 1400 to 1600. 1024 rows of 8 experts, d 512, f 2048, nothing in L2: gate_and_up 160 -> 46 us,
// both products 250 -> 77 us (packed FMA on the CUDA cores before; 45 and 75 without the look for infinities). Error of h
// and y against 64 bits, in the 2-norm, at 2 to 4096 rows: 1.8e-7 and 0.9e-7 to 1.4e-7 (before: 2.3e-7 to 4.2e-7 and
// 1.6e-7).
#include <cuda.h>
#include <cfloat>
#include "common.cuh"
#include "tc_ptx.cuh"

namespace moe {

namespace {

using namespace tc;

constexpr int kRowsA = 128;      // weight rows per tile = accumulator lanes
constexpr int kMaxN = 160;       // tokens per tile; 2 * 160 + 3 * 48 columns of tensor memory
constexpr int BK = 32;
constexpr int kRawStages = 3, kConvStages = 3;
constexpr int kRawA = kRowsA * BK * 4;            // 16 KiB, rows of 128 bytes
constexpr int kRawBytes = kRawA + kMaxN * BK * 4;
constexpr int kPlane = kMaxN * BK * 2;            // one bf16 tile of the tokens, rows of 64 bytes
constexpr int kSplitWarps = 8, kEpiWarps = 8;       // split warps of a step
constexpr int kEpiFirst = 4 + 2 * kSplitWarps;
constexpr int kThreads = 32 * (kEpiFirst + kEpiWarps);
// Registers: 896 threads start with 72 each, 504 for the seven warps of a thread index
constexpr int kRegsLoad = 40, kRegsSplit = 48, kRegsEpi = 136;
static_assert(kRegsLoad + 4 * kRegsSplit + 2 * kRegsEpi <= 7 * 72, "a share above the launch's registers would wait for good");
constexpr int kMainCol = 0, kSmallCol = kMaxN, kACol = 2 * kMaxN;   // tensor memory columns
constexpr int kACols = 3 * BK / 2;                                  // of one stage of A
constexpr int kLargeSteps = 2, kSmallSteps = 8;   // steps of K after which an accumulator is read out and started again
constexpr int kGroups = kMaxN / 8 / 2;            // groups of eight tokens per epilogue warp
static_assert(kACol + kConvStages * kACols <= 512, "tensor memory");
static_assert((kMaxN / 8 + 4) * kRowsA * 32 <= kRawStages * kRawBytes, "sums of all ranges reuse the raw stages");

struct Control {
  uint64_t raw_full[kRawStages], raw_empty[kRawStages];
  uint64_t conv_full[kConvStages], conv_empty[kConvStages];
  uint64_t main_full, main_empty, small_full, small_empty;
  uint32_t tmem_base;
  int abort;
  int offsets[kMaxExperts + 1];
  int block_start[kMaxExperts + 1];   // token blocks of the experts before
};
constexpr size_t kSmemBytes = 1024 + (size_t)kRawStages * kRawBytes + kConvStages * 3 * kPlane + sizeof(Control);
static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");

struct Tile {
  int e, m;            // expert, tile of weight rows
  int row0, rows, n;   // tokens, their number, rounded up to 16
};
// Tiles go expert by expert, weight rows by weight rows: blocks of tokens that read the same weights are neighbours.
// An expert's tokens are cut into as few blocks as hold them, of equal size.
__device__ __forceinline__ Tile tile_of(const Control* ctl, int E, int m_tiles, int t) {
  int lo = 0, hi = E;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (ctl->block_start[mid] * m_tiles <= t) lo = mid; else hi = mid;
  }
  const int blocks = ctl->block_start[lo + 1] - ctl->block_start[lo];
  const int local = t - ctl->block_start[lo] * m_tiles;
  const int cnt = ctl->offsets[lo + 1] - ctl->offsets[lo];
  Tile tl;
  tl.e = lo;
  tl.m = local / blocks;
  const int b = local - tl.m * blocks;
  const int per = ((cnt + blocks - 1) / blocks + 15) & ~15;
  tl.row0 = ctl->offsets[lo] + b * per;
  tl.rows = min(per, cnt - b * per);
  tl.n = (tl.rows + 15) & ~15;
  return tl;
}

__device__ __forceinline__ void st_tmem4(uint32_t taddr, const uint32_t (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3])
               : "memory");
}
// For warps that stay together: all lanes have the same answer.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, Control* ctl, int32_t* status, int where) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, &ctl->abort, status, where)) != 0;
}
__device__ __forceinline__ void prefetch_tmap(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}
__device__ __forceinline__ void st_tmem_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void ld_tmem8(uint32_t taddr, uint32_t (&u)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
               : "r"(taddr));
}
__device__ __forceinline__ void st_tmem8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
template <int N>
__device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
// A in tensor memory (two bf16 per column, lane = row), B in shared memory
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// K-major tile of 32 bf16 (64 bytes) a row, 64-byte swizzle, 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t desc64(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3ffffu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}

// Two values cut off to bf16, NaN to NaN (whose upper half alone may be an infinity's).
__device__ __forceinline__ uint32_t cut_bf16x2(float lo, float hi) {
  uint32_t v;
  asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
  return v;
}
// Eight values into their three bf16 parts, exactly (where they are finite).
__device__ __forceinline__ void split8(const float (&x)[8], uint32_t (&p0)[4], uint32_t (&p1)[4], uint32_t (&p2)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t u0 = __float_as_uint(x[2 * i]), u1 = __float_as_uint(x[2 * i + 1]);
    p0[i] = cut_bf16x2(x[2 * i], x[2 * i + 1]);
    float r0 = x[2 * i] - __uint_as_float(u0 & 0xffff0000u);
    float r1 = x[2 * i + 1] - __uint_as_float(u1 & 0xffff0000u);
    p1[i] = pack_bf16x2(r0, r1);
    r0 -= bf16_lo(p1[i]);
    r1 -= bf16_hi(p1[i]);
    p2[i] = pack_bf16x2(r0, r1);
  }
}

// (a: the rows may come from the kernel before this one, so they are not read as constant data)
__device__ __forceinline__ float dot_f32(const float* a, const float* w, int k0, int k1) {
  float s = 0.f;
#pragma unroll 1
  for (int k = k0; k < k1; ++k) s = fmaf(__ldcg(a + k), w[k], s);
  return s;
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= FLT_MAX; }

// The sums of eight tokens have been used: those of the next eight take their place.
__device__ __forceinline__ void next_group(float (&acc)[kGroups][8]) {
#pragma unroll
  for (int g = 0; g + 1 < kGroups; ++g)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[g][i] = acc[g + 1][i];
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(cta));
  return r;
}
__device__ __forceinline__ void st_cluster4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// A: [rows, K] activations (sorted buffer); W_e: [Nw, K]; out [rows, Nout].
// GEGLU: Nw = 2 * Nout, gate rows [0, Nout), up rows [Nout, 2 * Nout).
// splits: CTAs of a cluster; with more than one a cluster has one tile at most.
template <bool GEGLU>
__global__ void __launch_bounds__(kThreads, 1)
ffn_f32_kernel(const __grid_constant__ CUtensorMap tmap_a,          // activations, 16-row boxes of 32 columns
               const CUtensorMap* __restrict__ tmap_w,              // [E], 64-row boxes of 32 columns
               const float* __restrict__ A, const int32_t* __restrict__ offsets, const void* const* __restrict__ Wp,
               const void* const* __restrict__ bp, int E, int K, int Nout, int splits, float* __restrict__ out,
               int32_t* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* planes = smem + (size_t)kRawStages * kRawBytes;      // [kConvStages][3] bf16 tiles of the tokens
  Control* ctl = reinterpret_cast<Control*>(planes + kConvStages * 3 * kPlane);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kFeatures = GEGLU ? 64 : 128;                    // output columns of a tile
  const int m_tiles = (Nout + kFeatures - 1) / kFeatures;
  const int rank = splits > 1 ? (int)cluster_rank() : 0;
  const int first = blockIdx.x / splits, step = gridDim.x / splits;
  const int kb_all = (K + BK - 1) / BK;
  const int kb_per = (kb_all + splits - 1) / splits;
  const int kb0 = min(kb_all, rank * kb_per), kn = min(kb_all, kb0 + kb_per) - kb0;   // this CTA's steps of K

  if (threadIdx.x == 0) {
    for (int s = 0; s < kRawStages; ++s) { mbar_init(&ctl->raw_full[s], 1); mbar_init(&ctl->raw_empty[s], kSplitWarps); }
    for (int c = 0; c < kConvStages; ++c) { mbar_init(&ctl->conv_full[c], kSplitWarps); mbar_init(&ctl->conv_empty[c], 1); }
    mbar_init(&ctl->main_full, 1);
    mbar_init(&ctl->main_empty, kEpiWarps);
    mbar_init(&ctl->small_full, 1);
    mbar_init(&ctl->small_empty, kEpiWarps);
    ctl->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  if (warp == 2) {
    if (lane == 0) prefetch_tmap(&tmap_a);
    for (int e = lane; e < E; e += 32) prefetch_tmap(tmap_w + e);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&ctl->tmem_base))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_wait();
  pdl_launch_dependents();
  for (int e = threadIdx.x; e <= E; e += kThreads) ctl->offsets[e] = __ldcg(&offsets[e]);
  __syncthreads();
  if (warp == 0) {
    int carry = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const int nb = e < E ? (ctl->offsets[e + 1] - ctl->offsets[e] + kMaxN - 1) / kMaxN : 0;
      int incl = nb;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      if (e < E) ctl->block_start[e] = carry + incl - nb;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) ctl->block_start[E] = carry;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctl->tmem_base);
  const int total = ctl->block_start[E] * m_tiles;

  if (warp < 4) {
    fewer_registers<kRegsLoad>();
    if (warp == 0 && elect_one()) {
      // ---------------- TMA producer ----------------
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = first; ok && t < total; t += step) {
        const Tile tl = tile_of(ctl, E, m_tiles, t);
        const CUtensorMap* tw = tmap_w + tl.e;
        const int r0 = tl.m * kFeatures, r1 = GEGLU ? Nout + r0 : r0 + 64;
        for (int i = 0; i < kn; ++i) {
          if (!mbar_wait(&ctl->raw_empty[s], phase ^ 1u, &ctl->abort, status, 51)) { ok = false; break; }
          uint8_t* dst = smem + (size_t)s * kRawBytes;
          const int k = (kb0 + i) * BK;
          mbar_expect_tx(&ctl->raw_full[s], (uint32_t)(kRawA + tl.n * BK * 4));
          tma_load_2d(dst, tw, &ctl->raw_full[s], k, r0);
          tma_load_2d(dst + kRawA / 2, tw, &ctl->raw_full[s], k, r1);
          for (int j = 0; j < tl.n; j += 16) tma_load_2d(dst + kRawA + j * BK * 4, &tmap_a, &ctl->raw_full[s], k, tl.row0 + j);
          if (++s == kRawStages) { s = 0; phase ^= 1u; }
        }
      }
    } else if (warp == 1) {
      // ---------------- products: the whole warp keeps step, so that addresses stay in uniform registers ----------------
      const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
      uint32_t phase = 0, larges = 0, smalls = 0;
      int c = 0;
      bool ok = true;
      for (int t = first; ok && t < total; t += step) {
        const Tile tl = tile_of(ctl, E, m_tiles, t);
        const uint32_t idesc = make_idesc(tl.n);
        for (int i = 0; i < kn; ++i) {
          if (!warp_wait(&ctl->conv_full[c], phase, ctl, status, 53)) { ok = false; break; }
          if (i % kLargeSteps == 0) {
            if (!warp_wait(&ctl->main_empty, (larges & 1u) ^ 1u, ctl, status, 54)) { ok = false; break; }
            ++larges;
          }
          tc_fence_after();
          const uint32_t a = tm + kACol + c * kACols;
          const uint64_t b = desc64(smem_u32(planes) + (uint32_t)(c * 3 * kPlane));
          constexpr uint64_t kP = kPlane / 16;
          const bool large_ends = (i + 1) % kLargeSteps == 0 || i == kn - 1;
          const bool small_ends = (i + 1) % kSmallSteps == 0 || i == kn - 1;
          // the large products first: their sums are read out while the small products run
          if (elect_one()) {
            mma_ts(tm + kMainCol, a, b, idesc, i % kLargeSteps != 0 ? 1u : 0u);
            mma_ts(tm + kMainCol, a + 8, b + 2, idesc, 1u);
            if (large_ends) tc_commit(&ctl->main_full);
          }
          __syncwarp();
          if (i % kSmallSteps == 0) {
            if (!warp_wait(&ctl->small_empty, (smalls & 1u) ^ 1u, ctl, status, 52)) { ok = false; break; }
            tc_fence_after();
            ++smalls;
          }
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
              const uint32_t ak = a + kk * 8;
              const uint64_t bk = b + kk * 2;
              mma_ts(tm + kSmallCol, ak + 32, bk, idesc, (i % kSmallSteps | kk) != 0 ? 1u : 0u);   // a2 b0
              mma_ts(tm + kSmallCol, ak, bk + 2 * kP, idesc, 1u);                                  // a0 b2
              mma_ts(tm + kSmallCol, ak + 16, bk + kP, idesc, 1u);                                 // a1 b1
              mma_ts(tm + kSmallCol, ak + 16, bk, idesc, 1u);                                      // a1 b0
              mma_ts(tm + kSmallCol, ak, bk + kP, idesc, 1u);                                      // a0 b1
            }
            if (small_ends) tc_commit(&ctl->small_full);
            tc_commit(&ctl->conv_empty[c]);
          }
          __syncwarp();
          if (++c == kConvStages) { c = 0; phase ^= 1u; }
        }
      }
    }
    __syncwarp();
    if (splits > 1) { cluster_sync(); cluster_sync(); }
  } else if (warp < kEpiFirst) {
    // ---------------- split ----------------
    fewer_registers<kRegsSplit>();
    const int quad = warp & 3, part = ((warp - 4) >> 2) & 1;   // lanes of tensor memory; half of the step's K
    const int group = (warp - 4) / kSplitWarps;
    const int et = (threadIdx.x - 128) % (32 * kSplitWarps);
    // the row of the raw tile that goes to this lane. GEGLU: gate and up of a feature in one warp, 16 lanes apart
    const int r = GEGLU ? (lane & 15) + quad * 16 + (lane >> 4) * 64 : quad * 32 + lane;
    static_assert(kRawStages == kConvStages, "one stage counter for both");
    int s = 0, turn = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = first; ok && t < total; t += step) {
      const Tile tl = tile_of(ctl, E, m_tiles, t);
      for (int i = 0; i < kn; ++i, turn ^= 1) {
        const int c = s;
        const uint32_t ph = phase;
        if (++s == kRawStages) { s = 0; phase ^= 1u; }
        if (turn != group) continue;
        // In this order: boxes may land out of order, and with the other group's last turn on this stage still to come its
        // barrier would be a phase behind and this parity would look done. The products of that turn are done first.
        if (!warp_wait(&ctl->conv_empty[c], ph ^ 1u, ctl, status, 56)) { ok = false; break; }
        if (!warp_wait(&ctl->raw_full[c], ph, ctl, status, 55)) { ok = false; break; }
        tc_fence_after();
        const uint8_t* raw = smem + (size_t)c * kRawBytes;
        const uint32_t ta = tmem + ((uint32_t)(quad * 32) << 16) + kACol + c * kACols + part * 8;
        // 16-byte piece p of row r of a raw tile lies at p ^ (r mod 8)
        auto load8_at = [&](const uint8_t* row, int rr, int p, float (&x)[8]) {
          const float4 v0 = *reinterpret_cast<const float4*>(row + ((p ^ (rr & 7)) << 4));
          const float4 v1 = *reinterpret_cast<const float4*>(row + (((p + 1) ^ (rr & 7)) << 4));
          x[0] = v0.x; x[1] = v0.y; x[2] = v0.z; x[3] = v0.w;
          x[4] = v1.x; x[5] = v1.y; x[6] = v1.z; x[7] = v1.w;
        };
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float x[8];
          uint32_t p0[4], p1[4], p2[4];
          load8_at(raw + r * 128, r, part * 4 + j * 2, x);
          split8(x, p0, p1, p2);
          st_tmem4(ta + j * 4, p0);
          st_tmem4(ta + 16 + j * 4, p1);
          st_tmem4(ta + 32 + j * 4, p2);
        }
        uint8_t* pl = planes + (size_t)c * 3 * kPlane;
        for (int q = et; q < tl.n * 4; q += 32 * kSplitWarps) {      // a token's eight values at a time
          const int rr = q >> 2, p = q & 3;
          float x[8];
          uint32_t p0[4], p1[4], p2[4];
          load8_at(raw + kRawA + rr * 128, rr, p * 2, x);
          split8(x, p0, p1, p2);
          uint8_t* d = pl + rr * 64 + ((p ^ ((rr >> 1) & 3)) << 4);
          *reinterpret_cast<uint4*>(d) = make_uint4(p0[0], p0[1], p0[2], p0[3]);
          *reinterpret_cast<uint4*>(d + kPlane) = make_uint4(p1[0], p1[1], p1[2], p1[3]);
          *reinterpret_cast<uint4*>(d + 2 * kPlane) = make_uint4(p2[0], p2[1], p2[2], p2[3]);
        }
        st_tmem_wait();
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&ctl->conv_full[c]);
          mbar_arrive(&ctl->raw_empty[c]);
        }
      }
    }
    __syncwarp();
    if (splits > 1) { cluster_sync(); cluster_sync(); }
  } else {
    // ---------------- sums and epilogue: lane = weight row, columns = tokens ----------------
    more_registers<kRegsEpi>();
    const int quad = warp & 3, part = (warp - kEpiFirst) >> 2;   // this warp: token groups part, part + 2, ...
    const uint32_t ta = tmem + ((uint32_t)(quad * 32) << 16) + part * 8;
    uint32_t larges = 0, smalls = 0;
    bool ok = true, sent = false;
    for (int t = first; ok && t < total; t += step) {
      const Tile tl = tile_of(ctl, E, m_tiles, t);
      float acc[kGroups][8];
#pragma unroll
      for (int g = 0; g < kGroups; ++g)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[g][i] = 0.f;
      uint64_t again = 0;      // a bit per sum of this thread whose small products were not finite, ...
      uint32_t again_hi = 0;   // ... from the ninth group on
      auto add = [&](int col) {
        // (groups past n hold old sums; they are not used)
#pragma unroll
        for (int g0 = 0; g0 < kGroups; g0 += 4) {
          if ((g0 * 2 + part) * 8 >= tl.n) break;
          uint32_t v[4][8];
#pragma unroll
          for (int g = 0; g < 4; ++g)
            if (g0 + g < kGroups) ld_tmem8(ta + col + (g0 + g) * 16, v[g]);
          tc_ld_wait();
#pragma unroll
          for (int g = 0; g < 4; ++g)
            if (g0 + g < kGroups) {
#pragma unroll
              for (int i = 0; i < 8; ++i) acc[g0 + g][i] += __uint_as_float(v[g][i]);
            }
        }
      };
      // Small products that are not finite become zero, in tensor memory, and are noted.
      auto keep_finite = [&]() {
        static_assert(kGroups % 2 == 0 && kGroups <= 12, "two groups at a time, 96 bits");
#pragma unroll 1
        for (int g0 = 0; (g0 * 2 + part) * 8 < tl.n; g0 += 2) {
          uint32_t v[2][8];
          ld_tmem8(ta + kSmallCol + g0 * 16, v[0]);
          ld_tmem8(ta + kSmallCol + g0 * 16 + 16, v[1]);
          tc_ld_wait();
          float probe[2] = {0.f, 0.f};      // times zero: NaN where one is not finite
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            probe[0] = fmaf(__uint_as_float(v[0][i]), 0.f, probe[0]);
            probe[1] = fmaf(__uint_as_float(v[1][i]), 0.f, probe[1]);
          }
          if (__any_sync(0xffffffffu, probe[0] + probe[1] != 0.f)) {
            uint32_t bits = 0;
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (!finite(__uint_as_float(v[i >> 3][i & 7]))) {
                v[i >> 3][i & 7] = 0u;
                bits |= 1u << i;
              }
            st_tmem8(ta + kSmallCol + g0 * 16, v[0]);
            st_tmem8(ta + kSmallCol + g0 * 16 + 16, v[1]);
            st_tmem_wait();
            if (g0 < 8) again |= (uint64_t)bits << (g0 * 8); else again_hi |= bits << (g0 * 8 - 64);
          }
        }
      };
      for (int i = 1; i <= kn; ++i) {
        if (i % kLargeSteps == 0 || i == kn) {
          if (!warp_wait(&ctl->main_full, larges & 1u, ctl, status, 57)) { ok = false; break; }
          ++larges;
          tc_fence_after();
          add(kMainCol);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->main_empty);
        }
        if (i % kSmallSteps == 0 || i == kn) {
          if (!warp_wait(&ctl->small_full, smalls & 1u, ctl, status, 58)) { ok = false; break; }
          ++smalls;
          tc_fence_after();
          keep_finite();
          add(kSmallCol);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->small_empty);
        }
      }
      if (!ok && splits <= 1) break;
      const float* W = static_cast<const float*>(Wp[tl.e]);
      const int feat = tl.m * kFeatures + (GEGLU ? quad * 16 + (lane & 15) : quad * 32 + lane);
      const bool feat_ok = feat < Nout;
      // The sums at hand, of eight tokens from c0 on: those that lack their small products and are finite without them are
      // formed again, over this CTA's range of K.
      auto form_again = [&](int c0) {
        const uint32_t bits = (uint32_t)again & 0xffu;
        again = again >> 8 | (uint64_t)again_hi << 56;
        again_hi >>= 8;
        if (bits != 0u && feat_ok) {
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = acc[0][i];
          const float* w = W + (int64_t)(GEGLU && lane >= 16 ? Nout + feat : feat) * K;
#pragma unroll 1
          for (int i = 0; i < 8 && c0 + i < tl.rows; ++i)
            if ((bits >> i & 1u) != 0u && finite(v[i]))
              v[i] = dot_f32(A + (int64_t)(tl.row0 + c0 + i) * K, w, kb0 * BK, min(K, (kb0 + kn) * BK));
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[0][i] = v[i];
        }
        __syncwarp();
      };
      if (splits > 1) {
        // Eight tokens at a time go to the CTAs in turn, which keep them as [eight][source][128 rows][8 tokens] in
        // their raw stages.
        __syncwarp();
        cluster_sync();    // no CTA reads its raw stages any more
        const uint32_t mine = smem_u32(smem) + (uint32_t)((rank * kRowsA + quad * 32 + lane) * 32);
#pragma unroll 1
        for (int g = part; g * 8 < tl.n; g += 2, next_group(acc)) {
          form_again(g * 8);
          const uint32_t to = map_to_cta(mine, g & (splits - 1)) + (uint32_t)((g & -splits) * kRowsA * 32);
          st_cluster4(to, acc[0][0], acc[0][1], acc[0][2], acc[0][3]);
          st_cluster4(to + 16, acc[0][4], acc[0][5], acc[0][6], acc[0][7]);
        }
        sent = true;
        break;
      }
      const float* bias = static_cast<const float*>(bp[tl.e]);
      const float b0 = feat_ok ? __ldg(bias + feat) : 0.f;
      const float b1 = GEGLU && feat_ok ? __ldg(bias + Nout + feat) : 0.f;
      // rolled, and the sums moved up: unrolled, 60 KB of code that runs from a cold instruction cache took 30000 clk
#pragma unroll 1
      for (int c0 = part * 8; c0 < tl.rows; c0 += 16, next_group(acc)) {
        form_again(c0);
        float* o = out + (int64_t)(tl.row0 + c0) * Nout + feat;
        if (GEGLU) {
          // lanes 0-15 (gate) take tokens c0 + i, lanes 16-31 (up) tokens c0 + i + 1, i even
          const int upper = lane >> 4;
          float v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float other = __shfl_xor_sync(0xffffffffu, upper ? acc[0][2 * i] : acc[0][2 * i + 1], 16);
            const float gate = upper ? other : acc[0][2 * i], up = upper ? acc[0][2 * i + 1] : other;
            v[i] = gelu_tanh_precise(gate + b0) * (up + b1);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (c0 + 2 * i + upper < tl.rows && feat_ok) o[(int64_t)(2 * i + upper) * Nout] = v[i];
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (c0 + i < tl.rows && feat_ok) o[(int64_t)i * Nout] = acc[0][i] + b0;
        }
      }
    }
    if (splits > 1) {
      __syncwarp();
      if (!sent) cluster_sync();     // (a cluster without a tile)
      cluster_sync();                // the sums of all ranges are there (or a wait ran out, and the status says so)
      if (first < total) {
        const Tile tl = tile_of(ctl, E, m_tiles, first);
        const float* bias = static_cast<const float*>(bp[tl.e]);
        auto sum4 = [&](const float* p, float (&v)[4]) {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = 0.f;
          for (int q = 0; q < splits; ++q, p += kRowsA * 8) {
            const float4 u = *reinterpret_cast<const float4*>(p);
            v[0] += u.x; v[1] += u.y; v[2] += u.z; v[3] += u.w;
          }
        };
        // a thread: one feature of four tokens
        const int et = threadIdx.x - 32 * kEpiFirst, j = et & (kFeatures - 1), half = et / kFeatures;
        const int feat = tl.m * kFeatures + j;
        const int r = GEGLU ? (j >> 4) * 32 + (j & 15) : j;
        if (half < 2 && feat < Nout) {
          const float b0 = __ldg(bias + feat), b1 = GEGLU ? __ldg(bias + Nout + feat) : 0.f;
          for (int g = rank; g * 8 < tl.rows; g += splits) {
            const int c0 = g * 8 + half * 4;
            const float* p = reinterpret_cast<const float*>(smem) + ((g & -splits) * kRowsA + r) * 8 + half * 4;
            float v[8];
            sum4(p, reinterpret_cast<float(&)[4]>(v[0]));
            if (GEGLU) sum4(p + 16 * 8, reinterpret_cast<float(&)[4]>(v[4]));
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (c0 + i < tl.rows)
                out[(int64_t)(tl.row0 + c0 + i) * Nout + feat] =
                    GEGLU ? gelu_tanh_precise(v[i] + b0) * (v[4 + i] + b1) : v[i] + b0;
          }
        }
      }
    }
  }

  // ---------------- teardown ----------------
  __syncwarp();
  if (*reinterpret_cast<volatile int*>(&ctl->abort)) {
    unsigned long long t0 = global_ns();
    while (global_ns() - t0 < 1000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// CTAs that share a tile: while all clusters still run at once (74 of two CTAs, 32 of four and 12 of eight do), with four
// steps of K or more each. The host does not know the routing: every expert that can have rows is taken to have them.
int pick_splits(int64_t tiles, int K) {
  const int kb = (K + BK - 1) / BK;
  if (tiles <= 12 && kb >= 32) return 8;
  if (tiles <= 32 && kb >= 16) return 4;
  if (tiles <= 74 && kb >= 8) return 2;
  return 1;
}

template <bool GEGLU>
int launch(const float* A, const int32_t* offsets, const void* tmaps_w, const void* const* W, const void* const* b,
           int64_t M, int K, int Nout, int E, float* out, int32_t* status, cudaStream_t s) {
  static PerDeviceOnce once;
  int rc = ensure_dynamic_smem(once, ffn_f32_kernel<GEGLU>, kSmemBytes);
  if (rc) return rc;
  alignas(64) CUtensorMap tm;
  rc = encode_tmap_2d_f32(&tm, A, (uint64_t)M, (uint64_t)K, 16);
  if (rc) return rc;
  int sms = 0;
  rc = sm_count(&sms);
  if (rc) return rc;
  const int64_t m_tiles = (Nout + (GEGLU ? 64 : 128) - 1) / (GEGLU ? 64 : 128);
  const int64_t hit = M < E ? M : E, full = (M + kMaxN - 1) / kMaxN;
  const int splits = pick_splits((hit > full ? hit : full) * m_tiles, K);
  const int64_t most = (M / kMaxN + hit) * m_tiles;        // tiles there can be
  const unsigned grid = splits > 1 ? (unsigned)(most * splits) : (unsigned)(most < sms ? most : sms);
  MOE_CUDA_CHECK(launch_pdl_cluster(ffn_f32_kernel<GEGLU>, dim3(grid), dim3(kThreads), splits, kSmemBytes, s, tm,
                                    static_cast<const CUtensorMap*>(tmaps_w), A, offsets, W, b, E, K, Nout, splits, out,
                                    status));
  return 0;
}

}  // namespace

int launch_experts_f32(const void* perm, const int32_t* offsets, const void* plan, int64_t M, int d, int f, int E, void* h,
                       void* y, int32_t* status, cudaStream_t s) {
  if (M == 0) return 0;
  PlanView pv = plan_view(plan, E);
  int rc = launch<true>(static_cast<const float*>(perm), offsets, pv.tmap_W1, pv.W1, pv.b1, M, d, f, E,
                        static_cast<float*>(h), status, s);
  if (rc) return rc;
  return launch<false>(static_cast<const float*>(h), offsets, pv.tmap_W2, pv.W2, pv.b2, M, f, d, E,
                       static_cast<float*>(y), status, s);
}

}  // namespace moe
