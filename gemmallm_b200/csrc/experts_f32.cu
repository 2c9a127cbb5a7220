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
//   warp 0       loads boxes by TMA, three or four stages ahead
//   warp 1       one lane issues the products (A from tensor memory, B from shared memory), two steps at a time
//   then split warps, half of them on even and half on odd steps: their row of A into tensor memory (tcgen05.st)
//   and epilogue warps, which add up the products, then bias, GELU and the store
// In whole calls (PLANES) the tokens come as three bf16 planes, split once by the kernel in front (front_small.cuh) and by
// the GEGLU pass's epilogue: one box a step brings all three, and 8 split and 16 epilogue warps are at work. Where h is the
// caller's fp32 tensor, or the rows come from the dispatch kernel, 16 split warps also turn the tokens' boxes into three bf16
// tiles, and 8 warps are left for the epilogue.
// Where tiles are few K is split: the GEGLU pass over a cluster of up to eight CTAs, every one of which sends each other one
// its sums of that one's tokens through distributed shared memory, to be added in rank order; the down pass on planes over
// blocks that leave partial sums to the combine kernel (the exchange took 6 of that pass's 26 us).
//
// What bounds it (clk of 1.9 GHz, 512 tokens, d 512, f 2048, 8 experts, top-2): a step takes 1000 to 1100 for 768 of products
// at N 128; a pass's first step is done 7000 to 9000 after the routing is known, most of it code that runs for the first time;
// the epilogue 5000 to 8000, stores and again code that is cold. The call 95.4 -> 81.8 us: a step 1500 -> 1100 (tokens split
// once, 1024 tokens 145.9 -> 134; the issuing lane looking at half as many barriers), epilogue warps and partial sums the
// rest; 1 / 16 / 128 / 2048 tokens 38.1 -> 35.2, 61.5 -> 57.2, 71.3 -> 65.6, 243 -> 228. Error of h and y against 64 bits, in
// the 2-norm, at 2 to 4096 rows: 1.8e-7 and 0.9e-7 to 1.4e-7.
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
constexpr int kRawA = kRowsA * BK * 4;            // 16 KiB, rows of 128 bytes
constexpr int kRawB = kMaxN * BK * 4;
constexpr int kPlane = kMaxN * BK * 2;            // one bf16 tile of the tokens, rows of 64 bytes
constexpr int kThreads = 896;
constexpr int kMaxStages = 4;
// PLANES: the tokens come as three bf16 planes, and only the weights are split here: half as many warps do, and the others
// are epilogue warps.
template <bool PLANES>
struct Cfg {
  static constexpr int kStages = PLANES ? 4 : 3;
  static constexpr int kRawBytes = kRawA + (PLANES ? 0 : kRawB);
  static constexpr int kSplitWarps = PLANES ? 4 : 8;        // of a step; as many on even as on odd steps
  static constexpr int kEpiFirst = 4 + 2 * kSplitWarps;
  static constexpr int kEpiWarps = kThreads / 32 - kEpiFirst;
  static constexpr int kParts = kEpiWarps / 4;              // warps that share the tile's tokens, eight at a time in turn
  static constexpr int kGroups = (kMaxN / 8 + kParts - 1) / kParts;   // groups of eight tokens per epilogue warp
  // Registers: 896 threads start with 72 each, 504 for the seven warps of a thread index
  static constexpr int kRegsLoad = PLANES ? 56 : 40, kRegsSplit = 48, kRegsEpi = PLANES ? 88 : 136;
  static_assert(kRegsLoad + kSplitWarps / 2 * kRegsSplit + kParts * kRegsEpi <= 7 * 72,
                "a share above the launch's registers would wait for good");
  static constexpr size_t kStageBytes = (size_t)kStages * (kRawBytes + 3 * kPlane);
};
constexpr int kMainCol = 0, kSmallCol = kMaxN, kACol = 2 * kMaxN;   // tensor memory columns
constexpr int kACols = 3 * BK / 2;                                  // of one stage of A
constexpr int kLargeSteps = 2, kSmallSteps = 8;   // steps of K after which an accumulator is read out and started again
static_assert(kACol + kMaxStages * kACols <= 512, "tensor memory");
static_assert((kMaxN / 8 + 4) * kRowsA * 32 <= Cfg<false>::kStages * Cfg<false>::kRawBytes &&
              (kMaxN / 8 + 4) * kRowsA * 32 <= Cfg<true>::kStageBytes, "sums of all ranges reuse the stages");

struct Control {
  uint64_t raw_full[kMaxStages], raw_empty[kMaxStages];
  uint64_t conv_full[kMaxStages], conv_empty[kMaxStages];
  uint64_t main_full, main_empty, small_full, small_empty;
  uint32_t tmem_base;
  int abort;
  int offsets[kMaxExperts + 1];
  int block_start[kMaxExperts + 1];   // token blocks of the experts before
};
template <bool PLANES>
constexpr size_t kSmemBytes = 1024 + Cfg<PLANES>::kStageBytes + sizeof(Control);
static_assert(kSmemBytes<false> <= 227 * 1024 && kSmemBytes<true> <= 227 * 1024, "shared memory of one CTA");

// The activations. Split in the kernel: 16-row boxes of 32 columns in rows[0]. PLANES: [3][M][K] bf16, boxes of 32 columns
// of 32, 64, ..., 160 rows of all planes.
struct TokenMaps {
  CUtensorMap rows[kMaxN / 32];
};

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

__device__ __forceinline__ void split8(const float (&x)[8], uint32_t (&p0)[4], uint32_t (&p1)[4], uint32_t (&p2)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) split2(x[2 * i], x[2 * i + 1], p0[i], p1[i], p2[i]);
}

// (a: the rows may come from the kernel before this one, so they are not read as constant data)
__device__ __forceinline__ float dot_f32(const float* a, const float* w, int k0, int k1) {
  float s = 0.f;
#pragma unroll 1
  for (int k = k0; k < k1; ++k) s = fmaf(__ldcg(a + k), w[k], s);
  return s;
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= FLT_MAX; }

// Row `a` of three bf16 planes: what they are the parts of (an infinity's other parts are NaN).
__device__ __forceinline__ float join(const __nv_bfloat16* a, int64_t plane) {
  const float p0 = __bfloat162float(__ldcg(a));
  return fabsf(p0) <= FLT_MAX ? p0 + (__bfloat162float(__ldcg(a + plane)) + __bfloat162float(__ldcg(a + 2 * plane))) : p0;
}
__device__ __forceinline__ float dot_planes(const __nv_bfloat16* a, int64_t plane, const float* w, int k0, int k1) {
  float s = 0.f;
#pragma unroll 1
  for (int k = k0; k < k1; ++k) s = fmaf(join(a + k, plane), w[k], s);
  return s;
}

// The sums of eight tokens have been used: those of the next eight take their place.
template <int kGroups>
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

__device__ __forceinline__ void tma_load_planes(void* dst, const void* tmap, uint64_t* bar, int k, int row) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(k), "r"(row), "r"(0)
      : "memory");
}

// A: [M, K] activations (sorted buffer); W_e: [Nw, K]; out [M, Nout].
// GEGLU: Nw = 2 * Nout, gate rows [0, Nout), up rows [Nout, 2 * Nout).
// PLANES: the activations are read as bf16 planes, and the GEGLU pass writes its own so; A is read again where a sum is
// formed again, fp32 rows in the GEGLU pass, planes in the down pass.
// splits: CTAs of a cluster; with more than one a cluster has one tile at most.
template <bool GEGLU, bool PLANES>
__global__ void __launch_bounds__(kThreads, 1)
ffn_f32_kernel(const __grid_constant__ TokenMaps tmap_a, const CUtensorMap* __restrict__ tmap_w,   // [E], 64-row boxes of 32
               const void* __restrict__ A, const int32_t* __restrict__ offsets, const void* const* __restrict__ Wp,
               const void* const* __restrict__ bp, int64_t M, int E, int K, int Nout, int splits, void* __restrict__ out_raw,
               int32_t* __restrict__ status) {
  using C = Cfg<PLANES>;
  constexpr int kStages = C::kStages, kRawBytes = C::kRawBytes, kEpiFirst = C::kEpiFirst, kParts = C::kParts, kGroups = C::kGroups;
  float* out = static_cast<float*>(out_raw);
  __nv_bfloat16* out_planes = static_cast<__nv_bfloat16*>(out_raw);     // PLANES && GEGLU: [3][M][Nout]
  const int64_t plane_out = M * Nout;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* planes = smem + (size_t)kStages * kRawBytes;         // [kStages][3] bf16 tiles of the tokens
  Control* ctl = reinterpret_cast<Control*>(planes + kStages * 3 * kPlane);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kFeatures = GEGLU ? 64 : 128;                    // output columns of a tile
  const int m_tiles = (Nout + kFeatures - 1) / kFeatures;
  // K over a cluster that adds its sums up, or (the down pass on planes) over blocks that leave them to the combine kernel
  constexpr bool kParted = PLANES && !GEGLU;
  const bool clustered = !kParted && splits > 1;
  const int rank = kParted ? (int)(blockIdx.x % splits) : clustered ? (int)cluster_rank() : 0;
  const int first = blockIdx.x / splits, step = gridDim.x / splits;
  const int kb_all = (K + BK - 1) / BK;
  const int kb_per = (kb_all + splits - 1) / splits;
  const int kb0 = min(kb_all, rank * kb_per), kn = min(kb_all, kb0 + kb_per) - kb0;   // this CTA's steps of K

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&ctl->raw_full[s], 1);
      mbar_init(&ctl->raw_empty[s], C::kSplitWarps);
      mbar_init(&ctl->conv_full[s], C::kSplitWarps + (PLANES ? 1 : 0));   // and the planes
      mbar_init(&ctl->conv_empty[s], 1);
    }
    mbar_init(&ctl->main_full, 1);
    mbar_init(&ctl->main_empty, C::kEpiWarps);
    mbar_init(&ctl->small_full, 1);
    mbar_init(&ctl->small_empty, C::kEpiWarps);
    ctl->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  if (warp == 2) {
    if (lane < (PLANES ? kMaxN / 32 : 1)) prefetch_tmap(&tmap_a.rows[lane]);
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
    fewer_registers<C::kRegsLoad>();
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
          mbar_expect_tx(&ctl->raw_full[s], (uint32_t)(kRawA + (PLANES ? 0 : tl.n * BK * 4)));
          tma_load_2d(dst, tw, &ctl->raw_full[s], k, r0);
          tma_load_2d(dst + kRawA / 2, tw, &ctl->raw_full[s], k, r1);
          if constexpr (PLANES) {
            if (!mbar_wait(&ctl->conv_empty[s], phase ^ 1u, &ctl->abort, status, 59)) { ok = false; break; }
            const int boxes = (tl.n + 31) >> 5;
            mbar_expect_tx(&ctl->conv_full[s], (uint32_t)(boxes * 32 * 3 * BK * 2));
            tma_load_planes(planes + (size_t)s * 3 * kPlane, &tmap_a.rows[boxes - 1], &ctl->conv_full[s], k, tl.row0);
          } else {
            for (int j = 0; j < tl.n; j += 16)
              tma_load_2d(dst + kRawA + j * BK * 4, &tmap_a.rows[0], &ctl->raw_full[s], k, tl.row0 + j);
          }
          if (++s == kStages) { s = 0; phase ^= 1u; }
        }
      }
    } else if (warp == 1 && elect_one()) {
      // ---------------- products ----------------
      uint32_t phase = 0, larges = 0, smalls = 0;
      int c = 0;
      bool ok = true;
      for (int t = first; ok && t < total; t += step) {
        const Tile tl = tile_of(ctl, E, m_tiles, t);
        const uint32_t idesc = make_idesc(tl.n);
        // 16-byte units from one plane of the tokens to the next
        const uint64_t kP = PLANES ? (uint64_t)((tl.n + 31) >> 5) * (32 * BK * 2 / 16) : (uint64_t)(kPlane / 16);
        // Two steps at a time, their large products first: those sums are read out while the small products run, and the
        // thread that issues has to look at barriers half as often (46 clk a product, 60 to 100 a barrier or commit).
        // (of three stages, which the split of tokens here leaves, two would be taken: there a step at a time; d 512, f 2048, 8 experts,
        // 2049 / 4000 / 8000 tokens 267 / 443 / 746 us in pairs, 253 / 420 / 712 so)
        static_assert(kLargeSteps == 2 && kSmallSteps % 2 == 0, "steps go in pairs");
        auto small_products = [&](uint32_t a, uint64_t b, bool more) {
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            const uint32_t ak = a + kk * 8;
            const uint64_t bk = b + kk * 2;
            mma_ts(tmem + kSmallCol, ak + 32, bk, idesc, more || kk != 0 ? 1u : 0u);   // a2 b0
            mma_ts(tmem + kSmallCol, ak, bk + 2 * kP, idesc, 1u);                      // a0 b2
            mma_ts(tmem + kSmallCol, ak + 16, bk + kP, idesc, 1u);                     // a1 b1
            mma_ts(tmem + kSmallCol, ak + 16, bk, idesc, 1u);                          // a1 b0
            mma_ts(tmem + kSmallCol, ak, bk + kP, idesc, 1u);                          // a0 b1
          }
        };
        for (int i = 0; !PLANES && i < kn; ++i) {
          if (!mbar_wait(&ctl->conv_full[c], phase, &ctl->abort, status, 53)) { ok = false; break; }
          if (i % kLargeSteps == 0 && !mbar_wait(&ctl->main_empty, (larges++ & 1u) ^ 1u, &ctl->abort, status, 54)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a = tmem + kACol + c * kACols;
          const uint64_t b = desc64(smem_u32(planes) + (uint32_t)(c * 3 * kPlane));
          mma_ts(tmem + kMainCol, a, b, idesc, i % kLargeSteps != 0 ? 1u : 0u);
          mma_ts(tmem + kMainCol, a + 8, b + 2, idesc, 1u);
          if ((i + 1) % kLargeSteps == 0 || i + 1 == kn) tc_commit(&ctl->main_full);
          if (i % kSmallSteps == 0) {
            if (!mbar_wait(&ctl->small_empty, (smalls++ & 1u) ^ 1u, &ctl->abort, status, 52)) { ok = false; break; }
            tc_fence_after();
          }
          small_products(a, b, i % kSmallSteps != 0);
          if ((i + 1) % kSmallSteps == 0 || i + 1 == kn) tc_commit(&ctl->small_full);
          tc_commit(&ctl->conv_empty[c]);
          if (++c == kStages) { c = 0; phase ^= 1u; }
        }
        for (int i = 0; PLANES && i < kn; i += 2) {
          const bool two = i + 1 < kn;
          const int c1 = c + 1 == kStages ? 0 : c + 1;
          const uint32_t phase1 = c + 1 == kStages ? phase ^ 1u : phase;
          if (!mbar_wait(&ctl->conv_full[c], phase, &ctl->abort, status, 53)) { ok = false; break; }
          if (!mbar_wait(&ctl->main_empty, (larges++ & 1u) ^ 1u, &ctl->abort, status, 54)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a0 = tmem + kACol + c * kACols, a1 = tmem + kACol + c1 * kACols;
          const uint64_t b0 = desc64(smem_u32(planes) + (uint32_t)(c * 3 * kPlane));
          const uint64_t b1 = desc64(smem_u32(planes) + (uint32_t)(c1 * 3 * kPlane));
          mma_ts(tmem + kMainCol, a0, b0, idesc, 0u);
          mma_ts(tmem + kMainCol, a0 + 8, b0 + 2, idesc, 1u);
          if (two) {
            if (!mbar_wait(&ctl->conv_full[c1], phase1, &ctl->abort, status, 53)) { ok = false; break; }
            tc_fence_after();
            mma_ts(tmem + kMainCol, a1, b1, idesc, 1u);
            mma_ts(tmem + kMainCol, a1 + 8, b1 + 2, idesc, 1u);
          }
          tc_commit(&ctl->main_full);
          if (i % kSmallSteps == 0) {
            if (!mbar_wait(&ctl->small_empty, (smalls++ & 1u) ^ 1u, &ctl->abort, status, 52)) { ok = false; break; }
            tc_fence_after();
          }
          small_products(a0, b0, i % kSmallSteps != 0);
          tc_commit(&ctl->conv_empty[c]);
          if (two) {
            small_products(a1, b1, true);
            tc_commit(&ctl->conv_empty[c1]);
          }
          if ((i + 2) % kSmallSteps == 0 || i + 2 >= kn) tc_commit(&ctl->small_full);
          if (two) { c = c1; phase = phase1; }
          if (++c == kStages) { c = 0; phase ^= 1u; }
        }
      }
    }
    __syncwarp();
    if (clustered) { cluster_sync(); cluster_sync(); }
  } else if (warp < kEpiFirst) {
    // ---------------- split ----------------
    fewer_registers<C::kRegsSplit>();
    constexpr int kSplitWarps = C::kSplitWarps;
    const int quad = warp & 3, part = PLANES ? 0 : ((warp - 4) >> 2) & 1;   // lanes of tensor memory; half of the step's K
    const int group = (warp - 4) / kSplitWarps;
    const int et = (threadIdx.x - 128) % (32 * kSplitWarps);
    // the row of the raw tile that goes to this lane. GEGLU: gate and up of a feature in one warp, 16 lanes apart
    const int r = GEGLU ? (lane & 15) + quad * 16 + (lane >> 4) * 64 : quad * 32 + lane;
    int s = 0, turn = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = first; ok && t < total; t += step) {
      const Tile tl = tile_of(ctl, E, m_tiles, t);
      for (int i = 0; i < kn; ++i, turn ^= 1) {
        const int c = s;
        const uint32_t ph = phase;
        if (++s == kStages) { s = 0; phase ^= 1u; }
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
        for (int j = 0; j < 16 / kSplitWarps; ++j) {
          float x[8];
          uint32_t p0[4], p1[4], p2[4];
          load8_at(raw + r * 128, r, part * 4 + j * 2, x);
          split8(x, p0, p1, p2);
          st_tmem4(ta + j * 4, p0);
          st_tmem4(ta + 16 + j * 4, p1);
          st_tmem4(ta + 32 + j * 4, p2);
        }
        uint8_t* pl = planes + (size_t)c * 3 * kPlane;
        for (int q = et; !PLANES && q < tl.n * 4; q += 32 * kSplitWarps) {      // a token's eight values at a time
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
        if (!PLANES) fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&ctl->conv_full[c]);
          mbar_arrive(&ctl->raw_empty[c]);
        }
      }
    }
    __syncwarp();
    if (clustered) { cluster_sync(); cluster_sync(); }
  } else {
    // ---------------- sums and epilogue: lane = weight row, columns = tokens ----------------
    more_registers<C::kRegsEpi>();
    const int quad = warp & 3, part = (warp - kEpiFirst) >> 2;   // this warp: token groups part, part + kParts, ...
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
      const int feat = tl.m * kFeatures + (GEGLU ? quad * 16 + (lane & 15) : quad * 32 + lane);
      const bool feat_ok = feat < Nout;
      // (asked for here: behind the products their way from memory took longer than the rest of the epilogue)
      const bool biased = !clustered && !(kParted && splits > 1);
      const float* bias = biased && feat_ok ? static_cast<const float*>(bp[tl.e]) : nullptr;
      const float b0 = bias != nullptr ? __ldg(bias + feat) : 0.f;
      const float b1 = GEGLU && bias != nullptr ? __ldg(bias + Nout + feat) : 0.f;
      uint64_t again = 0;      // a bit per sum of this thread whose small products were not finite, ...
      uint32_t again_hi = 0;   // ... from the ninth group on
      auto add = [&](int col) {
        // (groups past n hold old sums; they are not used)
        constexpr int kAtOnce = PLANES ? 3 : 4;
#pragma unroll
        for (int g0 = 0; g0 < kGroups; g0 += kAtOnce) {
          if ((g0 * kParts + part) * 8 >= tl.n) break;
          uint32_t v[kAtOnce][8];
#pragma unroll
          for (int g = 0; g < kAtOnce; ++g)
            if (g0 + g < kGroups) ld_tmem8(ta + col + (g0 + g) * 8 * kParts, v[g]);
          tc_ld_wait();
#pragma unroll
          for (int g = 0; g < kAtOnce; ++g)
            if (g0 + g < kGroups) {
#pragma unroll
              for (int i = 0; i < 8; ++i) acc[g0 + g][i] += __uint_as_float(v[g][i]);
            }
        }
      };
      // Small products that are not finite become zero and are noted.
      auto add_small = [&]() {
        if constexpr (PLANES) {
          constexpr int kAtOnce = 3;
          static_assert(kGroups <= 8, "bits of `again`");
#pragma unroll
          for (int g0 = 0; g0 < kGroups; g0 += kAtOnce) {
            if ((g0 * kParts + part) * 8 >= tl.n) break;
            uint32_t v[kAtOnce][8];
#pragma unroll
            for (int g = 0; g < kAtOnce; ++g)
              if (g0 + g < kGroups) ld_tmem8(ta + kSmallCol + (g0 + g) * 8 * kParts, v[g]);
            tc_ld_wait();
#pragma unroll
            for (int g = 0; g < kAtOnce; ++g)
              if (g0 + g < kGroups) {
                float probe[2] = {0.f, 0.f};      // times zero: NaN where one is not finite
#pragma unroll
                for (int i = 0; i < 8; ++i) probe[i & 1] = fmaf(__uint_as_float(v[g][i]), 0.f, probe[i & 1]);
                if (probe[0] + probe[1] != 0.f) {
#pragma unroll
                  for (int i = 0; i < 8; ++i)
                    if (!finite(__uint_as_float(v[g][i]))) {
                      v[g][i] = 0u;
                      again |= 1ull << ((g0 + g) * 8 + i);
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[g0 + g][i] += __uint_as_float(v[g][i]);
              }
          }
        } else {
          // (in tensor memory: twenty groups in registers leave no room to do it on the way)
          static_assert(PLANES || (kGroups % 2 == 0 && kGroups <= 12), "two groups at a time, 96 bits");
#pragma unroll 1
          for (int g0 = 0; (g0 * kParts + part) * 8 < tl.n; g0 += 2) {
            uint32_t v[2][8];
            ld_tmem8(ta + kSmallCol + g0 * 8 * kParts, v[0]);
            ld_tmem8(ta + kSmallCol + (g0 + 1) * 8 * kParts, v[1]);
            tc_ld_wait();
            float probe[2] = {0.f, 0.f};
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
              st_tmem8(ta + kSmallCol + g0 * 8 * kParts, v[0]);
              st_tmem8(ta + kSmallCol + (g0 + 1) * 8 * kParts, v[1]);
              st_tmem_wait();
              if (g0 < 8) again |= (uint64_t)bits << (g0 * 8); else again_hi |= bits << (g0 * 8 - 64);
            }
          }
          add(kSmallCol);
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
          add_small();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->small_empty);
        }
      }
      if (!ok && !clustered) break;
      // The sums at hand, of eight tokens from c0 on: those that lack their small products and are finite without them are
      // formed again, over this CTA's range of K.
      auto form_again = [&](int c0) {
        if ((again | again_hi) == 0) return;       // none of this thread's; nothing below needs the warp
        const uint32_t bits = (uint32_t)again & 0xffu;
        again = again >> 8 | (uint64_t)again_hi << 56;
        again_hi >>= 8;
        if (bits != 0u && feat_ok) {
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = acc[0][i];
          const float* w = static_cast<const float*>(Wp[tl.e]) + (int64_t)(GEGLU && lane >= 16 ? Nout + feat : feat) * K;
#pragma unroll 1
          for (int i = 0; i < 8 && c0 + i < tl.rows; ++i)
            if ((bits >> i & 1u) != 0u && finite(v[i]))
            {
              const int64_t at = (int64_t)(tl.row0 + c0 + i) * K;
              const int k0 = kb0 * BK, k1 = min(K, (kb0 + kn) * BK);
              v[i] = PLANES && !GEGLU ? dot_planes(static_cast<const __nv_bfloat16*>(A) + at, M * K, w, k0, k1)
                                      : dot_f32(static_cast<const float*>(A) + at, w, k0, k1);
            }
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[0][i] = v[i];
        }
      };
      if (clustered) {
        // Eight tokens at a time go to the CTAs in turn, which keep them as [eight][source][128 rows][8 tokens] in
        // their raw stages.
        __syncwarp();
        cluster_sync();    // no CTA reads its raw stages any more
        const uint32_t mine = smem_u32(smem) + (uint32_t)((rank * kRowsA + quad * 32 + lane) * 32);
#pragma unroll 1
        for (int g = part; g * 8 < tl.n; g += kParts, next_group(acc)) {
          form_again(g * 8);
          __syncwarp();
          const uint32_t to = map_to_cta(mine, g & (splits - 1)) + (uint32_t)((g & -splits) * kRowsA * 32);
          st_cluster4(to, acc[0][0], acc[0][1], acc[0][2], acc[0][3]);
          st_cluster4(to + 16, acc[0][4], acc[0][5], acc[0][6], acc[0][7]);
        }
        sent = true;
        break;
      }
      // rolled, and the sums moved up: unrolled, 60 KB of code that runs from a cold instruction cache took 30000 clk
#pragma unroll 1
      for (int c0 = part * 8; c0 < tl.rows; c0 += 8 * kParts, next_group(acc)) {
        form_again(c0);
        __syncwarp();
        float* o = out + ((kParted ? rank * M : 0) + tl.row0 + c0) * Nout + feat;
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
          if constexpr (PLANES) {
            // lanes of even features take the first two of their tokens for both features, the others the last two
            const int odd = lane & 1;
            const float r0 = __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[2], 1);
            const float r1 = __shfl_xor_sync(0xffffffffu, odd ? v[1] : v[3], 1);
            const float pair[2][2] = {{odd ? r0 : v[0], odd ? v[2] : r0}, {odd ? r1 : v[1], odd ? v[3] : r1}};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int token = c0 + 4 * odd + 2 * i + upper;
              if (token < tl.rows && feat_ok) {
                uint32_t p0, p1, p2;
                split2(pair[i][0], pair[i][1], p0, p1, p2);
                __nv_bfloat16* q = out_planes + (int64_t)(tl.row0 + token) * Nout + (feat - odd);
                *reinterpret_cast<uint32_t*>(q) = p0;
                *reinterpret_cast<uint32_t*>(q + plane_out) = p1;
                *reinterpret_cast<uint32_t*>(q + 2 * plane_out) = p2;
              }
            }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (c0 + 2 * i + upper < tl.rows && feat_ok) o[(int64_t)(2 * i + upper) * Nout] = v[i];
          }
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (c0 + i < tl.rows && feat_ok) o[(int64_t)i * Nout] = acc[0][i] + b0;
        }
      }
    }
    if (clustered) {
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
        // a thread: one feature of four tokens at a time
        constexpr int kUnits = 32 * C::kEpiWarps / kFeatures;
        const int et = threadIdx.x - 32 * kEpiFirst, j = et & (kFeatures - 1);
        const int feat = tl.m * kFeatures + j;
        const int r = GEGLU ? (j >> 4) * 32 + (j & 15) : j;
        if (feat < Nout) {
          const float b0 = __ldg(bias + feat), b1 = GEGLU ? __ldg(bias + Nout + feat) : 0.f;
          for (int u = et / kFeatures;; u += kUnits) {
            const int g = rank + (u >> 1) * splits, half = u & 1;
            if (g * 8 >= tl.rows) break;
            const int c0 = g * 8 + half * 4;
            const float* p = reinterpret_cast<const float*>(smem) + ((g & -splits) * kRowsA + r) * 8 + half * 4;
            float v[8];
            sum4(p, reinterpret_cast<float(&)[4]>(v[0]));
            if (GEGLU) sum4(p + 16 * 8, reinterpret_cast<float(&)[4]>(v[4]));
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (c0 + i < tl.rows) {
                const float o = GEGLU ? gelu_tanh_precise(v[i] + b0) * (v[4 + i] + b1) : v[i] + b0;
                const int64_t at = (int64_t)(tl.row0 + c0 + i) * Nout + feat;
                if constexpr (GEGLU && PLANES) {
                  uint32_t p0, p1, p2;
                  split2(o, 0.f, p0, p1, p2);
                  reinterpret_cast<uint16_t*>(out_planes)[at] = (uint16_t)p0;
                  reinterpret_cast<uint16_t*>(out_planes)[at + plane_out] = (uint16_t)p1;
                  reinterpret_cast<uint16_t*>(out_planes)[at + 2 * plane_out] = (uint16_t)p2;
                } else {
                  out[at] = o;
                }
              }
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

}  // namespace

// Ranges of K of the down pass on planes, a part of the sums each: those with which the rounds of tiles take the fewest
// steps, a tile's start, epilogue and partial sums counted as five. (The host does not know the routing: every expert that
// can have rows is taken to have them.)
int f32_down_splits(int64_t M, int d, int f, int E) {
  const int64_t hit = M < E ? M : E, full = (M + kMaxN - 1) / kMaxN, kb = (f + BK - 1) / BK;
  const int64_t tiles = (hit > full ? hit : full) * ((d + 127) / 128);
  int best = 1;
  int64_t least = 0;
  for (int s = 1; s <= 8 && (s == 1 || kb >= 4 * s); ++s) {
    const int64_t cost = (tiles * s + kNumSMs - 1) / kNumSMs * ((kb + s - 1) / s + 5);
    if (s == 1 || cost < least) { best = s; least = cost; }
  }
  return best;
}

namespace {

// A: fp32 rows; planes: [3][M][K] bf16, or nullptr and A is split in the kernel.
template <bool GEGLU, bool PLANES>
int launch(const void* A, const void* planes, const int32_t* offsets, const void* tmaps_w, const void* const* W,
           const void* const* b, int64_t M, int K, int Nout, int E, void* out,
           int32_t* status, cudaStream_t s) {
  static PerDeviceOnce once;
  auto kernel = ffn_f32_kernel<GEGLU, PLANES>;
  int rc = ensure_dynamic_smem(once, kernel, kSmemBytes<PLANES>);
  if (rc) return rc;
  alignas(64) TokenMaps tm;
  if (PLANES) {
    for (int i = 0; i < kMaxN / 32 && rc == 0; ++i)
      if (i * 32 < M) rc = encode_tmap_planes(&tm.rows[i], planes, (uint64_t)M, (uint64_t)K, 32 * (i + 1));
      else tm.rows[i] = tm.rows[0];         // no block has more tokens than there are rows
  } else {
    rc = encode_tmap_2d_f32(&tm.rows[0], A, (uint64_t)M, (uint64_t)K, 16);
  }
  if (rc) return rc;
  int sms = 0;
  rc = sm_count(&sms);
  if (rc) return rc;
  const int64_t m_tiles = (Nout + (GEGLU ? 64 : 128) - 1) / (GEGLU ? 64 : 128);
  const int64_t hit = M < E ? M : E, full = (M + kMaxN - 1) / kMaxN;
  constexpr bool kParted = PLANES && !GEGLU;
  const int splits = kParted ? f32_down_splits(M, Nout, K, E) : pick_splits((hit > full ? hit : full) * m_tiles, K);
  const int64_t most = (M / kMaxN + hit) * m_tiles;        // tiles there can be
  const int64_t at_once = kParted ? sms / splits : splits > 1 ? most : sms;     // a cluster has one tile at most
  const unsigned grid = (unsigned)((most < at_once || at_once < 1 ? most : at_once) * splits);
  MOE_CUDA_CHECK(launch_pdl_cluster(kernel, dim3(grid), dim3(kThreads), kParted ? 1 : splits, kSmemBytes<PLANES>, s, tm,
                                    static_cast<const CUtensorMap*>(tmaps_w), PLANES && !GEGLU ? planes : A, offsets, W, b, M,
                                    E, K, Nout, splits, out, status));
  return 0;
}

}  // namespace

int launch_experts_f32(const void* perm, const int32_t* offsets, const void* plan, int64_t M, int d, int f, int E, void* h,
                       void* y, int32_t* status, cudaStream_t s) {
  if (M == 0) return 0;
  PlanView pv = plan_view(plan, E);
  int rc = launch<true, false>(perm, nullptr, offsets, pv.tmap_W1, pv.W1, pv.b1, M, d, f, E, h, status, s);
  if (rc) return rc;
  return launch<false, false>(h, nullptr, offsets, pv.tmap_W2, pv.W2, pv.b2, M, f, d, E, y, status, s);
}

// The same with perm in three bf16 planes [3][M, d] as well, and h [3][M, f] kept in planes only. y: [M, d], or with more
// than one of f32_down_splits() the partial sums [splits][M, d] without down.bias.
int launch_experts_f32_planes(const void* perm, const void* perm_planes, const int32_t* offsets, const void* plan, int64_t M,
                              int d, int f, int E, void* h_planes, void* y, int32_t* status, cudaStream_t s) {
  if (M == 0) return 0;
  PlanView pv = plan_view(plan, E);
  int rc = launch<true, true>(perm, perm_planes, offsets, pv.tmap_W1, pv.W1, pv.b1, M, d, f, E, h_planes, status, s);
  if (rc) return rc;
  return launch<false, true>(nullptr, h_planes, offsets, pv.tmap_W2, pv.W2, pv.b2, M, f, d, E, y, status, s);
}

}  // namespace moe
