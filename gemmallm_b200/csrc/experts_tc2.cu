// Grouped expert GEMMs with CTA pairs (tcgen05 cta_group::2): two neighbouring
// SMs share one 256-row x 256-column output tile. Each CTA stages its own 128
// rows of the activation operand and HALF of the weight tile (for the GEGLU
// pass CTA 0 holds the 128 gate rows, CTA 1 the 128 up rows); the pair's MMA
// (M=256, N=256, K=16), issued by the even CTA, reads both halves, and each
// CTA's TMEM receives the 128x256 accumulator of its own rows. Per 128x256x64
// step a CTA therefore pulls 32 KiB from L2 and shared memory instead of the
// 48 KiB a single CTA with a 128x256 tile would need: operand delivery, not the
// tensor pipe, is what bounds a one-CTA kernel of this shape.
//
// Synchronisation inside the pair (all mbarriers, all waits bounded):
//   full[s]       lives in the even CTA; both CTAs' TMA loads complete on it
//                 (cp.async.bulk.tensor ... cta_group::2, no multicast);
//   empty[s]      one per CTA; the MMA thread commits to its own and, through
//                 the cluster-mapped address, to its peer's;
//   tmem_full[a]  one per CTA, committed the same way;
//   tmem_empty[a] in the even CTA; the 16 epilogue warps of the pair arrive on
//                 it (the odd CTA's warps through the cluster-mapped address).
// Math and epilogue (tc_epilogue.cuh): reference model.py:174,180-184.
//
// The same kernel serves the backward pass (the reference trains through this block with
// torch.autograd, train.py:140). The input gradients are two more row-grouped products whose
// weights are read as they lie in memory: their rows are the contraction index there, so the B
// operand is MN-major in shared memory (B_MN; 64 x 64 boxes, see make_smem_desc_mn) and no
// transposed copy of the weights is made. The weight gradients dW_e = dY_e^T X_e (COLS) contract
// over an expert's rows: both operands are MN-major tiles of the activation buffers, a group is
// a range of rows, and every expert has the same output tiles. An expert's last 64-row block holds
// rows of the next expert; an eleventh warp (the "fixer") waits for such a block itself, zeroes
// those rows in shared memory up to the next multiple of 16, which is where the products of that
// block stop, and passes the stage on. (Only there do the two CTAs arrive on a common barrier: an
// arrival across the pair for every block halved the rate, 680 instead of 1280 TFLOP/s.)
//
// SPLIT > 1 (kPlain, kDx): products of few tiles and a long contraction. A tile of 256 x 256 takes 0.31 us per
// 64 of K however few of them run (shared memory's rate: 580 clk), so 28 tiles of K = 4096 left 46 pairs idle for 20 us.
// SPLIT pairs in one cluster take a range of K each, put their fp32 accumulators into shared memory (the stages are free by
// then: a cluster has one tile) and each adds up and stores 256 / SPLIT columns, in the order of the ranges. (128-column
// tiles instead gained nothing when the load loop still set the pace, 640 clk a step whatever the columns; they have not
// been measured since it does not.)
//
// kLinear, kLinearSkip: the Linears around the attention core (model.py:104, 139, 150), QKV and head gate as one product, the
// output Linear with the skip connection behind it (model.py:308), whose pieces are asked for before a tile's accumulator is
// awaited (in the epilogue's stores they made it the bound: 100 us, now 60 to 75). 32768 tokens, d 1024, 16 heads, one KV
// head: QKV and gate 75 us as two library products, 56 here; output Linear and addition 87, 65. A decoder layer, 8 experts,
// torch's Linears -> these: 512 tokens 108.6 -> 104.7 us, 1024 125.4 -> 120.3, 4096 236 -> 225, 6528 341 -> 328, 32768 1560 to 1629
// -> 1528 to 1591 (three runs each).
#include <cuda.h>
#include "common.cuh"
#include "tc_ptx.cuh"
#include "tc_pair.cuh"
#include "tc_epilogue.cuh"
#include "ep_sync.cuh"

namespace moe {

namespace {

using namespace tc;

constexpr int BM = 128;           // rows per CTA = TMEM lanes
constexpr int kPairRows = 256;    // rows per tile (both CTAs)
constexpr int BK = 64;
constexpr int BN = 256;
constexpr int kMaxStages = 6;
constexpr int kABytes = BM * BK * 2;         // 16 KiB: this CTA's rows
constexpr int kBBytes = (BN / 2) * BK * 2;   // 16 KiB: this CTA's half of the weight tile
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kTmemCols = 2 * BN;
constexpr int kPartPitch = BN + 4;       // SPLIT: floats per row of a partial tile in shared memory
constexpr int kHalfTile = 64 * BK * 2;   // one 64 x 64 box of an MN-major operand: 8 KiB

// What a launch computes. Rows of A are grouped by expert except in kWgrad.
enum Kind {
  kGeglu,        // h = gelu(x Wg^T + bg) * (x Wu^T + bu)
  kGegluTrain,   // the same with dropout, keeping the derivatives of h (TrainArgs)
  kGegluTrainPre,   // ... keeping pre-activations and mask (LoRA steps)
  kPlain,        // y = h W2^T + b2
  kScatter,      // the same into the token owners' buffers (expert parallelism)
  kDx,           // out = A B, B [K, Nout] as it lies in memory
  kDhGeglu,      // dh = dy W2 as kDx, times the derivatives of h in the epilogue
  kDhGegluBf16,  // from pre-activations and mask, with dh rounded to bf16 and the column sums over rounded values (LoRA steps)
  kWgrad,        // out_e [Ra, Nout] = A[rows of e]^T B[rows of e]
  kLinear,       // one group of rows, one or two weights: out = A W^T + b of both, column after column (LinearArgs)
  kLinearSkip    // ... of one, plus the skip connection
};
// The Linears around the attention core. 128 columns, a CTA's share of a tile's weights and an epilogue warp's of its
// columns, belong to one of the two.
struct LinearArgs {
  const __nv_bfloat16* bias[2];
  __nv_bfloat16* out[2];       // [rows, cols]
  int cols[2];
  int rows;
  const __nv_bfloat16* skip;   // kLinearSkip: [rows, cols[0]]
  __host__ __device__ int halves(int i) const { return (cols[i] + 127) / 128; }
  // (no index: parameters that are indexed are copied to local memory)
  __device__ __forceinline__ const __nv_bfloat16* bias_of(int i) const { return i ? bias[1] : bias[0]; }
  __device__ __forceinline__ __nv_bfloat16* out_of(int i) const { return i ? out[1] : out[0]; }
  __device__ __forceinline__ int cols_of(int i) const { return i ? cols[1] : cols[0]; }
};
// Where the 128 columns `half` of the tiles lie.
struct LinearHalf {
  int which, col, limit;       // limit: columns of the output; 0: none of these exist
  __device__ __forceinline__ LinearHalf(const LinearArgs& la, int half) {
    const int h0 = la.halves(0);
    which = half < h0 || la.cols[1] == 0 ? 0 : 1;
    col = (which ? half - h0 : half) * 128;
    limit = col < la.cols_of(which) ? la.cols_of(which) : 0;
  }
};
template <int KIND>
struct Traits {
  static constexpr bool TRAIN = KIND == kGegluTrain || KIND == kGegluTrainPre;
  static constexpr bool PRE = KIND == kGegluTrainPre;
  static constexpr bool GEGLU = KIND == kGeglu || TRAIN;
  static constexpr bool COLS = KIND == kWgrad;
  static constexpr bool DH = KIND == kDhGeglu || KIND == kDhGegluBf16;
  static constexpr bool LIN = KIND == kLinear || KIND == kLinearSkip;
  static constexpr bool A_MN = COLS;
  static constexpr bool B_MN = KIND == kDx || DH || COLS;
  // The training epilogues do 10 to 20 instructions per accumulator element and move as much again as the
  // products' operands: sixteen warps, and further ones for what does not need the accumulator.
  static constexpr int kEpiWarps = TRAIN || DH ? 16 : 8;
  static constexpr int kHelpers = TRAIN ? 4 : (DH || COLS ? 1 : 0);
  static constexpr int kThreads = 64 + 32 * (kEpiWarps + kHelpers);
  // (kGegluTrain at 16384 tokens, d 1024, f 4096: 149 / 126 / 116 us above the inference pass with 3 / 4 / 5
  // stages, so one box per epilogue warp and a fifth stage instead of two boxes)
  static constexpr int kStages = TRAIN ? 5 : (DH ? 4 : 6);
  // room behind the stages (boxes want 1 KiB alignment): a box for each epilogue warp, or two chunks of gate and up
  static constexpr int kBoxes = TRAIN ? 16 * kBoxBytes : (DH ? 2 * 2 * GegluBwd::kBoxBytes : 0);
  // and behind Control: staging of the epilogue warps; biases and mask bits; column sums of the lane quadrants
  static constexpr int kExtra =
      TRAIN ? 16 * 256 + 2 * BM * 16 : (DH ? 4 * 2 * BN * 4 : 8 * kStgBytes);
};

// M = 256 across the pair: M/16 at bit 24
constexpr uint32_t kIdesc2 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                             ((256u >> 4) << 24);

struct Control {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t tail[kMaxStages];   // COLS: this CTA's half of a block that has to be cut has arrived
  uint64_t peer_cut[kMaxStages];   // COLS, even CTA: the odd CTA's half has been cut
  uint64_t aux_full[2];    // kGegluTrain: mask bits of a tile drawn; kDhGeglu: a chunk of derivatives there
  uint64_t aux_empty[2];   // kGegluTrain: they have been read; kDhGeglu: replaced by their gradients
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int abort;
  int tile_start[kMaxExperts + 1];
  int offsets[kMaxExperts + 1];
};

// [stages][boxes][Control][extra]
constexpr size_t kControlBytes = (sizeof(Control) + 15) & ~(size_t)15;
template <int KIND>
constexpr size_t smem_bytes() {
  using T = Traits<KIND>;
  return 1024 + (size_t)T::kStages * kStageBytes + T::kBoxes + kControlBytes + T::kExtra;
}

// COLS = false: groups are row ranges [offsets[e], offsets[e+1]) of A; B_e = tmap_b[e]; K fixed.
// COLS = true : groups are the same row ranges, contracted over; A has Ra columns, B (one map,
//               tmap_bc) has Nout columns; out [E][Ra][Nout], zero for experts without rows.
template <int KIND, int SPLIT>
__global__ void __launch_bounds__(Traits<KIND>::kThreads, 1)
grouped_gemm_tc2_kernel(const __grid_constant__ CUtensorMap tmap_a,
                        const __grid_constant__ CUtensorMap tmap_bc,
                        const __grid_constant__ CUtensorMap tmap_h,    // kGegluTrain: h, 32 x 32 boxes
                        const __grid_constant__ CUtensorMap tmap_gu,   // training: gu
                        const CUtensorMap* __restrict__ tmap_b,  // [E], 128-row (B_MN: 64-row) boxes
                        const int32_t* __restrict__ offsets,
                        const void* const* __restrict__ bias_ptrs, int E, int K, int Nout,
                        __nv_bfloat16* __restrict__ out, const EpScatter sc, const TrainArgs tr,
                        const EpSync sy, int Ra, const LinearArgs la, int32_t* __restrict__ status) {
  using T = Traits<KIND>;
  constexpr bool GEGLU = T::GEGLU, COLS = T::COLS, A_MN = T::A_MN, B_MN = T::B_MN;
  constexpr int kStages = T::kStages, kEpiWarps = T::kEpiWarps;
  constexpr uint32_t kIdesc = kIdesc2 | (A_MN ? 1u << 15 : 0u) | (B_MN ? 1u << 16 : 0u);
  // descriptor step of one K = 16 product: 32 bytes along a row, or sixteen 128-byte rows
  constexpr uint64_t kStepA = A_MN ? 16 * 128 / 16 : 2, kStepB = B_MN ? 16 * 128 / 16 : 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~(uintptr_t)1023);
  uint8_t* boxes = smem + (size_t)kStages * kStageBytes;
  Control* ctl = reinterpret_cast<Control*>(boxes + T::kBoxes);
  uint8_t* extra = boxes + T::kBoxes + kControlBytes;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  static_assert(SPLIT == 1 || KIND == kPlain || KIND == kDx || T::LIN, "kinds with a split form");
  static_assert(SPLIT == 1 || BM * kPartPitch * 4 <= kStages * kStageBytes, "the partial tile reuses the stages");
  const uint32_t rank = cluster_ctarank();
  const uint32_t cta = rank & 1u;           // 0 = even CTA: issues the MMAs, owns full/tmem_empty
  const uint32_t lead = SPLIT > 1 ? rank & ~1u : 0u;      // the pair's even CTA
  // the tiles of this pair: t = pair, pair + num_pairs, ... (SPLIT: of its cluster, one tile at most)
  const int pair = blockIdx.x / (2 * SPLIT);
  const int num_pairs = gridDim.x / (2 * SPLIT);
  constexpr int kTileN = GEGLU ? BN / 2 : BN;
  const int n_tiles = T::LIN ? (la.halves(0) + la.halves(1) + 1) / 2 : (Nout + kTileN - 1) / kTileN;
  const int k_blocks_all = (K + BK - 1) / BK;
  const int k_blocks_per = (k_blocks_all + SPLIT - 1) / SPLIT;
  const int kb_first = SPLIT > 1 ? (int)(rank >> 1) * k_blocks_per : 0;       // this pair's range of K
  const int k_blocks_rows = min(k_blocks_per, k_blocks_all - kb_first);
  const int m_tiles_cols = (Ra + kPairRows - 1) / kPairRows;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
      mbar_init(&ctl->tail[s], 1);
      mbar_init(&ctl->peer_cut[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&ctl->tmem_full[a], 1);
      mbar_init(&ctl->tmem_empty[a], 2 * kEpiWarps);
      mbar_init(&ctl->aux_full[a], T::TRAIN ? T::kHelpers : 1);
      mbar_init(&ctl->aux_empty[a], kEpiWarps);
    }
    ctl->abort = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&ctl->tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  // everything above is independent of the kernels before this one in the stream
  pdl_wait();
  pdl_launch_dependents();
  // expert-parallel: the rows this kernel reads were pushed by the other ranks; wait for all of
  // them (bounded), then order those peer writes before this CTA's TMA reads
  const bool arrived = epsync::block_wait(sy, status, 24);
  if (sy.wait_flags != nullptr) asm volatile("fence.proxy.async;" ::: "memory");
  if (threadIdx.x == 0) {
    int acc = 0;
    int beg = T::LIN ? 0 : offsets[0];
    ctl->offsets[0] = beg;
    for (int e = 0; e < E; ++e) {
      ctl->tile_start[e] = acc;
      const int end = T::LIN ? la.rows : offsets[e + 1];
      ctl->offsets[e + 1] = end;
      acc += (COLS ? m_tiles_cols : (end - beg + kPairRows - 1) / kPairRows) * n_tiles;
      beg = end;
    }
    ctl->tile_start[E] = arrived ? acc : 0;   // a peer never arrived: nothing to do
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();   // both CTAs' barriers exist before anything signals across the pair
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&ctl->tmem_base);
  const int total_tiles = ctl->tile_start[E];

  if (warp == 0) {
    // ---------------- TMA producer (each CTA loads its own rows and its half of B) -------------
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      int e = 0;
      bool ok = true;
      for (int t = pair; ok && t < total_tiles; t += num_pairs) {
        while (t >= ctl->tile_start[e + 1]) ++e;
        const int local = t - ctl->tile_start[e];
        const int mt = local / n_tiles, nt = local - mt * n_tiles;
        const int row0 = (COLS ? 0 : ctl->offsets[e]) + mt * kPairRows + (int)cta * BM;
        int brow = GEGLU ? (cta == 0 ? nt * kTileN : Nout + nt * kTileN)
                         : nt * kTileN + (int)cta * (BN / 2);
        const CUtensorMap* tb = COLS ? &tmap_bc : tmap_b + e;
        if constexpr (T::LIN) {
          const LinearHalf lh(la, nt * 2 + (int)cta);
          tb = lh.which ? &tmap_h : &tmap_bc;
          brow = lh.col;
        }
        const int k0 = COLS ? ctl->offsets[e] : 0;
        const int k_rows = COLS ? ctl->offsets[e + 1] - k0 : 0;
        const int k_blocks = COLS ? (k_rows + BK - 1) / BK : k_blocks_rows;
        for (int kb = 0; kb < k_blocks; ++kb) {
          {
            if (!mbar_wait(&ctl->empty[stage], phase ^ 1u, &ctl->abort, status, 31)) { ok = false; break; }
          }
          uint8_t* sa = smem + (size_t)stage * kStageBytes;
          const uint32_t full0 = map_to_cta(smem_u32(&ctl->full[stage]), lead);
          uint32_t bar = full0;
          if (COLS && (kb + 1) * BK > k_rows) {
            mbar_expect_tx(&ctl->tail[stage], kStageBytes);     // the fixer passes it on
            bar = map_to_cta(smem_u32(&ctl->tail[stage]), rank);
          } else if (cta == 0) {
            mbar_expect_tx(&ctl->full[stage], 2 * kStageBytes);
          }
          const int kc = k0 + (kb_first + kb) * BK;
          if (A_MN) {
            tma_load_2d_pair(sa, &tmap_a, bar, row0, kc);
            tma_load_2d_pair(sa + kHalfTile, &tmap_a, bar, row0 + 64, kc);
          } else {
            tma_load_2d_pair(sa, &tmap_a, bar, kc, row0);
          }
          if (B_MN) {
            tma_load_2d_pair(sa + kABytes, tb, bar, brow, kc);
            tma_load_2d_pair(sa + kABytes + kHalfTile, tb, bar, brow + 64, kc);
          } else {
            tma_load_2d_pair(sa + kABytes, tb, bar, kc, brow);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (even CTA only) ----------------
    if (cta == 0 && elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase = 0;
      int it = 0;
      int e = 0;
      bool ok = true;
      for (int t = pair; ok && t < total_tiles; t += num_pairs) {
        int k_blocks = k_blocks_rows, k_rows = 0;
        if (COLS) {
          while (t >= ctl->tile_start[e + 1]) ++e;
          k_rows = ctl->offsets[e + 1] - ctl->offsets[e];
          k_blocks = (k_rows + BK - 1) / BK;
          if (k_blocks == 0) continue;     // nothing to add up: the epilogue stores zeros
        }
        const int a = it & 1;
        {
          if (!mbar_wait(&ctl->tmem_empty[a], acc_phase ^ 1u, &ctl->abort, status, 32)) { ok = false; break; }
        }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(a * BN);
        for (int kb = 0; kb < k_blocks; ++kb) {
          {
            if (!mbar_wait(&ctl->full[stage], phase, &ctl->abort, status, 33)) { ok = false; break; }
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + (size_t)stage * kStageBytes);
          const uint64_t adesc = A_MN ? make_smem_desc_mn(sa) : make_smem_desc(sa);
          const uint64_t bdesc = B_MN ? make_smem_desc_mn(sa + kABytes) : make_smem_desc(sa + kABytes);
          const int left = COLS ? k_rows - kb * BK : BK;    // rows of this expert in the block
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            if (!COLS || kk * 16 < left)
              tc_mma_pair(tmem_d, adesc + (uint64_t)kk * kStepA, bdesc + (uint64_t)kk * kStepB, kIdesc,
                          (kb | kk) != 0 ? 1u : 0u);
          // the stage is free in both CTAs once these MMAs have read it
          const uint32_t e_local = smem_u32(&ctl->empty[stage]);
          tc_commit_pair(map_to_cta(e_local, lead));
          tc_commit_pair(map_to_cta(e_local, lead + 1));
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        const uint32_t f_local = smem_u32(&ctl->tmem_full[a]);
        tc_commit_pair(map_to_cta(f_local, lead));
        tc_commit_pair(map_to_cta(f_local, lead + 1));
        if (a == 1) acc_phase ^= 1u;
        ++it;
      }
    }
  } else if (COLS && warp == 2 + kEpiWarps) {
    // ---------------- fixer: blocks that run past the expert's last row ----------------
    int blocks = 0;             // K blocks of this CTA's tiles so far
    uint32_t parity = 0;        // bit s: parity of the next use of tail[s]
    int e = 0;
    for (int t = pair; t < total_tiles; t += num_pairs) {
      while (t >= ctl->tile_start[e + 1]) ++e;
      const int k_rows = ctl->offsets[e + 1] - ctl->offsets[e];
      const int k_blocks = (k_rows + BK - 1) / BK;
      const int left = k_rows - (k_blocks - 1) * BK;        // rows of the last block, 1 .. 64
      blocks = (blocks + k_blocks) % kStages;
      if (k_blocks == 0 || left == BK) continue;
      const int s = (blocks + kStages - 1) % kStages;       // the stage of the last block
      if (!mbar_wait(&ctl->tail[s], (parity >> s) & 1u, &ctl->abort, status, 35)) break;
      uint8_t* sa = smem + (size_t)s * kStageBytes;
      // rows [left, next multiple of 16) of the four 64 x 64 boxes; a row is 128 bytes
      const int pieces = (((left + 15) & ~15) - left) * 8;
      for (int i = lane; i < 4 * pieces; i += 32) {
        const int box = i / pieces, p = i - box * pieces;
        *reinterpret_cast<uint4*>(sa + box * kHalfTile + (size_t)left * 128 + p * 16) = make_uint4(0, 0, 0, 0);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (cta == 1) {
        if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&ctl->peer_cut[s]), 0));
      } else {
        if (!mbar_wait_cluster(&ctl->peer_cut[s], (parity >> s) & 1u, &ctl->abort, status, 36)) break;
        if (lane == 0) mbar_arrive(&ctl->full[s]);
      }
      parity ^= 1u << s;
    }
  } else if (T::TRAIN && warp >= 2 + kEpiWarps) {
    // ---------------- dropout mask: four warps, 32 rows of the tile each ----------------
    int it = 0, e = 0;
    for (int t = pair; tr.thresh != 0u && t < total_tiles; t += num_pairs, ++it) {
      while (t >= ctl->tile_start[e + 1]) ++e;
      const int local = t - ctl->tile_start[e];
      const int mt = local / n_tiles, nt = local - mt * n_tiles;
      const int row_cta = ctl->offsets[e] + mt * kPairRows + (int)cta * BM;
      const int a = it & 1;
      if (!mbar_wait(&ctl->aux_empty[a], ((uint32_t)(it >> 1) & 1u) ^ 1u, &ctl->abort, status, 37)) break;
      uint32_t* s_mask = reinterpret_cast<uint32_t*>(extra + kEpiWarps * 256) + a * BM * 4;
      const int rl = (warp - 2 - kEpiWarps) * 32 + lane;
      draw_mask<T::PRE>(tr, row_cta + rl, row_cta + rl < ctl->offsets[e + 1], nt * kTileN, Nout, s_mask + rl * 4);
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->aux_full[a]);
    }
  } else if (T::DH && warp == 2 + kEpiWarps) {
    // ---------------- derivatives after gate and up: two chunks ahead, stored again as gradients ----------------
    if (elect_one()) {
      struct Place { int col, row; bool boxes; } place[2];
      int ci = 0, e = 0;
      auto put_back = [&](int b, int use) {      // use: how many times the buffer has been filled before
        if (!mbar_wait(&ctl->aux_empty[b], (uint32_t)use & 1u, &ctl->abort, status, 38)) return false;
        const Place& p = place[b];
        if (p.boxes) {
          uint8_t* box = boxes + b * 2 * GegluBwd::kBoxBytes;
          tma_store_2d(&tmap_gu, box, p.col, p.row);
          tma_store_2d(&tmap_gu, box + GegluBwd::kBoxBytes, Nout + p.col, p.row);
        }
        bulk_commit();
        return true;
      };
      bool ok = true;
      for (int t = pair; ok && t < total_tiles; t += num_pairs) {
        while (t >= ctl->tile_start[e + 1]) ++e;
        const int local = t - ctl->tile_start[e];
        const int mt = local / n_tiles, nt = local - mt * n_tiles;
        const int row_cta = ctl->offsets[e] + mt * kPairRows + (int)cta * BM;
        const bool rows_full = ctl->offsets[e + 1] - row_cta >= BM;
        for (int c = 0; ok && c < BN / GegluBwd::kChunk; ++c, ++ci) {
          const int b = ci & 1;
          const int col = nt * kTileN + c * GegluBwd::kChunk;
          if (ci >= 2) {
            ok = put_back(b, (ci >> 1) - 1);
            bulk_wait_read<0>();
            if (!ok) break;
          }
          // a box must lie inside gate or up: the last columns of an odd width are stored by the epilogue
          place[b] = Place{col, row_cta, rows_full && col + GegluBwd::kChunk <= Nout};
          uint8_t* box = boxes + b * 2 * GegluBwd::kBoxBytes;
          mbar_expect_tx(&ctl->aux_full[b], 2 * GegluBwd::kBoxBytes);
          tma_load_2d(box, &tmap_gu, &ctl->aux_full[b], col, row_cta);
          tma_load_2d(box + GegluBwd::kBoxBytes, &tmap_gu, &ctl->aux_full[b], Nout + col, row_cta);
        }
      }
      for (int q = ci > 2 ? ci - 2 : 0; ok && q < ci; ++q) ok = put_back(q & 1, q >> 1);
      bulk_wait_all();
    }
  } else {
    // ---------------- epilogue: one accumulator row per thread ----------------
    const int quad = warp & 3;
    const int part = (warp - 2) >> 2;  // the warps of a TMEM lane quadrant split the columns
    const int r = quad * 32 + lane;
    uint32_t acc_phase = 0;
    int it = 0;
    int e = 0;
    bool ok = true;
    BoxOut box{boxes + (warp - 2) * kBoxBytes};    // kGegluTrain
    for (int t = pair; ok && t < total_tiles; t += num_pairs) {
      while (t >= ctl->tile_start[e + 1]) ++e;
      const int local = t - ctl->tile_start[e];
      const int mt = local / n_tiles, nt = local - mt * n_tiles;
      const int row_end = COLS ? Ra : ctl->offsets[e + 1];
      const int row_cta = (COLS ? 0 : ctl->offsets[e]) + mt * kPairRows + (int)cta * BM;
      const int row_warp = row_cta + quad * 32;
      const int rows = min(32, row_end - row_warp);   // rows of this warp to store (may be negative)
      const int n0 = nt * kTileN;
      const __nv_bfloat16* bias =
          bias_ptrs != nullptr ? static_cast<const __nv_bfloat16*>(bias_ptrs[e]) : nullptr;
      __nv_bfloat16* out_e = COLS ? out + (size_t)e * Ra * Nout : out;
      if (COLS && ctl->offsets[e + 1] == ctl->offsets[e]) {
        store_zero_tile(out_e, row_warp, rows, Nout, n0 + part * 128, lane);
        continue;
      }
      const int a = it & 1;
      float* s_bias = reinterpret_cast<float*>(extra + (warp - 2) * 256);
      if constexpr (T::TRAIN) GegluTrain<T::PRE>::start(n0, Nout, bias, s_bias, lane, part);
      uint32_t keep[4];
      if constexpr (KIND == kDhGegluBf16) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          keep[c] = GegluBwd::mask_bits(tr, row_warp + lane, lane < rows, n0 + c * 64 + part * 16, Nout);
      }
      uint4 skip[KIND == kLinearSkip ? 2 : 1][8];
      if constexpr (KIND == kLinearSkip) {
        const LinearHalf lh(la, nt * 2 + part);
#pragma unroll
        for (int q = 0; q < 2; ++q) load_skip64(skip[q], la.skip, row_warp, rows, la.cols[0], lh.col + q * 64, lh.limit, lane);
      }
      ok = mbar_wait(&ctl->tmem_full[a], acc_phase, &ctl->abort, status, 34);
      if (!T::DH && !ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(a * BN);
      auto release = [&]() {     // this warp has read its part of the accumulator
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(&ctl->tmem_empty[a]), lead));
      };
      if constexpr (T::TRAIN) {
        uint32_t bits = 0xffffffffu;
        if (tr.thresh != 0u) {
          ok = mbar_wait(&ctl->aux_full[a], acc_phase, &ctl->abort, status, 39);
          if (!ok) break;
          bits = reinterpret_cast<const uint32_t*>(extra + kEpiWarps * 256)[(a * BM + r) * 4 + part];
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->aux_empty[a]);
        }
        GegluTrain<T::PRE>::finish(taddr, row_warp, rows, n0, Nout, out_e, tr, &tmap_h, &tmap_gu, s_bias, bits, box, lane, part,
                           release);
      } else if constexpr (T::DH) {
        float* s_col = reinterpret_cast<float*>(extra);
#pragma unroll 1
        for (int c = 0; ok && c < 4; ++c) {
          const int b = c & 1;
          // two uses of either buffer per tile
          ok = mbar_wait(&ctl->aux_full[b], (uint32_t)(c >> 1), &ctl->abort, status, 40);
          if (!ok) break;
          const int n = n0 + c * 64 + part * 16;
          uint32_t v[16];
          tc_ld16(taddr + c * 64 + part * 16, v);
          tc_ld_wait();
          if (c == 3) release();
          const bool as_boxes = row_end - row_cta >= BM && n0 + c * 64 + 64 <= Nout;
          __nv_bfloat16* direct = as_boxes ? nullptr : tr.gu + (int64_t)(row_warp + lane) * 2 * Nout + n;
          uint32_t bits = 0;
          if constexpr (KIND == kDhGegluBf16) {
            bits = keep[0];
            bits = c == 1 ? keep[1] : bits;
            bits = c == 2 ? keep[2] : bits;
            bits = c == 3 ? keep[3] : bits;
          }
          GegluBwd::chunk<KIND == kDhGegluBf16>(v, boxes + b * 2 * GegluBwd::kBoxBytes, bits, tr.scale, lane < rows, direct,
                          Nout, Nout - n, s_col + quad * 2 * BN + c * 64 + part * 16, BN, quad, part, lane);
          fence_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->aux_empty[b]);
        }
        // column sums of this CTA's 128 rows: the four lane quadrants in order. A warp whose wait
        // ran out still comes to the barrier, and all leave together.
        ok = barrier_and(1, 32 * kEpiWarps, ok);
        if (!ok) break;
        const int c = (int)threadIdx.x - 64;
        const int col = n0 + (c & (BN - 1));
        if (col < Nout) {
          const float sum = (s_col[c] + s_col[2 * BN + c]) + (s_col[4 * BN + c] + s_col[6 * BN + c]);
          const int64_t slot = (int64_t)(ctl->tile_start[e] / n_tiles + mt) * 2 + (int)cta;
          tr.col_part[slot * 2 * Nout + (c >= BN ? Nout : 0) + col] = sum;
        }
        barrier_and(1, 32 * kEpiWarps, true);
      } else if constexpr (SPLIT > 1) {
        float* mine = reinterpret_cast<float*>(smem) + r * kPartPitch + part * (BN / 2);
#pragma unroll 1
        for (int c = 0; c < BN / 2; c += 32) {
          uint32_t v[32];
          tc_ld32(taddr + part * (BN / 2) + c, v);
          tc_ld_wait();
#pragma unroll
          for (int q = 0; q < 32; q += 4)
            *reinterpret_cast<uint4*>(mine + c + q) = make_uint4(v[q], v[q + 1], v[q + 2], v[q + 3]);
        }
      } else if constexpr (T::LIN) {
        const LinearHalf lh(la, nt * 2 + part);
        store_tile<false, false, KIND == kLinearSkip>(
            taddr, row_cta + r, row_cta + r < row_end, lh.col - part * 128, lh.limit, la.bias_of(lh.which), la.out_of(lh.which), sc,
            extra + (warp - 2) * kStgBytes, lane, part, release, la.cols_of(lh.which), skip);
      } else {
        store_tile<GEGLU, KIND == kScatter>(taddr, row_cta + r, row_cta + r < row_end, n0, Nout, bias, out_e, sc,
                                            extra + (warp - 2) * kStgBytes, lane, part, release);
      }
      if (a == 1) acc_phase ^= 1u;
      ++it;
    }
    if (T::TRAIN && lane == 0) bulk_wait_all();
    if (KIND == kScatter) __threadfence_system();
  }
  if constexpr (SPLIT > 1) {
    __syncwarp();
    cluster_sync();       // the partial tiles of all ranges are there (or a wait ran out, and the status says so)
    if (pair < total_tiles) {
      int e = 0;
      while (pair >= ctl->tile_start[e + 1]) ++e;
      const int local = pair - ctl->tile_start[e];
      const int mt = local / n_tiles, nt = local - mt * n_tiles;
      const int row_cta = ctl->offsets[e] + mt * kPairRows + (int)cta * BM;
      const int rows = min(BM, ctl->offsets[e + 1] - row_cta);
      const __nv_bfloat16* bias = bias_ptrs != nullptr ? static_cast<const __nv_bfloat16*>(bias_ptrs[e]) : nullptr;
      __nv_bfloat16* to = out;
      int width = Nout;
      constexpr int kPieces = BN / SPLIT / 8;          // of eight columns, per row
      const int c0 = (int)(rank >> 1) * (BN / SPLIT);
      for (int i = threadIdx.x; i < rows * kPieces; i += T::kThreads) {
        const int rr = i / kPieces, c = c0 + (i % kPieces) * 8;
        int n = nt * kTileN + c;
        if constexpr (T::LIN) {
          const LinearHalf lh(la, nt * 2 + (c >> 7));
          n = lh.col + (c & 127);
          if (n >= lh.limit) continue;
          bias = la.bias_of(lh.which);
          to = la.out_of(lh.which);
          width = la.cols_of(lh.which);
        } else if (n >= Nout) {
          continue;
        }
        const uint32_t at = smem_u32(smem) + (uint32_t)(rr * kPartPitch + c) * 4;
        float o[8] = {};
#pragma unroll
        for (int q = 0; q < SPLIT; ++q) {
          const uint32_t from = map_to_cta(at, 2 * q + cta);
          float4 v0, v1;
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(v0.x), "=f"(v0.y), "=f"(v0.z), "=f"(v0.w) : "r"(from) : "memory");
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(v1.x), "=f"(v1.y), "=f"(v1.z), "=f"(v1.w) : "r"(from + 16) : "memory");
          o[0] += v0.x; o[1] += v0.y; o[2] += v0.z; o[3] += v0.w;
          o[4] += v1.x; o[5] += v1.y; o[6] += v1.z; o[7] += v1.w;
        }
        if (bias != nullptr) {
          float b[8];
          load8_ldg(bias + n, b);
#pragma unroll
          for (int q = 0; q < 8; ++q) o[q] += b[q];
        }
        const int64_t at_out = (int64_t)(row_cta + rr) * width + n;
        if constexpr (KIND == kLinearSkip) {
          float k[8];
          load8(la.skip + at_out, k);
#pragma unroll
          for (int q = 0; q < 8; ++q) o[q] = __bfloat162float(__float2bfloat16_rn(o[q])) + k[q];
        }
        store8(to + at_out, o);
      }
    }
  }
  // expert-parallel down pass: the last CTA to get here tells every rank that this rank's
  // outputs have been stored
  epsync::grid_signal(sy);

  // ---------------- teardown ----------------
  __syncwarp();
  if (*reinterpret_cast<volatile int*>(&ctl->abort)) {
    unsigned long long t0 = global_ns();
    while (global_ns() - t0 < 1000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();   // the peer may still signal this CTA's barriers or read its shared memory
  tc_fence_after();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(kTmemCols)
                 : "memory");
  }
}

// SPLIT > 1: max_tiles is an upper bound of the launch's tiles, one cluster each (those without one leave).
template <int KIND, int SPLIT = 1>
int launch_pair(const CUtensorMap& tm_a, const CUtensorMap& tm_bc, const void* tmap_b, const int32_t* offsets,
                const void* const* bias, int E, int K, int Nout, void* out, const EpScatter& sc,
                const TrainArgs& tr, const EpSync& sy, int Ra, int32_t* status, int sms, cudaStream_t s,
                const CUtensorMap* tm_h = nullptr, const CUtensorMap* tm_gu = nullptr, int64_t max_tiles = 0,
                const LinearArgs& la = {}) {
  static PerDeviceOnce once;
  auto fn = grouped_gemm_tc2_kernel<KIND, SPLIT>;
  constexpr size_t smem = smem_bytes<KIND>();
  static_assert(smem <= 227 * 1024, "shared memory of one CTA");
  int rc = ensure_dynamic_smem(once, fn, smem);
  if (rc) return rc;
  const unsigned grid = SPLIT > 1 ? (unsigned)max_tiles * 2 * SPLIT : (unsigned)(sms & ~1);
  MOE_CUDA_CHECK(launch_pdl_cluster(fn, dim3(grid), dim3(Traits<KIND>::kThreads), 2 * SPLIT, smem, s, tm_a, tm_bc,
                                    tm_h != nullptr ? *tm_h : tm_a, tm_gu != nullptr ? *tm_gu : tm_a,
                                    static_cast<const CUtensorMap*>(tmap_b), offsets, bias, E, K, Nout,
                                    static_cast<__nv_bfloat16*>(out), sc, tr, sy, Ra, la, status));
  return 0;
}

// How many pairs share a tile of a row-grouped product: as many as the tiles leave idle, where each still has a
// range of eight blocks of K or more. The host does not know the routing: every expert that can have rows is taken
// to end in half a tile. The tiles must fit in one round of clusters, and clusters stay inside a group of SMs: 32
// clusters of four CTAs and 12 of eight did, 36 and 16 did not. The feed-forward with E 1, d 1024, f 4096, without
// and with the split (us, nothing in L2): 1 row 48 / 32, 512 rows (8 tiles, four ranges) 50 / 40, 1024 rows (16 tiles)
// 58 / 62 with four ranges, 1100 rows (20 tiles, two ranges) 63 / 54, 2048 (32 tiles) 73 / 64, 2304 (36) 73 / 83.
int k_splits(int64_t M, int E, int K, int Nout) {
  const int64_t n_tiles = (Nout + BN - 1) / BN;
  const int64_t tiles = ((M + kPairRows - 1) / kPairRows + (E > 1 ? (M < E ? M : E) / 2 : 0)) * n_tiles;
  const int kb = (K + BK - 1) / BK;
  if (tiles <= 12 && kb >= 32) return 4;
  if (tiles <= 32 && kb >= 16) return 2;
  return 1;
}
int64_t max_tiles(int64_t M, int E, int Nout) {
  return ((M + kPairRows - 1) / kPairRows + (M < E ? M : E)) * ((Nout + BN - 1) / BN);
}

}  // namespace

int launch_experts_tc2(const void* perm, const int32_t* offsets, const void* plan, int64_t M, int d,
                       int f, int E, void* h, void* y, const EpScatter* sc, int32_t* status,
                       cudaStream_t s, const TrainArgs* train, const EpSync* ep_wait,
                       const EpSync* ep_signal) {
  // expert-parallel ranks take part in the hand-shakes even when they own no rows
  if ((M == 0 || E == 0) && ep_wait == nullptr && ep_signal == nullptr) return 0;
  PlanView pv = plan_view(plan, E);
  alignas(64) CUtensorMap tm_x, tm_h;
  const uint64_t rows = M > 0 ? (uint64_t)M : 1;   // a rank without rows still launches (hand-shakes)
  int rc = encode_tmap_2d(&tm_x, perm, rows, (uint64_t)d, BM);
  if (rc) return rc;
  rc = encode_tmap_2d(&tm_h, h, rows, (uint64_t)f, BM);
  if (rc) return rc;
  int sms = 0;
  rc = sm_count(&sms);
  if (rc) return rc;
  const EpScatter none = {};
  const TrainArgs eval = {};
  const EpSync nosync = {};
  const EpSync& sy1 = ep_wait != nullptr ? *ep_wait : nosync;
  const EpSync& sy2 = ep_signal != nullptr ? *ep_signal : nosync;
  if (train != nullptr) {
    alignas(64) CUtensorMap tm_hb, tm_gu;
    rc = encode_tmap_2d(&tm_hb, h, rows, (uint64_t)f, 32, 32);
    if (rc) return rc;
    rc = encode_tmap_2d(&tm_gu, train->gu, rows, (uint64_t)2 * f, 32, 32);
    if (rc) return rc;
    rc = train->keep_pre
             ? launch_pair<kGegluTrainPre>(tm_x, tm_x, pv.tmap_W1, offsets, pv.b1, E, d, f, h, none, *train, sy1, 0, status,
                                           sms, s, &tm_hb, &tm_gu)
             : launch_pair<kGegluTrain>(tm_x, tm_x, pv.tmap_W1, offsets, pv.b1, E, d, f, h, none, *train, sy1, 0, status,
                                        sms, s, &tm_hb, &tm_gu);
  } else {
    rc = launch_pair<kGeglu>(tm_x, tm_x, pv.tmap_W1, offsets, pv.b1, E, d, f, h, none, eval, sy1, 0, status, sms, s);
  }
  if (rc) return rc;
  if (sc != nullptr)
    return launch_pair<kScatter>(tm_h, tm_h, pv.tmap_W2, offsets, pv.b2, E, f, d, nullptr, *sc, eval, sy2, 0, status,
                                 sms, s);
  const int split = ep_signal == nullptr && M > 0 ? k_splits(M, E, f, d) : 1;
  if (split == 4)
    return launch_pair<kPlain, 4>(tm_h, tm_h, pv.tmap_W2, offsets, pv.b2, E, f, d, y, none, eval, sy2, 0, status, sms,
                                  s, nullptr, nullptr, max_tiles(M, E, d));
  if (split == 2)
    return launch_pair<kPlain, 2>(tm_h, tm_h, pv.tmap_W2, offsets, pv.b2, E, f, d, y, none, eval, sy2, 0, status, sms,
                                  s, nullptr, nullptr, max_tiles(M, E, d));
  return launch_pair<kPlain>(tm_h, tm_h, pv.tmap_W2, offsets, pv.b2, E, f, d, y, none, eval, sy2, 0, status, sms, s);
}

int launch_grouped_dx(const void* A, int64_t M, int K, const void* tmaps_b, const int32_t* offsets, int E, int Nout,
                      void* out, const TrainArgs* geglu_bwd, bool round_dh, int32_t* status, cudaStream_t s) {
  if (M == 0 || E == 0) return 0;
  alignas(64) CUtensorMap tm_a;
  int rc = encode_tmap_2d(&tm_a, A, (uint64_t)M, (uint64_t)K, BM);
  if (rc) return rc;
  int sms = 0;
  rc = sm_count(&sms);
  if (rc) return rc;
  const EpScatter none = {};
  const TrainArgs eval = {};
  const EpSync nosync = {};
  if (geglu_bwd != nullptr) {
    alignas(64) CUtensorMap tm_gu;
    rc = encode_tmap_2d(&tm_gu, geglu_bwd->gu, (uint64_t)M, (uint64_t)2 * Nout, BM);
    if (rc) return rc;
    if (round_dh)
      return launch_pair<kDhGegluBf16>(tm_a, tm_a, tmaps_b, offsets, nullptr, E, K, Nout, nullptr, none, *geglu_bwd,
                                       nosync, 0, status, sms, s, nullptr, &tm_gu);
    return launch_pair<kDhGeglu>(tm_a, tm_a, tmaps_b, offsets, nullptr, E, K, Nout, nullptr, none, *geglu_bwd,
                                 nosync, 0, status, sms, s, nullptr, &tm_gu);
  }
  const int split = k_splits(M, E, K, Nout);
  if (split == 4)
    return launch_pair<kDx, 4>(tm_a, tm_a, tmaps_b, offsets, nullptr, E, K, Nout, out, none, eval, nosync, 0, status,
                               sms, s, nullptr, nullptr, max_tiles(M, E, Nout));
  if (split == 2)
    return launch_pair<kDx, 2>(tm_a, tm_a, tmaps_b, offsets, nullptr, E, K, Nout, out, none, eval, nosync, 0, status,
                               sms, s, nullptr, nullptr, max_tiles(M, E, Nout));
  return launch_pair<kDx>(tm_a, tm_a, tmaps_b, offsets, nullptr, E, K, Nout, out, none, eval, nosync, 0, status, sms,
                          s);
}

namespace {
template <int KIND>
int linear_tiles(const CUtensorMap& a, const CUtensorMap& w0, const CUtensorMap& w1, int64_t N, int K, const LinearArgs& la,
                 int32_t* status, int sms, cudaStream_t s) {
  const int cols = (la.halves(0) + la.halves(1)) * 128;
  const EpScatter none = {};
  const TrainArgs eval = {};
  const EpSync nosync = {};
  const int64_t tiles = max_tiles(N, 1, cols);
  switch (k_splits(N, 1, K, cols)) {
    case 4: return launch_pair<KIND, 4>(a, w0, nullptr, nullptr, nullptr, 1, K, cols, nullptr, none, eval, nosync, 0, status,
                                        sms, s, &w1, nullptr, tiles, la);
    case 2: return launch_pair<KIND, 2>(a, w0, nullptr, nullptr, nullptr, 1, K, cols, nullptr, none, eval, nosync, 0, status,
                                        sms, s, &w1, nullptr, tiles, la);
    default: return launch_pair<KIND, 1>(a, w0, nullptr, nullptr, nullptr, 1, K, cols, nullptr, none, eval, nosync, 0, status,
                                         sms, s, &w1, nullptr, 0, la);
  }
}
}  // namespace

// All buffers 16-byte aligned, K and the numbers of rows of W multiples of 8.
int launch_linear_tiles(const void* x, const LinearRows& first, const LinearRows& second, const void* skip, int64_t N, int K,
                        int32_t* status, cudaStream_t s) {
  if (N == 0) return 0;
  alignas(64) CUtensorMap a, w0, w1;
  int rc = encode_tmap_2d(&a, x, (uint64_t)N, (uint64_t)K, BM);
  if (!rc) rc = encode_tmap_2d(&w0, first.W, (uint64_t)first.rows, (uint64_t)K, BN / 2);
  if (!rc && second.rows > 0) rc = encode_tmap_2d(&w1, second.W, (uint64_t)second.rows, (uint64_t)K, BN / 2);
  if (rc) return rc;
  if (second.rows == 0) w1 = w0;
  int sms = 0;
  rc = sm_count(&sms);
  if (rc) return rc;
  LinearArgs la = {};
  int i = 0;
  for (const LinearRows* l : {&first, &second}) {
    la.bias[i] = static_cast<const __nv_bfloat16*>(l->b);
    la.out[i] = static_cast<__nv_bfloat16*>(l->out);
    la.cols[i++] = l->rows;
  }
  la.rows = (int)N;
  la.skip = static_cast<const __nv_bfloat16*>(skip);
  return skip != nullptr ? linear_tiles<kLinearSkip>(a, w0, w1, N, K, la, status, sms, s)
                         : linear_tiles<kLinear>(a, w0, w1, N, K, la, status, sms, s);
}

int launch_grouped_wgrad(const void* A, const void* B, int64_t M, int Ra, int Rb, const int32_t* offsets, void* out,
                         int E, int32_t* status, cudaStream_t s) {
  if (M == 0 || E == 0) return 0;
  alignas(64) CUtensorMap tm_a, tm_b;
  int rc = encode_tmap_2d(&tm_a, A, (uint64_t)M, (uint64_t)Ra, BK);
  if (rc) return rc;
  rc = encode_tmap_2d(&tm_b, B, (uint64_t)M, (uint64_t)Rb, BK);
  if (rc) return rc;
  int sms = 0;
  rc = sm_count(&sms);
  if (rc) return rc;
  const EpScatter none = {};
  const TrainArgs eval = {};
  const EpSync nosync = {};
  return launch_pair<kWgrad>(tm_a, tm_b, nullptr, offsets, nullptr, E, 0, Rb, out, none, eval, nosync, Ra, status,
                             sms, s);
}

}  // namespace moe
