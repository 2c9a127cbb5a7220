// Both products of the experts in one launch, for calls between the decode and the prefill sizes (and, with more experts
// than the decode kernels take, the smallest): reference model.py:174,180-184.
//   gate_and_up tile: h[row][feature] = gelu_tanh(g + bg) * (u + bu), 128 features of up to 256 tokens of one expert
//   down tile:        y[row][feature] = h W2^T + b2, 256 features
// The weights are the 256 rows of a CTA pair's product (M, 128 a CTA, cta_group::2), the tokens its columns (N, each CTA
// loads half of them), so that a tile costs what its tokens are: an expert's tokens are cut into as few blocks as hold them,
// of equal size, N a multiple of 32. In experts_tc2.cu, where a tile has 256 rows of tokens whatever it holds, 293 rows an
// expert (the average of 1173 tokens, 8 experts, two slots) made 57 % of the products real ones.
// Weights come as they lie in memory; those of gate_and_up through a map that gives a box gate and up rows in turn, so that
// neighbouring lanes of the accumulator hold a feature's pair and each takes every other token.
//
// One persistent pair of CTAs for two SMs. Tiles are claimed in order from a counter, all of gate_and_up before the first of
// the down product; a down tile waits until its expert's h is there, which tiles claimed earlier by running pairs write, so
// that the waits end whatever else runs on the GPU. (The tiles dealt out in turn, with no counter, were 1 us faster at 1173
// tokens, but wait for pairs that may not be running; a cooperative launch of that form was 3 us slower than the counter.)
//   warp 0       loads weights              warp 10      loads tokens, or rows of h
//   warp 1       issues the products (even CTA)
//   warps 2-9    epilogue: two groups of four, 32 tokens at a time each
//   warp 11      makes stored tiles of h known       warp 12      claims tiles and hands them to all roles of the pair
//
// What bounds it: from some 150 rows an expert on, shared memory: a step of 64 of K brings in 16 KiB of weights and n/2 x 128
// bytes of tokens a CTA and the products read both again; 500 clk at N = 160 and 580 at 256, for 320 and 512 of products.
// Below, the stream of the weights. Kept from the two launches it replaces: nothing of the second's start and of the first's
// last tiles, 7 us. Block, d 1024, f 4096, 8 experts, two slots, weights not in L2, whole calls one after the other, us, with
// the streaming kernel (up to 2048 tokens) or the 256-row tiles / with this one: 384 tokens 62.2 / 62.2, 512 70.7 / 63.2, 640
// 79.7 / 64.6, 1024 94.1 / 74.9, 2048 127 / 104, 4096 193 / 180, 8192 349 / 319. 64 experts, d 2048, f 1408, four slots: 1
// token 99 / 58, 16 1163 / 147, 64 929 / 207, 512 225 / 219, 4096 396 / 332, 16384 998 / 999.
// Tried and taken back: prefetches of weights into L2 ahead of their load (the SM's TMA unit takes as long for one as for a
// load: 94 -> 100 us at 1173 tokens); the down product cut into equal ranges of K for all pairs, with partial sums handed
// on through L2 (64 tiles for 74 pairs: the exchange took 5 us, as much as it gave; 1024 tokens 81 -> 87 us).
#include <cuda.h>
#include <cmath>
#include "common.cuh"
#include "tc_ptx.cuh"
#include "tc_pair.cuh"

namespace moe {

namespace {

using namespace tc;

constexpr int kRowsA = 128;       // weight rows per CTA = accumulator lanes
constexpr int kMaxTok = 256;      // tokens per tile
constexpr int BK = 64;
constexpr int kStages = 6;
constexpr int kABytes = kRowsA * BK * 2;             // 16 KiB of weights
constexpr int kBBytes = kMaxTok / 2 * BK * 2;        // up to 16 KiB: this CTA's half of the tile's tokens
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kTmemCols = 2 * kMaxTok;
constexpr int kEpiWarps = 8;
constexpr int kThreads = 160 + 32 * kEpiWarps;
constexpr int kFeat1 = 64, kFeat2 = 128;             // features of a CTA's tile: gate and up of 64; 128
constexpr int kMaxE = kMaxExperts;
constexpr int kGroup = 16;        // blocks of tokens that take turns on a tile of weights: 4096 rows of 4 KiB stay in L2
constexpr int kRing = 4;
constexpr int kReaders = kEpiWarps + 3;              // of a claimed tile in a CTA, besides the even one's issuer of products

// A tile as its roles need it.
struct alignas(16) Item {
  int e, nt;             // expert, tile of features
  int row0, rows;        // tokens
  int n;                 // their number rounded up to 32
  int kb;                // blocks of K; 0: no more tiles
  int down;
  int pad;
};

struct Control {
  Item ring[kRing];
  uint64_t full[kStages], empty[kStages];
  uint64_t tmem_full[2], tmem_empty[2];
  uint64_t stored[kRing];           // the epilogue has stored the tile of h in ring[slot]
  uint64_t want;                    // even CTA: the next tile can be claimed
  uint64_t ring_full[kRing];        // ring[slot] has been written
  uint64_t ring_empty[kRing];       // all roles of this CTA have read it
  uint64_t ring_peer[kRing];        // even CTA: all roles of the odd one have
  uint32_t tmem_base;
  int abort;
  int offsets[kMaxE + 1];
  int blocks[kMaxE + 1];      // token blocks of the experts before
};
constexpr int kPitch1 = 160, kPitch2 = 272;             // bytes per staged token
constexpr int kStgBytes = 32 * kPitch1;                 // one of a group's two staging buffers
static_assert(16 * kPitch2 <= kStgBytes, "16 tokens of 128 features");
constexpr size_t kSmemBytes = 1024 + (size_t)kStages * kStageBytes + sizeof(Control) + 16 + 4 * kStgBytes;
static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");

// M = 256 across the pair, bf16 x bf16 -> fp32, N at bit 17
__device__ __forceinline__ uint32_t idesc_pair(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((256u >> 4) << 24);
}
__device__ __forceinline__ bool try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void load_2d(uint32_t dst, const void* tmap, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void load_3d(uint32_t dst, const void* tmap, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tma_prefetch_3d(const void* tmap, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(
                   reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// What all roles know of the call.
struct Work {
  int n1, n2;            // tiles of features: gate_and_up, down
  int kb1, kb2;          // blocks of K
  int tiles1, tiles;     // tiles of gate_and_up; of both products
  int E;
};

// The tile of a number: gate_and_up first, expert by expert. An expert's tokens are cut into as few blocks as hold them, of equal
// size; blocks that read the same weights are neighbours, as far as kGroup blocks go.
__device__ __forceinline__ Item item_of(const Control* ctl, const Work& w, int t) {
  Item it;
  if (t >= w.tiles) {
    it.e = it.nt = it.row0 = it.rows = it.n = it.kb = it.down = it.pad = 0;
    return it;
  }
  it.pad = 0;
  it.down = t >= w.tiles1;
  if (it.down) t -= w.tiles1;
  it.kb = it.down ? w.kb2 : w.kb1;
  const int tiles = it.down ? w.n2 : w.n1;
  int lo = 0, hi = w.E;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (ctl->blocks[mid] * tiles <= t) lo = mid; else hi = mid;
  }
  const int local = t - ctl->blocks[lo] * tiles;
  const int nb = ctl->blocks[lo + 1] - ctl->blocks[lo], cnt = ctl->offsets[lo + 1] - ctl->offsets[lo];
  const int g = local / (kGroup * tiles), of_group = min(kGroup, nb - g * kGroup), in_group = local - g * kGroup * tiles;
  const int per = ((cnt + nb - 1) / nb + 31) & ~31;
  it.e = lo;
  it.nt = in_group / of_group;
  const int b = g * kGroup + in_group - it.nt * of_group;
  it.row0 = ctl->offsets[lo] + b * per;
  it.rows = min(per, cnt - b * per);
  it.n = (it.rows + 31) & ~31;
  return it;
}

// A role's place in the ring of claimed tiles.
struct Ring {
  int slot = 0;
  uint32_t phase = 0;
  // The next tile. arrive(): this role has read it.
  __device__ __forceinline__ Item take(Control* ctl, uint32_t cta, int32_t* status) {
    const bool ok = cta == 0 ? mbar_wait(&ctl->ring_full[slot], phase, &ctl->abort, status, 65)
                             : mbar_wait_cluster(&ctl->ring_full[slot], phase, &ctl->abort, status, 65);
    Item it = ctl->ring[slot];
    if (!ok) it.kb = 0;
    return it;
  }
  __device__ __forceinline__ void arrive(Control* ctl) {
    mbar_arrive(&ctl->ring_empty[slot]);
  }
  __device__ __forceinline__ void step() {
    if (++slot == kRing) { slot = 0; phase ^= 1u; }
  }
};

__global__ void __launch_bounds__(kThreads, 1)
experts_mid_kernel(const __grid_constant__ CUtensorMap tmap_x64, const __grid_constant__ CUtensorMap tmap_x16,
                   const __grid_constant__ CUtensorMap tmap_h64, const __grid_constant__ CUtensorMap tmap_h16,
                   const CUtensorMap* __restrict__ tmap_w1, const CUtensorMap* __restrict__ tmap_w2,
                   const int32_t* __restrict__ offsets, const void* const* __restrict__ b1, const void* const* __restrict__ b2,
                   int E, int d, int f, int ahead, __nv_bfloat16* __restrict__ h, __nv_bfloat16* __restrict__ y,
                   int* __restrict__ ready, int32_t* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  Control* ctl = reinterpret_cast<Control*>(smem + (size_t)kStages * kStageBytes);
  uint8_t* stg_all = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ctl + 1) + 15) & ~(uintptr_t)15);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();
  Work w;
  w.E = E;
  w.n1 = (f + 2 * kFeat1 - 1) / (2 * kFeat1);
  w.n2 = (d + 2 * kFeat2 - 1) / (2 * kFeat2);
  w.kb1 = (d + BK - 1) / BK;
  w.kb2 = (f + BK - 1) / BK;
  int* claimed = ready + (MOE_B200_READY_INTS - 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&ctl->full[s], 1); mbar_init(&ctl->empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&ctl->tmem_full[a], 1); mbar_init(&ctl->tmem_empty[a], 2 * kEpiWarps); }
    mbar_init(&ctl->want, 1);
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&ctl->stored[i], kEpiWarps);
      mbar_init(&ctl->ring_full[i], 1);
       mbar_init(&ctl->ring_empty[i], kReaders + (cta == 0 ? 1 : 0));
      mbar_init(&ctl->ring_peer[i], 1);
    }
    ctl->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)),
                 "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (ahead && warp == 2 && elect_one()) {
    // the first weights into L2 while the routing still runs, which they do not depend on: 28 MiB in all
    for (int i = 0, t = blockIdx.x >> 1; i < 12 && t < E * w.n1; t += gridDim.x >> 1) {
      const int e = t / w.n1, nt = t - e * w.n1;
      for (int kb = 0; kb < w.kb1 && i < 12; ++kb, ++i) tma_prefetch_3d(tmap_w1 + e, kb * BK, 0, (nt * 2 + (int)cta) * kFeat1);
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();   // both CTAs' barriers exist before anything signals across the pair
  tc_fence_after();
  pdl_wait();
  pdl_launch_dependents();
  int claim = 0;
  if (warp == 4 + kEpiWarps && cta == 0 && elect_one()) claim = atomicAdd(claimed, 1);
  if (warp == 0) {
    int carry = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const int o0 = e < E ? __ldcg(&offsets[e]) : 0, o1 = e < E ? __ldcg(&offsets[e + 1]) : 0;
      const int nb = (o1 - o0 + kMaxTok - 1) / kMaxTok;
      int incl = nb;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      if (e < E) {
        ctl->offsets[e + 1] = o1;
        ctl->blocks[e + 1] = carry + incl;
        if (e == 0) {
          ctl->offsets[0] = o0;
          ctl->blocks[0] = 0;
        }
      }
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __syncthreads();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&ctl->tmem_base);
  w.tiles1 = ctl->blocks[E] * w.n1;
  w.tiles = w.tiles1 + ctl->blocks[E] * w.n2;

  if (warp == 0) {
    // ---------------- weights ----------------
    if (elect_one()) {
      const uint32_t u_smem = smem_u32(smem), u_full = smem_u32(ctl->full), u_empty = smem_u32(ctl->empty);
      const uint32_t u_full0 = map_to_cta(u_full, 0);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      Ring ring;
      while (ok) {
        const Item it = ring.take(ctl, cta, status);
        ring.arrive(ctl);
        ring.step();
        if (it.kb == 0) break;
        const uint32_t bytes = (uint32_t)(2 * kABytes + it.n * BK * 2);
        const CUtensorMap* tw = (it.down ? tmap_w2 : tmap_w1) + it.e;
        const int feat = (it.nt * 2 + (int)cta) * (it.down ? kFeat2 : kFeat1);
        // the next tile is claimed a few steps before the end: late enough that nobody hoards tiles, early enough that the
        // answer is there in time
        const int claim_kb = max(0, it.kb - 8);
        if (it.down) {
#pragma unroll 1
          for (int kb = 0; kb < it.kb; ++kb) {
            if (cta == 0 && kb == claim_kb) mbar_arrive(&ctl->want);
            if (!try_wait(u_empty + stage * 8, phase ^ 1u) &&
                !mbar_wait(&ctl->empty[stage], phase ^ 1u, &ctl->abort, status, 61)) { ok = false; break; }
            const uint32_t sa = u_smem + (uint32_t)stage * kStageBytes, bar = u_full0 + stage * 8;
            if (cta == 0) expect_tx(u_full + stage * 8, bytes);
            load_2d(sa, tw, bar, kb * BK, feat);
            if (++stage == kStages) { stage = 0; phase ^= 1u; }
          }
        } else {
#pragma unroll 1
          for (int kb = 0; kb < it.kb; ++kb) {
            if (cta == 0 && kb == claim_kb) mbar_arrive(&ctl->want);
            if (!try_wait(u_empty + stage * 8, phase ^ 1u) &&
                !mbar_wait(&ctl->empty[stage], phase ^ 1u, &ctl->abort, status, 61)) { ok = false; break; }
            const uint32_t sa = u_smem + (uint32_t)stage * kStageBytes, bar = u_full0 + stage * 8;
            if (cta == 0) expect_tx(u_full + stage * 8, bytes);
            load_3d(sa, tw, bar, kb * BK, 0, feat);
            if (++stage == kStages) { stage = 0; phase ^= 1u; }
          }
        }
      }
    }
  } else if (warp == 2 + kEpiWarps) {
    // ---------------- tokens ----------------
    if (elect_one()) {
      const uint32_t u_smem = smem_u32(smem) + kABytes, u_empty = smem_u32(ctl->empty);
      const uint32_t u_full0 = map_to_cta(smem_u32(ctl->full), 0);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int seen = -1;       // the last expert whose h has been waited for
      Ring ring;
      while (ok) {
        const Item it = ring.take(ctl, cta, status);
        ring.arrive(ctl);
        ring.step();
        if (it.kb == 0) break;
        if (it.down && it.e != seen) {
          seen = it.e;
          const int want = 2 * w.n1 * (ctl->blocks[it.e + 1] - ctl->blocks[it.e]);
          const unsigned long long t0 = global_ns();
          for (uint32_t i = 0; ld_acquire_gpu(&ready[it.e]) < want; ++i) {
            if ((i & 63u) == 63u) {
              if (*reinterpret_cast<volatile int*>(&ctl->abort)) { ok = false; break; }
              if (global_ns() - t0 > kWaitLimitNs) {
                *reinterpret_cast<volatile int*>(&ctl->abort) = 1;
                atomicMax(&status[0], MOE_B200_DEV_TIMEOUT);
                status[1] = 67;
                status[2] = (int)blockIdx.x;
                ok = false;
                break;
              }
            }
          }
          if (!ok) break;
          asm volatile("fence.proxy.async;" ::: "memory");
        }
        const int half = it.n >> 1;
        const int row = it.row0 + (int)cta * half;
        const CUtensorMap* t64 = it.down ? &tmap_h64 : &tmap_x64;
        const CUtensorMap* t16 = it.down ? &tmap_h16 : &tmap_x16;
#pragma unroll 2
        for (int kb = 0; kb < it.kb; ++kb) {
          if (!try_wait(u_empty + stage * 8, phase ^ 1u) &&
              !mbar_wait(&ctl->empty[stage], phase ^ 1u, &ctl->abort, status, 66)) { ok = false; break; }
          const uint32_t sb = u_smem + (uint32_t)stage * kStageBytes, bar = u_full0 + stage * 8;
          int r = 0;
          for (; r + 64 <= half; r += 64) load_2d(sb + r * 128, t64, bar, kb * BK, row + r);
          for (; r < half; r += 16) load_2d(sb + r * 128, t16, bar, kb * BK, row + r);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- products ----------------
    if (cta == 0 && elect_one()) {
      const uint32_t u_smem = smem_u32(smem), u_full = smem_u32(ctl->full);
      const uint32_t u_e0 = map_to_cta(smem_u32(ctl->empty), 0), u_e1 = map_to_cta(smem_u32(ctl->empty), 1);
      int stage = 0;
      uint32_t phase = 0, acc_phase = 0;
      int a = 0;
      bool ok = true;
      Ring ring;
      while (ok) {
        const Item it = ring.take(ctl, cta, status);
        ring.arrive(ctl);
        ring.step();
        if (it.kb == 0) break;
        const uint32_t idesc = idesc_pair(it.n);
        if (!mbar_wait(&ctl->tmem_empty[a], acc_phase ^ 1u, &ctl->abort, status, 62)) break;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(a * kMaxTok);
#pragma unroll 2
        for (int kb = 0; kb < it.kb; ++kb) {
          if (!try_wait(u_full + stage * 8, phase) &&
              !mbar_wait(&ctl->full[stage], phase, &ctl->abort, status, 63)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = u_smem + (uint32_t)stage * kStageBytes;
          const uint64_t adesc = make_smem_desc(sa), bdesc = make_smem_desc(sa + kABytes);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            tc_mma_pair(tmem_d, adesc + (uint64_t)kk * 2, bdesc + (uint64_t)kk * 2, idesc, (kb | kk) != 0 ? 1u : 0u);
          tc_commit_pair(u_e0 + stage * 8);
          tc_commit_pair(u_e1 + stage * 8);
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        const uint32_t f_local = smem_u32(&ctl->tmem_full[a]);
        tc_commit_pair(map_to_cta(f_local, 0));
        tc_commit_pair(map_to_cta(f_local, 1));
        if (a == 1) acc_phase ^= 1u;
        a ^= 1;
      }
    }
  } else if (warp == 4 + kEpiWarps) {
    // ---------------- tiles are claimed and handed to all roles of the pair ----------------
    if (cta == 0 && elect_one()) {
      const uint32_t u_ring1 = map_to_cta(smem_u32(ctl->ring), 1), u_ring_full1 = map_to_cta(smem_u32(ctl->ring_full), 1);
      Ring ring;
      uint32_t phase = 0;
      for (;;) {
        const Item it = item_of(ctl, w, claim);
        if (!mbar_wait(&ctl->ring_empty[ring.slot], ring.phase ^ 1u, &ctl->abort, status, 69) ||
            !mbar_wait_cluster(&ctl->ring_peer[ring.slot], ring.phase ^ 1u, &ctl->abort, status, 69)) break;
        ctl->ring[ring.slot] = it;
        const uint32_t to = u_ring1 + ring.slot * (uint32_t)sizeof(Item);
        asm volatile("st.shared::cluster.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(it.e), "r"(it.nt), "r"(it.row0),
                     "r"(it.rows) : "memory");
        asm volatile("st.shared::cluster.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(to + 16), "r"(it.n), "r"(it.kb), "r"(it.down),
                     "r"(0) : "memory");
        mbar_arrive(&ctl->ring_full[ring.slot]);
        mbar_arrive_cluster(u_ring_full1 + ring.slot * 8);
        ring.step();
        if (it.kb == 0) break;
        if (!mbar_wait(&ctl->want, phase, &ctl->abort, status, 60)) break;
        phase ^= 1u;
        claim = atomicAdd(claimed, 1);
      }
    } else if (cta != 0 && elect_one()) {
      // (an arrival across the pair that releases waits for the warp's stores: no epilogue warp should)
      Ring ring;
      for (;;) {
        const Item it = ring.take(ctl, cta, status);
        if (!mbar_wait(&ctl->ring_empty[ring.slot], ring.phase, &ctl->abort, status, 69)) break;
        mbar_arrive_cluster(map_to_cta(smem_u32(&ctl->ring_peer[ring.slot]), 0));
        ring.step();
        if (it.kb == 0) break;
      }
    }
  } else if (warp == 3 + kEpiWarps) {
    // ---------------- stored tiles are made known: the fence waits for the memory, and no epilogue warp should ----------------
    if (elect_one()) {
      // (the slot is given back when its tile is known, so that no epilogue warp gets a round ahead on stored[slot])
      Ring ring;
      for (;;) {
        const Item it = ring.take(ctl, cta, status);
        if (it.kb > 0 && !it.down) {
          if (!mbar_wait(&ctl->stored[ring.slot], ring.phase, &ctl->abort, status, 68)) break;
          __threadfence();
          atomicAdd(&ready[it.e], 1);
        }
        ring.arrive(ctl);
        ring.step();
        if (it.kb == 0) break;
      }
    }
  } else {
    // ---------------- epilogue: two groups of four warps, a chunk of 32 tokens at a time each ----------------
    const int quad = warp & 3, group = (warp - 2) >> 2;
    const int gt = (int)threadIdx.x - 64 - group * 128;
    uint8_t* stg = stg_all + group * 2 * kStgBytes;
    int buf = 0;
    uint32_t acc_phase = 0;
    int a = 0;
    Ring ring;
    for (;;) {
      const Item it = ring.take(ctl, cta, status);
      const int slot = ring.slot;
      __syncwarp();
      if (lane == 0) ring.arrive(ctl);
      ring.step();
      if (!barrier_and(1 + group, 128, it.kb > 0)) break;      // the group leaves together
      const int feat0 = (it.nt * 2 + (int)cta) * (it.down ? kFeat2 : kFeat1);      // first feature of this CTA's tile
      const int feat = feat0 + (it.down ? quad * 32 + lane : quad * 16 + (lane >> 1));
      const int Nout = it.down ? d : f;
      float bias0 = 0.f, bias1 = 0.f;
      if (feat < Nout) {
        const __nv_bfloat16* b = static_cast<const __nv_bfloat16*>((it.down ? b2 : b1)[it.e]);
        bias0 = __bfloat162float(__ldg(b + feat));
        if (!it.down) bias1 = __bfloat162float(__ldg(b + f + feat));
      }
      // (where a wait runs out the tiles go on, so that all meet at the barriers below; the status says what they are worth)
      mbar_wait(&ctl->tmem_full[a], acc_phase, &ctl->abort, status, 64);
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(a * kMaxTok);
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(&ctl->tmem_empty[a]), 0));
      };
      if (group * 32 >= it.n) release();
      if (!it.down) {
#pragma unroll 1
        for (int c = group * 32; c < it.n; c += 64) {
          uint32_t v[32];
          tc_ld32(taddr + c, v);
          tc_ld_wait();
          if (c + 64 >= it.n) release();
          // even lanes hold gate, odd lanes up of a feature: each takes every other token
          uint8_t* s = stg + buf * kStgBytes + (lane & 1) * kPitch1 + (quad * 16 + (lane >> 1)) * 2;
          const bool odd = lane & 1;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? v[2 * i] : v[2 * i + 1], 1);
            const float g = __uint_as_float(odd ? other : v[2 * i]) + bias0;
            const float u = __uint_as_float(odd ? v[2 * i + 1] : other) + bias1;
            *reinterpret_cast<__nv_bfloat16*>(s + 2 * i * kPitch1) = __float2bfloat16_rn(gelu_tanh_fast(g) * u);
          }
          named_barrier(1 + group, 128);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int tok = j * 16 + (gt >> 3), piece = gt & 7, n = feat0 + piece * 8;
            if (c + tok < it.rows && n < f)
              *reinterpret_cast<uint4*>(h + (int64_t)(it.row0 + c + tok) * f + n) =
                  *reinterpret_cast<const uint4*>(stg + buf * kStgBytes + tok * kPitch1 + piece * 16);
          }
          buf ^= 1;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->stored[slot]);
      } else {
#pragma unroll 1
        for (int c = group * 32; c < it.n; c += 64) {
          uint32_t v[32];
          tc_ld32(taddr + c, v);
          tc_ld_wait();
          if (c + 64 >= it.n) release();
#pragma unroll
          for (int hc = 0; hc < 2; ++hc) {
            uint8_t* s = stg + buf * kStgBytes + (quad * 32 + lane) * 2;
#pragma unroll
            for (int i = 0; i < 16; ++i)
              *reinterpret_cast<__nv_bfloat16*>(s + i * kPitch2) = __float2bfloat16_rn(__uint_as_float(v[hc * 16 + i]) + bias0);
            named_barrier(1 + group, 128);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int tok = j * 8 + (gt >> 4), piece = gt & 15, n = feat0 + piece * 8;
              if (c + hc * 16 + tok < it.rows && n < d)
                *reinterpret_cast<uint4*>(y + (int64_t)(it.row0 + c + hc * 16 + tok) * d + n) =
                    *reinterpret_cast<const uint4*>(stg + buf * kStgBytes + tok * kPitch2 + piece * 16);
            }
            buf ^= 1;
          }
        }
      }
      if (a == 1) acc_phase ^= 1u;
      a ^= 1;
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
  cluster_sync();
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  // the last CTA to leave puts the counters back to zero for the next call
  if (threadIdx.x == 0) {
    int* exit_count = ready + (MOE_B200_READY_INTS - 2);
    __threadfence();
    if (atomicAdd(exit_count, 1) == (int)gridDim.x - 1) {
      for (int e = 0; e < E; ++e) ready[e] = 0;
      *claimed = 0;
      *exit_count = 0;
    }
  }
}

}  // namespace

// Whether a call of M rows is better off here than with the kernels it would take else.
// More than 32 experts, up to 256 rows: the matrix-vector kernel goes row by row (64 experts, d 2048, f 1408, four slots, us:
// 4 rows 99 / here 58, 64 rows 1163 / 147). Up to 32 experts the streaming kernel is as fast below 96 rows an expert (600
// rows of 8 experts 60 / 62) and, with one or two experts, below 1536 rows.
// Up to 4096 rows the streaming kernel remains (experts_decode_spec.cu, sorted rows), which cuts the down product's K into
// ranges for all SMs. Here that product takes whole rounds of all K on pairs of SMs, and where d is small and f large its
// few tiles are the longest part of the call (d 256, f 8192, 8 experts, 768 rows: 51.8 / here 68.3 us, 3 experts 45.4 /
// 67.9), while the streaming kernel's GEGLU product reads weights once per 128 rows. So the two are compared by what
// differs, rounds x steps of 64 of K under balanced routing, in us: a step of the down product here, up to 0.31 with 256
// tokens, and 0.75 a round of GEGLU epilogues; there 0.30 a step of GEGLU with 128 rows, 0.27 one of a range of down's K, and
// what the fp32 sums of the ranges cost. Fitted to whole calls of both kernels: 1 to 200 experts, d 64 to 4096, f 264 to
// 16384, 2012 sizes. The kernel that is chosen takes 0.4 % longer than the faster one on average (always here: 4 %), and is
// the slower one by more than 3 % at 106 sizes (by 4.4 % in the middle of them, by 15 % at most). One or two experts with f
// beyond 4 d are told apart by d alone, where the estimate is least good (3000 rows of two: d 512, f 8192 105 / here 118, d
// 1024, f 8192 174 / 148).
// Beyond, the 256-row tiles remain (experts_tc2.cu), to which remainders no longer count at 2048 rows an expert (8 experts,
// d 1024, f 4096 there: 349 / here 319). With K of the down product more than four times that of gate_and_up a tile's
// epilogue is the bound, and theirs is the faster: up to 2 d rows an expert this one is still ahead (d 256, f 2048, 24
// experts, 320 rows each 93.9 / 87.3; d 256, f 8192, 8 experts, 2048 rows each 262 / 292).
bool experts_mid_chosen(int64_t M, int d, int f, int E) {
  if (M <= kDecodeMaxRows) return E > 32 && M > 0;
  const int64_t least = E > 32 ? 0 : E > 2 ? (int64_t)96 * E : 1536;
  const int64_t most = E > 2 ? (int64_t)2048 * E : kRowsPathMaxRows;
  if (M < least || M > most) return false;
  if (E <= 2 && f > 4 * (int64_t)d + 64) return d >= 1024;
  if (M > kRowsPathMaxRows || !rows_supported(M, E)) return f <= 4 * (int64_t)d + 64 || M <= (int64_t)2 * d * E;
  auto up = [](int64_t a, int64_t b) { return (a + b - 1) / b; };
  auto rounds = [](int64_t tiles, int units) { return fmax(1., (double)tiles / units + .5); };
  const int64_t hit = M < E ? M : E, share = up(M, hit);          // experts with rows, rows of one
  const int64_t cut = up(share, kMaxTok), n = up(up(share, cut), 32) * 32;
  const int64_t n1 = up(f, 128), n2 = up(d, 256), kb1 = up(d, BK), kb2 = up(f, BK);
  const int NP = rows_block(M, E), ks = rows_splits(M, d, f, E);
  const int64_t blocks = hit * up(share, NP);                     // of the streaming kernel
  const double here = rounds(hit * cut * n2, kNumSMs / 2) * kb2 * (0.078 + 0.232 * n / kMaxTok) +
                      0.75 * rounds(hit * cut * n1, kNumSMs / 2) - 1.3;
  const double there = 0.30 * rounds(blocks * n1, kNumSMs) * kb1 * NP / 128 +
                       0.27 * rounds(blocks * n2 * ks, kNumSMs) * up(kb2, ks) + 1.5e-6 * M * d * ks;
  return here < there;
}

int launch_experts_mid(const void* perm, const int32_t* offsets, const void* plan, int64_t M, int d, int f, int E, void* h,
                       void* y, int* ready, int32_t* status, cudaStream_t s) {
  if (M == 0) return 0;
  PlanView pv = plan_view(plan, E);
  int sms = 0;
  int rc = sm_count(&sms);
  if (rc) return rc;
  static PerDeviceOnce once;
  rc = ensure_dynamic_smem(once, experts_mid_kernel, kSmemBytes);
  if (rc) return rc;
  alignas(64) CUtensorMap x64, x16, h64, h16;
  rc = encode_tmap_2d(&x64, perm, (uint64_t)M, (uint64_t)d, 64);
  if (!rc) rc = encode_tmap_2d(&x16, perm, (uint64_t)M, (uint64_t)d, 16);
  if (!rc) rc = encode_tmap_2d(&h64, h, (uint64_t)M, (uint64_t)f, 64);
  if (!rc) rc = encode_tmap_2d(&h16, h, (uint64_t)M, (uint64_t)f, 16);
  if (rc) return rc;
  // with fewer rows many experts have none, and their weights would come for nothing (64 experts: 1 token 102.2 -> 99.7 us,
  // 12 tokens 148.3 -> 147.2; the same at 64)
  const int ahead = M >= 2 * (int64_t)E ? 1 : 0;
  MOE_CUDA_CHECK(launch_pdl_cluster(experts_mid_kernel, dim3((unsigned)(sms & ~1)), dim3(kThreads), 2, kSmemBytes, s, x64,
                                    x16, h64, h16, static_cast<const CUtensorMap*>(pv.tmap_W1_pairs),
                                    static_cast<const CUtensorMap*>(pv.tmap_W2), offsets, pv.b1, pv.b2, E, d, f, ahead,
                                    static_cast<__nv_bfloat16*>(h), static_cast<__nv_bfloat16*>(y), ready, status));
  return 0;
}

}  // namespace moe
