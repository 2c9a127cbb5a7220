// Expert feed-forward on CUDA cores: the fp32 implementation of
// FeedForward.forward (reference model.py:173-190, fine_tuning=False, eval):
//   h = gelu_tanh(x W1[:f]^T + b1[:f]) * (x W1[f:]^T + b1[f:])   (model.py:174,180-182)
//   y = h W2^T + b2                                               (model.py:184)
// grouped over experts by the row offsets the dispatch kernel wrote.
//
// fp32 needs max-abs 1e-4 against the reference, which single-pass TF32
// tensor-core math does not give after two chained products, so this path is
// fp32 FMA with fp32 accumulation, and the FMA pipe is what bounds it.
//   Block: 128 threads, 64 rows x 128 weight rows (GEGLU: 64 gate and the 64 up
//   rows of the same features), K in steps of 32 through three cp.async stages.
//   Both operands stay as they lie in memory, [row][k], and a thread multiplies
//   its 8 x 8 tile four k at a time: sixteen 16-byte reads of shared memory for
//   256 products. fma.rn.f32x2 takes two neighbouring k, so operands are register
//   pairs as loaded; even and odd k are summed apart and added at the end. The
//   pipe takes a pair in the time of one plain FMA (the same tiles with fmaf, at
//   twice the warps an SM, took 1.15 times as long).
//   Rows of 36 floats: the eight rows a quarter-warp reads lie in eight
//   different groups of four banks.
//   Warps whose 32 rows lie behind the expert's last row only load.
//   A cluster of up to eight blocks shares one tile and splits K where tiles are
//   few; partial tiles meet in shared memory and are summed in rank order, each
//   block for its share of the rows.
// 1024 rows of 8 experts, d 512, f 2048: gate_and_up 178 -> 160 us, down 184 -> 90 us
// (before: 64 x 64 tiles of 4 x 4 per thread, no split of K). Left: the FMA pipe is
// busy 45% of the time, with two warps a scheduler that wait for their operands.
#include "common.cuh"

namespace moe {

namespace {

constexpr int BM = 64, BN = 128, BK = 32;
constexpr int kPitch = BK + 4;                     // floats
constexpr int kStages = 3;
constexpr int kThreads = 128;
constexpr int kStageFloats = (BM + BN) * kPitch;
constexpr int kOutPitch = BN + 4;
constexpr size_t kSmemBytes = (size_t)kStages * kStageFloats * sizeof(float);
static_assert(BM * kOutPitch <= kStages * kStageFloats, "the partial tile reuses the stages");

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// invalid: fills with zeros and reads nothing
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool valid) {
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(dst);
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa), "l"(src), "r"(bytes) : "memory");
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
__device__ __forceinline__ float ld_cluster(const float* p, uint32_t rank) {
  uint32_t addr = (uint32_t)__cvta_generic_to_shared(p), remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}

// One K step of a warp: the first 4 * MI of its rows (row ty + 4 i) times its 64 columns (tx + 8 j).
template <int MI>
__device__ __forceinline__ void multiply(const float* a, const float* b, uint64_t (&acc)[8][8]) {
#pragma unroll 2
  for (int kk = 0; kk < BK; kk += 4) {
    ulonglong2 av[MI];
#pragma unroll
    for (int i = 0; i < MI; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(a + 4 * i * kPitch + kk);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const ulonglong2 bv = *reinterpret_cast<const ulonglong2*>(b + 8 * j * kPitch + kk);
#pragma unroll
      for (int i = 0; i < MI; ++i) acc[i][j] = fma2(av[i].x, bv.x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < MI; ++i) acc[i][j] = fma2(av[i].y, bv.y, acc[i][j]);
    }
  }
}

// A: [rows, K] activations (sorted buffer); W: per-expert [Nw, K]; out [rows, Nout].
// GEGLU: Nw = 2*Nout, gate rows [0,Nout), up rows [Nout, 2*Nout).
// grid (row tiles, column tiles, splits of K = cluster size)
template <bool GEGLU>
__global__ void __launch_bounds__(kThreads, 2)
grouped_ffn_kernel(const float* __restrict__ A, const int32_t* __restrict__ offsets,
                   const void* const* __restrict__ Wp, const void* const* __restrict__ bp, int E,
                   int K, int Nout, float* __restrict__ out) {
  extern __shared__ __align__(16) float smem[];
  __shared__ int s_off[kMaxExperts + 1];
  // all offsets at once: one thread walking them in memory is a chain of up to E trips to L2
  for (int i = threadIdx.x; i <= E; i += kThreads) s_off[i] = offsets[i];
  __syncthreads();
  int e = 0, row0 = 0, rows = 0;
  for (int tile = blockIdx.x; e < E; ++e) {
    const int beg = s_off[e], cnt = s_off[e + 1] - beg;
    const int tiles = (cnt + BM - 1) / BM;
    if (tile < tiles) { row0 = beg + tile * BM; rows = min(BM, cnt - tile * BM); break; }
    tile -= tiles;
  }
  if (e == E) return;    // the whole cluster: its blocks share blockIdx.x
  constexpr int kCols = GEGLU ? BN / 2 : BN;     // output columns of a tile
  const int n0 = blockIdx.y * kCols;
  const float* W = static_cast<const float*>(Wp[e]);
  const float* bias = static_cast<const float*>(bp[e]);
  const uint32_t splits = gridDim.z, rank = splits > 1 ? cluster_rank() : 0u;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = warp & 1, wn = warp >> 1;       // 32 rows, 64 columns
  const int ty = lane >> 3, tx = lane & 7;

  // loads: eight threads per row of 32 k, sixteen rows at a time (4 passes over A, 8 over W)
  const int lr = tid >> 3, lk = (tid & 7) * 4;
  const float* srcA = A + (int64_t)(row0 + lr) * K + lk;
  const float* srcW = W + (int64_t)(n0 + lr) * K + lk;
  const int64_t step = (int64_t)16 * K;                  // sixteen rows
  const int64_t to_up = (int64_t)(Nout - 64) * K;        // GEGLU: from the last gate rows to the first up rows
  const int kb_all = (K + BK - 1) / BK;
  const int per = (kb_all + (int)splits - 1) / (int)splits;
  const int kb0 = min(kb_all, (int)rank * per), kb1 = min(kb_all, kb0 + per);
  auto fetch = [&](int kb) {
    if (kb < kb1) {
      float* dst = smem + (size_t)((kb - kb0) % kStages) * kStageFloats + lr * kPitch + lk;
      const int k = kb * BK;
      const bool k_ok = k + lk < K;                // K is a multiple of 4: a piece is whole or absent
      const float* q = srcA + k;                   // rows that do not exist are filled, not read
#pragma unroll
      for (int p = 0; p < BM / 16; ++p, q += step) cp_async16(dst + p * 16 * kPitch, q, k_ok && p * 16 + lr < rows);
      q = srcW + k;
#pragma unroll
      for (int p = 0; p < BN / 16; ++p, q += step) {
        if (GEGLU && p == 4) q += to_up;
        cp_async16(dst + (BM + p * 16) * kPitch, q, k_ok && n0 + (GEGLU ? p & 3 : p) * 16 + lr < Nout);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  uint64_t acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  const int my_rows = rows - wm * 32;              // of this warp; uniform in it
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) fetch(kb0 + s);
  for (int kb = kb0; kb < kb1; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();      // stage kb is there for all; stage kb - 1 has been read by all
    fetch(kb + kStages - 1);
    const float* st = smem + (size_t)((kb - kb0) % kStages) * kStageFloats;
    const float* a = st + (wm * 32 + ty) * kPitch;
    const float* b = st + (BM + wn * 64 + tx) * kPitch;
    if (my_rows > 8) multiply<8>(a, b, acc);
    else if (my_rows > 0) multiply<2>(a, b, acc);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // ---- the (partial) tile in shared memory, summed over the cluster, act and store ----
  if (my_rows > 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 v = *reinterpret_cast<const float2*>(&acc[i][j]);
        smem[(wm * 32 + ty + 4 * i) * kOutPitch + wn * 64 + tx + 8 * j] = v.x + v.y;
      }
  }
  if (splits > 1) cluster_sync(); else __syncthreads();
  const int share = BM / (int)splits;
  const int r_begin = (int)rank * share, r_end = min(rows, r_begin + share);
  auto total = [&](int r, int c) {
    const float* p = smem + r * kOutPitch + c;
    if (splits == 1) return *p;
    float v = ld_cluster(p, 0);
    for (uint32_t q = 1; q < splits; ++q) v += ld_cluster(p, q);
    return v;
  };
  for (int i = tid; i < (r_end - r_begin) * kCols; i += kThreads) {
    const int r = r_begin + i / kCols, c = i % kCols, n = n0 + c;
    if (n >= Nout) continue;
    float val = total(r, c) + bias[n];
    if (GEGLU) val = gelu_tanh_precise(val) * (total(r, c + 64) + bias[Nout + n]);
    out[(int64_t)(row0 + r) * Nout + n] = val;
  }
  if (splits > 1) cluster_sync();     // no block leaves while another reads its tile
}

// Splits of K: until there are four rounds of the blocks that are resident together (two an SM), so that the
// last round is a small part, but at least four K steps (128) each.
int pick_splits(int64_t tiles, int K) {
  const int kb = (K + BK - 1) / BK;
  int s = 1;
  while (s < 8 && tiles * s < 4 * 2 * kNumSMs && kb >= 8 * s) s *= 2;
  return s;
}

template <bool GEGLU>
int launch(const float* A, const int32_t* offsets, const void* const* W, const void* const* b, int64_t M, int K,
           int Nout, int E, float* out, cudaStream_t s) {
  static PerDeviceOnce once;
  int rc = ensure_dynamic_smem(once, grouped_ffn_kernel<GEGLU>, kSmemBytes);
  if (rc) return rc;
  const int64_t n_tiles = (Nout + (GEGLU ? BN / 2 : BN) - 1) / (GEGLU ? BN / 2 : BN);
  // the host does not know the routing: every expert that can have rows ends in half a tile
  const int64_t expected = (M + BM - 1) / BM + (M < E ? M : E) / 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((M + BM - 1) / BM + E), (unsigned)n_tiles,
                     (unsigned)pick_splits(expected * n_tiles, K));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = cfg.gridDim.z;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MOE_CUDA_CHECK(cudaLaunchKernelEx(&cfg, grouped_ffn_kernel<GEGLU>, A, offsets, W, b, E, K, Nout, out));
  return 0;
}

}  // namespace

int launch_experts_simt(const void* perm, const int32_t* offsets, const void* plan, int64_t M,
                        int d, int f, int E, void* h, void* y, cudaStream_t s) {
  if (M == 0) return 0;
  PlanView pv = plan_view(plan, E);
  int rc = launch<true>(static_cast<const float*>(perm), offsets, pv.W1, pv.b1, M, d, f, E, static_cast<float*>(h), s);
  if (rc) return rc;
  return launch<false>(static_cast<const float*>(h), offsets, pv.W2, pv.b2, M, f, d, E, static_cast<float*>(y), s);
}

}  // namespace moe
