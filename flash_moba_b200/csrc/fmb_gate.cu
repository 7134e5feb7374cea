// Stage G: fused gating.  scores = Q . centroid^T (fp32, unscaled) -> causal chunk rule ->
// per-row top-k, in one kernel; the score matrix never reaches HBM.
//
// Replaces csrc/flash_topk/src/flash_topk_kernel.h:31-357 of the reference (one thread per
// row doing a serial insertion over every score of every tile).  Two kernels:
//   * gate_topk_tc_kernel (head dims 64 / 128, top-k <= 32): the score tile is a tcgen05 MMA with
//     the accumulator in TMEM; TMEM lane = query row, so a thread reads its row's scores straight
//     from TMEM and keeps the row's list in registers as 64-bit ordered keys;
//   * gate_topk_kernel (other shapes, and the cross-check of the first): CUDA-core score tile in
//     shared memory, a warp per row, the list distributed over the lanes.
// Ordering rule = the reference's: descending score, and on equal scores the higher chunk id
// first (csrc/flash_topk/src/flash_topk_kernel.h:261-285).
#include <type_traits>

#include "fmb_common.cuh"
#include "fmb_tma.cuh"

namespace fmb {

int sm_count();   // SMs of the current device (fmb_attn_common.cu)

constexpr int kGateM = 128;          // query rows per CTA
constexpr int kGateN = 128;          // centroids per score tile
constexpr int kGateThreads = 256;
constexpr int kGateDSlab = 128;      // head-dim slab staged in shared memory
constexpr int kGateSStride = kGateN + 4;

struct GateParams {
  const void* q; int64_t q_rs, q_hs;
  const void* km;
  const int32_t *cu_q, *cu_k, *cu_km;
  int32_t* topk_idx; float* topk_val; int64_t t_rs, t_hs;
  int heads, heads_k, d, topk, chunk, causal;
};

// true if entry a ranks ahead of entry b
__device__ __forceinline__ bool ranks_ahead(float va, int ia, float vb, int ib) {
  return va > vb || (va == vb && ia > ib);
}

// Sorted list of one row, distributed over the warp: lane j holds ranks j and j+32.
struct RowList {
  float v0, v1;
  int i0, i1;
};

template <bool kTwoHalves>
__device__ __forceinline__ void list_insert(RowList& L, float v, int n, int topk, int lane) {
  const unsigned full = 0xffffffffu;
  const unsigned m0 = __ballot_sync(full, ranks_ahead(L.v0, L.i0, v, n));
  int pos = __popc(m0);
  if (kTwoHalves) pos += __popc(__ballot_sync(full, ranks_ahead(L.v1, L.i1, v, n)));
  // shift the tail down by one rank and drop the new entry in at `pos`
  const float pv0 = __shfl_up_sync(full, L.v0, 1);
  const int pi0 = __shfl_up_sync(full, L.i0, 1);
  if (kTwoHalves) {
    const float cv = __shfl_sync(full, L.v0, 31);
    const int ci = __shfl_sync(full, L.i0, 31);
    float pv1 = __shfl_up_sync(full, L.v1, 1);
    int pi1 = __shfl_up_sync(full, L.i1, 1);
    if (lane == 0) { pv1 = cv; pi1 = ci; }
    const int r1 = lane + 32;
    if (r1 == pos) { L.v1 = v; L.i1 = n; }
    else if (r1 > pos) { L.v1 = pv1; L.i1 = pi1; }
    if (r1 >= topk) { L.v1 = -CUDART_INF_F; L.i1 = -1; }
  }
  if (lane == pos) { L.v0 = v; L.i0 = n; }
  else if (lane > pos) { L.v0 = pv0; L.i0 = pi0; }
  if (lane >= topk) { L.v0 = -CUDART_INF_F; L.i0 = -1; }
}

// Offer 32 scores (one per lane) of one row to its list.
template <bool kTwoHalves>
__device__ __forceinline__ void list_offer(RowList& L, float v, int n, bool eligible, int topk, int lane) {
  const unsigned full = 0xffffffffu;
  const int kl = (topk - 1) & 31;
  float tv = __shfl_sync(full, (kTwoHalves && topk > 32) ? L.v1 : L.v0, kl);
  int ti = __shfl_sync(full, (kTwoHalves && topk > 32) ? L.i1 : L.i0, kl);
  bool cand = eligible && v > -CUDART_INF_F && ranks_ahead(v, n, tv, ti);
  unsigned m = __ballot_sync(full, cand);
  while (m) {
    const int src = __ffs(m) - 1;
    const float nv = __shfl_sync(full, v, src);
    const int nn = __shfl_sync(full, n, src);
    list_insert<kTwoHalves>(L, nv, nn, topk, lane);
    tv = __shfl_sync(full, (kTwoHalves && topk > 32) ? L.v1 : L.v0, kl);
    ti = __shfl_sync(full, (kTwoHalves && topk > 32) ? L.i1 : L.i0, kl);
    cand = cand && lane != src && ranks_ahead(v, n, tv, ti);
    m = __ballot_sync(full, cand);
  }
}

// One score tile (rows x ncols in sS) offered to the rows' lists; warp w owns rows w*R..,
// R = 128 / number of warps.
template <bool kTwoHalves>
__device__ __forceinline__ void select_tile(const float* sS, float* sTV, int* sTI, int r0, int rows, int n0,
                                            int ncols, int shift, int topk, int chunk, int causal) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows_per_warp = kGateM / (blockDim.x >> 5);
  for (int rr = 0; rr < rows_per_warp; ++rr) {
    const int r = warp * rows_per_warp + rr;
    if (r >= rows) break;
    const int pos = r0 + r + shift;
    RowList L;
    L.v0 = lane < topk ? sTV[r * topk + lane] : -CUDART_INF_F;
    L.i0 = lane < topk ? sTI[r * topk + lane] : -1;
    L.v1 = -CUDART_INF_F; L.i1 = -1;
    if (kTwoHalves && lane + 32 < topk) { L.v1 = sTV[r * topk + lane + 32]; L.i1 = sTI[r * topk + lane + 32]; }
    for (int g = 0; g < kGateN; g += 32) {
      if (g >= ncols) break;
      const int n = n0 + g + lane;
      const float v = sS[r * kGateSStride + g + lane];
      const bool ok = (g + lane < ncols) && (!causal || ((n + 1) * chunk - 1 < pos));
      list_offer<kTwoHalves>(L, v, n, ok, topk, lane);
    }
    if (lane < topk) { sTV[r * topk + lane] = L.v0; sTI[r * topk + lane] = L.i0; }
    if (kTwoHalves && lane + 32 < topk) { sTV[r * topk + lane + 32] = L.v1; sTI[r * topk + lane + 32] = L.i1; }
  }
}

// CUDA-core score tile: S[128][128] = Qt^T . Kt over one head-dim slab (operands transposed
// in shared memory so that each thread reads 16 contiguous bytes per operand per step).
template <typename T>
__device__ __forceinline__ void score_tile_fma(const T* sQt, const T* sKt, int dlen, float (&acc)[8][8]) {
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  for (int dd = 0; dd < dlen; ++dd) {
    float a[8], b[8];
    unpack8<T>(*reinterpret_cast<const uint4*>(sQt + dd * kGateM + ty * 8), a);
    unpack8<T>(*reinterpret_cast<const uint4*>(sKt + dd * kGateN + tx * 8), b);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
  }
}

// stage rows [r0, r0+128) x dims [d0, d0+dlen) of a (rows, stride) matrix, transposed
template <typename T>
__device__ __forceinline__ void stage_transposed(T* dst, const T* src, int64_t row_stride, int rows_valid,
                                                 int d0, int dlen) {
  // lane -> row (conflict-free transposed stores), loop over 16-byte column groups
  const int ngroups = dlen / 8;
  for (int e = threadIdx.x; e < 128 * ngroups; e += blockDim.x) {
    const int r = e & 127, g = e >> 7;
    uint4 u = make_uint4(0, 0, 0, 0);
    if (r < rows_valid) u = ldg_nc_16(src + (int64_t)r * row_stride + d0 + g * 8);
    const T* x = reinterpret_cast<const T*>(&u);
#pragma unroll
    for (int i = 0; i < 8; ++i) dst[(g * 8 + i) * 128 + r] = x[i];
  }
}

template <typename T, bool kTwoHalves>
__global__ void __launch_bounds__(kGateThreads) gate_topk_kernel(GateParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sQt = reinterpret_cast<T*>(smem_raw);                         // [128 dd][128 rows]
  T* sKt = sQt + kGateDSlab * kGateM;                              // [128 dd][128 centroids]
  float* sS = reinterpret_cast<float*>(sKt + kGateDSlab * kGateN); // [128][132]
  float* sTV = sS + kGateM * kGateSStride;                         // [128][topk]
  int* sTI = reinterpret_cast<int*>(sTV + kGateM * p.topk);        // [128][topk]

  // late row tiles see the most candidate chunks under a causal mask: they are scheduled first
  const int mt = gridDim.x - 1 - blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int q0 = p.cu_q[b], len_q = p.cu_q[b + 1] - q0;
  const int len_k = p.cu_k[b + 1] - p.cu_k[b];
  const int km0 = p.cu_km[b], nchunks = p.cu_km[b + 1] - km0;
  const int r0 = mt * kGateM;
  if (r0 >= len_q) return;
  const int rows = min(kGateM, len_q - r0);
  const int hk = h / (p.heads / p.heads_k);
  const int shift = len_k - len_q;
  const int topk = p.topk;

  // initial lists: empty, or the row's own chunk pinned at rank 0 under the causal rule
  for (int e = threadIdx.x; e < kGateM * topk; e += blockDim.x) {
    const int r = e / topk, j = e - r * topk;
    float v = -CUDART_INF_F;
    int i = -1;
    const int pos = r0 + r + shift;
    if (p.causal && j == 0 && r < rows && pos >= 0 && nchunks > 0) { v = CUDART_INF_F; i = pos / p.chunk; }
    sTV[e] = v;
    sTI[e] = i;
  }

  // centroids that any row of this CTA may still select
  int n_end = nchunks;
  if (p.causal) {
    const int pmax = r0 + rows - 1 + shift;
    n_end = pmax < 0 ? 0 : min(nchunks, pmax / p.chunk);   // candidate n: (n+1)*chunk <= p
  }
  const T* qbase = static_cast<const T*>(p.q) + (int64_t)(q0 + r0) * p.q_rs + (int64_t)h * p.q_hs;
  const T* kmbase = static_cast<const T*>(p.km) + ((int64_t)km0 * p.heads_k + hk) * p.d;
  const int64_t km_rs = (int64_t)p.heads_k * p.d;
  const bool single_slab = p.d <= kGateDSlab;
  if (single_slab && n_end > 0) stage_transposed<T>(sQt, qbase, p.q_rs, rows, 0, p.d);
  __syncthreads();

  for (int n0 = 0; n0 < n_end; n0 += kGateN) {
    const int ncols = min(kGateN, n_end - n0);
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    for (int d0 = 0; d0 < p.d; d0 += kGateDSlab) {
      const int dlen = min(kGateDSlab, p.d - d0);
      if (!single_slab) stage_transposed<T>(sQt, qbase, p.q_rs, rows, d0, dlen);
      stage_transposed<T>(sKt, kmbase + (int64_t)n0 * km_rs, km_rs, ncols, d0, dlen);
      __syncthreads();
      score_tile_fma<T>(sQt, sKt, dlen, acc);
      __syncthreads();
    }
    {
      const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float* dst = sS + (ty * 8 + i) * kGateSStride + tx * 8;
        *reinterpret_cast<float4*>(dst) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
      }
    }
    __syncthreads();
    select_tile<kTwoHalves>(sS, sTV, sTI, r0, rows, n0, ncols, shift, topk, p.chunk, p.causal);
    __syncthreads();
  }
  __syncthreads();
  // write the lists
  for (int e = threadIdx.x; e < rows * topk; e += blockDim.x) {
    const int r = e / topk, j = e - r * topk;
    const int64_t o = (int64_t)(q0 + r0 + r) * p.t_rs + (int64_t)h * p.t_hs + j;
    p.topk_idx[o] = sTI[e];
    if (p.topk_val) p.topk_val[o] = sTV[e];
  }
}

// ---------------------------------------------------------------------------------------
// Tensor-core variant (head_dim 64, 128 or 256, top-k <= 32).  The score tile is a tcgen05 MMA
// with the accumulator in TMEM; TMEM lane = query row, so thread t reads row t's scores
// straight from TMEM (no shared-memory staging of scores) and keeps that row's top-k list
// in registers: val[] = order-preserving 32-bit images of the fp32 scores, descending, and
// idx[] = their chunk ids.  A thread meets its candidates in ascending chunk order, so "the
// higher chunk id ranks first on equal scores" (the reference's rule) is simply: a candidate
// goes ahead of every entry it is greater than OR EQUAL to, one 32-bit compare per slot; the
// values move with a min/max pair, the ids with two selects.  Slots that must never be
// displaced (the row's own chunk, and the unused head of a list shorter than KMAX) hold the image
// 0xffffffff, which no score that passes the "> -inf" test can reach; the empty slot holds the
// image of -inf.  Q is staged once; centroid tiles and TMEM accumulators are double-buffered so
// the MMA of tile n+1 runs under the selection of tile n; two CTAs share an SM.  All waits are
// bounded (status word g_gate_status).
// ---------------------------------------------------------------------------------------
__device__ int g_gate_status = 0;

__device__ __forceinline__ uint32_t score_to_ordered(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ordered_to_score(uint32_t o) {
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// NQ threads share a row (TMEM lane): warps w, w+4, w+8, ... may all read lane quarter w%4, so
// each of them scans 128/NQ of a tile's columns into a private list; the NQ lists of a row are
// merged once at the end.  More warps per row hide the latency of the (divergent) insertions.
template <typename T, int D, int KMAX, int NQ>
__global__ void __launch_bounds__(128 * NQ) gate_topk_tc_kernel(GateParams p) {
  using namespace tc;
  constexpr uint32_t kBlock = 128 * 128;       // bytes between 64-element blocks of a 128-row tile
  constexpr uint32_t kTile = 128 * D * 2;
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t bar[2];
  __shared__ uint32_t tmem_base_s;
  // the two threads of a row tell each other the eight best images they hold (NQ == 2)
  __shared__ uint32_t sX[NQ == 2 ? 2 : 1][NQ == 2 ? 8 : 1][NQ == 2 ? 128 : 1];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* sQ = smem;
  unsigned char* sKM = sQ + kTile;             // two buffers

  // late row tiles see the most candidate chunks under a causal mask: they are scheduled first
  const int mt = gridDim.x - 1 - blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int q0 = p.cu_q[b], len_q = p.cu_q[b + 1] - q0;
  const int len_k = p.cu_k[b + 1] - p.cu_k[b];
  const int km0 = p.cu_km[b], nchunks = p.cu_km[b + 1] - km0;
  const int r0 = mt * kGateM;
  if (r0 >= len_q) return;
  const int rows = min(kGateM, len_q - r0);
  const int hk = h / (p.heads / p.heads_k);
  const int shift = len_k - len_q;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int lt = tid & 127, qd = tid >> 7;     // row, and which share of the columns
  const int topk = p.topk;

  // this thread's row: list of KMAX keys, descending; the first KMAX-topk are sentinels
  const int pos = r0 + lt + shift;
  const bool row_ok = lt < rows;
  int nlim = nchunks;                          // candidate chunks of the row: n < nlim
  if (p.causal) nlim = pos < 0 ? 0 : min(nchunks, pos / p.chunk);
  if (!row_ok) nlim = 0;
  constexpr uint32_t kFixed = 0xffffffffu;     // image of a slot no candidate may displace
  constexpr uint32_t kEmptyVal = 0x007fffffu;  // image of -inf: the empty slot
  constexpr int kBlockedId = -2;               // id of the unused head of a list shorter than KMAX
  const bool own = p.causal && row_ok && pos >= 0 && nchunks > 0 && qd == 0;
  uint32_t val[KMAX];
  int idx[KMAX];
#pragma unroll
  for (int j = 0; j < KMAX; ++j) {   // static indices only: the list must stay in registers
    const bool blocked = j < KMAX - topk, is_own = (j == KMAX - topk) && own;
    val[j] = (blocked || is_own) ? kFixed : kEmptyVal;
    idx[j] = blocked ? kBlockedId : (is_own ? pos / p.chunk : -1);
  }
  // val[j] for a j that depends on the run-time top-k (selects: the list must stay in registers)
  auto val_at = [&](int j) {
    if (topk == KMAX) return val[j < KMAX ? j : 0];   // (callers pass compile-time j: no selects in the common case)
    uint32_t x = val[0];
#pragma unroll
    for (int y = 1; y < KMAX; ++y) x = (j == y) ? val[y] : x;
    return x;
  };
  // candidate (image ox, chunk n) into the list; every entry already there has a lower chunk id
  auto insert = [&](uint32_t ox, int n) {
    bool ge[KMAX];
#pragma unroll
    for (int y = 0; y < KMAX; ++y) ge[y] = ox >= val[y];
#pragma unroll
    for (int y = KMAX - 1; y > 0; --y) {
      idx[y] = ge[y - 1] ? idx[y - 1] : (ge[y] ? n : idx[y]);
      val[y] = min(val[y - 1], max(val[y], ox));
    }
    idx[0] = ge[0] ? n : idx[0];
    val[0] = max(val[0], ox);
  };

  int n_end = nchunks;
  if (p.causal) {
    const int pmax = r0 + rows - 1 + shift;
    n_end = pmax < 0 ? 0 : min(nchunks, pmax / p.chunk);
  }
  const int ntiles = (n_end + kGateN - 1) / kGateN;
  if (ntiles > 0) {   // CTA-uniform
    if (warp == 0) tmem_alloc(&tmem_base_s, 256);
    if (tid == 0) {
      mbar_init(&bar[0], 1);
      mbar_init(&bar[1], 1);
      mbar_fence_init();
    }
    const T* qbase = static_cast<const T*>(p.q) + (int64_t)(q0 + r0) * p.q_rs + (int64_t)h * p.q_hs;
    const T* kmbase = static_cast<const T*>(p.km) + ((int64_t)km0 * p.heads_k + hk) * p.d;
    const int64_t km_rs = (int64_t)p.heads_k * p.d;
    // The Q tile and the first two centroid tiles are copied with cp.async (no registers, all in
    // flight at once); inside the loop the tile two steps ahead is copied while this step's scores
    // are examined, and its MMA is issued at the step's end, so that neither a copy nor an MMA is
    // waited for in the steady state.
    auto stage_km = [&](int t) {
      const int n1 = t * kGateN, nc = min(kGateN, n_end - n1);
      dense_cp_async<T, D / 8, kGateN, 128 * NQ>(tid, sKM + (t & 1) * kTile, kBlock, kmbase + (int64_t)n1 * km_rs, km_rs, nc);
    };
    dense_cp_async<T, D / 8, kGateM, 128 * NQ>(tid, sQ, kBlock, qbase, p.q_rs, rows);
    stage_km(0);
    if (ntiles > 1) stage_km(1);
    cp_async_wait_all();
    fence_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_s;
    const uint32_t sQ_a = smem_u32(sQ), sKM_a = smem_u32(sKM);
    constexpr uint32_t idesc = make_idesc(FmtOf<T>::v, 128, 128, 0, 0);
    auto issue = [&](int buf) {
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        const uint32_t o = (ks >> 2) * kBlock + (ks & 3) * 32;
        umma_ss(tmem_base + buf * 128, make_desc_sw128(sQ_a + o, 16, 1024),
                make_desc_sw128(sKM_a + buf * kTile + o, 16, 1024), idesc, ks > 0);
      }
      umma_commit(&bar[buf]);
    };
    if (tid == 0) {
      issue(0);
      if (ntiles > 1) issue(1);
    }
    uint32_t phases = 0;   // bit b = parity to wait for on bar[b]
    float floor_thr_row = -CUDART_INF_F;   // what the k-th best of the row is known to reach
    for (int t = 0; t < ntiles; ++t) {
      const int buf = t & 1;
      const int n0 = t * kGateN;
      const bool ok = mbar_wait(&bar[buf], (phases >> buf) & 1u, &g_gate_status, 1);
      phases ^= 1u << buf;
      if (!__syncthreads_and(ok)) break;
      tc_fence_after_sync();
      // MMA t has completed: its centroid buffer takes the tile two steps ahead
      const bool ahead = t + 2 < ntiles;
      if (ahead) stage_km(t + 2);
      constexpr int kCols = kGateN / NQ;        // columns of a tile examined by this thread
      const uint32_t taddr = tmem_base + buf * 128 + qd * kCols + ((uint32_t)((warp & 3) * 32) << 16);
      // 16 scores per step; the next 16 are fetched while these are examined.  A step first marks,
      // without branching, the scores that reach the row's current k-th best (a superset of the
      // scores that enter the list: the threshold is not updated inside the step).  Then every lane
      // works through ITS OWN marked scores, so the (long) insertion code runs max-over-lanes of
      // the marked counts times per step instead of once per position that any lane marked.
      const bool tail = n0 + kGateN > nlim;     // this tile crosses the row's candidate limit
      // A list that is still empty lets every score in.  For the first tile of a row the thread
      // therefore first finds a floor for its k-th best: the maxima of its groups of 4 scores are
      // different candidates, so their k-th largest cannot exceed the k-th largest score (lists of
      // 8 with 16 or 32 groups, lists of 16 with 32 groups).  Only the scores that reach the floor
      // are then looked at one by one, a dozen instead of some forty while a list of 8 fills (the
      // scores are read from TMEM a second time for it).
      float floor_thr = floor_thr_row;
      constexpr int kGroups = kCols / 4;
      constexpr bool kColdFloor = (KMAX == 8 && kGroups == 16) || (KMAX == 16 && kGroups == 32);
      if (kColdFloor && t == 0) {
        float gm[kGroups];
#pragma unroll
        for (int i = 0; i < kCols / 16; ++i) {
          float w[16];
          tmem_ld16(taddr + i * 16, w);
          tmem_ld_wait();
          if (tail) {
            const int left = nlim - (n0 + qd * kCols + i * 16);
#pragma unroll
            for (int j = 0; j < 16; ++j) w[j] = j < left ? w[j] : -CUDART_INF_F;
          }
#pragma unroll
          for (int g4 = 0; g4 < 4; ++g4)
            gm[i * 4 + g4] = fmaxf(fmaxf(fmaxf(w[g4 * 4], w[g4 * 4 + 1]), fmaxf(w[g4 * 4 + 2], w[g4 * 4 + 3])),
                                   -CUDART_INF_F);   // (a group of NaNs counts as -inf: fmaxf drops NaN operands)
        }
        // descending sorting networks on registers: 8 values in 19 compare-exchanges; 16 values as
        // two sorted eights and a bitonic merge
#define FMB_CE(x, i, j) { const float hi_ = fmaxf(x[i], x[j]), lo_ = fminf(x[i], x[j]); x[i] = hi_; x[j] = lo_; }
        auto sort8 = [](float* x) {
          FMB_CE(x, 0, 1) FMB_CE(x, 2, 3) FMB_CE(x, 4, 5) FMB_CE(x, 6, 7)
          FMB_CE(x, 0, 2) FMB_CE(x, 1, 3) FMB_CE(x, 4, 6) FMB_CE(x, 5, 7)
          FMB_CE(x, 1, 2) FMB_CE(x, 5, 6) FMB_CE(x, 0, 4) FMB_CE(x, 3, 7)
          FMB_CE(x, 1, 5) FMB_CE(x, 2, 6)
          FMB_CE(x, 1, 4) FMB_CE(x, 3, 6)
          FMB_CE(x, 2, 4) FMB_CE(x, 3, 5)
          FMB_CE(x, 3, 4)
        };
        auto sort16 = [&](float* x) {
          sort8(x);
          sort8(x + 8);
#pragma unroll
          for (int i = 0; i < 8; ++i) FMB_CE(x, i, 15 - i)
#pragma unroll
          for (int h8 = 0; h8 < 16; h8 += 8) {
#pragma unroll
            for (int i = 0; i < 4; ++i) FMB_CE(x, h8 + i, h8 + i + 4)
#pragma unroll
            for (int i = 0; i < 8; i += 4) { FMB_CE(x, h8 + i, h8 + i + 2) FMB_CE(x, h8 + i + 1, h8 + i + 3) }
#pragma unroll
            for (int i = 0; i < 8; i += 2) FMB_CE(x, h8 + i, h8 + i + 1)
          }
        };
        float kth = CUDART_INF_F;
        if constexpr (KMAX == 8) {
          // 8th largest of the 16 group maxima: both halves sorted, then min over i of max(a[i], b[7 - i]);
          // those eight maxima, sorted, are also what the row's other thread needs
          sort8(gm);
          sort8(gm + 8);
          float c8[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) c8[i] = fmaxf(gm[i], gm[15 - i]);
          if constexpr (NQ == 2) {
            // the 8th largest of the 32 groups of the whole tile is the floor for both threads
            sort8(c8);
#pragma unroll
            for (int i = 0; i < 8; ++i) sX[qd][i][lt] = __float_as_uint(c8[i]);
            bar_sync(1 + (warp & 3), 64);         // warps w and w + 4 hold the same rows
#pragma unroll
            for (int i = 0; i < 8; ++i) kth = fminf(kth, fmaxf(c8[i], __uint_as_float(sX[qd ^ 1][7 - i][lt])));
            bar_sync(1 + (warp & 3), 64);         // both have read before the buffer is written again
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) kth = fminf(kth, c8[i]);
          }
        } else {
          // 16th largest of the 32 group maxima
          sort16(gm);
          sort16(gm + 16);
#pragma unroll
          for (int i = 0; i < 16; ++i) kth = fminf(kth, fmaxf(gm[i], gm[31 - i]));
        }
#undef FMB_CE
        floor_thr = kth;
        floor_thr_row = kth;
      }
      float v[2][16];
      tmem_ld16(taddr, v[0]);
#pragma unroll 1
      for (int i = 0; i < kCols / 16; i += 2) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          tmem_ld_wait();
          if (i + half + 1 < kCols / 16) tmem_ld16(taddr + (i + half + 1) * 16, v[half ^ 1]);
          const int nb = n0 + qd * kCols + (i + half) * 16;
          const float thr = val[KMAX - 1] == kFixed ? CUDART_INF_F : fmaxf(floor_thr, ordered_to_score(val[KMAX - 1]));
          uint32_t m = 0;
#pragma unroll
          for (int j = 0; j < 16; ++j) m |= (v[half][j] >= thr) ? (1u << j) : 0u;
          if (tail) {
            const int left = nlim - nb;           // candidates are n < nlim
            m = left <= 0 ? 0u : (left >= 16 ? m : (m & ((1u << left) - 1u)));
          }
          while (__any_sync(0xffffffffu, m != 0u)) {
            if (m != 0u) {
              const int j = __ffs(m) - 1;
              m &= m - 1u;
              // v[half][j] for a run-time j: a 4-level select tree (the array must stay in registers)
              float a8[8], a4[4];
#pragma unroll
              for (int e = 0; e < 8; ++e) a8[e] = (j & 8) ? v[half][8 + e] : v[half][e];
#pragma unroll
              for (int e = 0; e < 4; ++e) a4[e] = (j & 4) ? a8[4 + e] : a8[e];
              const float a2a = (j & 2) ? a4[2] : a4[0], a2b = (j & 2) ? a4[3] : a4[1];
              const float x = (j & 1) ? a2b : a2a;
              const uint32_t ox = score_to_ordered(x);
              if (x > -CUDART_INF_F && ox >= val[KMAX - 1]) insert(ox, nb + j);
            }
          }
        }
      }
      if (ahead) {             // CTA-uniform
        if (NQ == 2 && KMAX == 8) {   // this thread's list without the slots of a list shorter than KMAX
#pragma unroll
          for (int j = 0; j < 8; ++j) sX[qd][j][lt] = (j + (KMAX - topk) < KMAX) ? val_at(j + (KMAX - topk)) : kEmptyVal;
        }
        cp_async_wait_all();
        fence_async_smem();
        tc_fence_before_sync();
        __syncthreads();       // tile t + 2 staged; every thread has finished reading TMEM buffer buf
        if (tid == 0) {
          tc_fence_after_sync();
          issue(buf);
        }
        if (NQ == 2 && KMAX == 8) {
          // The k-th best of the row so far is at least the k-th largest of the two threads' lists
          // together (both sorted: min over i of max(a[i], b[k - 1 - i])): a floor for the next tiles
          // that roughly halves the scores each thread still has to look at one by one.  (The
          // barrier at the top of the next tile separates these reads from the next writes.)
          uint32_t kth = kFixed;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t mine = (i + (KMAX - topk) < KMAX) ? val_at(i + (KMAX - topk)) : kEmptyVal;
            kth = min(kth, max(mine, sX[qd ^ 1][7 - i][lt]));
          }
          if (kth != kFixed) floor_thr_row = fmaxf(floor_thr_row, ordered_to_score(kth));
        }
      }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, 256);
    if (NQ > 1) {   // merge the row's NQ lists (the centroid buffers are free: every MMA has completed)
      uint64_t* sMerge = reinterpret_cast<uint64_t*>(sKM);
      if (qd > 0) {
#pragma unroll
        for (int j = 0; j < KMAX; ++j) sMerge[((qd - 1) * KMAX + j) * 128 + lt] = ((uint64_t)val[j] << 32) | (uint32_t)idx[j];
      }
      __syncthreads();
      if (qd == 0) {
        for (int e = 0; e < (NQ - 1) * KMAX; ++e) {
          const uint64_t cand = sMerge[e * 128 + lt];
          const uint32_t ox = (uint32_t)(cand >> 32);
          const int n = (int)(uint32_t)cand;
          // blocked and empty slots of the other lists are skipped.  The lists meet in no particular
          // chunk order, so the order is the full one here: score first, then the higher chunk id.
          if (n >= 0 && (ox > val[KMAX - 1] || (ox == val[KMAX - 1] && n > idx[KMAX - 1]))) {
            bool gt[KMAX];
#pragma unroll
            for (int y = 0; y < KMAX; ++y) gt[y] = ox > val[y] || (ox == val[y] && n > idx[y]);
#pragma unroll
            for (int y = KMAX - 1; y > 0; --y) {
              idx[y] = gt[y - 1] ? idx[y - 1] : (gt[y] ? n : idx[y]);
              val[y] = gt[y - 1] ? val[y - 1] : (gt[y] ? ox : val[y]);
            }
            idx[0] = gt[0] ? n : idx[0];
            val[0] = gt[0] ? ox : val[0];
          }
        }
      }
    }
  }
  if (row_ok && qd == 0) {
    const int64_t o = (int64_t)(q0 + r0 + lt) * p.t_rs + (int64_t)h * p.t_hs;
#pragma unroll
    for (int j = 0; j < KMAX; ++j) {
      const int slot = j - (KMAX - topk);
      if (slot >= 0) {
        p.topk_idx[o + slot] = idx[j];
        if (p.topk_val) p.topk_val[o + slot] = val[j] == kFixed ? CUDART_INF_F : ordered_to_score(val[j]);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------
// Two-sweep selection (top-k <= 16, sizes of q and km known): the kernel of the usual shapes.
//
// What bounds gating is the selection on the CUDA cores, not the score product: with a list kept while
// the scores stream by (the kernel above) a thread handled some 33 insertions per row of 512
// candidates, each a divergent loop of 40-odd instructions: 65 instructions per score.  Here the scores are
// looked at twice instead, straight-line both times:
//   sweep 1  only keeps maxima of groups of scores (strided groups: neighbouring chunks may score
//            alike) and, every few tiles, merges them into a sorted list of the K largest by a sorting network.
//            Group maxima are different candidates' scores, so the k-th largest of them is a floor no
//            member of the row's top-k lies under; only some 9 scores of a row (k = 8) reach it;
//   sweep 2  appends the scores that reach the floor to a short queue in shared memory (predicated
//            stores, no branch).  Each of a row's two threads then sorts its own queue: 32-bit keys, the upper 26 bits of the
//            score and the entry's place in the queues, through a network of min / max pairs; the first thread merges the
//            two lists and writes the row's.  Neighbours that agree in those 26 bits are compared exactly and exchanged; where
//            more than two agree, or the last place and what was dropped (masses of equal scores), the pair of warps
//            takes the long way: a candidate's place is the number of the row's candidates ahead of it, counted by comparing
//            all with all (out of line: with that code in the kernel 64K tokens took 495 instead of 471 us, lists of 16 3 % more).
// The score tiles of sweep 2 are those of sweep 1, still in TMEM, for up to 256 candidates; beyond that the
// products are computed again (the tensor pipe is idle otherwise).  A queue that runs full (masses of
// equal scores) is cut down to its k best, the last of which then is the floor.
// Persistent CTAs, two per SM.  Warp 8 loads Q and the centroid tiles by TMA, warp 9 issues the MMAs, both running
// ahead into the next item (row tile, head, sequence) while warps 0-7 (two threads per row, alternate halves of a
// tile's columns) are still in sweep 2: with a CTA per item, start-up and Q's way from HBM were a third of its time.  With one
// thread for loads and MMAs a centroid tile was requested only when the MMAs before it had been issued, one tile in flight at a
// time: 1 us a step, which is what long sequences took (64K tokens, 32 heads 605 / 549 us with one / two warps).
// Measured (B200, d 128; the kernel above / two sweeps, all compared with all / sorted keys): 64K tokens, 32 heads, chunk 128, top-k 8
// 1020 / 605 / 471 us; 8 x 8K tokens 580 / 256 / 178; 32K tokens, 16 heads 185 / 97 / 78; 317K tokens in 16 sequences, chunk 64, top-k 16
// 7400 / 3430 / 2928; 512K tokens, 4 heads, chunk 256, top-k 16 - / 2106 / 1824; d 64, 9K tokens, 12 heads, no mask - / 31 / 22.  All scores
// equal, the long way throughout: 16K tokens, 8 heads 84 / 88 us, top-k 16 198 / 130; no mask 161 / 166 and 440 / 247.  Scores that are smooth from chunk
// to chunk (correlation 0.95): 32K tokens, 16 heads 111 / 92, chunk 64, top-k 16 304 / 300, no mask 512 / 454.
// What bounds it now: instructions at 60 % issue (32K tokens: 1,900 a warp and row tile before, 1,600 with sorted keys; the min / max pipe is busy
// for 58 %), fetching them where lists are of 16, at 64K also the MMAs (128 x 64 x 16: 52 cycles, of which A's and B's way from shared memory takes 48).
// ---------------------------------------------------------------------------------------
constexpr int kSelN = 64;            // centroids per score tile
constexpr int kSelBufs = 4;          // score tiles in TMEM
constexpr int kSelRing = 2;          // centroid tiles in shared memory
constexpr int kSelThreads = 256 + 64;  // selection, loads, MMAs

// descending sorting networks on registers: 8 values in 19 compare-exchanges; 16 as two sorted eights
// and a bitonic merge
__device__ __forceinline__ void sel_ce(float& a, float& b) {
  const float hi = fmaxf(a, b), lo = fminf(a, b);
  a = hi;
  b = lo;
}
__device__ __forceinline__ void sel_ce(uint32_t& a, uint32_t& b) {
  const uint32_t hi = max(a, b), lo = min(a, b);
  a = hi;
  b = lo;
}
template <typename V>
__device__ __forceinline__ void sel_sort8(V* x) {
  sel_ce(x[0], x[1]); sel_ce(x[2], x[3]); sel_ce(x[4], x[5]); sel_ce(x[6], x[7]);
  sel_ce(x[0], x[2]); sel_ce(x[1], x[3]); sel_ce(x[4], x[6]); sel_ce(x[5], x[7]);
  sel_ce(x[1], x[2]); sel_ce(x[5], x[6]); sel_ce(x[0], x[4]); sel_ce(x[3], x[7]);
  sel_ce(x[1], x[5]); sel_ce(x[2], x[6]);
  sel_ce(x[1], x[4]); sel_ce(x[3], x[6]);
  sel_ce(x[2], x[4]); sel_ce(x[3], x[5]);
  sel_ce(x[3], x[4]);
}
// x bitonic -> descending
template <int N, typename V>
__device__ __forceinline__ void sel_bitonic(V* x) {
#pragma unroll
  for (int o = N / 2; o; o >>= 1)
#pragma unroll
    for (int i = 0; i < N; ++i)
      if ((i & o) == 0) sel_ce(x[i], x[i + o]);
}
template <int N, typename V>
__device__ __forceinline__ void sel_sort(V* x) {
  if constexpr (N == 8) {
    sel_sort8(x);
  } else {
    static_assert(N == 16, "8 or 16");
    sel_sort8(x);
    sel_sort8(x + 8);
#pragma unroll
    for (int i = 0; i < 8; ++i) sel_ce(x[i], x[15 - i]);
    sel_bitonic<8>(x);
    sel_bitonic<8>(x + 8);
  }
}

// candidate as one number: descending score, on equal scores the higher chunk id first
__device__ __forceinline__ uint64_t sel_key(float2 c) { return ((uint64_t)score_to_ordered(c.x) << 32) | (uint32_t)__float_as_int(c.y); }

// A thread's queue (entries 64 apart) cut down to its `keep` best, in order.  Rare (see above) and long:
// kept out of line.
__device__ __noinline__ void sel_compact(float2* queue, int cnt, int keep) {
  for (int i = 0; i < keep; ++i) {
    float2 x = queue[i * 64];
    const float2 first = x;
    int best = i;
    uint64_t kb = sel_key(x);
#pragma unroll 4
    for (int j = i + 1; j < cnt; ++j) {
      const float2 y = queue[j * 64];
      const uint64_t kj = sel_key(y);
      if (kj > kb) { kb = kj; best = j; x = y; }
    }
    queue[i * 64] = x;
    queue[best * 64] = first;
  }
}
// The same for lists of 16, of which few have to go: the worst are taken out one by one; returns the score of the worst that stays.  (16K tokens,
// 8 heads, top-k 16, no mask, all scores equal, the best put in order / the worst taken out: 561 / 252 us.  Lists of eight, where more have to go
// than stay, 91 / 104.)
__device__ __noinline__ float sel_cut(float2* queue, int cnt, int keep) {
  for (;; --cnt) {
    int worst = 0;
    float2 w = queue[0];
    uint64_t kw = sel_key(w);
#pragma unroll 4
    for (int j = 1; j < cnt; ++j) {
      const float2 x = queue[j * 64];
      const uint64_t kj = sel_key(x);
      if (kj < kw) { kw = kj; worst = j; w = x; }
    }
    if (cnt <= keep) return w.x;
    queue[worst * 64] = queue[(cnt - 1) * 64];
  }
}

// Four scores, of columns col ... col + 3, for a thread's queue of `cnt` of `cap` entries, for warps in which four more may be too many for
// some thread: one score at a time, queues cut down (as above) whenever one of the warp is full.  Returns entries and floor.  (Cut down inside the
// kernel, as lists of eight are: 317K tokens, lists of 16 3210 us, this way 2946; 512K 1963 / 1850: less code to fetch.)
__device__ __noinline__ float2 sel_append4(float2* queue, int cnt, int cap, int keep, float thr, float4 v, int col) {
  for (int j = 0; j < 4; ++j) {
    if (__any_sync(0xffffffffu, cnt == cap)) {
      if (cnt > keep) {
        thr = fmaxf(thr, sel_cut(queue, cnt, keep));
        cnt = keep;
      }
      __syncwarp();
    }
    if (v.x >= thr) queue[cnt++ * 64] = make_float2(v.x, __int_as_float(col + j));
    v = make_float4(v.y, v.z, v.w, v.x);
  }
  return make_float2(__int_as_float(cnt), thr);
}

// A row's list by exact comparisons of all candidates with all: the place of a candidate is the number of those ahead of it.  The queues of the
// row's two threads start at `queue` and 32 entries behind it, c0 and c - c0 entries; a thread ranks every second candidate from `first` on and
// writes what is among the first `topk`.  By whole warps; rare and long like sel_compact, so that the kernel's own code stays small (inlined: see
// gate_select_kernel).
constexpr int kSelOwn = 8;
__device__ __noinline__ void sel_rank_all(const float2* queue, int c0, int c, int first, int places, int topk, int32_t* out, float* val) {
  const int most = __reduce_max_sync(0xffffffffu, c);
#pragma unroll 1
  for (; first < most; first += 2 * kSelOwn) {
    uint64_t key[kSelOwn];
    int rank[kSelOwn];
#pragma unroll
    for (int m = 0; m < kSelOwn; ++m) {
      const int i = first + 2 * m;
      rank[m] = topk;
      key[m] = ~0ull;
      if (i < c) {
        key[m] = sel_key(queue[i < c0 ? i * 64 : (i - c0) * 64 + 32]);
        rank[m] = places;
      }
    }
    const float2* at = queue;
    for (int i = 0; i < most; ++i) {
      if (i == c0) at = queue + 32;
      const uint64_t k = i < c ? sel_key(*at) : 0ull;
      at += 64;
#pragma unroll
      for (int m = 0; m < kSelOwn; ++m) rank[m] += k > key[m] ? 1 : 0;
    }
#pragma unroll
    for (int m = 0; m < kSelOwn; ++m) {
      if (rank[m] < topk) {
        out[rank[m]] = (int)(uint32_t)key[m];
        if (val) val[rank[m]] = ordered_to_score((uint32_t)(key[m] >> 32));
      }
    }
  }
}

// n / d for 0 <= n < 2^31: one multiplication with a reciprocal from the host, rounded up, which is exact
// for these n (d = 1 is its own case)
struct FastDiv {
  uint32_t mul, shift, d;
};
__device__ __forceinline__ int fast_div(int n, const FastDiv& f) {
  return f.d == 1 ? n : (int)(__umulhi((uint32_t)n, f.mul) >> f.shift);
}

// Queue entries per thread: what two CTAs per SM leave room for.  A row has some 9 (k = 8) or 19 (k = 16)
// candidates, a thread half of them on average; more than 12 or 15 in one thread's queue are rare where scores are independent (with
// room for 16 the queues of k = 8 ran full all the time: 0.82 ms instead of 0.65 at 64K), not where neighbouring chunks score alike or equal.
template <int KMAX> __host__ __device__ constexpr int sel_cap() { return KMAX == 8 ? 20 : 19; }
// Scores between two looks at the queues' lengths, after which no queue has more than CAP - STEP entries, or `need` of them where that is more.  A
// full list of 16 and four scores do not fit: sel_append4.
template <int KMAX> __host__ __device__ constexpr int sel_step() { return KMAX == 8 ? 8 : 4; }

constexpr int kSelSeqs = 64;         // sequences whose bounds are kept in shared memory
constexpr size_t kSelStatic = 1280;  // at least what the kernel declares in static shared memory

template <typename T, int D, int KMAX>
__global__ void __launch_bounds__(kSelThreads, D <= 128 ? 2 : 1)
gate_select_kernel(GateParams p, const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_km,
                   int batch, int row_tiles, FastDiv by_chunk, FastDiv by_tile, FastDiv by_heads) {
  using namespace tc;
  follow_on();
  constexpr uint32_t kQTile = kGateM * D * 2, kKTile = kSelN * D * 2;
  constexpr int CAP = sel_cap<KMAX>();                   // queue entries per thread
  constexpr bool kByEight = KMAX == 8;                   // see mask8
  constexpr int STEP = sel_step<KMAX>();                 // scores between two looks at the queue's length
  constexpr bool kOneByOne = KMAX + STEP > CAP;          // a queue that has been cut has no room for a step's scores
  static_assert(KMAX < CAP && CAP <= 32 && (!kOneByOne || STEP == 4), "a queue that has been cut has room; places have five bits; sel_append4");
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t bar_q, bar_qfree, bar_kfull[kSelRing], bar_kfree[kSelRing], bar_tfull[kSelBufs], bar_tfree[kSelBufs];
  __shared__ uint32_t tmem_base_s;
  __shared__ uint8_t sCount[256];
  __shared__ int sCu[3][kSelSeqs + 1];
  static_assert((2 + 2 * kSelRing + 2 * kSelBufs) * 8 + 4 + sizeof(sCount) + sizeof(sCu) + 64 <= kSelStatic, "see gate_select_launch");
  unsigned char* sQ = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* sKM = sQ + kQTile;
  unsigned char* sQueue = sKM + kSelRing * kKTile;       // per warp pair [CAP][64] (score, chunk); also the pair's exchange area
  uint32_t* sKeys = reinterpret_cast<uint32_t*>(sQueue + CAP * 256 * 8);   // per warp pair [KMAX + 1][32] sorted keys of the rows' second threads

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int topk = p.topk;
  const bool small_batch = batch <= kSelSeqs;
  const bool vec_out = (reinterpret_cast<uintptr_t>(p.topk_idx) & 15) == 0 && (p.t_hs & 3) == 0;
  if (small_batch)
    for (int i = tid; i <= batch; i += kSelThreads) { sCu[0][i] = p.cu_q[i]; sCu[1][i] = p.cu_k[i]; sCu[2][i] = p.cu_km[i]; }
  if (warp == 0) tmem_alloc(&tmem_base_s, kSelBufs * kSelN);
  if (tid == 0) {
    mbar_init(&bar_q, 1);
    mbar_init(&bar_qfree, 1);
    for (int i = 0; i < kSelRing; ++i) { mbar_init(&bar_kfull[i], 1); mbar_init(&bar_kfree[i], 1); }
    for (int i = 0; i < kSelBufs; ++i) { mbar_init(&bar_tfull[i], 1); mbar_init(&bar_tfree[i], 8); }
    mbar_fence_init();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;

  // items: the last row tiles (most candidates under a causal mask) first, all heads and sequences of a
  // row tile before the next, so that the CTAs running at the same time have equally long items
  const int per_tile = p.heads * batch, n_items = row_tiles * per_tile;
  struct Item { int h, r0, q0, rows, shift, km0, nchunks, nt; };
  auto decode = [&](int item, Item& I) -> bool {
    const int x = fast_div(item, by_tile), y = item - x * per_tile, b = fast_div(y, by_heads);
    int len_k, km1;
    I.h = y - b * p.heads;
    I.r0 = (row_tiles - 1 - x) * kGateM;
    if (small_batch) {
      I.q0 = sCu[0][b]; I.rows = sCu[0][b + 1]; len_k = sCu[1][b + 1] - sCu[1][b]; I.km0 = sCu[2][b]; km1 = sCu[2][b + 1];
    } else {
      I.q0 = p.cu_q[b]; I.rows = p.cu_q[b + 1]; len_k = p.cu_k[b + 1] - p.cu_k[b]; I.km0 = p.cu_km[b]; km1 = p.cu_km[b + 1];
    }
    const int len_q = I.rows - I.q0;
    I.rows = min(kGateM, len_q - I.r0);
    if (I.rows <= 0) return false;                       // past the sequence's last row
    I.shift = len_k - len_q;
    I.nchunks = km1 - I.km0;
    int n_end = I.nchunks;                               // candidates of any row of the tile: n < n_end
    if (p.causal) {
      const int pmax = I.r0 + I.rows - 1 + I.shift;
      n_end = pmax < 0 ? 0 : min(I.nchunks, fast_div(pmax, by_chunk));
    }
    I.nt = (n_end + kSelN - 1) / kSelN;
    return true;
  };

  if (warp == 8) {
    // =============================================================== loads
    if (lane == 0) {
      const int group = p.heads / p.heads_k;
      uint32_t gs = 0, qn = 0;                           // steps and items with candidates so far
      bool ok = true;
#pragma unroll 1
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
        Item I;
        if (!decode(item, I) || I.nt == 0) continue;
        const int nt = I.nt, steps = nt <= kSelBufs ? nt : 2 * nt, hk = I.h / group;
        if (qn > 0) ok = mbar_wait(&bar_qfree, (qn - 1) & 1, &g_gate_status, 2);   // the last item's MMAs have read Q
        if (!ok) break;
        mbar_expect_tx(&bar_q, kQTile);
#pragma unroll
        for (int hb = 0; hb < D / 64; ++hb) tma_load_3d(sQ + hb * (kGateM * 128), &map_q, hb * 64, I.h, I.q0 + I.r0, &bar_q);
#pragma unroll 1
        for (int s = 0; s < steps && ok; ++s) {          // centroid tiles, each as soon as its ring slot is free
          const uint32_t n = gs + s, slot = n % kSelRing;
          if (n >= kSelRing) ok = mbar_wait(&bar_kfree[slot], (n / kSelRing - 1) & 1, &g_gate_status, 2);
          if (!ok) break;
          const int row = I.km0 + (s < nt ? s : s - nt) * kSelN;
          mbar_expect_tx(&bar_kfull[slot], kKTile);
#pragma unroll
          for (int hb = 0; hb < D / 64; ++hb)
            tma_load_3d(sKM + slot * kKTile + hb * (kSelN * 128), &map_km, hb * 64, hk, row, &bar_kfull[slot]);
        }
        gs += steps;
        ++qn;
      }
    }
  } else if (warp == 9) {
    // =============================================================== MMAs
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc(FmtOf<T>::v, kGateM, kSelN, 0, 0);
      const uint32_t hi = desc_hi_sw128(1024), q_km = desc_lo_sw128(smem_u32(sQ), 16);
      uint32_t gs = 0, qn = 0;
      bool ok = true;
#pragma unroll 1
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
        Item I;
        if (!decode(item, I) || I.nt == 0) continue;
        const int steps = I.nt <= kSelBufs ? I.nt : 2 * I.nt;
        ok = mbar_wait(&bar_q, qn & 1, &g_gate_status, 2);
#pragma unroll 1
        for (int s = 0; s < steps && ok; ++s) {
          const uint32_t n = gs + s, slot = n % kSelRing, buf = n % kSelBufs;
          ok = mbar_wait(&bar_kfull[slot], (n / kSelRing) & 1, &g_gate_status, 2);
          if (ok && n >= kSelBufs) ok = mbar_wait(&bar_tfree[buf], (n / kSelBufs - 1) & 1, &g_gate_status, 2);
          if (!ok) break;
          tc_fence_after_sync();
          umma_gemm<D / 16>(tmem_base + buf * kSelN, q_km, hi, 2, (kGateM * 128) >> 4,
                            desc_lo_sw128(smem_u32(sKM) + slot * kKTile, 16), hi, 2, (kSelN * 128) >> 4, idesc, 0);
          umma_commit(&bar_tfull[buf]);
          umma_commit(&bar_kfree[slot]);
        }
        umma_commit(&bar_qfree);
        gs += steps;
        ++qn;
      }
      // nobody waits for the last tiles' bar_kfree: their arrivals land before the CTA's shared memory is given up
      if (ok && qn > 0) mbar_wait(&bar_qfree, (qn - 1) & 1, &g_gate_status, 2);
    }
  } else {
    // =============================================================== selection
    const int lt = tid & 127, qd = (tid >> 7) & 1;       // row, and which half of a tile's columns
    const int pair = 1 + (warp & 3);                     // barrier of warps w and w + 4, which hold the same rows
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    unsigned char* mine = sQueue + (warp & 3) * (CAP * 64 * 8);   // the pair's own part of the area
    float2* queue = reinterpret_cast<float2*>(mine) + qd * 32 + lane;
    bool good = true;
    uint32_t gs = 0;
#pragma unroll 1
    for (int item = blockIdx.x; item < n_items && good; item += gridDim.x) {
      Item I;
      if (!decode(item, I)) continue;
      const int nt = I.nt;
      const bool resident = nt <= kSelBufs;              // sweep 2 finds every score tile where sweep 1 left it
      const int pos = I.r0 + lt + I.shift;
      const bool row_ok = lt < I.rows;
      int nlim = I.nchunks;                              // candidate chunks of the row: n < nlim
      const int pos_chunk = pos < 0 ? 0 : fast_div(pos, by_chunk);
      if (p.causal) nlim = min(I.nchunks, pos_chunk);
      if (!row_ok) nlim = 0;
      const bool own = p.causal && row_ok && pos >= 0 && I.nchunks > 0;
      const int need = topk - (own ? 1 : 0);
      const int nlim_warp = __reduce_max_sync(0xffffffffu, nlim), nlim_all = __reduce_min_sync(0xffffffffu, nlim);

      // this thread's 32 scores of score tile s
      auto fetch = [&](uint32_t n, int s, bool wait, bool release, float (&v)[32]) {
        const int buf = n % kSelBufs;
        if (wait && good) good = mbar_wait(&bar_tfull[buf], (n / kSelBufs) & 1, &g_gate_status, 1);
        good = __all_sync(0xffffffffu, good);
        tc_fence_after_sync();
        tmem_ld16(tmem_base + buf * kSelN + qd * 16 + lane_sel, v);          // columns 0-15 and 32-47, or 16-31 and 48-63
        tmem_ld16(tmem_base + buf * kSelN + 32 + qd * 16 + lane_sel, v + 16);
        tmem_ld_wait();
        if (release) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar_tfree[buf]);
        }
        const int left = nlim - (s * kSelN + qd * 16);
        if (!kByEight && __any_sync(0xffffffffu, left < 48)) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = j + (j & 16) < left ? v[j] : -CUDART_INF_F;
        }
      };
      // Columns at or past a row's limit read as -inf.  Lists of eight: eight columns at a time, those past every row of the warp are left
      // out, those before every row's limit need no mask (chunks and row tiles mostly end together, so that one group of an
      // item does).  Lists of 16 mask whole tiles: their code is too long as it is.  Measured, whole tiles / by eight: 8 x 8K tokens x 32 heads
      // 198.8 / 185.7 us, 32K x 16 83.0 / 82.0, d 64, 9K x 12 23.0 / 22.2, 64K x 32 493.8 / 497.6; lists of 16, 317K 3297 / 3396, 512K x 4 1990 / 2064
      auto mask8 = [&](float* v, int first) {
        if (first + 8 > nlim_all) {
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = first + j < nlim ? v[j] : -CUDART_INF_F;
        }
      };
      // ---- sweep 1: the KMAX largest group maxima of this thread's columns
      float top[KMAX];
      {
        float gm[KMAX];
        const int period = max(1, nt / 2);
        int since = 0;
#pragma unroll
        for (int j = 0; j < KMAX; ++j) { top[j] = -CUDART_INF_F; gm[j] = -CUDART_INF_F; }
#pragma unroll 1
        for (int s = 0; s < nt; ++s) {
          float v[32];
          fetch(gs + s, s, true, !resident, v);
          const int nb = s * kSelN + qd * 16;
          if (!kByEight || nb + 48 <= nlim_all) {
#pragma unroll
            for (int j = 0; j < 32; ++j) gm[j % KMAX] = fmaxf(gm[j % KMAX], v[j]);   // (fmaxf drops NaN operands)
          } else {
#pragma unroll
            for (int js = 0; js < 32; js += 8) {
              const int first = nb + js + (js & 16);
              if (first >= nlim_warp) break;             // warp-uniform
              mask8(v + js, first);
#pragma unroll
              for (int j = js; j < js + 8; ++j) gm[j % KMAX] = fmaxf(gm[j % KMAX], v[j]);
            }
          }
          if (++since == period || s + 1 == nt) {
            since = 0;
            sel_sort<KMAX>(gm);
#pragma unroll
            for (int j = 0; j < KMAX; ++j) top[j] = fmaxf(top[j], gm[KMAX - 1 - j]);
            sel_bitonic<KMAX>(top);
#pragma unroll
            for (int j = 0; j < KMAX; ++j) gm[j] = -CUDART_INF_F;
          }
        }
      }
      // floor: the need-th largest of the two threads' lists together (both sorted: min over i of
      // max(a[i], b[need - 1 - i]))
      float thr = CUDART_INF_F;
      {
        float* sX = reinterpret_cast<float*>(mine);
#pragma unroll
        for (int j = 0; j < KMAX; ++j) sX[(qd * KMAX + j) * 32 + lane] = top[j];
        bar_sync(pair, 64);
#pragma unroll
        for (int j = 0; j < KMAX; ++j)
          if (j < need) thr = fminf(thr, fmaxf(top[j], sX[((qd ^ 1) * KMAX + need - 1 - j) * 32 + lane]));
        thr = fmaxf(thr, -3.402823466e38f);              // a score of -inf is no candidate
        bar_sync(pair, 64);                              // both have read before the queue is written
      }

      // ---- sweep 2
      const uint32_t q_first = smem_u32(queue);
      uint32_t q_next = q_first;                         // where the next candidate goes
#pragma unroll 1
      for (int s = 0; s < nt; ++s) {
        float v[32];
        fetch(resident ? gs + s : gs + nt + s, s, !resident, true, v);
        const int nb = s * kSelN + qd * 16;
#pragma unroll
        for (int js = 0; js < 32; js += STEP) {
          if (nb + js + (js & 16) >= nlim_warp) break;   // warp-uniform
          if (kByEight) mask8(v + js, nb + js + (js & 16));
          if (__any_sync(0xffffffffu, q_next > q_first + (CAP - STEP) * 512)) {
            const int cnt = (q_next - q_first) / 512;
            if constexpr (kOneByOne) {
              const float2 x = sel_append4(queue, cnt, CAP, need, thr, make_float4(v[js], v[js + 1], v[js + 2], v[js + 3]), nb + js + (js & 16));
              q_next = q_first + __float_as_int(x.x) * 512;
              thr = x.y;
              continue;
            }
            if (cnt > need) {
              sel_compact(queue, cnt, need);
              q_next = q_first + need * 512;
              if (need > 0) thr = fmaxf(thr, queue[(need - 1) * 64].x);
            }
            __syncwarp();
          }
#pragma unroll
          for (int j = js; j < js + STEP; ++j)
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ge.f32 p, %1, %2;\n\t"
                "@p st.shared.v2.b32 [%0], {%3, %4};\n\t"
                "@p add.u32 %0, %0, 512;\n\t}"
                : "+r"(q_next)
                : "f"(v[j]), "f"(thr), "r"(__float_as_uint(v[j])), "r"(nb + j + (j & 16))
                : "memory");
        }
      }
      gs += resident ? nt : 2 * nt;
      const int cnt = (q_next - q_first) / 512;
      sCount[tid] = (uint8_t)cnt;
      // ---- the list, short way: 32-bit keys of the score's upper bits and the candidate's place in its queue, sorted by each
      // thread for its own queue; the first thread of a row merges the two lists
      uint32_t key[KMAX], dropped = 0;                   // dropped: the largest key that is in no list any more
#pragma unroll
      for (int j = 0; j < KMAX; ++j) {
        const uint32_t k = (score_to_ordered(queue[j * 64].x) & ~63u) | (uint32_t)(qd * 32 + j);
        key[j] = j < cnt ? k : 0u;
      }
      sel_sort<KMAX>(key);
      for (int j = KMAX; __any_sync(0xffffffffu, j < cnt); ++j) {
        const uint32_t k = (score_to_ordered(queue[j * 64].x) & ~63u) | (uint32_t)(qd * 32 + j);
        uint32_t x = j < cnt ? k : 0u;
#pragma unroll
        for (int i = 0; i < KMAX; ++i) sel_ce(key[i], x);
        dropped = max(dropped, x);
      }
      uint32_t* keys = sKeys + (warp & 3) * ((KMAX + 1) * 32) + lane;
      if (qd == 1) {
#pragma unroll
        for (int j = 0; j < KMAX; ++j) keys[j * 32] = key[j];
        keys[KMAX * 32] = dropped;
      }
      bar_sync(pair, 64);                                // both queues are complete, the second thread's list is there
      const int first_place = own ? 1 : 0;
      bool close = false;
      auto candidate = [&](uint32_t k) { return reinterpret_cast<const float2*>(mine) + (k & 31u) * 64 + (k & 32u) + lane; };
      if (qd == 0) {
        uint32_t low = max(dropped, keys[KMAX * 32]);
#pragma unroll
        for (int j = 0; j < KMAX; ++j) {
          const uint32_t o = keys[(KMAX - 1 - j) * 32];
          low = max(low, min(key[j], o));
          key[j] = max(key[j], o);
        }
        sel_bitonic<KMAX>(key);
        // neighbours that may agree in the bits that the keys hold (less one: keys differ, but for the empty ones, which do not count:
        // with them 8 x 8K tokens, top-k 4 / 12 took 177 / 365 us instead of 173 / 351)
        uint32_t gap = ~0u;
#pragma unroll
        for (int j = 0; j + 1 < KMAX; ++j) gap = min(gap, key[j] - key[j + 1] - 1u);
        if (need == KMAX) gap = min(gap, key[KMAX - 1] - low - 1u);
        if (__any_sync(0xffffffffu, gap < 63u)) {
          uint32_t near = 0;
#pragma unroll
          for (int j = 0; j + 1 < KMAX; ++j) near |= key[j] - key[j + 1] < 64u ? 1u << j : 0u;
          const int c = min(KMAX, cnt + (int)sCount[tid ^ 128]);
          near &= (1u << max(c - 1, 0)) - 1u;
          if (low != 0u && key[KMAX - 1] - low < 64u) near |= 1u << (KMAX - 1);
          close = (near & (near >> 1)) != 0 || (need == KMAX && (near >> (KMAX - 1)) != 0);
          // pairs are put right one by one, anything more is left to the long way below
#pragma unroll
          for (int j = 0; j < KMAX; ++j) keys[j * 32] = key[j];
          for (near &= (1u << (KMAX - 1)) - 1u; near != 0 && !close; near &= near - 1) {
            uint32_t* pair_at = keys + (__ffs(near) - 1) * 32;
            const uint32_t x = pair_at[0], y = pair_at[32];
            if (sel_key(*candidate(y)) > sel_key(*candidate(x))) {
              pair_at[0] = y;
              pair_at[32] = x;
            }
          }
#pragma unroll
          for (int j = 0; j < KMAX; ++j) key[j] = keys[j * 32];
        }
        const int64_t row_at = (int64_t)(I.q0 + I.r0 + lt) * p.t_rs + (int64_t)I.h * p.t_hs;
        if (row_ok) {
          int id[KMAX];
#pragma unroll
          for (int j = 0; j < KMAX; ++j) {
            id[j] = key[j] != 0u ? __float_as_int(candidate(key[j])->y) : -1;
          }
          if (topk == KMAX && p.t_rs == KMAX && vec_out) {
            int4* dst = reinterpret_cast<int4*>(p.topk_idx + row_at);
#pragma unroll
            for (int j = 0; j < KMAX; j += 4) {
              int4 x;
              x.x = own ? (j == 0 ? pos_chunk : id[j > 0 ? j - 1 : 0]) : id[j];
              x.y = own ? id[j] : id[j + 1];
              x.z = own ? id[j + 1] : id[j + 2];
              x.w = own ? id[j + 2] : id[j + 3];
              dst[j / 4] = x;
            }
          } else {
            if (own) p.topk_idx[row_at] = pos_chunk;
#pragma unroll
            for (int j = 0; j < KMAX; ++j)
              if (j + first_place < topk) p.topk_idx[row_at + j + first_place] = id[j];
          }
          if (p.topk_val) {
            if (own) p.topk_val[row_at] = CUDART_INF_F;
#pragma unroll
            for (int j = 0; j < KMAX; ++j) {
              if (j + first_place < topk) p.topk_val[row_at + j + first_place] = key[j] != 0u ? candidate(key[j])->x : -CUDART_INF_F;
            }
          }
        }
      }
      if (bar_and(pair, 64, good && !close)) continue;   // the pair goes on, or leaves, together; its areas are free
      good = bar_and(pair, 64, good);
      if (!good) break;
      // ---- the list, long way
      {
        const int other = sCount[tid ^ 128], c = cnt + other;
        const int64_t row_at = (int64_t)(I.q0 + I.r0 + lt) * p.t_rs + (int64_t)I.h * p.t_hs;
        float* val = p.topk_val ? p.topk_val + row_at : nullptr;
        sel_rank_all(reinterpret_cast<const float2*>(mine) + lane, qd == 0 ? cnt : other, c, qd, first_place, topk, p.topk_idx + row_at, val);
        if (qd == 0 && row_ok) {                         // the row's own chunk first, nothing after the last candidate
          if (own) {
            p.topk_idx[row_at] = pos_chunk;
            if (val) val[0] = CUDART_INF_F;
          }
          for (int j = c + first_place; j < topk; ++j) {
            p.topk_idx[row_at + j] = -1;
            if (val) val[j] = -CUDART_INF_F;
          }
        }
      }
      good = bar_and(pair, 64, good);                    // the pair goes on, or leaves, together; its areas are free
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 0) tmem_dealloc(tmem_base, kSelBufs * kSelN);
}

static int g_gate_engine = 1;
void set_gate_engine(int e) { g_gate_engine = e; }
bool gate_tc_supported(int d, int topk) { return (d == 64 || d == 128 || d == 256) && topk <= 32; }

// reads the word (synchronising) and clears it, so that one expired wait is reported once
int read_gate_status(int* out) {
  FMB_CUDA(cudaMemcpyFromSymbol(out, g_gate_status, sizeof(int)));
  if (*out != 0) {
    const int zero = 0;
    FMB_CUDA(cudaMemcpyToSymbol(g_gate_status, &zero, sizeof(int)));
  }
  return FMB_OK;
}

template <typename T, int D, int KMAX, int NQ>
static int gate_tc_launch(const GateParams& p, int batch, int max_q, cudaStream_t s) {
  // 2 CTAs per SM at most (256 TMEM columns each): keep dynamic shared memory above a third of the SM's
  size_t smem = 1024 + (size_t)3 * 128 * D * 2;
  if (smem < 80 * 1024) smem = 80 * 1024;
  static_assert(NQ == 1 || (size_t)(NQ - 1) * KMAX * 128 * 8 <= (size_t)2 * 128 * D * 2, "merge buffer fits the centroid tiles");
  auto kern = gate_topk_tc_kernel<T, D, KMAX, NQ>;
  FMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<dim3(ceil_div(max_q, kGateM), p.heads, batch), 128 * NQ, smem, s>>>(p);
  FMB_LAUNCH_CHECK("gate_topk_tc_kernel");
  return FMB_OK;
}
template <typename T, int D>
static int gate_tc_pick(const GateParams& p, int batch, int max_q, cudaStream_t s) {
  // threads per row (each scans its share of a tile's columns with its own list, merged at the
  // end).  Measured at 64K tokens, top-k 8: 1.77 ms with one, 1.67 ms with two, 2.68 ms with four.
  if (p.topk <= 8) return gate_tc_launch<T, D, 8, 2>(p, batch, max_q, s);
  if (p.topk <= 16) return gate_tc_launch<T, D, 16, 1>(p, batch, max_q, s);
  return gate_tc_launch<T, D, 32, 1>(p, batch, max_q, s);
}

template <typename T, int D, int KMAX>
static int gate_select_launch(const GateParams& p, const CUtensorMap& mq, const CUtensorMap& mk, int batch, int max_q, cudaStream_t s) {
  constexpr int kCap = sel_cap<KMAX>();
  constexpr size_t smem = 1024 + (size_t)kGateM * D * 2 + (size_t)kSelRing * kSelN * D * 2 + (size_t)kCap * 256 * 8 + (size_t)4 * (KMAX + 1) * 32 * 4;
  static_assert(D > 128 || 2 * (smem + kSelStatic + 1024) <= 228 * 1024, "two CTAs per SM, each with 1 KB that the system takes");
  static_assert(2 * KMAX * 32 * 4 <= kCap * 64 * 8, "a pair's exchange area fits its queues");
  auto divider = [](int d) {
    FastDiv fd{0, 0, (uint32_t)d};
    if (d > 1) {                       // 2^(32 + shift) / d rounded up, shift = ceil(log2(d)) - 1
      while ((2u << fd.shift) < fd.d) ++fd.shift;
      fd.mul = (uint32_t)((((uint64_t)1 << (32 + fd.shift)) + fd.d - 1) / fd.d);
    }
    return fd;
  };
  auto kern = gate_select_kernel<T, D, KMAX>;
  FMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int row_tiles = ceil_div(max_q, kGateM);
  const int64_t items = (int64_t)row_tiles * p.heads * batch;
  const int64_t ctas = (int64_t)sm_count() * (D <= 128 ? 2 : 1);
  launch_follow_on(kern, dim3((unsigned)(items < ctas ? items : ctas)), dim3(kSelThreads), smem, s, p, mq, mk, batch, row_tiles,
                   divider(p.chunk), divider(p.heads * batch), divider(p.heads));
  FMB_LAUNCH_CHECK("gate_select_kernel");
  return FMB_OK;
}
// The two-sweep kernel where its tensor maps can be made; *done = false: left to the other kernels
template <typename T>
static int gate_select_try(const GateParams& p, int batch, int max_q, int64_t total_q, int64_t km_rows, cudaStream_t s, bool* done) {
  *done = false;
  if (total_q <= 0 || km_rows <= 0 || p.topk > 16 || p.q_rs <= 0 || p.q_hs <= 0) return FMB_OK;
  if ((int64_t)ceil_div(max_q, kGateM) * p.heads * batch >= (1 << 30)) return FMB_OK;
  CUtensorMap mq, mk;
  const int dt = std::is_same<T, __nv_bfloat16>::value ? FMB_BF16 : FMB_FP16;
  if (make_tmap_3d(&mq, p.q, dt, p.d, p.heads, total_q, (uint64_t)p.q_hs * 2, (uint64_t)p.q_rs * 2, kGateM) != FMB_OK ||
      make_tmap_3d(&mk, p.km, dt, p.d, p.heads_k, km_rows, (uint64_t)p.d * 2, (uint64_t)p.heads_k * p.d * 2, kSelN) != FMB_OK)
    return FMB_OK;
  *done = true;
#define FMB_SEL(D_) \
  return p.topk <= 8 ? gate_select_launch<T, D_, 8>(p, mq, mk, batch, max_q, s) : gate_select_launch<T, D_, 16>(p, mq, mk, batch, max_q, s)
  if (p.d <= 64) FMB_SEL(64);
  if (p.d <= 128) FMB_SEL(128);
  FMB_SEL(256);
#undef FMB_SEL
}

template <typename T>
static int gate_dispatch(const GateParams& p, int batch, int max_q, int64_t total_q, int64_t km_rows, cudaStream_t s) {
  if (g_gate_engine == 1) {
    bool done = false;
    const int rc = gate_select_try<T>(p, batch, max_q, total_q, km_rows, s, &done);
    if (done) return rc;
  }
  const size_t smem = (size_t)kGateDSlab * (kGateM + kGateN) * sizeof(T) +
                      (size_t)kGateM * kGateSStride * sizeof(float) + (size_t)kGateM * p.topk * 8;
  dim3 grid(ceil_div(max_q, kGateM), p.heads, batch);
  if (g_gate_engine == 1 && gate_tc_supported(p.d, p.topk)) {
    if (p.d == 64) return gate_tc_pick<T, 64>(p, batch, max_q, s);
    if (p.d == 128) return gate_tc_pick<T, 128>(p, batch, max_q, s);
    return gate_tc_pick<T, 256>(p, batch, max_q, s);     // one CTA per SM: Q and two centroid tiles are 192 KB
  }
  if (p.topk > 32) {
    auto kern = gate_topk_kernel<T, true>;
    FMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<grid, kGateThreads, smem, s>>>(p);
  } else {
    auto kern = gate_topk_kernel<T, false>;
    FMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<grid, kGateThreads, smem, s>>>(p);
  }
  FMB_LAUNCH_CHECK("gate_topk_kernel");
  return FMB_OK;
}

int launch_gate_topk(const GateArgs& a, cudaStream_t s) {
  if (a.batch == 0 || a.max_q == 0 || a.heads == 0) return FMB_OK;
  GateParams p;
  p.q = a.q; p.q_rs = a.q_rs; p.q_hs = a.q_hs; p.km = a.km;
  p.cu_q = a.cu_q; p.cu_k = a.cu_k; p.cu_km = a.cu_km;
  p.topk_idx = a.topk_idx; p.topk_val = a.topk_val; p.t_rs = a.t_rs; p.t_hs = a.t_hs;
  p.heads = a.heads; p.heads_k = a.heads_k; p.d = a.d; p.topk = a.topk; p.chunk = a.chunk; p.causal = a.causal;
  prof_begin(2, s);
  const int rc = a.dtype == FMB_BF16 ? gate_dispatch<__nv_bfloat16>(p, a.batch, a.max_q, a.total_q, a.km_rows, s)
                                     : gate_dispatch<__half>(p, a.batch, a.max_q, a.total_q, a.km_rows, s);
  prof_end(2, s);
  return rc;
}

}  // namespace fmb
