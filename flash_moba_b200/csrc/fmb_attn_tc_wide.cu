// tcgen05 main kernels of the block-sparse attention for head dim 256 (the host pads 129 ... 255 up to it).
//
// The kernels of fmb_attn_tc.cu keep dK and dV of a 128-key block in the SM's 512 TMEM columns,
// which a head dim of 128 already fills, and their shared-memory tiles assume d <= 128.  Wider heads
// run here (forward: key blocks of 128 keys where the chunk allows, else 64; backward: 64): one CTA per
// work item (key block, head or kv head, sequence), warp-specialised, described at each kernel.  Same workspace
// contract (slots, per-entry partials) and the same merge kernels as the other engines.  Every mbarrier
// wait is bounded (status word of the workspace).
//
// dK and dV are accumulated TRANSPOSED (TMEM lane = head-dim index, two halves of 128; column = key), which takes
// 2 x 128 columns instead of the 2 x 256 of a key-per-lane layout.
// Measured (B200, 16K tokens in three sequences, 16 / 4 heads, chunk 128, top-k 8; the kernels before, in which every
// thread took part in every phase / these): forward 790 / 446 us, backward 1830 / 1120 us.  Of that: gathers that read their
// row numbers ahead of the copies 3 - 5 %; long columns first 5 - 7 %; MMA issue in turns of four instructions, not
// fully unrolled, 17 % of the backward (sixteen unrolled ones took 2850 cycles to issue, in turns 1050).
#include "fmb_attn.cuh"
#include "fmb_tc.cuh"

namespace fmb {

using namespace tc;

namespace {

constexpr int kM = 128;               // gathered rows per tile = TMEM lanes
constexpr int kC = 64;                // keys per block
constexpr float kLog2e = 1.4426950408889634f;

struct WideParams {
  const void *q, *k, *v, *dout;
  int64_t q_rs, q_hs, k_rs, k_hs, v_rs, v_hs, do_rs, do_hs;
  void *dk, *dv; int64_t dk_rs, dk_hs, dv_rs, dv_hs;
  const float *lse, *softmax_d;
  PassParams ps;
  const int32_t *cu_q, *k_begin, *k_end;
  void* part_o; float* part_lse; int* status;
  int heads, heads_k; int64_t total_q;
  float scale; int causal;
  // one CTA per item (key block, head or kv head, sequence); the first `items_heavy` key blocks of every head (under a
  // causal mask the longest columns) come before all others, which follow one head after the other
  int items_x, items_y, items_z, items_heavy;
  int item_heads;                               // forward: q heads per item
};

struct WideItem { int c, sb, y, b; };           // chunk, key block in it, head or kv head of the pass, sequence
__device__ __forceinline__ WideItem wide_item(const WideParams& p) {
  const int yz = p.items_y * p.items_z, heavy = p.items_heavy * yz, item = blockIdx.x;
  int bx, rem;
  if (item < heavy) {
    bx = item / yz;
    rem = item - bx * yz;
  } else {
    const int rest = p.items_x - p.items_heavy;
    rem = (item - heavy) / rest;
    bx = p.items_heavy + (item - heavy - rem * rest);
  }
  return WideItem{bx / p.ps.nsub, bx % p.ps.nsub, rem % p.items_y, rem / p.items_y};
}

// 16 rows of NCHUNK*16 bytes gathered by one warp: lanes 0-15 (and again 16-31) hold the rows' numbers (-1 = zero fill);
// see gather_rows32().  FULL: without tests where all rows are there (backward 1,140 / 1,090 us at 16,389 tokens, 16 / 4 heads; the forward, where
// the code is longer than what it saves, 102 / 107 us at 16,892 tokens, 2 heads)
template <int NCHUNK, bool FULL, typename T>
__device__ __forceinline__ void gather_rows16(int lane, unsigned char* tile, uint32_t block_stride, const T* base, int64_t rs, int row) {
  static_assert(NCHUNK == 32, "a warp copies a row at a time");
  constexpr int GB = 4;                         // copies per turn of the loop
  const uint32_t dst = smem_u32(tile + (lane >> 3) * block_stride);
  const T* src = base + lane * 8;
  if (FULL && __all_sync(0xffffffffu, row >= 0)) {   // every tile but a column's last
#pragma unroll 1
    for (int i0 = 0; i0 < 16; i0 += GB) {
      int o[GB];
#pragma unroll
      for (int i = 0; i < GB; ++i) o[i] = __shfl_sync(0xffffffffu, row, i0 + i);
#pragma unroll
      for (int i = 0; i < GB; ++i) {
        const int r = i0 + i;
        const uint32_t d = dst + r * 128 + ((((uint32_t)lane & 7) ^ (r & 7)) << 4);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + (int64_t)o[i] * rs) : "memory");
      }
    }
    return;
  }
#pragma unroll 1
  for (int i0 = 0; i0 < 16; i0 += GB) {
    int o[GB];
#pragma unroll
    for (int i = 0; i < GB; ++i) o[i] = __shfl_sync(0xffffffffu, row, i0 + i);
#pragma unroll
    for (int i = 0; i < GB; ++i) {
      const int r = i0 + i;
      const uint32_t d = dst + r * 128 + ((((uint32_t)lane & 7) ^ (r & 7)) << 4);
      const bool ok = o[i] >= 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src + (int64_t)(ok ? o[i] : 0) * rs), "r"(ok ? 16u : 0u)
                   : "memory");
    }
  }
}

// ---- forward
// Work item = key block of one (sequence, several q heads of a kv head); one CTA per item, which walks the 128-row tiles
// of the heads' columns; 768 threads, warp-specialised:
//   warps 0-7    compute: two groups of 4 warps take the tiles in turn, a thread per row (TMEM lane): row maximum in one
//                pass over the scores in TMEM, P in a second one.
//   warps 8-11   drain: O / l of the tile from TMEM to the entries' slots, from registers, 32 bytes a store.
//   warp 12      one thread issues every MMA.
//   warps 16-23  loaders: each fetches 16 of a tile's Q rows as soon as S of the tile before has completed.
// S is double-buffered in TMEM, O is not: its two halves of the head dim are computed and drained one after the other.
// K, V, one Q tile and one P tile fill the shared memory at 128 keys.  What bounds it is the chain gather -> S -> P -> P.V with one
// tile of each (the drain's stores a row per lane or a line per four lanes: 454 / 453 us at 16,389 tokens, 16 / 4 heads).
constexpr int kFwDrainWarp = 8, kFwIssuerWarp = 12, kFwLoadWarp = 16, kFwLoaders = 8, kFwThreads = 768;

template <typename T, int C, int D>
__global__ void __launch_bounds__(kFwThreads, 1) fwd_wide_tc_kernel(WideParams p) {
  static_assert(D == 256 && (C == 64 || C == 128), "head dim 256, key blocks of 64 or 128");
  follow_on();
  constexpr int NCH = D / 8;                    // 16-byte chunks of a row
  constexpr uint32_t kKBlock = C * 128;         // bytes between 64-element blocks of the K / V tiles
  constexpr uint32_t kQBlock = kM * 128;        // same for the 128-row Q and P tiles
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ uint64_t bar_fullq, bar_k, bar_v, bar_s[2], bar_pready[2], bar_o[2][2], bar_ofree[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ float sInv[2][kM];                 // 1 / l of the tile's rows, per group

  // with 128-key blocks the tiles and the arrays above fill the 227 KB: no room for alignment padding
  unsigned char* smem = smem_raw;
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(p.status, 0, 9);
    return;
  }
  unsigned char* sK = smem;                     // [C][D]
  unsigned char* sV = sK + C * D * 2;           // [C][D]
  unsigned char* sQ = sV + C * D * 2;           // [128][D]
  unsigned char* sP = sQ + kM * D * 2;          // [128][C]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const WideItem item = wide_item(p);
  const int c = item.c, h0 = p.ps.h0 + item.y * p.item_heads, b = item.b;
  // The item's tiles as one sequence over its heads and the 128-row tiles of each head's column
  struct Tile { int hg, t0, nnz; int64_t off, slot; bool valid; };
  auto seek = [&](Tile& t) {                    // first head >= t.hg with a column; t.t0 = 0
    t.valid = false;
    for (; t.hg < p.item_heads; ++t.hg) {
      const ColRef col = column_of(p.ps, b, h0 + t.hg, c);
      if (col.nnz > 0) { t.nnz = col.nnz; t.off = col.off; t.slot = col.slot; t.t0 = 0; t.valid = true; return; }
    }
  };
  auto first = [&] {
    Tile t{0, 0, 0, 0, 0, false};
    seek(t);
    return t;
  };
  auto advance = [&](Tile& t) {
    t.t0 += kM;
    if (t.t0 >= t.nnz) { ++t.hg; seek(t); }
  };
  uint32_t ntiles = 0;
  for (int hg = 0; hg < p.item_heads; ++hg) ntiles += (uint32_t)((column_of(p.ps, b, h0 + hg, c).nnz + kM - 1) / kM);
  if (ntiles == 0) return;                      // CTA-uniform
  const int64_t plane = (int64_t)item.sb * p.ps.cap;
  const int q0 = p.cu_q[b], len_q = p.cu_q[b + 1] - q0;
  const int k0 = p.k_begin[b], len_k = p.k_end[b] - k0;
  const int key0 = c * p.ps.chunk + item.sb * C;
  const int keys_valid = max(0, min(C, len_k - key0));
  const int hk = h0 / (p.heads / p.heads_k);
  const int shift = len_k - len_q;

  if (warp == 0) tmem_alloc(&tmem_base_s, 512);
  if (tid == 0) {
    mbar_init(&bar_fullq, kFwLoaders);          // one arrival per loader warp
    mbar_init(&bar_k, 8); mbar_init(&bar_v, 8); // one arrival per warp that copies
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_s[i], 1);                  // per group
      mbar_init(&bar_pready[i], 4);
      mbar_init(&bar_o[i][0], 1); mbar_init(&bar_o[i][1], 1);   // per group and half of the head dim
      mbar_init(&bar_ofree[i], 4);              // per half
    }
    mbar_fence_init();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  const uint32_t tO = tmem_base + 256;          // S of group i at columns 128 i
  auto wait_all = [&](uint64_t* bar, uint32_t parity, int where) -> bool {   // the same answer for the whole warp
    return __all_sync(0xffffffffu, mbar_wait(bar, parity & 1u, p.status, where));
  };

  // K is copied by the drain and issuer warpgroups, V by the compute warps, each on its way to its role
  auto stage = [&](unsigned char* tile, const void* src, int64_t rs, int64_t hs, int t, uint64_t* bar) {
    dense_cp_async<T, NCH, C, 256>(t, tile, kKBlock, static_cast<const T*>(src) + (int64_t)(k0 + key0) * rs + (int64_t)hk * hs, rs,
                                   keys_valid);
    cp_async_wait_all();
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
  };
  if (warp < kFwDrainWarp) stage(sV, p.v, p.v_rs, p.v_hs, tid, &bar_v);
  else if (warp < kFwLoadWarp) stage(sK, p.k, p.k_rs, p.k_hs, tid - kFwDrainWarp * 32, &bar_k);

  if (warp >= kFwLoadWarp) {
    // =============================================================== loaders
    const int row0 = (warp - kFwLoadWarp) * 16, i = row0 + (lane & 15);   // this lane's row (lanes in pairs)
    uint32_t g = 0;
    Tile t = first();
    auto entry = [&](const Tile& x) { return x.valid && x.t0 + i < x.nnz ? ldg_s32_here(p.ps.indices + x.off + x.t0 + i) : -1; };
    int raw = entry(t);
#pragma unroll 1
    for (; t.valid; ++g) {
      const int r = (raw < 0 || raw >= len_q) ? -1 : raw;
      const T* qbase = static_cast<const T*>(p.q) + (int64_t)q0 * p.q_rs + (int64_t)(h0 + t.hg) * p.q_hs;
      advance(t);
      raw = entry(t);                           // the next tile's, in flight meanwhile
      if (g > 0 && !wait_all(&bar_s[(g - 1) & 1], (g - 1) >> 1, 5)) break;   // S of the tile before has read the Q tile
      gather_rows16<NCH, false>(lane, sQ + row0 * 128, kQBlock, qbase, p.q_rs, r);
      cp_async_wait_all();
      fence_async_smem();                       // the copies are generic-proxy writes; the MMAs read through the async proxy
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_fullq);
    }
  } else if (warp >= kFwIssuerWarp) {
    // =============================================================== MMA issuer
    if (warp == kFwIssuerWarp && elect_one()) {
      constexpr uint32_t idesc_s = make_idesc(FmtOf<T>::v, kM, C, 0, 0);
      constexpr uint32_t idesc_o = make_idesc(FmtOf<T>::v, kM, 128, 0, 1);
      const uint32_t hi = desc_hi_sw128(1024);
      const uint32_t q_km = desc_lo_sw128(smem_u32(sQ), 16), k_km = desc_lo_sw128(smem_u32(sK), 16);
      const uint32_t v_mn = desc_lo_sw128(smem_u32(sV), kKBlock), p_km = desc_lo_sw128(smem_u32(sP), 16);
      bool ok = mbar_wait(&bar_k, 0, p.status, 6);
#pragma unroll 1
      for (uint32_t g = 0; g <= ntiles && ok; ++g) {
        if (g < ntiles) {                       // S(g); its columns were read before P(g - 2) was ready
          if (!(ok = mbar_wait(&bar_fullq, g & 1, p.status, 6))) break;
          tc_fence_after_sync();
          umma_gemm<D / 16>(tmem_base + (g & 1) * 128, q_km, hi, 2, kQBlock >> 4, k_km, hi, 2, kKBlock >> 4, idesc_s, 0);
          umma_commit(&bar_s[g & 1]);
        }
        if (g == 0) {
          ok = mbar_wait(&bar_v, 0, p.status, 6);
          continue;
        }
        const uint32_t m = g - 1;               // O(m) = P.V per half of the head dim, once O(m - 1) has been read out
        if (!(ok = mbar_wait(&bar_pready[m & 1], (m >> 1) & 1, p.status, 6))) break;
#pragma unroll 1
        for (int hh = 0; hh < 2; ++hh) {
          if (m > 0 && !(ok = mbar_wait(&bar_ofree[hh], (m - 1) & 1, p.status, 6))) break;
          tc_fence_after_sync();
          umma_gemm<C / 16>(tO + hh * 128, p_km, hi, 2, kQBlock >> 4, v_mn + hh * (2 * kKBlock >> 4), hi, 128, 512, idesc_o, 0);
          umma_commit(&bar_o[m & 1][hh]);
        }
      }
    }
  } else if (warp >= kFwDrainWarp) {
    // =============================================================== drain warps
    const uint32_t at = (uint32_t)((warp & 3) * 32) << 16;
    T* part_o = static_cast<T*>(p.part_o);
    bool good = true;
    uint32_t g = 0;
#pragma unroll 1
    for (Tile t = first(); t.valid && good; advance(t), ++g) {
      const int row = (warp & 3) * 32 + (lane >> 2), left = t.nnz - t.t0 - row;
      T* dst = part_o + (plane + t.slot + t.t0 + row) * D + (lane & 3) * 16;
      if (!(good = wait_all(&bar_pready[g & 1], g >> 1, 4))) break;   // (for 1 / l)
      float inv[4];                    // (at once: the group's next tile but one replaces them)
#pragma unroll
      for (int i = 0; i < 4; ++i) inv[i] = sInv[g & 1][row + i * 8];
      // ---- normalised partial O, halves of the head dim, 16 rows of the warp at a time: a thread has a quarter of a line of
      // two rows (part_col)
#pragma unroll 1
      for (int hh = 0; hh < 2; ++hh) {
        if (!(good = wait_all(&bar_o[g & 1][hh], g >> 1, 4))) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (int r16 = 0; r16 < 32; r16 += 16) {
          const float ia = r16 ? inv[2] : inv[0], ib = r16 ? inv[3] : inv[1];
#pragma unroll 1
          for (int c = hh * 128; c < hh * 128 + 128; c += 64) {
            float o[32];
            tmem_ld_16x64(tO + at + ((uint32_t)r16 << 16) + c, o);
            tmem_ld_wait();
            if (r16 == 16 && (c & 64)) {
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&bar_ofree[hh]);
            }
            if (left > r16) store_part<T>(dst + r16 * D + c, o, ia);
            if (left > r16 + 8) store_part<T>(dst + (r16 + 8) * D + c, o + 2, ib);
          }
        }
      }
    }
  } else {
    // =============================================================== compute groups
    const int grp = warp >> 2, lt = tid & (kM - 1);
    const uint32_t tS = tmem_base + grp * 128 + ((uint32_t)((warp & 3) * 32) << 16);
    const float scale_log2 = p.scale * kLog2e;
    uint32_t g = 0;
    Tile t = first();
    if (grp == 1 && t.valid) { advance(t); ++g; }
    auto entry = [&](const Tile& x) { return x.valid && x.t0 + lt < x.nnz ? ldg_s32_here(p.ps.indices + x.off + x.t0 + lt) : -1; };
    int raw = entry(t);
#pragma unroll 1
    for (; t.valid; g += 2) {
      const int lim = (raw < 0 || raw >= len_q) ? 0 : (p.causal ? min(keys_valid, raw + shift - key0 + 1) : keys_valid);
      const bool mine = lt < t.nnz - t.t0;
      const int64_t slot = plane + t.slot + t.t0 + lt;
      advance(t);
      if (t.valid) advance(t);
      raw = entry(t);                           // the group's next tile's, in flight meanwhile
      if (!wait_all(&bar_s[grp], g >> 1, 1)) break;
      tc_fence_after_sync();
      // ---- chunk-local softmax of row `lt`
      float mx = -CUDART_INF_F;
#pragma unroll 1
      for (int q4 = 0; q4 < C / 32; ++q4) {
        float s[32];
        tmem_ld32(tS + q4 * 32, s);
        tmem_ld_wait();
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) mx = fmaxf(mx, q4 * 32 + jj < lim ? s[jj] : -CUDART_INF_F);
      }
      const float mref = lim > 0 ? mx * scale_log2 : 0.f;
      // P.V of the tile before (the other group's) has read the P tile
      if (g > 0 && !wait_all(&bar_o[grp ^ 1][1], (g - 1) >> 1, 1)) break;
      float sum = 0.f;
#pragma unroll 1
      for (int q4 = 0; q4 < C / 32; ++q4) {
        float s[32];
        tmem_ld32(tS + q4 * 32, s);
        tmem_ld_wait();
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) {
          const float e = exp2f(s[jj] * scale_log2 - mref);
          s[jj] = q4 * 32 + jj < lim ? e : 0.f;
          sum += s[jj];
        }
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
          *reinterpret_cast<uint4*>(sP + sw128_offset(lt, q4 * 4 + jj, kQBlock)) = pack8<T>(s + jj * 8);
      }
      sInv[grp][lt] = sum > 0.f ? 1.f / sum : 0.f;
      if (mine) p.part_lse[slot] = sum > 0.f ? mx * p.scale + logf(sum) : -CUDART_INF_F;
      fence_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_pready[grp]);   // S has been read, P is in shared memory
    }
  }
  cp_async_wait_all();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
}

// ---- backward
// Work item = key block of 64 keys of one (sequence, kv head); one CTA per item; 768 threads, warp-specialised:
//   warps 0-7    compute: TMEM lane = gathered row, warps w and w + 4 split the keys in halves.  P and dS of a tile; at
//                the end the item's dK and dV.
//   warps 8-11   drain: the tile's two dQ halves from TMEM to the entries' slots, from registers, 32 bytes a store.
//   warp 12      one thread issues every MMA.
//   warps 16-23  loaders: each fetches 16 of a tile's Q rows and 16 of its dO rows.
// Q and dO of one tile, K, V, P and dS fill the shared memory, so a tile's rows can only be fetched once the GEMMs that
// read the tile before have completed: dK^T += Q^T.dS is issued first (Q is what the next tile starts with), dV^T += dO^T.P
// behind it, then dQ, whose two halves share 128 TMEM columns: the second is issued behind the next tile's dP.
// What bounds it is that cycle: gather of Q, S, P (dP beside it), dS, dK.
// Q's copies and dO's arrive on their own, and the issuing thread tests its barriers (16,389 tokens, 16 / 4 heads, us: Q announced behind dO's issue,
// waits / this 1,150 / 1,090; with an elected thread 1,120).
constexpr int kBwDrainWarp = 8, kBwIssuerWarp = 12, kBwLoadWarp = 16, kBwLoaders = 8, kBwThreads = 768;
// registers per thread: launched with 80 (65536 / 768 rounded down to a multiple of 8)
constexpr int kBwRegsLaunch = 80, kBwRegsCompute = 112, kBwRegsOther = 64;
static_assert(2 * (kBwRegsCompute - kBwRegsLaunch) <= 4 * (kBwRegsLaunch - kBwRegsOther), "registers requested <= registers released");

template <typename T, int D>
__global__ void __launch_bounds__(kBwThreads, 1) bwd_wide_tc_kernel(WideParams p) {
  static_assert(D == 256, "two head-dim halves of 128 TMEM lanes");
  follow_on();
  constexpr int NCH = D / 8;
  constexpr uint32_t kKBlock = kC * 128;
  constexpr uint32_t kQBlock = kM * 128;
  constexpr uint32_t kQTile = kM * D * 2;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ uint64_t bar_fullq, bar_fulldo, bar_s, bar_p, bar_ds, bar_dk, bar_dv, bar_dq[2], bar_dqfree, bar_fin;
  __shared__ uint32_t tmem_base_s;
  __shared__ int sRow[kM];                      // query rows of the tile
  __shared__ float sLse[kM], sDsum[kM];         // their log-sum-exps and dO.O sums

  // the tiles fill the 227 KB together with the static arrays above: no room for alignment padding
  unsigned char* smem = smem_raw;
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(p.status, 0, 9);
    return;
  }
  unsigned char* sK = smem;                     // [64][D]
  unsigned char* sV = sK + kC * D * 2;          // [64][D]
  unsigned char* sQ = sV + kC * D * 2;          // [128][D]
  unsigned char* sdO = sQ + kQTile;             // [128][D]
  unsigned char* sP = sdO + kQTile;             // [128][64]
  unsigned char* sdS = sP + kM * kC * 2;        // [128][64]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int group = p.heads / p.heads_k;
  const WideItem item = wide_item(p);
  const int c = item.c, sb = item.sb, hk = p.ps.h0 / group + item.y, b = item.b;
  const int64_t plane = (int64_t)sb * p.ps.cap;
  const int q0 = p.cu_q[b], len_q = p.cu_q[b + 1] - q0;
  const int k0 = p.k_begin[b], len_k = p.k_end[b] - k0;
  const int key0 = c * p.ps.chunk + sb * kC;
  T* part_dq = static_cast<T*>(p.part_o);
  if (key0 >= len_k) {                          // CTA-uniform: the key block starts past the sequence's last key
    zero_dq_partials<T>(p.ps, part_dq, plane, b, hk, group, c, D);
    return;
  }
  const int keys_valid = min(kC, len_k - key0);
  const int shift = len_k - len_q;

  if (warp == 0) tmem_alloc(&tmem_base_s, 512);
  if (tid == 0) {
    mbar_init(&bar_fullq, kBwLoaders * 33); mbar_init(&bar_fulldo, kBwLoaders * 32);   // one arrival per thread of the loader warps, and one per warp
    mbar_init(&bar_s, 1); mbar_init(&bar_p, 1); mbar_init(&bar_dk, 1); mbar_init(&bar_dv, 1);
    mbar_init(&bar_dq[0], 1); mbar_init(&bar_dq[1], 1); mbar_init(&bar_fin, 1);
    mbar_init(&bar_ds, 8);                      // one arrival per compute warp
    mbar_init(&bar_dqfree, 4);                  // one arrival per drain warp
    mbar_fence_init();
  }
  if (tid < 512) {
    const T* kbase = static_cast<const T*>(p.k) + (int64_t)(k0 + key0) * p.k_rs + (int64_t)hk * p.k_hs;
    const T* vbase = static_cast<const T*>(p.v) + (int64_t)(k0 + key0) * p.v_rs + (int64_t)hk * p.v_hs;
    dense_cp_async<T, NCH, kC, 512>(tid, sK, kKBlock, kbase, p.k_rs, keys_valid);
    dense_cp_async<T, NCH, kC, 512>(tid, sV, kKBlock, vbase, p.v_rs, keys_valid);
    cp_async_wait_all();
    fence_async_smem();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_s;
  const uint32_t tS = tmem_base, tdP = tmem_base + 64, tdQ = tmem_base + 128;
  const uint32_t tdK = tmem_base + 256, tdV = tmem_base + 384;                // [half][64 keys]

  // The item's tiles as one sequence over the q heads of the group and the 128-row tiles of each head's column
  struct Tile { int hg, t0, nnz; int64_t off, slot; bool valid; };
  auto seek = [&](Tile& t) {                    // first head >= t.hg with a column; t.t0 = 0
    t.valid = false;
    for (; t.hg < group; ++t.hg) {
      const ColRef col = column_of(p.ps, b, hk * group + t.hg, c);
      if (col.nnz > 0) { t.nnz = col.nnz; t.off = col.off; t.slot = col.slot; t.t0 = 0; t.valid = true; return; }
    }
  };
  auto first = [&] {
    Tile t{0, 0, 0, 0, 0, false};
    seek(t);
    return t;
  };
  auto advance = [&](Tile& t) {
    t.t0 += kM;
    if (t.t0 >= t.nnz) { ++t.hg; seek(t); }
  };
  auto count = [&] {                            // tiles of the item
    int n = 0;
    for (int hg = 0; hg < group; ++hg) n += (column_of(p.ps, b, hk * group + hg, c).nnz + kM - 1) / kM;
    return n;
  };
  auto wait_all = [&](uint64_t* bar, uint32_t parity, int where) -> bool {   // the same answer for the whole warp
    return __all_sync(0xffffffffu, mbar_wait(bar, parity & 1u, p.status, where));
  };

  if (warp >= kBwLoadWarp) {
    // =============================================================== loaders
    reg_dec<kBwRegsOther>();
    const int row0 = (warp - kBwLoadWarp) * 16, i = row0 + (lane & 15);   // this lane's row (lanes in pairs)
    uint32_t g = 0;
    Tile t = first();
    auto entry = [&](const Tile& x) { return x.valid && x.t0 + i < x.nnz ? ldg_s32_here(p.ps.indices + x.off + x.t0 + i) : -1; };
    int raw = entry(t);
#pragma unroll 1
    for (; t.valid; ++g) {
      const int r = (raw < 0 || raw >= len_q) ? -1 : raw, h = hk * group + t.hg;
      const T* qbase = static_cast<const T*>(p.q) + (int64_t)q0 * p.q_rs + (int64_t)h * p.q_hs;
      const T* obase = static_cast<const T*>(p.dout) + (int64_t)q0 * p.do_rs + (int64_t)h * p.do_hs;
      float l = CUDART_INF_F, dd = 0.f;
      if (r >= 0) {
        const int64_t at = (int64_t)h * p.total_q + q0 + r;
        l = p.lse[at];
        dd = p.softmax_d[at];
      }
      advance(t);
      raw = entry(t);                           // the next tile's, in flight meanwhile
      // dK of the tile before has read the Q tile (and, before that, the compute warps the row data)
      if (g > 0 && !wait_all(&bar_dk, g - 1, 5)) break;
      if (lane < 16) { sRow[i] = r; sLse[i] = l; sDsum[i] = dd; }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_fullq);             // (for the row data)
      gather_rows16<NCH, true>(lane, sQ + row0 * 128, kQBlock, qbase, p.q_rs, r);
      cp_async_arrive(&bar_fullq);                        // Q does not wait for dO
      if (g > 0 && !wait_all(&bar_dv, g - 1, 5)) break;   // dV has read the dO tile
      gather_rows16<NCH, true>(lane, sdO + row0 * 128, kQBlock, obase, p.do_rs, r);
      cp_async_arrive(&bar_fulldo);
    }
    cp_async_wait_all();
  } else if (warp >= kBwIssuerWarp) {
    // =============================================================== MMA issuer
    reg_dec<kBwRegsOther>();
    if (warp == kBwIssuerWarp && lane == 0) {
      constexpr uint32_t idesc_s = make_idesc(FmtOf<T>::v, kM, kC, 0, 0);         // rows x keys
      constexpr uint32_t idesc_t = make_idesc(FmtOf<T>::v, 128, kC, 1, 1);        // head-dim half x keys, both M/N-major
      constexpr uint32_t idesc_dq = make_idesc(FmtOf<T>::v, kM, 128, 0, 1);       // rows x head-dim half
      const uint32_t hi = desc_hi_sw128(1024);
      const uint32_t k_km = desc_lo_sw128(smem_u32(sK), 16), v_km = desc_lo_sw128(smem_u32(sV), 16);
      const uint32_t k_mn = desc_lo_sw128(smem_u32(sK), kKBlock);
      const uint32_t q_km = desc_lo_sw128(smem_u32(sQ), 16), do_km = desc_lo_sw128(smem_u32(sdO), 16);
      const uint32_t q_mn = desc_lo_sw128(smem_u32(sQ), kQBlock), do_mn = desc_lo_sw128(smem_u32(sdO), kQBlock);
      const uint32_t ds_km = desc_lo_sw128(smem_u32(sdS), 16);
      const uint32_t p_mn = desc_lo_sw128(smem_u32(sP), kQBlock), ds_mn = desc_lo_sw128(smem_u32(sdS), kQBlock);
      const uint32_t ntiles = (uint32_t)count();
      bool ok = true;
      // the second dQ half of tile g, once the first has been read out
      auto dq_second = [&] {
        if (!mbar_spin(&bar_dqfree, 0, p.status, 6)) return false;   // phase 2 g: the first half of tile g
        tc_fence_after_sync();
        umma_gemm<kC / 16>(tdQ, ds_km, hi, 2, 0, k_mn + (2 * kKBlock >> 4), hi, 128, 512, idesc_dq, 0);
        umma_commit(&bar_dq[1]);
        return true;
      };
#pragma unroll 1
      for (uint32_t g = 0; g <= ntiles && ok; ++g) {
        if (g < ntiles) {
          // S(g) and dP(g): their columns were read before dS(g - 1) was ready
          if (!(ok = mbar_spin(&bar_fullq, g & 1, p.status, 6))) break;
          fence_async_smem();                   // the gathers are generic-proxy writes; the MMAs read through the async proxy
          tc_fence_after_sync();
          umma_gemm<D / 16>(tS, q_km, hi, 2, kQBlock >> 4, k_km, hi, 2, kKBlock >> 4, idesc_s, 0);
          umma_commit(&bar_s);
          if (!(ok = mbar_spin(&bar_fulldo, g & 1, p.status, 6))) break;
          fence_async_smem();
          tc_fence_after_sync();
          umma_gemm<D / 16>(tdP, do_km, hi, 2, kQBlock >> 4, v_km, hi, 2, kKBlock >> 4, idesc_s, 0);
          umma_commit(&bar_p);
        }
        if (g > 0 && !(ok = dq_second())) break;
        if (g == ntiles) break;
        if (!(ok = mbar_spin(&bar_ds, g & 1, p.status, 6))) break;
        tc_fence_after_sync();
        const uint32_t acc = g > 0 ? 1u : 0u;   // the item's first tile starts the accumulators
        // dK^T[half] += Q^T.dS, dV^T[half] += dO^T.P : M = 128 head-dim columns, N = keys, K = the rows
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
          umma_gemm<kM / 16>(tdK + hh * 64, q_mn + hh * (2 * kQBlock >> 4), hi, 128, 512, ds_mn, hi, 128, 512, idesc_t, acc);
        umma_commit(&bar_dk);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
          umma_gemm<kM / 16>(tdV + hh * 64, do_mn + hh * (2 * kQBlock >> 4), hi, 128, 512, p_mn, hi, 128, 512, idesc_t, acc);
        umma_commit(&bar_dv);
        // first half of dQ = dS.K, once the second half of the tile before has been read out (phase 2 g - 1 of bar_dqfree)
        if (g > 0 && !(ok = mbar_spin(&bar_dqfree, 1, p.status, 6))) break;
        tc_fence_after_sync();
        umma_gemm<kC / 16>(tdQ, ds_km, hi, 2, 0, k_mn, hi, 128, 512, idesc_dq, 0);
        umma_commit(&bar_dq[0]);
      }
      if (ok) umma_commit(&bar_fin);
    }
  } else if (warp >= kBwDrainWarp) {
    // =============================================================== drain warps
    reg_dec<kBwRegsOther>();
    const uint32_t at = (uint32_t)((warp & 3) * 32) << 16;
    bool good = true;
    uint32_t g = 0;
#pragma unroll 1
    for (Tile t = first(); t.valid && good; advance(t), ++g) {
      const int row = (warp & 3) * 32 + (lane >> 2), left = t.nnz - t.t0 - row;
      T* dst = part_dq + (plane + t.slot + t.t0 + row) * D + (lane & 3) * 16;
      // ---- dQ partial: scaled, rounded, halves of the head dim, 16 rows of the warp at a time: a thread has a quarter of a
      // line of two rows (part_col)
#pragma unroll 1
      for (int hh = 0; hh < 2; ++hh) {
        if (!(good = wait_all(&bar_dq[hh], g, 4))) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (int r16 = 0; r16 < 32; r16 += 16) {
#pragma unroll 1
          for (int c = 0; c < 128; c += 64) {
            float o[32];
            tmem_ld_16x64(tdQ + at + ((uint32_t)r16 << 16) + c, o);
            tmem_ld_wait();
            if (r16 == 16 && c == 64) {
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&bar_dqfree);
            }
            if (left > r16) store_part<T>(dst + r16 * D + hh * 128 + c, o, p.scale);
            if (left > r16 + 8) store_part<T>(dst + (r16 + 8) * D + hh * 128 + c, o + 2, p.scale);
          }
        }
      }
    }
  } else {
    // =============================================================== compute warps
    reg_inc<kBwRegsCompute>();
    const int lt = tid & (kM - 1), hf = tid >> 7;
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    const float scale_log2 = p.scale * kLog2e;
    const uint32_t ntiles = (uint32_t)count();
    bool good = true;
#pragma unroll 1
    for (uint32_t g = 0; g < ntiles; ++g) {
      // ---- P of row `lt`, this thread's 32 keys (Q's barrier: for the row data)
      if (!(good = wait_all(&bar_fullq, g, 3) && wait_all(&bar_s, g, 3))) break;
      tc_fence_after_sync();
      const int r = sRow[lt];
      const float lse2 = sLse[lt] * kLog2e, dd = sDsum[lt];
      const int lim = (r < 0 ? 0 : (p.causal ? min(keys_valid, r + shift - key0 + 1) : keys_valid)) - hf * 32;
      float pr[32], dp[32];
      tmem_ld32(tS + lane_sel + hf * 32, pr);
      tmem_ld_wait();
#pragma unroll
      for (int jj = 0; jj < 32; ++jj) pr[jj] = jj < lim ? exp2f(pr[jj] * scale_log2 - lse2) : 0.f;
      if (g > 0 && !(good = wait_all(&bar_dv, g - 1, 3))) break;    // dV of the tile before has read P
#pragma unroll
      for (int jj = 0; jj < 4; ++jj)
        *reinterpret_cast<uint4*>(sP + sw128_offset(lt, hf * 4 + jj, kQBlock)) = pack8<T>(pr + jj * 8);
      // ---- dS
      if (!(good = wait_all(&bar_p, g, 3))) break;
      tc_fence_after_sync();
      tmem_ld32(tdP + lane_sel + hf * 32, dp);
      tmem_ld_wait();
      tc_fence_before_sync();
#pragma unroll
      for (int jj = 0; jj < 32; ++jj) dp[jj] = pr[jj] * (dp[jj] - dd);
      if (g > 0 && !(good = wait_all(&bar_dq[1], g - 1, 3))) break;   // dQ of the tile before has read dS
#pragma unroll
      for (int jj = 0; jj < 4; ++jj)
        *reinterpret_cast<uint4*>(sdS + sw128_offset(lt, hf * 4 + jj, kQBlock)) = pack8<T>(dp + jj * 8);
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_ds);      // S, dP and the row data have been read, P and dS are in shared memory
    }
    // ---- dK (scaled) and dV of this key block: TMEM lane = head-dim index of this thread's half,
    // column = key; consecutive lanes write consecutive elements of a key's row
    if (good) good = wait_all(&bar_fin, 0, 4);
    if (good) {
      tc_fence_after_sync();
      T* dkp = static_cast<T*>(p.dk) + (int64_t)(k0 + key0) * p.dk_rs + (int64_t)hk * p.dk_hs + hf * 128 + lt;
      T* dvp = static_cast<T*>(p.dv) + (int64_t)(k0 + key0) * p.dv_rs + (int64_t)hk * p.dv_hs + hf * 128 + lt;
#pragma unroll 1
      for (int i2 = 0; i2 < 2; ++i2) {
        float a[32], bq[32];
        if (ntiles > 0) {
          tmem_ld32(tdK + hf * 64 + lane_sel + i2 * 32, a);
          tmem_ld32(tdV + hf * 64 + lane_sel + i2 * 32, bq);
          tmem_ld_wait();
        } else {                                 // no tile at all: the gradients of these keys are zero
#pragma unroll
          for (int jj = 0; jj < 32; ++jj) { a[jj] = 0.f; bq[jj] = 0.f; }
        }
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) {
          const int kk = i2 * 32 + jj;
          if (kk < keys_valid) {
            dkp[(int64_t)kk * p.dk_rs] = Elem<T>::from_f(a[jj] * p.scale);
            dvp[(int64_t)kk * p.dv_rs] = Elem<T>::from_f(bq[jj]);
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
}

WideParams make_wide_params(const AttnArgs& a, const AttnWorkspace& w, const PassParams& ps, int nchunk, int items_y) {
  WideParams p;
  p.q = a.q; p.k = a.k; p.v = a.v; p.dout = a.dout;
  p.q_rs = a.q_rs; p.q_hs = a.q_hs; p.k_rs = a.k_rs; p.k_hs = a.k_hs; p.v_rs = a.v_rs; p.v_hs = a.v_hs;
  p.do_rs = a.do_rs; p.do_hs = a.do_hs;
  p.dk = a.dk; p.dv = a.dv; p.dk_rs = a.dk_rs; p.dk_hs = a.dk_hs; p.dv_rs = a.dv_rs; p.dv_hs = a.dv_hs;
  p.lse = a.lse; p.softmax_d = a.softmax_d;
  p.ps = ps;
  p.cu_q = a.cu_q; p.k_begin = a.k_begin; p.k_end = a.k_end;
  p.part_o = w.part_o; p.part_lse = w.part_lse; p.status = w.status;
  p.heads = a.heads; p.heads_k = a.heads_k; p.total_q = a.total_q;
  p.scale = a.scale; p.causal = a.causal;
  p.items_x = nchunk * ps.nsub; p.items_y = items_y; p.items_z = a.batch;
  p.items_heavy = a.causal ? min(p.items_x, 16 * ps.nsub) : 0;
  return p;
}

template <typename T, int C, int D>
int fwd_wide_launch(const AttnArgs& a, const AttnWorkspace& w, const PassParams& ps, cudaStream_t s) {
  WideParams p = make_wide_params(a, w, ps, a.ncol, ps.nh);
  // q heads per item: a divisor of the kv head's group.  More of them share the staging of K and V and the start of
  // the pipeline, but a small problem needs its items to fill the SMs evenly.
  const int group = a.heads / a.heads_k;
  const int64_t cols = (int64_t)p.items_x * ps.nh * a.batch;
  for (p.item_heads = group; p.item_heads > 1; --p.item_heads)
    if (group % p.item_heads == 0 && cols >= (int64_t)p.item_heads * 8 * sm_count()) break;
  p.items_y = ps.nh / p.item_heads;
  const size_t smem = (size_t)2 * C * D * 2 + (size_t)kM * D * 2 + (size_t)kM * C * 2;   // K, V, Q, P
  auto kern = fwd_wide_tc_kernel<T, C, D>;
  FMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_follow_on(kern, dim3(p.items_x * p.items_y * p.items_z), dim3(kFwThreads), smem, s, p);
  FMB_LAUNCH_CHECK("fwd_wide_tc_kernel");
  return FMB_OK;
}

template <typename T, int D>
int bwd_wide_launch(const AttnArgs& a, const AttnWorkspace& w, const PassParams& ps, cudaStream_t s) {
  const WideParams p = make_wide_params(a, w, ps, max(a.ncol, ceil_div(a.max_k, a.chunk)), ps.nh / (a.heads / a.heads_k));
  // K, V, Q, dO, P, dS: with d = 256 that and the kernel's static arrays are the 227 KB a CTA may have
  const size_t smem = (size_t)2 * kC * D * 2 + (size_t)2 * kM * D * 2 + (size_t)2 * kM * kC * 2;
  auto kern = bwd_wide_tc_kernel<T, D>;
  // the hand-over of registers inside the kernel counts on the launch's share per thread
  static const int regs = [kern] {
    cudaFuncAttributes at;
    return cudaFuncGetAttributes(&at, kern) == cudaSuccess ? at.numRegs : 0;
  }();
  if (regs != kBwRegsLaunch)
    return fail(FMB_ERR_CUDA, "wide-head backward: built with %d registers per thread (%d expected)", regs, kBwRegsLaunch);
  FMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch_follow_on(kern, dim3(p.items_x * p.items_y * p.items_z), dim3(kBwThreads), smem, s, p);
  FMB_LAUNCH_CHECK("bwd_wide_tc_kernel");
  return FMB_OK;
}

}  // namespace

bool tc_wide_supported(const AttnArgs& a, bool backward) {
  if (a.chunk % 64 != 0) return false;
  return a.d == 256;
}

int launch_bwd_main_tc_wide(const AttnArgs& a, const AttnWorkspace& w, const PassParams& ps, cudaStream_t s) {
  if (a.batch == 0 || a.heads == 0) return FMB_OK;
  if (w.kb != kC) return fail(FMB_ERR_UNSUPPORTED, "wide-head backward: key block %d (64 expected)", w.kb);
  if (a.d == 256)
    return a.dtype == FMB_BF16 ? bwd_wide_launch<__nv_bfloat16, 256>(a, w, ps, s) : bwd_wide_launch<__half, 256>(a, w, ps, s);
  return fail(FMB_ERR_UNSUPPORTED, "wide-head backward: head_dim %d not built", a.d);
}

int launch_fwd_main_tc_wide(const AttnArgs& a, const AttnWorkspace& w, const PassParams& ps, cudaStream_t s) {
  if (a.ncol == 0 || a.batch == 0 || a.heads == 0) return FMB_OK;
  if (a.d == 256 && w.kb == 128)
    return a.dtype == FMB_BF16 ? fwd_wide_launch<__nv_bfloat16, 128, 256>(a, w, ps, s)
                               : fwd_wide_launch<__half, 128, 256>(a, w, ps, s);
  if (a.d == 256 && w.kb == 64)
    return a.dtype == FMB_BF16 ? fwd_wide_launch<__nv_bfloat16, 64, 256>(a, w, ps, s)
                               : fwd_wide_launch<__half, 64, 256>(a, w, ps, s);
  return fail(FMB_ERR_UNSUPPORTED, "wide-head forward: key block %d / head_dim %d not built", w.kb, a.d);
}

}  // namespace fmb
