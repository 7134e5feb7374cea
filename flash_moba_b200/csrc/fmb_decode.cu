// Few query rows against long key sequences (decoding, short blocks of new rows): gating and
// attention of a row in ONE launch.
//
// The key-chunk-major kernels are built for columns of many rows: with one row per column a tile of
// 128 gathered rows is 127 rows of padding, and the work items are the columns of every sequence and
// head, nearly all of them empty (16 sequences of up to 32K keys, 32 heads: 129,000 items for 4,096
// (row, chunk) entries, 0.83 ms).  Here a thread-block cluster owns one query row of HG q heads of a kv
// head and does everything for it, row-major:
//   1. scores of the row against the centroids of its candidate chunks (fp32), a warp per 32
//      centroids (16 at head dim 256); each head's scores are collected in the shared memory of one CTA of the cluster
//   2. top-k of each head by one warp (descending score, on equal scores the higher chunk id, the
//      row's own chunk first under the causal rule: the order of the other gating kernels); the list
//      goes to every CTA of the cluster
//   3. attention over the selected chunks, a warp per 32 (16) keys: fp32 scores, online softmax, fp32
//      accumulation; the warps' results meet in the owner CTA's shared memory and are merged in warp
//      order, so that the result does not depend on timing (its last bits do on how many CTAs share a row,
//      which goes by the number of rows)
// No pattern, no partials in global memory, no merge launch.  What bounds it: the selected K and V
// rows, each read once per (row, head) from L2 or HBM.
//
// One row per head leaves a tensor-core tile nearly empty, but the warp-level MMA still is the
// cheapest way through the arithmetic: with CUDA cores (unpack, FMA, butterfly reduction) a group of 32
// keys took 1,500 instructions and the kernel waited on its own instruction stream (26 M instructions,
// 88 us for 16 rows x 32 heads); here it takes about 250.  Keys (and centroids) are the M side of the
// score product, so a score needs no reduction across lanes: a thread loads 16-byte chunks of rows
// g and g + 8 (g = lane / 4) and uses them as A fragments as they are, the order of the head dimension
// inside the product being the same for q.  The values are the A operand of the second product (M =
// head dim): pairs of key rows are interleaved with byte permutes.  P is used as the sum of two
// 16-bit numbers (hi in column 0, lo in column 1 of the otherwise unused N side): 16 bits of it in bf16, 22
// in fp16, where the key-chunk-major kernels keep 8 and 11.
// All loads of a group (8 KB per warp at d 64, else 16 KB) are issued before its arithmetic; CTAs of 4 warps, four per
// SM at d 64, else two.
// Measured (B200, 32 / 8 heads, d 128, chunk 128, top-k 8): see decode_preferred().
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "fmb_common.cuh"

namespace fmb {

namespace cg = cooperative_groups;

constexpr int kDecThreads = 128, kDecWarps = kDecThreads / 32;
constexpr float kLog2eDec = 1.4426950408889634f;
// Candidates of a lane that are kept in registers while a list is made: four of them for rows of up to 128 candidates, else sixteen (every look
// goes over all places, used or not).  One row, us, all looked up in shared memory / 16 / 4 or 16: 2 chunks 7.7 / 8.0 / 7.4, d 64, 20 chunks
// 7.3 / 7.4 / 7.0; two rows, 125 chunks 14.6 / 14.3 / 13.4.  With 8 in place of 4: 235 chunks 12.0 / 11.4, but 125 13.4 / 13.8 and 8 8.6 / 8.8;
// with 24 in place of 16: 703 chunks 13.4 / 12.5, but 508 12.3 / 12.8 and 313 10.7 / 11.5
constexpr int kDecFew = 4, kDecHeld = 16;

struct DecodeParams {
  const void *q, *k, *v, *km;
  int64_t q_rs, q_hs, k_rs, k_hs, v_rs, v_hs, o_rs, o_hs;
  void* out;
  const int32_t *cu_q, *cu_k, *cu_km;
  int batch, heads, heads_k, d, topk, chunk, causal, hg, ncap;
  float scale;
};

// Geometry of a warp's group of keys at padded head dim D
template <int D> struct DecGeo {
  static constexpr int KC = D / 32;             // 16-byte chunks of a key row per thread
  static constexpr int VC = D / 64;             // 16-byte chunks of a value row per thread
  static constexpr int KB = D == 256 ? 1 : 2;   // 16-key blocks per group: 8 KB of K and V at d = 64, else 16 KB
  static constexpr int CTAS = D == 64 ? 4 : 2;  // resident CTAs per SM
  static constexpr int GK = 16 * KB;            // keys per group (chunks are multiples of 64)
};

template <typename T> struct DecMma;
template <> struct DecMma<__nv_bfloat16> {
  static __device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};
template <> struct DecMma<__half> {
  static __device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};
template <typename T>
__device__ __forceinline__ uint32_t dec_pack(float a, float b) {
  const typename Elem<T>::T2 x = Elem<T>::from_f2(a, b);
  return *reinterpret_cast<const uint32_t*>(&x);
}

// Key (or centroid) rows as A fragments: rows g, g + 8 of every 16-row block, chunks t, t + 4, ...
// of the row (g = lane / 4, t = lane % 4).  base: the first row's first byte; nothing is read at or
// past row `rows` or chunk `nch`.
template <int D>
__device__ __forceinline__ void dec_load_k(uint4 (&u)[DecGeo<D>::KB][2][DecGeo<D>::KC], const char* base, int64_t row_bytes,
                                           int rows, int nch, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int kb = 0; kb < DecGeo<D>::KB; ++kb) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int r = kb * 16 + half * 8 + g;
      const char* row = base + (int64_t)r * row_bytes + t * 16;
#pragma unroll
      for (int i = 0; i < DecGeo<D>::KC; ++i)
        u[kb][half][i] = (r < rows && t + 4 * i < nch) ? ldg_16(row + i * 64) : make_uint4(0, 0, 0, 0);
    }
  }
}
// c: scores of rows g (c[0], c[1]) and g + 8 (c[2], c[3]) of block kb against the columns 2t, 2t + 1
template <typename T, int D>
__device__ __forceinline__ void dec_mma_k(float (&c)[4], const uint4 (&u)[2][DecGeo<D>::KC], const uint4 (&q)[DecGeo<D>::KC]) {
  c[0] = c[1] = c[2] = c[3] = 0.f;
#pragma unroll
  for (int i = 0; i < DecGeo<D>::KC; ++i) {
    DecMma<T>::mma(c, u[0][i].x, u[1][i].x, u[0][i].y, u[1][i].y, q[i].x, q[i].y);
    DecMma<T>::mma(c, u[0][i].z, u[1][i].z, u[0][i].w, u[1][i].w, q[i].z, q[i].w);
  }
}

template <typename T, int D>
__global__ void __launch_bounds__(kDecThreads, DecGeo<D>::CTAS) decode_kernel(DecodeParams p) {
  using Geo = DecGeo<D>;
  follow_on();
  constexpr int KC = Geo::KC, VC = Geo::VC, KB = Geo::KB, GK = Geo::GK;
  extern __shared__ __align__(16) unsigned char dec_smem[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), S = (int)cluster.num_blocks();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, tq = lane & 3;
  const int HG = p.hg, topk = p.topk;
  const int hpr = (HG + S - 1) / S;             // heads whose scores, lists and results a CTA owns
  const int wph = kDecWarps * S / HG;           // warps per head
  float* sAcc = reinterpret_cast<float*>(dec_smem);           // [hpr][wph][D]
  float* sML = sAcc + hpr * wph * D;                          // [hpr][wph][2]
  int* sList = reinterpret_cast<int*>(sML + hpr * wph * 2);   // [HG][topk]
  float* sScore = reinterpret_cast<float*>(sList + HG * topk);// [hpr][ncap]

  const int t = blockIdx.z, h0 = blockIdx.y * HG, hk = h0 / (p.heads / p.heads_k);
  int b = 0;                                    // the sequence of row t: the last b with cu_q[b] <= t
  {
    int lo = 0, hi = p.batch;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (p.cu_q[mid] <= t) lo = mid; else hi = mid;
    }
    b = lo;
  }
  const int q0 = p.cu_q[b], len_q = p.cu_q[b + 1] - q0;
  if (t < q0 || t >= q0 + len_q) {              // a row of no sequence (uniform over the cluster) sees no key
    for (int i = rank * kDecThreads + tid; i < HG * p.d; i += S * kDecThreads)
      static_cast<T*>(p.out)[(int64_t)t * p.o_rs + (int64_t)(h0 + i / p.d) * p.o_hs + i % p.d] = Elem<T>::from_f(0.f);
    return;
  }
  const int k0 = p.cu_k[b], len_k = p.cu_k[b + 1] - k0;
  const int km0 = p.cu_km[b];
  const int nchunks = min((len_k + p.chunk - 1) / p.chunk, p.ncap);
  const int pos = len_k - len_q + (t - q0);
  const int own = p.causal ? (pos >= 0 && nchunks > 0 ? pos / p.chunk : -1) : -1;
  const int ncand = p.causal ? (pos < 0 ? 0 : min(nchunks, pos / p.chunk)) : nchunks;
  const int key_end = p.causal ? min(len_k, pos + 1) : len_k;
  const int nch = p.d / 8;                      // 16-byte chunks of a row in use
  // q of head h as a B fragment: chunks t, t + 4, ... of its row
  auto load_q = [&](uint4 (&q)[KC], int h, bool ok) {
    const T* row = static_cast<const T*>(p.q) + (int64_t)t * p.q_rs + (int64_t)(h0 + h) * p.q_hs + tq * 8;
#pragma unroll
    for (int i = 0; i < KC; ++i) q[i] = (ok && tq + 4 * i < nch) ? ldg_16(row + i * 32) : make_uint4(0, 0, 0, 0);
  };
  const int my_warp = rank * kDecWarps + warp, n_warps = S * kDecWarps;

  cluster.sync();                               // every CTA of the cluster runs: its shared memory may be written

  // ---- 1. scores: the N side of the product is the cluster's heads
  {
    uint4 q[KC];
    load_q(q, gr, gr < HG);
    const int64_t km_row = (int64_t)p.heads_k * p.d * (int64_t)sizeof(T);
    for (int n0 = my_warp * GK; n0 < ncand; n0 += n_warps * GK) {
      const int rows = min(GK, ncand - n0);
      uint4 u[KB][2][KC];
      dec_load_k<D>(u, reinterpret_cast<const char*>(static_cast<const T*>(p.km) + ((int64_t)(km0 + n0) * p.heads_k + hk) * p.d),
                    km_row, rows, nch, lane);
#pragma unroll
      for (int kb = 0; kb < KB; ++kb) {
        float c[4];
        dec_mma_k<T, D>(c, u[kb], q);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int h = 2 * tq + (x & 1), r = kb * 16 + (x >> 1) * 8 + gr;
          if (h < HG && r < rows) cluster.map_shared_rank(sScore, h % S)[(int64_t)(h / S) * p.ncap + n0 + r] = c[x];
        }
      }
    }
  }
  cluster.sync();

  // ---- 2. lists
  for (int h = rank + warp * S; h < HG; h += kDecWarps * S) {
    float* sc = sScore + (int64_t)(h / S) * p.ncap;
    int j = 0;
    if (own >= 0) {
      if (lane < S) cluster.map_shared_rank(sList, lane)[h * topk] = own;
      j = 1;
    }
    // Every lane knows the best of its candidates (n = lane, lane + 32, ...); a round takes the best of the lanes' and only
    // the lane it came from looks for its next.  Scores as ordered integers (+0 and -0 alike, though no sum that starts at +0 is -0), 0: none
    // (-inf, NaN).  Up to kDecHeld candidates a lane are held in registers, for a look in shared memory at all of them takes a round as long as the reductions;
    // more are looked up there.  (With a scan of all candidates and ten shuffles in every round: one row of 32 heads
    // and 65,001 keys 17.7 us, 16 rows of 16 sequences 54.6; looks in shared memory 16.3 and 52.7.  Since then, looks in shared
    // memory / in registers: one row 14.6 / 13.7, two of 16,000 keys 14.8 / 14.5, 16 54.0 / 53.7, d 64, eight rows 19.8 / 19.35.
    // Looks in shared memory compare floats and make an integer of the best one only: with one made of every score, one row
    // of 4 heads and 50,894 keys (795 chunks, top 12) took 18.7 us instead of 16.6)
    auto ordered = [](float x) {
      const uint32_t u = __float_as_uint(x + 0.f);
      return !(x > -CUDART_INF_F) ? 0u : (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    };
    auto rounds = [&](auto look, auto take) {
      uint32_t best;
      int at;
      look(best, at);
      for (; j < topk; ++j) {
        const uint32_t top = __reduce_max_sync(0xffffffffu, best);
        const int pick = __reduce_max_sync(0xffffffffu, best == top ? at : -1);
        if (pick >= 0 && pick == at) {
          take(at);
          look(best, at);
        }
        if (lane < S) cluster.map_shared_rank(sList, lane)[h * topk + j] = pick;
      }
    };
    auto held = [&](auto most) {
      constexpr int N = decltype(most)::value;
      uint32_t u[N];
#pragma unroll
      for (int i = 0; i < N; ++i) u[i] = lane + 32 * i < ncand ? ordered(sc[lane + 32 * i]) : 0u;
      rounds(
          [&](uint32_t& best, int& at) {
            best = 0u;
            at = 0;
#pragma unroll
            for (int i = 0; i < N; ++i)
              if (u[i] >= best) { best = u[i]; at = lane + 32 * i; }   // ascending n: the higher id on equal scores
            if (best == 0u) at = -1;
          },
          [&](int at) {
#pragma unroll
            for (int i = 0; i < N; ++i)
              if (at == lane + 32 * i) u[i] = 0u;
          });
    };
    if (ncand <= 32 * kDecFew) {
      held(std::integral_constant<int, kDecFew>{});
    } else if (ncand <= 32 * kDecHeld) {
      held(std::integral_constant<int, kDecHeld>{});
    } else {
      rounds(
          [&](uint32_t& best, int& at) {
            float m = -CUDART_INF_F;
            at = -1;
            for (int n = lane; n < ncand; n += 32) {
              const float x = sc[n];
              if (x >= m && x > -CUDART_INF_F) { m = x; at = n; }
            }
            best = at < 0 ? 0u : ordered(m);
          },
          [&](int at) { sc[at] = -CUDART_INF_F; });
    }
  }
  cluster.sync();

  // ---- 3. attention: this warp's head, every wph-th group of GK keys of its list
  const int h = my_warp % HG, wh = my_warp / HG;
  uint4 q[KC];
  load_q(q, h, true);                           // the same in all 8 columns: every thread of a row gets the score
  float acc[D / 16][4];                         // element j of chunk g: [j][0..1] (hi and lo part); of its partner: [j][2..3]
  float m = -CUDART_INF_F, l = 0.f;
#pragma unroll
  for (int j = 0; j < D / 16; ++j) { acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f; }
  const float scale_log2 = p.scale * kLog2eDec;
  const int gpc = p.chunk / GK, groups = topk * gpc;
  const int64_t k_row = p.k_rs * (int64_t)sizeof(T), v_row = p.v_rs * (int64_t)sizeof(T);
#pragma unroll 1
  for (int g = wh; g < groups; g += wph) {
    const int li = g / gpc;
    const int c = sList[h * topk + li];
    if (c < 0) continue;
    const int key0 = c * p.chunk + (g - li * gpc) * GK;
    const int rows = min(GK, key_end - key0);
    if (rows <= 0) continue;
    uint4 uk[KB][2][KC], uv[KB][4][VC];
    dec_load_k<D>(uk, reinterpret_cast<const char*>(static_cast<const T*>(p.k) + (int64_t)(k0 + key0) * p.k_rs + (int64_t)hk * p.k_hs),
                  k_row, rows, nch, lane);
    {
      // value rows 2t, 2t + 1, 2t + 8, 2t + 9 of every block, chunks g, g + 8, ...
      const char* vb = reinterpret_cast<const char*>(static_cast<const T*>(p.v) + (int64_t)(k0 + key0) * p.v_rs + (int64_t)hk * p.v_hs) + gr * 16;
#pragma unroll
      for (int kb = 0; kb < KB; ++kb)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int r = kb * 16 + 2 * tq + (x & 1) + (x >> 1) * 8;
#pragma unroll
          for (int i = 0; i < VC; ++i)
            uv[kb][x][i] = (r < rows && gr + 8 * i < nch) ? ldg_16(vb + (int64_t)r * v_row + i * 128) : make_uint4(0, 0, 0, 0);
        }
    }
    float s[KB][2], mx = -CUDART_INF_F;
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) {
      float cc[4];
      dec_mma_k<T, D>(cc, uk[kb], q);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        s[kb][half] = kb * 16 + half * 8 + gr < rows ? cc[half * 2] * scale_log2 : -CUDART_INF_F;
        mx = fmaxf(mx, s[kb][half]);
      }
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (mx > m) {                               // warp-uniform
      const float keep = exp2f(m - mx);
      m = mx;
      l *= keep;
#pragma unroll
      for (int j = 0; j < D / 16; ++j) { acc[j][0] *= keep; acc[j][1] *= keep; acc[j][2] *= keep; acc[j][3] *= keep; }
    }
    const float mref = m > -CUDART_INF_F ? m : 0.f;   // nothing but scores of -inf (no weight) or NaN so far
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) {
      const float p0 = exp2f(s[kb][0] - mref), p1 = exp2f(s[kb][1] - mref);
      l += p0 + p1;
      // P of this thread's value rows: column 0 the rounded value, column 1 what the rounding left
      const float w0 = __shfl_sync(0xffffffffu, p0, 8 * tq), w1 = __shfl_sync(0xffffffffu, p0, 8 * tq + 4);
      const float w2 = __shfl_sync(0xffffffffu, p1, 8 * tq), w3 = __shfl_sync(0xffffffffu, p1, 8 * tq + 4);
      uint32_t b0 = dec_pack<T>(w0, w1), b1 = dec_pack<T>(w2, w3);
      {
        using T2 = typename Elem<T>::T2;
        const float2 f0 = Elem<T>::to_f2(*reinterpret_cast<const T2*>(&b0)), f1 = Elem<T>::to_f2(*reinterpret_cast<const T2*>(&b1));
        const uint32_t l0 = dec_pack<T>(w0 - f0.x, w1 - f0.y), l1 = dec_pack<T>(w2 - f1.x, w3 - f1.y);
        b0 = gr == 0 ? b0 : gr == 1 ? l0 : 0u;
        b1 = gr == 0 ? b1 : gr == 1 ? l1 : 0u;
      }
      auto word = [](const uint4& u, int i) { return i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w; };
      if constexpr (D == 64) {                  // rows of the product: element j of chunk g and element j + 4 of chunk g
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;
          const int w = j >> 1;
          DecMma<T>::mma(acc[j], __byte_perm(word(uv[kb][0][0], w), word(uv[kb][1][0], w), sel),
                         __byte_perm(word(uv[kb][0][0], w + 2), word(uv[kb][1][0], w + 2), sel),
                         __byte_perm(word(uv[kb][2][0], w), word(uv[kb][3][0], w), sel),
                         __byte_perm(word(uv[kb][2][0], w + 2), word(uv[kb][3][0], w + 2), sel), b0, b1);
        }
      } else {                                  // element j of chunk g + 16i and of chunk g + 16i + 8
#pragma unroll
        for (int i = 0; i < VC / 2; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;
            const int w = j >> 1;
            DecMma<T>::mma(acc[i * 8 + j], __byte_perm(word(uv[kb][0][2 * i], w), word(uv[kb][1][2 * i], w), sel),
                           __byte_perm(word(uv[kb][0][2 * i + 1], w), word(uv[kb][1][2 * i + 1], w), sel),
                           __byte_perm(word(uv[kb][2][2 * i], w), word(uv[kb][3][2 * i], w), sel),
                           __byte_perm(word(uv[kb][2][2 * i + 1], w), word(uv[kb][3][2 * i + 1], w), sel), b0, b1);
          }
      }
    }
  }
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  {
    float* dA = cluster.map_shared_rank(sAcc, h % S) + ((h / S) * wph + wh) * D;
    float* dM = cluster.map_shared_rank(sML, h % S) + ((h / S) * wph + wh) * 2;
    if (tq == 0) {                              // columns 0 and 1
#pragma unroll
      for (int j = 0; j < D / 16; ++j) {
        // an infinite value makes the hi part infinite, and the lo part infinite the other way or NaN
        const float x = fabsf(acc[j][0]) < CUDART_INF_F ? acc[j][0] + acc[j][1] : acc[j][0];
        const float y = fabsf(acc[j][2]) < CUDART_INF_F ? acc[j][2] + acc[j][3] : acc[j][2];
        if constexpr (D == 64) {
          dA[gr * 8 + j] = x;
          dA[gr * 8 + j + 4] = y;
        } else {
          dA[(j / 8) * 128 + gr * 8 + j % 8] = x;
          dA[(j / 8) * 128 + 64 + gr * 8 + j % 8] = y;
        }
      }
    }
    if (lane == 0) { dM[0] = m; dM[1] = l; }
  }
  cluster.sync();                               // (the last access to another CTA's shared memory lies before it)

  // ---- 4. merge of the heads this CTA owns, in warp order
  for (int i = tid; i < hpr * D; i += kDecThreads) {
    const int hr = i / D, c = i % D, hh = hr * S + rank;
    if (hh >= HG || c >= p.d) continue;
    const float* M = sML + hr * wph * 2;
    float mm = -CUDART_INF_F;
    for (int w = 0; w < wph; ++w) mm = fmaxf(mm, M[2 * w]);
    float num = 0.f, den = 0.f;
    for (int w = 0; w < wph; ++w) {
      const float f = exp2f(M[2 * w] - mm);
      num = fmaf(f, sAcc[(hr * wph + w) * D + c], num);
      den = fmaf(f, M[2 * w + 1], den);
    }
    // zero only for a row that sees no key (an empty list): NaN in its scores or values stays visible
    static_cast<T*>(p.out)[(int64_t)t * p.o_rs + (int64_t)(h0 + hh) * p.o_hs + c] = Elem<T>::from_f(sList[hh * topk] >= 0 ? num / den : 0.f);
  }
}

struct DecodeShape { int hg, S, ncap; size_t smem; };

static DecodeShape decode_shape(int64_t total_q, int heads, int heads_k, int d, int max_k, int topk, int chunk) {
  DecodeShape r;
  const int dp = d <= 64 ? 64 : d <= 128 ? 128 : 256, keys = d <= 64 ? DecGeo<64>::GK : d <= 128 ? DecGeo<128>::GK : DecGeo<256>::GK;
  const int group = heads / heads_k;
  // heads per cluster: a divisor of the group and of the warps of one CTA (every head has a warp)
  static_assert(kDecWarps == 4, "4, 2 or 1 heads per cluster");
  r.hg = group % 4 == 0 ? 4 : group % 2 == 0 ? 2 : 1;
  // With few rows: fewer heads per cluster and clusters of more CTAs, until the device is full or a
  // warp would be left without a group of keys; of eight CTAs only where with four a warp would have four groups or more: clusters of
  // eight find their places later, and are no longer brought up early (below).  Measured, eight / four, one row: 32 / 8 heads, d 128, top-k 8,
  // 65,001 keys 15.8 / 13.1 us, 4,000 keys 13.8 / 11.6; 16 / 4 heads, d 64 11.2 / 10.0; two rows, 16 / 8 heads, chunk 64, top-k 16 19.5 / 16.7 (two
  // groups a warp with four CTAs, all of them); 8 heads, chunk 256, top-k 8 (four groups) 13.0 / 13.7; 32 / 16 heads, d 64, chunk 256, top-k 16
  // (eight) 17.7 / 20.2.
  const int64_t want = 148 * (d <= 64 ? DecGeo<64>::CTAS : DecGeo<128>::CTAS);
  while (r.hg > 1 && total_q * (heads / r.hg) * 8 < want) r.hg /= 2;
  r.S = 1;
  while (r.S < 8 && total_q * (heads / r.hg) * r.S * 2 <= want && (int64_t)r.hg * topk * (chunk / keys) >= (r.S < 4 ? 2 : 4) * r.S * kDecWarps)
    r.S *= 2;
  r.ncap = (max_k + chunk - 1) / chunk;
  if (r.ncap < 1) r.ncap = 1;
  const int hpr = (r.hg + r.S - 1) / r.S, wph = kDecWarps * r.S / r.hg;
  r.smem = sizeof(float) * ((size_t)hpr * wph * (dp + 2) + (size_t)r.hg * topk + (size_t)hpr * r.ncap);
  return r;
}

constexpr size_t kDecSmemMost = 100 * 1024;

bool decode_supported(int64_t total_q, int heads, int heads_k, int d, int max_k, int topk, int chunk) {
  if (total_q > 65535 || heads > 65535 || topk > 64 || chunk % 64 != 0 || d % 8 != 0 || d > 256) return false;
  return decode_shape(total_q, heads, heads_k, d, max_k, topk, chunk).smem <= kDecSmemMost;
}

// Where the line lies: both ways' times in microseconds, estimated from what bounds them, fitted to a
// sweep on a B200 (1 to 64 sequences of 2,000 and 16,000 keys, 1 to 32 new rows each, 8 to 32 heads, chunk 64 to 256,
// top-k 8 and 16, d 64 to 256).  This kernel: the selected keys and values of every (row, head) at 6.5 TB/s,
// whoever else selects them too.  The key-chunk-major way: gating, pattern and launches, then 6 ns
// for every column (128-key block) of every head and 20 ns more for one that any row selects, whatever
// the number of its rows; the share of such columns as for independent selections.
// Measured, this kernel / the other (d 128, 32 / 8 heads, chunk 128, top-k 8): 16 sequences of 16,000
// keys, 1 row each 56 / 522 us, 4 rows 183 / 673, 16 rows 615 / 1222; 4 sequences of 2,000 keys, 4 rows each
// 43 / 96, 16 rows 140 / 99; one row and 65,001 keys 19 / 149.
bool decode_preferred(int64_t total_q, int64_t total_k, int batch, int heads, int heads_k, int d, int max_k, int topk, int chunk) {
  if (!decode_supported(total_q, heads, heads_k, d, max_k, topk, chunk)) return false;
  const double keys_per_row = std::min((double)topk * chunk, (double)total_k / batch);
  const double row_major = 12.0 + (double)total_q * heads * keys_per_row * d * 4.0 / 6.5e6;
  const double columns = (double)total_k / chunk + batch;
  const double in_use = columns * (1.0 - std::exp(-(double)total_q * topk / columns));
  const double blocks = heads * std::max(1.0, chunk / 128.0);
  const double chunk_major = 45.0 + blocks * (columns * 0.006 + in_use * 0.02);
  return row_major < chunk_major;
}

template <typename T, int D>
static int decode_launch(const DecodeParams& p, const DecodeShape& sh, int64_t total_q, cudaStream_t s) {
  auto kern = decode_kernel<T, D>;
  FMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDecSmemMost));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sh.S, p.heads / sh.hg, (unsigned)total_q);
  cfg.blockDim = dim3(kDecThreads);
  cfg.dynamicSmemBytes = sh.smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  // Brought up beside the kernel before it (see follow_on()), but for clusters of eight CTAs: placed around those of a call
  // that still runs they may pile up on fewer SMs.  Measured, without / with, back to back; between elementwise kernels of torch
  // (32 / 8 heads): d 128, 32 rows (no clusters) 94.2 / 92.1; 94.3 / 91.1 us, 16 rows (of two) 56.0 / 54.4; 56.0 / 54.2, 8 rows (of
  // four) 34.8 / 32.8; 35.8 / 32.8, 4 rows (of four) 22.6 / 21.3; 23.6 / 22.0, one row (of four) and 65,001 keys 13.1 / 13.1; 12.8 / 12.7,
  // 4,000 keys 12.1 / 11.7; 11.7 / 11.4; d 64, 8 rows 22.5 / 20.2; 23.2 / 20.2, d 256, 4 rows 37.0 / 35.5; 37.7 / 35.9.  Of eight: one
  // row and 65,001 keys, when it was split that far, 18.5 / 25.7; 18.6 / 15.4; 8 heads, chunk 256, one row 13.1 / 12.6; 12.8 / 12.5;
  // 32 / 16 heads, d 64, chunk 256, top-k 16, one row 17.7 / 18.0; 17.5 / 17.3
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = sh.S;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = sh.S <= 4 ? 2 : 1;
  (void)cudaLaunchKernelEx(&cfg, kern, p);
  FMB_LAUNCH_CHECK("decode_kernel");
  return FMB_OK;
}

int launch_decode(const DecodeArgs& a, cudaStream_t s) {
  DecodeParams p;
  const DecodeShape sh = decode_shape(a.total_q, a.heads, a.heads_k, a.d, a.max_k, a.topk, a.chunk);
  p.q = a.q; p.k = a.k; p.v = a.v; p.km = a.km; p.out = a.o;
  p.q_rs = a.q_rs; p.q_hs = a.q_hs; p.k_rs = a.k_rs; p.k_hs = a.k_hs; p.v_rs = a.v_rs; p.v_hs = a.v_hs;
  p.o_rs = a.o_rs; p.o_hs = a.o_hs;
  p.cu_q = a.cu_q; p.cu_k = a.cu_k; p.cu_km = a.cu_km;
  p.batch = a.batch; p.heads = a.heads; p.heads_k = a.heads_k; p.d = a.d; p.topk = a.topk; p.chunk = a.chunk;
  p.causal = a.causal; p.scale = a.scale; p.hg = sh.hg; p.ncap = sh.ncap;
  const bool bf = a.dtype == FMB_BF16;
  if (a.d <= 64) return bf ? decode_launch<__nv_bfloat16, 64>(p, sh, a.total_q, s) : decode_launch<__half, 64>(p, sh, a.total_q, s);
  if (a.d <= 128) return bf ? decode_launch<__nv_bfloat16, 128>(p, sh, a.total_q, s) : decode_launch<__half, 128>(p, sh, a.total_q, s);
  return bf ? decode_launch<__nv_bfloat16, 256>(p, sh, a.total_q, s) : decode_launch<__half, 256>(p, sh, a.total_q, s);
}

}  // namespace fmb
