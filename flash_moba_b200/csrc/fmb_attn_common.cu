// Pass planning, slot and row lists (CSR transpose of the pattern), the row-major merge
// kernel and the forward / backward drivers shared by both attention engines.
#include "fmb_attn.cuh"

namespace fmb {

// ------------------------------------------------------------------ workspace layout / passes
static size_t scan_tmp_elems(int64_t n) { return (size_t)ceil_div64(n, 4096) + 1; }

static size_t layout(AttnWorkspace& w, void* base, const AttnArgs& a, size_t part_elem_bytes, bool with_lse, int nh) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    void* p = base ? static_cast<char*>(base) + off : nullptr;
    off += align_up(bytes, 256);
    return p;
  };
  w.nh = nh;
  w.fixed_k = 0;
  w.mirror = nullptr;
  // key block: 128 keys when the chunk is a multiple of 128, except in the backward pass of head
  // dim 256, whose dK and dV accumulators for 128 keys would not fit in TMEM (with_lse = forward)
  w.kb = (a.chunk % 128 == 0 && (a.d <= 128 || with_lse)) ? 128 : 64;
  w.nsub = a.chunk / w.kb;
  // one pass over all heads can never need more slots than the pattern has entries; a pass over a
  // share of the heads is given that share (exact for the top-k packing), rounded up
  w.cap = nh >= a.heads ? a.n_indices : ceil_div64(a.n_indices * nh, a.heads) + 128;
  w.cap = ceil_div64(w.cap, 8) * 8;
  const int64_t rows = a.total_q * nh;
  const int64_t ncols = (int64_t)a.batch * nh * a.ncol;
  w.status = static_cast<int*>(take(kStatusBytes));
  // the partials are stored 32 bytes at a time: a caller's workspace may start on any 16-byte boundary
  off += base ? (32 - (reinterpret_cast<uintptr_t>(base) + off) % 32) % 32 : 32;
  w.part_o = take((size_t)w.nsub * w.cap * a.d * part_elem_bytes);
  w.part_lse = static_cast<float*>(take(with_lse ? (size_t)w.nsub * w.cap * sizeof(float) : 0));
  w.lists_off = off;
  w.slot_base = static_cast<uint32_t*>(take((size_t)(ncols + 1) * sizeof(uint32_t)));
  w.row_ptr = static_cast<uint32_t*>(take((size_t)(rows + 1) * sizeof(uint32_t)));
  w.row_fill = static_cast<uint32_t*>(take((size_t)rows * sizeof(uint32_t)));
  w.row_pos = static_cast<uint32_t*>(take((size_t)w.cap * sizeof(uint32_t)));
  w.lists_bytes = off - w.lists_off;
  const int64_t longest = rows + 1 > ncols + 1 ? rows + 1 : ncols + 1;
  w.scan_tmp = static_cast<uint32_t*>(take(scan_tmp_elems(longest) * sizeof(uint32_t)));
  w.bytes = off;
  return off;
}

AttnWorkspace carve_attn_workspace(void* base, size_t bytes_available, const AttnArgs& a, size_t part_elem_bytes,
                                   bool with_lse, int heads_per_pass) {
  AttnWorkspace w;
  const int group = a.heads / a.heads_k;
  int nh = a.heads;
  if (heads_per_pass > 0) {
    nh = min(a.heads, max(group, heads_per_pass / group * group));
  } else if (base != nullptr) {   // the largest pass (whole kv-head groups) that fits what the caller gave
    while (nh > group && layout(w, nullptr, a, part_elem_bytes, with_lse, nh) > bytes_available) nh -= group;
  }
  layout(w, base, a, part_elem_bytes, with_lse, nh);
  return w;
}

size_t attn_workspace_bytes(int64_t total_q, int heads, int heads_k, int d, int64_t n_indices, int batch, int max_k,
                            int chunk, int heads_per_pass, bool backward) {
  AttnArgs a;
  memset(&a, 0, sizeof(a));
  a.total_q = total_q; a.heads = heads; a.heads_k = heads_k > 0 ? heads_k : heads; a.d = d; a.n_indices = n_indices;
  a.batch = batch; a.chunk = chunk > 0 ? chunk : 128; a.ncol = ceil_div(max_k, a.chunk);
  return carve_attn_workspace(nullptr, 0, a, 2, !backward, heads_per_pass > 0 ? heads_per_pass : heads)
      .bytes;
}

PassParams make_pass(const AttnArgs& a, const AttnWorkspace& w, int h0, int nh) {
  PassParams r;
  r.col_offsets = a.col_offsets; r.col_nnz = a.col_nnz; r.indices = a.indices; r.n_indices = a.n_indices;
  r.slot_base = w.slot_base;
  r.heads = a.heads; r.ncol = a.ncol; r.h0 = h0; r.nh = nh; r.nsub = w.nsub; r.kb = w.kb; r.chunk = a.chunk;
  r.cap = w.cap; r.status = w.status;
  r.slot_shift = w.fixed_k > 0 ? (int64_t)h0 * a.total_q * w.fixed_k : 0;
  return r;
}

// ------------------------------------------------------------------ slot and row lists
// slot_base[i + 1] = entries of the i-th column of the pass (0 if the column is malformed);
// an inclusive scan then turns the array into first slots
__global__ void __launch_bounds__(256) slot_count_kernel(PassParams r, uint32_t* slot_base, int batch) {
  const int64_t n = (int64_t)batch * r.nh * r.ncol;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) slot_base[0] = 0;
  if (i >= n) return;
  const int c = (int)(i % r.ncol);
  const int hr = (int)((i / r.ncol) % r.nh);
  const int b = (int)(i / ((int64_t)r.ncol * r.nh));
  const int64_t ci = ((int64_t)b * r.heads + r.h0 + hr) * r.ncol + c;
  const int nnz = r.col_nnz[ci];
  const int64_t off = r.col_offsets[ci];
  slot_base[i + 1] = (nnz > 0 && off >= 0 && off + nnz <= r.n_indices) ? (uint32_t)nnz : 0u;
}

struct RowListParams {
  PassParams r;
  const int32_t* cu_q;
  uint32_t *row_ptr, *row_fill, *row_pos;
  int64_t total_q;
};

// grid (ncol, nh, batch): one CTA per column of the pass
template <bool kFill>
__global__ void __launch_bounds__(256) row_list_kernel(RowListParams p) {
  const int c = blockIdx.x, hr = blockIdx.y, b = blockIdx.z;
  const ColRef col = column_of(p.r, b, p.r.h0 + hr, c);
  if (col.nnz <= 0) return;
  const int q0 = p.cu_q[b], len_q = p.cu_q[b + 1] - q0;
  const int64_t rbase = (int64_t)hr * p.total_q + q0;
  for (int j = threadIdx.x; j < col.nnz; j += blockDim.x) {
    const int r = p.r.indices[col.off + j];
    if (r < 0 || r >= len_q) continue;
    if (!kFill) {
      atomicAdd(&p.row_ptr[rbase + r + 1], 1u);     // counts, shifted by one for the scan
    } else {
      const uint32_t k = atomicAdd(&p.row_fill[rbase + r], 1u);
      p.row_pos[p.row_ptr[rbase + r] + k] = (uint32_t)(col.slot + j);
    }
  }
}

// The atomics of the fill leave a row's list in no particular order: put it in ascending slot order,
// which is the order of the merge.  A warp per row; lists of up to 32 by counting, longer ones by a
// direction-free bitonic network in place (every compare-exchange puts the smaller slot at the lower place).
__global__ void __launch_bounds__(256) sort_rows_kernel(const uint32_t* __restrict__ row_ptr, uint32_t* row_pos, int64_t rows) {
  const int64_t r = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= rows) return;
  uint32_t* a = row_pos + row_ptr[r];
  const int n = (int)(row_ptr[r + 1] - row_ptr[r]);
  if (n <= 32) {
    const uint32_t x = lane < n ? a[lane] : 0xffffffffu;
    int rank = 0;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const uint32_t y = __shfl_sync(0xffffffffu, x, i);
      rank += (y < x || (y == x && i < lane)) ? 1 : 0;
    }
    if (lane < n) a[rank] = x;
    return;
  }
  int N = 64;
  while (N < n) N <<= 1;
  for (int k = 2; k <= N; k <<= 1) {
    for (int j = k >> 1; j >= 1; j >>= 1) {
      const bool flip = j == (k >> 1);
      for (int i = lane; i < N; i += 32) {
        const int l = flip ? (i ^ (k - 1)) : (i ^ j);
        if (l > i && l < n) {
          const uint32_t x = a[i], y = a[l];
          if (x > y) { a[i] = y; a[l] = x; }
        }
      }
      __syncwarp();
    }
  }
}

// inclusive scan of u32 in place, three phases, 4096 items per block
constexpr int kScanItems = 4096;
__global__ void __launch_bounds__(1024) scan_block_kernel(uint32_t* data, int64_t n, uint32_t* block_sums) {
  __shared__ uint32_t wsum[32];
  const int64_t base = (int64_t)blockIdx.x * kScanItems + threadIdx.x * 4;
  uint32_t v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = (base + i < n) ? data[base + i] : 0u;
  v[1] += v[0]; v[2] += v[1]; v[3] += v[2];
  uint32_t x = v[3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  const uint32_t excl = (warp ? wsum[warp - 1] : 0u) + x - v[3];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (base + i < n) data[base + i] = v[i] + excl;
  if (threadIdx.x == 1023) block_sums[blockIdx.x] = wsum[31];
}
__global__ void __launch_bounds__(1024) scan_sums_kernel(uint32_t* block_sums, int nblocks) {
  // single block: serial over groups of 1024 with a running carry (exclusive result)
  __shared__ uint32_t wsum[32];
  __shared__ uint32_t carry_s;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int g = 0; g < nblocks; g += 1024) {
    const int i = g + threadIdx.x;
    const uint32_t v = i < nblocks ? block_sums[i] : 0u;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      wsum[lane] = w;
    }
    __syncthreads();
    const uint32_t carry = carry_s;
    if (i < nblocks) block_sums[i] = carry + (warp ? wsum[warp - 1] : 0u) + x - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry_s = carry + wsum[31];
    __syncthreads();
  }
}
__global__ void __launch_bounds__(1024) scan_add_kernel(uint32_t* data, int64_t n, const uint32_t* block_sums) {
  const int64_t base = (int64_t)blockIdx.x * kScanItems + threadIdx.x * 4;
  const uint32_t add = block_sums[blockIdx.x];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (base + i < n) data[base + i] += add;
}

static int inclusive_scan(uint32_t* data, int64_t n, uint32_t* tmp, cudaStream_t s) {
  const int nblocks = (int)ceil_div64(n, kScanItems);
  scan_block_kernel<<<nblocks, 1024, 0, s>>>(data, n, tmp);
  FMB_LAUNCH_CHECK("scan_block_kernel");
  if (nblocks > 1) {
    scan_sums_kernel<<<1, 1024, 0, s>>>(tmp, nblocks);
    FMB_LAUNCH_CHECK("scan_sums_kernel");
    scan_add_kernel<<<nblocks, 1024, 0, s>>>(data, n, tmp);
    FMB_LAUNCH_CHECK("scan_add_kernel");
  }
  return FMB_OK;
}

int build_row_lists(const AttnArgs& a, const AttnWorkspace& w, const PassParams& ps, cudaStream_t s) {
  const int64_t rows = a.total_q * ps.nh;
  const int64_t ncols = (int64_t)a.batch * ps.nh * a.ncol;
  // row_ptr and row_fill are neighbours in the workspace: one clear for both
  FMB_CUDA(cudaMemsetAsync(w.row_ptr, 0, (size_t)((char*)(w.row_fill + rows) - (char*)w.row_ptr), s));
  if (ncols == 0) return FMB_OK;
  slot_count_kernel<<<(unsigned)ceil_div64(ncols + 1, 256), 256, 0, s>>>(ps, w.slot_base, a.batch);
  FMB_LAUNCH_CHECK("slot_count_kernel");
  int rc = inclusive_scan(w.slot_base, ncols + 1, w.scan_tmp, s);
  if (rc) return rc;
  RowListParams p;
  p.r = ps; p.cu_q = a.cu_q; p.row_ptr = w.row_ptr; p.row_fill = w.row_fill; p.row_pos = w.row_pos;
  p.total_q = a.total_q;
  dim3 grid(a.ncol, ps.nh, a.batch);
  row_list_kernel<false><<<grid, 256, 0, s>>>(p);
  FMB_LAUNCH_CHECK("row_list_kernel<count>");
  rc = inclusive_scan(w.row_ptr, rows + 1, w.scan_tmp, s);
  if (rc) return rc;
  row_list_kernel<true><<<grid, 256, 0, s>>>(p);
  FMB_LAUNCH_CHECK("row_list_kernel<fill>");
  sort_rows_kernel<<<(unsigned)ceil_div64(rows, 8), 256, 0, s>>>(w.row_ptr, w.row_pos, rows);
  FMB_LAUNCH_CHECK("sort_rows_kernel");
  return FMB_OK;
}

// ------------------------------------------------------------------ merge of a row's partials
// What the merge kernel needs to know about the pass
struct MergeParams {
  const uint32_t* row_ptr; const uint32_t* row_pos;
  int64_t total_q, cap;
  int h0, nh, nsub;
  int fixed_k;     // > 0: row lists handed over by the pattern builder: row `rid` owns the fixed_k places
                   // row_pos[rid*fixed_k ..], empty places last (0xffffffff); row_ptr is not used
  int64_t slot_shift;               // handed-over rows hold positions in `indices`: slot = position - slot_shift
  const int* status; int* mirror;   // mirror != nullptr: the merge kernel of the call's last pass copies the
                                    // call's status word there (see attn_status_mirror)
};
constexpr uint32_t kNoSlot = 0xffffffffu;
constexpr int kMergeThreads = 256;
constexpr int kMergeBatch = 8;      // partial rows in flight per row

// From the order of a partial row (part_col) to a row's own: lane gl has columns 8 (4 (gl & 1) + k) + (gl & 6) and the next one of its
// 64, k = 0 .. 3; an exchange among the four lanes of the same parity gives it eight neighbouring ones, 16-byte chunk
// merged_place() of the row
__device__ __forceinline__ uint4 merged_chunk(uint4 u, int gl) {
  const bool odd = gl & 2, high = gl & 4;
  const uint32_t a = __shfl_xor_sync(0xffffffffu, odd ? u.x : u.y, 2), b = __shfl_xor_sync(0xffffffffu, odd ? u.z : u.w, 2);
  if (odd) { u.x = a; u.z = b; }
  else { u.y = a; u.w = b; }
  const uint32_t e = __shfl_xor_sync(0xffffffffu, high ? u.x : u.z, 4), f = __shfl_xor_sync(0xffffffffu, high ? u.y : u.w, 4);
  if (high) { u.x = e; u.y = f; }
  else { u.z = e; u.w = f; }
  return u;
}
__device__ __forceinline__ int merged_place(int gl) { return (gl & ~7) | (gl & 1) << 2 | ((gl >> 1) & 3); }

// Row lists are in ascending slot order (the pattern builder writes them so; sort_rows_kernel puts the
// lists of other patterns in order), so a row's partials are taken as they come: D/8 lanes per
// (head, token) row, one 16-byte chunk of every partial each, eight partials requested before anything
// waits, the next row's list requested before this row is worked on.  Merge order: plane by plane,
// ascending slots, whatever made the lists: results do not depend on it.  FWD weights the partials by
// exp(lse_j - max lse) and writes the row's log-sum-exp; the backward form is a plain sum.
// Bound: HBM (random 256-byte rows at d = 128), rows taken head by head.  With lists in the order of the
// gating lists, every lane group had to rank its row's places first and short lists left lanes idle; measured
// (B200, before / now, forward and backward): 64K tokens x 32 heads, top-k 8 1.19 / 0.82 and 0.93 / 0.78 ms (4.9 GB and
// 4.8 GB: 5.9 and 6.1 TB/s); 317K tokens, chunk 64, top-k 16 9.6 / 7.3 and 9.8 / 6.8 ms; 512K tokens x 4 heads, chunk 256,
// top-k 16 5.3 / 3.1 and 3.3 / 2.7 ms; d 64, 9,391 tokens x 12 heads 64 / 25 and 57 / 24 us.  Requesting a row's
// log-sum-exps before the output of the row before, not with its partials, is 10 % of the forward merge (0.915 -> 0.823).
template <typename T, int D, bool FWD>
__global__ void __launch_bounds__(kMergeThreads, 3) merge_kernel(const T* __restrict__ part, const float* __restrict__ part_lse,
                                                              MergeParams c, T* out, int64_t rs, int64_t hs, float* lse) {
  constexpr int LPR = D / 8, RPW = 32 / LPR, B = kMergeBatch;
  follow_on();
  if (c.mirror != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *c.mirror = *c.status;   // (the main kernel has completed)
  const int lane = threadIdx.x & 31, gl = lane % LPR;
  const int64_t n_rows = c.total_q * c.nh, stride = (int64_t)gridDim.x * (kMergeThreads / 32) * RPW;
  int64_t rid = ((int64_t)blockIdx.x * (kMergeThreads / 32) + (threadIdx.x >> 5)) * RPW + lane / LPR;
  const int64_t warp_first = rid - lane / LPR;

  // list of row r: its first place and length (an upper bound with empty places)
  auto span = [&](int64_t r, int64_t& p0, int& n) {
    p0 = 0;
    n = 0;
    if (r >= n_rows) return;
    if (c.fixed_k > 0) {
      p0 = r * c.fixed_k;
      n = c.fixed_k;
    } else {
      p0 = c.row_ptr[r];
      n = (int)(c.row_ptr[r + 1] - (uint32_t)p0);
    }
  };
  auto place = [&](int64_t p0, int n, int j) -> uint32_t { return j < n ? c.row_pos[p0 + j] : kNoSlot; };
  // slot in the pass of a place's content; kNoSlot also for what is no slot of this pass: nothing else is ever read.
  // (Applied at the use, not at the load, which is a row ahead.)
  auto slot_of = [&](uint32_t x) -> uint32_t {
    const uint32_t at = x - (uint32_t)c.slot_shift;
    return x != kNoSlot && at < c.cap ? at : kNoSlot;
  };
  auto lse_of = [&](uint32_t s, int sb) { return s == kNoSlot ? -CUDART_INF_F : part_lse[(int64_t)sb * c.cap + s]; };
  int64_t p0;
  int n;
  span(rid, p0, n);
  uint32_t next = place(p0, n, gl);             // this lane's place of the list, a row ahead
  float l_n = FWD ? lse_of(slot_of(next), 0) : 0.f;    // its log-sum-exp: requested ahead of the row before's output
#pragma unroll 1
  for (int64_t w0 = warp_first; w0 < n_rows; w0 += stride, rid += stride) {
    const int64_t q0 = p0;
    const int nr = n;
    const uint32_t slot = slot_of(next);
    span(rid + stride, p0, n);
    next = place(p0, n, gl);
    const int n_warp = __reduce_max_sync(0xffffffffu, nr);

    float m = -CUDART_INF_F, ssum = 0.f, acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    // places [b0, b0 + B) of the block of LPR places this lane's `s` belongs to, plane sb
    auto request = [&](uint32_t s, int sb, int b0, uint4 (&x)[B]) {
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const uint32_t sk = __shfl_sync(0xffffffffu, s, b0 + k, LPR);
        if (sk == kNoSlot) {
          x[k] = make_uint4(0, 0, 0, 0);
        } else {
          x[k] = ldg_nc_16(part + ((int64_t)sb * c.cap + sk) * D + gl * 8);
        }
      }
    };
    // the first batch is requested before the weights are known
    uint4 x[B];
    float l = l_n;
    request(slot, 0, 0, x);
    if (FWD) {
      m = l;
      for (int sb = 0; sb < c.nsub; ++sb)       // (longer lists and further planes)
        for (int j0 = sb == 0 ? LPR : 0; j0 < n_warp; j0 += LPR)
          m = fmaxf(m, lse_of(j0 == 0 ? slot : slot_of(place(q0, nr, j0 + gl)), sb));
#pragma unroll
      for (int o = LPR / 2; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    }
    for (int sb = 0; sb < c.nsub; ++sb) {
      for (int j0 = 0; j0 < n_warp; j0 += LPR) {
        const uint32_t s = j0 == 0 ? slot : slot_of(place(q0, nr, j0 + gl));
        float w = 1.f;
        if (FWD) {
          if (sb > 0 || j0 > 0) l = lse_of(s, sb);
          w = (s != kNoSlot && m > -CUDART_INF_F) ? __expf(l - m) : 0.f;
        }
#pragma unroll
        for (int b0 = 0; b0 < LPR; b0 += B) {
          if (j0 + b0 >= n_warp) break;         // warp-uniform
          if (sb > 0 || j0 > 0 || b0 > 0) request(s, sb, b0, x);
#pragma unroll
          for (int k = 0; k < B; ++k) {
            float f[8];
            unpack8<T>(x[k], f);
            if (FWD) {
              const float wk = __shfl_sync(0xffffffffu, w, b0 + k, LPR);
              ssum += wk;
#pragma unroll
              for (int e = 0; e < 8; ++e) acc[e] = fmaf(wk, f[e], acc[e]);
            } else {
#pragma unroll
              for (int e = 0; e < 8; ++e) acc[e] += f[e];
            }
          }
        }
      }
    }
    if (FWD) l_n = lse_of(slot_of(next), 0);
    if (FWD) {
      const float inv = ssum > 0.f ? 1.f / ssum : 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] *= inv;
    }
    const uint4 u = merged_chunk(pack8<T>(acc), gl);
    if (rid < n_rows) {
      const int hr = (int)(rid / c.total_q);
      const int64_t t = rid - (int64_t)hr * c.total_q;
      if (FWD) {
        if (gl == 0) lse[(int64_t)c.h0 * c.total_q + rid] = ssum > 0.f ? m + logf(ssum) : CUDART_INF_F;
      }
      *reinterpret_cast<uint4*>(out + t * rs + (int64_t)(c.h0 + hr) * hs + merged_place(gl) * 8) = u;
    }
  }
}

// The same merge for the builder's own lists of up to eight places, in one plane: the partials come by cp.async through a lane's own
// places in shared memory, the next row's requested before this one's are waited for, so that a warp has up to 8 KB on the way and
// the registers of one row.  Same sums in the same order.  Bound: HBM, 6.2 - 6.5 TB/s of partials at 64K tokens x 32 heads.
constexpr int kMergeStages = 2, kMergeStage = 32 * kMergeBatch * 16, kMergeSmem = kMergeThreads / 32 * kMergeStages * kMergeStage;
template <typename T, int D, bool FWD>
__global__ void __launch_bounds__(kMergeThreads, 3) merge_staged_kernel(const T* part, const float* part_lse, MergeParams c, T* out, int64_t rs,
                                                                     int64_t hs, float* lse) {
  constexpr int LPR = D / 8, RPW = 32 / LPR;
  follow_on();
  if (c.mirror != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *c.mirror = *c.status;   // (the main kernel has completed)
  extern __shared__ __align__(16) unsigned char merge_smem[];
  const int lane = threadIdx.x & 31, gl = lane % LPR;
  const uint32_t mine = (uint32_t)__cvta_generic_to_shared(merge_smem) + (threadIdx.x >> 5) * (kMergeStages * kMergeStage) + lane * 16;
  const int64_t n_rows = c.total_q * c.nh, stride = (int64_t)gridDim.x * (kMergeThreads / 32) * RPW;
  int64_t row = ((int64_t)blockIdx.x * (kMergeThreads / 32) + (threadIdx.x >> 5)) * RPW + lane / LPR;
  int64_t t;
  T* to;
  {
    const int64_t h = row / c.total_q;
    t = row - h * c.total_q;
    to = out + (c.h0 + h) * hs + merged_place(gl) * 8;
  }
  auto fetch = [&](int64_t r) { return r < n_rows && gl < c.fixed_k ? c.row_pos[r * c.fixed_k + gl] : kNoSlot; };
  // a place's content -> slot of the pass (kNoSlot also for what is none)
  auto slot_of = [&](uint32_t x) {
    const uint32_t at = x - (uint32_t)c.slot_shift;
    return x != kNoSlot && at < c.cap ? at : kNoSlot;
  };
  auto request = [&](uint32_t s, uint32_t stage) {
#pragma unroll
    for (int k = 0; k < kMergeBatch; ++k) {
      const uint32_t sk = __shfl_sync(0xffffffffu, s, k, LPR);
      const bool ok = sk != kNoSlot;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(mine + stage * kMergeStage + k * 512),
                   "l"(part + (int64_t)(ok ? sk : 0u) * D + gl * 8), "r"(ok ? 16u : 0u) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto lse_of = [&](uint32_t s) { return FWD && s != kNoSlot ? part_lse[s] : -CUDART_INF_F; };
  uint32_t slot = slot_of(fetch(row));
  float l = lse_of(slot);
  request(slot, 0);
  uint32_t next = fetch(row + stride), stage = 0;
#pragma unroll 1
  for (int64_t first = row - lane / LPR; first < n_rows; first += stride, row += stride) {
    const uint32_t s1 = slot_of(next);
    const float l1 = lse_of(s1);
    request(s1, stage ^ 1u);
    next = fetch(row + 2 * stride);
    float w = 1.f, m = l, ssum = 0.f, acc[8];
    if (FWD) {
#pragma unroll
      for (int o = kMergeBatch / 2; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));   // (lanes 0 - 7 of the row hold its list)
      w = slot != kNoSlot && m > -CUDART_INF_F ? __expf(l - m) : 0.f;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    asm volatile("cp.async.wait_group 1;" ::: "memory");   // (a lane reads back what it copied itself)
#pragma unroll
    for (int k = 0; k < kMergeBatch; ++k) {
      uint4 x;
      asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(mine + stage * kMergeStage + k * 512) : "memory");
      float f[8];
      unpack8<T>(x, f);
      if (FWD) {
        const float wk = __shfl_sync(0xffffffffu, w, k, LPR);
        ssum += wk;
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = fmaf(wk, f[e], acc[e]);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += f[e];
      }
    }
    if (FWD) {
      const float inv = ssum > 0.f ? 1.f / ssum : 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] *= inv;
      if (gl == 0 && row < n_rows) lse[(int64_t)c.h0 * c.total_q + row] = ssum > 0.f ? m + logf(ssum) : CUDART_INF_F;
    }
    const uint4 u = merged_chunk(pack8<T>(acc), gl);
    if (row < n_rows) *reinterpret_cast<uint4*>(to + t * rs) = u;
    for (t += stride; t >= c.total_q; t -= c.total_q) to += hs;
    slot = s1;
    l = l1;
    stage ^= 1u;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// D[h, t] = sum_d dO.O.  LPR = d / 8 lanes per row, each with one 16-byte load of dO and of O.  A thread's kDotRows rows are
// all in flight, and their tokens and heads follow from the first row's by counting: a 64-bit division per row made the
// kernel an arithmetic one.  Bound: HBM.  The first CTA also clears the call's status block, which the main kernel needs.
// Measured (B200, 64K tokens x 32 heads, d 128, 1.07 GB): one row and a division per thread 227 us, two rows 171 us
// (6.3 TB/s), four 204 us; d 256, 16K tokens x 16 heads 53 / 35 us.
constexpr int kDotRows = 2;
template <typename T, int LPR>
__global__ void __launch_bounds__(256) dot_do_o_kernel(const T* dout, int64_t do_rs, int64_t do_hs,
                                                       const T* o, int64_t o_rs, int64_t o_hs,
                                                       float* softmax_d, int64_t total_q, int heads, int* status) {
  constexpr int RPW = 32 / LPR;                  // rows of a warp at a time
  follow_on();
  if (blockIdx.x == 0 && threadIdx.x < kStatusBytes / 4) status[threadIdx.x] = 0;
  const int lane = threadIdx.x & 31, c = (lane % LPR) * 8;
  const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t row0 = wid * (RPW * kDotRows) + lane / LPR;   // rows in memory order: token, head
  int64_t t = row0 < 0x80000000ll ? (int64_t)((uint32_t)row0 / (uint32_t)heads) : row0 / heads;
  int h = (int)(row0 - t * heads);
  uint4 a[kDotRows], b[kDotRows];
  float* dst[kDotRows];
#pragma unroll
  for (int i = 0; i < kDotRows; ++i) {
    a[i] = b[i] = make_uint4(0, 0, 0, 0);
    dst[i] = nullptr;
    if (t < total_q) {
      a[i] = ldg_16(dout + t * do_rs + (int64_t)h * do_hs + c);
      b[i] = ldg_16(o + t * o_rs + (int64_t)h * o_hs + c);
      dst[i] = softmax_d + (int64_t)h * total_q + t;
    }
    for (h += RPW; h >= heads; h -= heads) ++t;
  }
#pragma unroll
  for (int i = 0; i < kDotRows; ++i) {
    float s = 0.f, x[8], y[8];
    unpack8<T>(a[i], x);
    unpack8<T>(b[i], y);
#pragma unroll
    for (int e = 0; e < 8; ++e) s = fmaf(x[e], y[e], s);
#pragma unroll
    for (int o2 = LPR / 2; o2; o2 >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o2);
    if (dst[i] != nullptr && lane % LPR == 0) *dst[i] = s;
  }
}

int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
    n = 148;
  return n;
}

template <typename T, int D, bool FWD>
static int merge_launch(const AttnArgs& a, const AttnWorkspace& w, const PassParams& ps, cudaStream_t s) {
  MergeParams c;
  c.row_ptr = w.row_ptr; c.row_pos = w.row_pos; c.total_q = a.total_q; c.cap = w.cap;
  c.h0 = ps.h0; c.nh = ps.nh; c.nsub = w.nsub;
  c.fixed_k = w.fixed_k;
  c.slot_shift = ps.slot_shift;
  if (w.fixed_k > 0) c.row_pos = w.row_pos + (int64_t)ps.h0 * a.total_q * w.fixed_k;   // the pass's heads
  c.status = w.status;
  c.mirror = (ps.h0 + ps.nh >= a.heads) ? w.mirror : nullptr;   // the call's last pass
  // persistent CTAs, as many as are resident
  const int64_t ctas = ceil_div64(a.total_q * ps.nh, (kMergeThreads / 32) * (32 / (D / 8))), most = (int64_t)sm_count() * 3;
  const unsigned grid = (unsigned)(ctas < most ? ctas : most);
  // Where the staged kernel is the better one: head dims of 128 and more; dQ, whose merge has less to do per row, from about a gigabyte of
  // partials on where lists are of eight, far earlier where they are shorter (a row's places are a smaller part of its work); the line lies
  // where lists of eight lose little.  dQ, from registers / staged, us: top-k 8, 234 MB 43.4 / 45.7, 402 MB 74.5 / 78.5, 537 MB 101 / 103, 671 MB
  // 125 / 127, 1.07 GB 201 / 199; d 256, 524 MB 167 / 166, 1.07 GB 344 / 342; top-k 6, 402 MB 81 / 78, 537 MB 106 / 105; top-k 4, 268 MB 74 / 64, 537
  // MB 141 / 114, 1.07 GB 281 / 219.  All: 64K tokens x 32 heads, d 128, top-k 8 828 / 780 forward, 790 / 750 backward; 8 x 8K 805 / 738
  // and 751 / 723; 32K x 16 213 / 207 and 202 / 202; 3.6K x 32 (235 MB) 51.7 / 47.6 and 43.5 / 47; d 64, 32K x 16 111 / 113 and 109 / 110.  Lists of 16, or
  // of two planes, with a staged kernel of several steps a row: 317K tokens 6.97 / 7.66 ms, 512K x 4 2.95 / 3.23.
  if constexpr (D >= 128) {
    if (c.fixed_k > 0 && c.fixed_k <= kMergeBatch && c.nsub == 1 &&
        (FWD || a.total_q * ps.nh * c.fixed_k * D * (int64_t)sizeof(T) >= (int64_t)1 << 29)) {
      auto kern = merge_staged_kernel<T, D, FWD>;
      FMB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMergeSmem));
      if (FWD) kern<<<grid, kMergeThreads, kMergeSmem, s>>>((const T*)w.part_o, w.part_lse, c, (T*)const_cast<void*>(a.o), a.o_rs, a.o_hs, a.lse);
      else kern<<<grid, kMergeThreads, kMergeSmem, s>>>((const T*)w.part_o, nullptr, c, (T*)a.dq, a.dq_rs, a.dq_hs, nullptr);
      FMB_LAUNCH_CHECK("merge_staged_kernel");
      return FMB_OK;
    }
  }
  // An ordinary launch: brought up early, on whatever SMs the kernel before leaves first, the CTAs would spread unevenly, and each
  // has its fixed share of the rows (64K tokens x 32 heads: a step 4 % slower)
  if (FWD) merge_kernel<T, D, true><<<grid, kMergeThreads, 0, s>>>((const T*)w.part_o, w.part_lse, c, (T*)const_cast<void*>(a.o), a.o_rs, a.o_hs, a.lse);
  else merge_kernel<T, D, false><<<grid, kMergeThreads, 0, s>>>((const T*)w.part_o, nullptr, c, (T*)a.dq, a.dq_rs, a.dq_hs, nullptr);
  FMB_LAUNCH_CHECK(FWD ? "merge_kernel<fwd>" : "merge_kernel<bwd>");
  return FMB_OK;
}
template <bool FWD>
static int launch_merge(const AttnArgs& a, const AttnWorkspace& w, const PassParams& ps, cudaStream_t s) {
  if (a.total_q * ps.nh == 0) return FMB_OK;
  const bool bf = a.dtype == FMB_BF16;
#define FMB_MERGE(D_) return bf ? merge_launch<__nv_bfloat16, D_, FWD>(a, w, ps, s) : merge_launch<__half, D_, FWD>(a, w, ps, s)
  if (a.d == 64) FMB_MERGE(64);
  if (a.d == 128) FMB_MERGE(128);
  if (a.d == 256) FMB_MERGE(256);
#undef FMB_MERGE
  return fail(FMB_ERR_UNSUPPORTED, "attention: head_dim %d not built (64, 128 or 256)", a.d);
}
int launch_fwd_combine(const AttnArgs& a, const AttnWorkspace& w, const PassParams& ps, cudaStream_t s) { return launch_merge<true>(a, w, ps, s); }
int launch_bwd_combine(const AttnArgs& a, const AttnWorkspace& w, const PassParams& ps, cudaStream_t s) { return launch_merge<false>(a, w, ps, s); }

template <typename T>
static int dot_do_o_dispatch(const AttnArgs& a, int* status, cudaStream_t s) {
  const int64_t rows = a.total_q * a.heads;
  const T* dout = (const T*)a.dout;
  const T* o = (const T*)a.o;
#define FMB_DOT(LPR_)                                                                                                \
  launch_follow_on(dot_do_o_kernel<T, LPR_>, dim3((unsigned)ceil_div64(rows, 8 * (32 / LPR_) * kDotRows)), dim3(256), 0, s, \
                   dout, a.do_rs, a.do_hs, o, a.o_rs, a.o_hs, a.softmax_d, a.total_q, a.heads, status)
  if (a.d == 128) FMB_DOT(16);
  else if (a.d == 64) FMB_DOT(8);
  else if (a.d == 256) FMB_DOT(32);
  else return fail(FMB_ERR_UNSUPPORTED, "attention: head_dim %d not built (64, 128 or 256)", a.d);
#undef FMB_DOT
  FMB_LAUNCH_CHECK("dot_do_o_kernel");
  return FMB_OK;
}

// also clears the call's status block
static int launch_dot_do_o(const AttnArgs& a, int* status, cudaStream_t s) {
  if (a.total_q * a.heads == 0) {
    FMB_CUDA(cudaMemsetAsync(status, 0, kStatusBytes, s));
    return FMB_OK;
  }
  return a.dtype == FMB_BF16 ? dot_do_o_dispatch<__nv_bfloat16>(a, status, s) : dot_do_o_dispatch<__half>(a, status, s);
}

// ------------------------------------------------------------------ drivers
// Each pass: slot and row lists of its heads, main kernel (partials), combine.  The status block
// is cleared once per call, so a failure in any pass stays visible.
static int check_pass_sizes(const char* op, const AttnArgs& a, const AttnWorkspace& w, size_t need_one_group) {
  if (a.ws == nullptr || a.ws_bytes < w.bytes)
    return fail(FMB_ERR_WORKSPACE, "%s: workspace too small (%zu bytes given; a pass over one kv-head group needs %zu)",
                op, a.ws_bytes, need_one_group);
  if ((int64_t)w.nsub * w.cap >= (int64_t)0xffffffffll)
    return fail(FMB_ERR_BAD_ARG, "%s: too many partial slots in one pass; give a smaller workspace", op);
  return FMB_OK;
}

// ------------------------------------------------------------------ rows handed over by the pattern builder
struct RowsTicket {
  const uint32_t* rows; int64_t total_q; int heads, topk; bool armed;
};
static thread_local RowsTicket g_rows = {nullptr, 0, 0, 0, false};

void attn_rows_offer(const uint32_t* row_slots, int64_t total_q, int heads, int topk) {
  g_rows = RowsTicket{row_slots, total_q, heads, topk, row_slots != nullptr && topk > 0};
}
// Consumes the ticket; true if this call (matching geometry; one pass over all heads, or a single
// sequence, whose heads lie one after the other in `indices`) runs on it: slots are positions in
// `indices` (less the pass's first), the row lists are the builder's.
static bool take_rows(const AttnArgs& a, AttnWorkspace& w) {
  const RowsTicket t = g_rows;
  g_rows.armed = false;
  w.fixed_k = 0;
  if (!t.armed || t.total_q != a.total_q || t.heads != a.heads || (w.nh < a.heads && a.batch != 1) ||
      (int64_t)t.total_q * t.heads * t.topk != a.n_indices || a.n_indices >= (int64_t)0xffffffffll)
    return false;
  w.fixed_k = t.topk;
  w.row_pos = const_cast<uint32_t*>(t.rows);
  w.slot_base = nullptr;
  return true;
}

// ------------------------------------------------------------------ status word mirrored for the host
static thread_local int* g_mirror = nullptr;
void attn_status_mirror(int* mirror) { g_mirror = mirror; }
static int* take_mirror() {
  int* m = g_mirror;
  g_mirror = nullptr;
  return m;
}

__global__ void clear_status_kernel(int* status) {
  follow_on();
  status[threadIdx.x] = 0;
}

int launch_attn_fwd(const AttnArgs& a, int engine, cudaStream_t s) {
  AttnWorkspace w = carve_attn_workspace(a.ws, a.ws_bytes, a, 2, true, 0);
  w.mirror = take_mirror();
  int rc = check_pass_sizes("attn_fwd", a, w, w.bytes);
  if (rc) return rc;
  const bool rows_given = take_rows(a, w);
  // A kernel in place of a memset, which would wait its turn and make the kernel behind wait (a training step of 3K tokens x
  // 8 heads, d 64 107.2 / 103.2 us, 3.6K new rows behind 66K cached keys 280 / 266 us with the memset / with it).  The backward's dO.O does it on the way.
  launch_follow_on(clear_status_kernel, dim3(1), dim3(kStatusBytes / 4), 0, s, w.status);
  FMB_LAUNCH_CHECK("clear_status_kernel");
  for (int h0 = 0; h0 < a.heads; h0 += w.nh) {
    const PassParams ps = make_pass(a, w, h0, min(w.nh, a.heads - h0));
    if (!rows_given && (rc = build_row_lists(a, w, ps, s))) return rc;
    prof_begin(0, s);
    if (engine == 1 && tc_supported(a, false)) rc = launch_fwd_main_tc(a, w, ps, s);
    else if (engine == 1 && tc_wide_supported(a, false)) rc = launch_fwd_main_tc_wide(a, w, ps, s);
    else rc = launch_fwd_main_simt(a, w, ps, s);
    prof_end(0, s);
    if (rc) return rc;
    prof_begin(4, s);
    rc = launch_fwd_combine(a, w, ps, s);
    prof_end(4, s);
    if (rc) return rc;
  }
  return FMB_OK;
}

// ------------------------------------------------------------------ lists handed from forward to backward
struct ListsTicket {
  const void* ws; int64_t total_q, n_indices; int heads, batch, ncol, chunk; bool armed;
};
static thread_local ListsTicket g_ticket = {nullptr, 0, 0, 0, 0, 0, 0, false};

size_t attn_lists_bytes(const AttnArgs& a) {
  return carve_attn_workspace(nullptr, 0, a, 2, false, a.heads).lists_bytes;
}
int attn_lists_save(const AttnArgs& a, void* dst, size_t dst_bytes, cudaStream_t s) {
  const AttnWorkspace w = carve_attn_workspace(a.ws, a.ws_bytes, a, 2, true, 0);
  if (a.ws == nullptr || a.ws_bytes < w.bytes || w.nh < a.heads) return 1;
  if (dst == nullptr || dst_bytes < w.lists_bytes)
    return fail(FMB_ERR_WORKSPACE, "attn_lists_save: buffer too small (%zu bytes given, %zu needed)", dst_bytes,
                w.lists_bytes);
  FMB_CUDA(cudaMemcpyAsync(dst, static_cast<const char*>(a.ws) + w.lists_off, w.lists_bytes,
                           cudaMemcpyDeviceToDevice, s));
  return FMB_OK;
}
int attn_lists_load(const AttnArgs& a, const void* src, size_t src_bytes, cudaStream_t s) {
  const AttnWorkspace w = carve_attn_workspace(a.ws, a.ws_bytes, a, 2, false, 0);
  if (a.ws == nullptr || a.ws_bytes < w.bytes || w.nh < a.heads) return 1;
  if (src == nullptr || src_bytes < w.lists_bytes)
    return fail(FMB_ERR_WORKSPACE, "attn_lists_load: buffer too small (%zu bytes given, %zu needed)", src_bytes,
                w.lists_bytes);
  FMB_CUDA(cudaMemcpyAsync(static_cast<char*>(a.ws) + w.lists_off, src, w.lists_bytes, cudaMemcpyDeviceToDevice, s));
  g_ticket = ListsTicket{a.ws, a.total_q, a.n_indices, a.heads, a.batch, a.ncol, a.chunk, true};
  return FMB_OK;
}

void attn_offers_end(bool backward) {
  g_rows.armed = false;
  g_mirror = nullptr;
  if (backward) g_ticket.armed = false;
}

int launch_attn_bwd(const AttnArgs& a, int engine, cudaStream_t s) {
  AttnWorkspace w = carve_attn_workspace(a.ws, a.ws_bytes, a, 2, false, 0);
  w.mirror = take_mirror();
  int rc = check_pass_sizes("attn_bwd", a, w, w.bytes);
  if (rc) return rc;
  // lists loaded into this very workspace for this very problem, one pass: no build of our own
  const bool lists_given = g_ticket.armed && g_ticket.ws == a.ws && g_ticket.total_q == a.total_q &&
                           g_ticket.n_indices == a.n_indices && g_ticket.heads == a.heads &&
                           g_ticket.batch == a.batch && g_ticket.ncol == a.ncol && g_ticket.chunk == a.chunk &&
                           w.nh >= a.heads;
  g_ticket.armed = false;
  const bool rows_given = take_rows(a, w);
  prof_begin(7, s);
  rc = launch_dot_do_o(a, w.status, s);
  prof_end(7, s);
  if (rc) return rc;
  for (int h0 = 0; h0 < a.heads; h0 += w.nh) {
    const PassParams ps = make_pass(a, w, h0, min(w.nh, a.heads - h0));
    if (!lists_given && !rows_given && (rc = build_row_lists(a, w, ps, s))) return rc;
    prof_begin(1, s);
    if (engine == 1 && tc_supported(a, true)) rc = launch_bwd_main_tc(a, w, ps, s);
    else if (engine == 1 && tc_wide_supported(a, true)) rc = launch_bwd_main_tc_wide(a, w, ps, s);
    else rc = launch_bwd_main_simt(a, w, ps, s);
    prof_end(1, s);
    if (rc) return rc;
    prof_begin(5, s);
    rc = launch_bwd_combine(a, w, ps, s);
    prof_end(5, s);
    if (rc) return rc;
  }
  return FMB_OK;
}

}  // namespace fmb
