// Host path of the PyTorch front end, in C++: argument checks, output and workspace allocation, the
// pattern -> attention hand-over, the autograd node.  Everything below it is the C ABI
// (include/flash_moba_b200.h); nothing here computes on tensors.
//
// Why native: a step is eleven kernel launches, and at small sizes (a few thousand tokens, a decode
// step) the kernels need 0.06-0.15 ms while the same host path in Python (ctypes calls of forty
// arguments, an autograd Function, two recorded events per attention call, a cache keyed by tuples)
// needed 0.25 ms per forward call and 0.5-0.6 ms per training step.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/extension.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <optional>
#include <thread>
#include <tuple>

#include "../../include/flash_moba_b200.h"
#include "fmb_status_ring.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

void check(int rc) {
  if (rc == FMB_OK) return;
  const char* msg = fmb_last_error();
  if (msg == nullptr || msg[0] == 0) TORCH_CHECK(false, "flash_moba_b200 error ", rc);
  TORCH_CHECK(false, msg);
}

bool env_is(const char* name, const char* unset, const char* value) {
  const char* e = std::getenv(name);
  return std::strcmp(e ? e : unset, value) == 0;
}
bool check_status_now() { return env_is("FMB_CHECK_STATUS", "0", "1"); }
bool share_lists() { return !env_is("FMB_SHARE_LISTS", "1", "0"); }

int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kBFloat16) return FMB_BF16;
  if (t.scalar_type() == at::kHalf) return FMB_FP16;
  TORCH_CHECK(false, "FlashMoBA only supports fp16 and bf16 data type");
}
void require_cuda(const Tensor& t) {
  TORCH_CHECK(t.is_cuda(), "flash_moba_b200: all tensors must be on a CUDA device (there is no CPU path)");
}
void last_contig(const Tensor& t, const char* name) {
  TORCH_CHECK(t.dim() == 3, name, " must have shape (tokens, heads, head_dim)");
  TORCH_CHECK(t.stride(-1) == 1, name, " must have contiguous last dimension");
}
const int32_t* i32c(const Tensor& t, const char* name) {
  TORCH_CHECK(t.scalar_type() == at::kInt, name, " must have dtype int32");
  TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
  return static_cast<const int32_t*>(t.data_ptr());
}
Tensor fix_last_stride(const Tensor& t) { return t.stride(-1) != 1 ? t.contiguous() : t; }
fmb_stream_t current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }
Tensor bytes_on(const Tensor& like, size_t n) {
  return at::empty({(int64_t)(n > 0 ? n : 1)}, like.options().dtype(at::kByte));
}

// ---------------------------------------------------------------------------- status words
// Every attention call leaves a device-side status word: 0, or which bounded wait gave up / 7 = the
// pattern did not fit the slots.  The library stores it straight into mapped pinned memory
// (fmb_attn_status_mirror) at the end of the call; the calls that follow look which words have
// arrived, without synchronising and without an event.  A failure is therefore raised one call late, never
// silently.  With FMB_CHECK_STATUS=1 every call synchronises and raises at once.
fmb::StatusRing& ring() {
  static fmb::StatusRing* r = [] {              // never destroyed: kernels may still write to it at exit
    void* p = nullptr;
    C10_CUDA_CHECK(cudaHostAlloc(&p, fmb::StatusRing::kSlots * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped));
    return new fmb::StatusRing(static_cast<volatile int*>(p));
  }();
  return *r;
}

void raise_for_status(int code, const char* what) {
  TORCH_CHECK(code != 7, "flash_moba_b200: ", what,
              ": the pattern does not fit the slots of a pass (overlapping columns, or raise FMB_WORKSPACE_GB)");
  TORCH_CHECK(code == 0, "flash_moba_b200: ", what, ": a bounded device-side wait expired (code ", code, ")");
}
void collect_status() {
  const fmb::StatusRing::Failure f = ring().collect();
  raise_for_status(f.code, f.what);
}

bool capturing() {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  C10_CUDA_CHECK(cudaStreamIsCapturing((cudaStream_t)current_stream(), &cap));
  return cap != cudaStreamCaptureStatusNone;
}

// A moment's rest while words are awaited: the words alone, no stream or device is waited for.  After a device
// error no word will come: the device's stream is asked for one.
void await_words(int device) {
  std::this_thread::sleep_for(std::chrono::microseconds(20));
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  if (capturing()) return;
  c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);   // (other threads may be capturing)
  const cudaError_t e = cudaStreamQuery((cudaStream_t)current_stream());
  if (e != cudaErrorNotReady) C10_CUDA_CHECK(e);
}

void check_pending_status() {
  const uint64_t bound = ring().now();
  for (;;) {
    collect_status();
    const int device = ring().outstanding(bound);
    if (device < 0) return;
    await_words(device);
  }
}

// The status word of the call about to be made.  Not mirrored if it is checked by synchronising, or if the stream is
// being captured into a graph, whose replays no host code looks at.
class StatusTicket {
 public:
  StatusTicket(const char* what, const Tensor& q, bool runs) : what_(what), runs_(runs) {
    if (!runs || check_status_now() || capturing()) return;
    const int device = q.device().index();
    for (;;) {
      collect_status();
      slot_ = ring().claim(what, device);
      if (slot_ >= 0) break;
      await_words(device);                      // 256 calls ahead of the GPU
    }
    check(fmb_attn_status_mirror(const_cast<int*>(ring().word(slot_))));
  }
  ~StatusTicket() {
    if (slot_ >= 0) ring().withdraw(slot_);     // the call was not made or failed
  }
  StatusTicket(const StatusTicket&) = delete;
  // the call has been made and returned rc
  void end(int rc, const Tensor& ws) {
    check(rc);
    if (slot_ >= 0) {
      ring().launched(slot_);
      slot_ = -1;
    } else if (runs_ && check_status_now()) {
      int code = 0;
      C10_CUDA_CHECK(cudaMemcpyAsync(&code, ws.data_ptr(), sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)current_stream()));
      C10_CUDA_CHECK(cudaStreamSynchronize((cudaStream_t)current_stream()));
      raise_for_status(code, what_);
    }
  }

 private:
  const char* what_;
  bool runs_;
  int slot_ = -1;
};

// ---------------------------------------------------------------------------- stages P, G, O/E/S
std::tuple<Tensor, Tensor> mean_pool(const Tensor& k, const Tensor& cu_k, int64_t max_k, int64_t chunk) {
  require_cuda(k);
  require_cuda(cu_k);
  last_contig(k, "k");
  const int32_t* cu = i32c(cu_k, "cu_seqlens_k");
  const int64_t total_k = k.size(0), hk = k.size(1), d = k.size(2), batch = cu_k.numel() - 1;
  TORCH_CHECK(chunk > 0, "mean_pool: chunk must be positive");
  c10::cuda::CUDAGuard guard(k.device());
  // no host sync: an upper bound of rows; rows [0, cu_seqlens_km[-1]) are valid
  Tensor km = at::empty({(total_k + chunk - 1) / chunk + batch, hk, d}, k.options());
  Tensor cu_km = at::empty({batch + 1}, k.options().dtype(at::kInt));
  check(fmb_mean_pool_offsets(k.data_ptr(), k.stride(0), k.stride(1), cu, static_cast<int32_t*>(cu_km.data_ptr()),
                              km.data_ptr(), (int)batch, (int)hk, (int)d, (int)max_k, (int)chunk, dtype_code(k),
                              current_stream()));
  return {km, cu_km};
}

// (lists as a head-major (H, T, K) buffer, scores in the same layout or undefined)
std::tuple<Tensor, OptTensor> gate_topk(const Tensor& q, const Tensor& km, const Tensor& cu_q, const Tensor& cu_k,
                                        const Tensor& cu_km, int64_t max_q, int64_t max_k, int64_t topk, int64_t chunk,
                                        bool causal, bool return_values) {
  require_cuda(q);
  require_cuda(km);
  last_contig(q, "q");
  TORCH_CHECK(km.is_contiguous(), "km must be contiguous");
  const int64_t total_q = q.size(0), h = q.size(1), d = q.size(2), hk = km.size(1), batch = cu_q.numel() - 1;
  c10::cuda::CUDAGuard guard(q.device());
  Tensor idx = at::empty({h, total_q, topk}, q.options().dtype(at::kInt));
  OptTensor val;
  if (return_values) val = at::empty({h, total_q, topk}, q.options().dtype(at::kFloat));
  check(fmb_gate_topk_sized(q.data_ptr(), q.stride(0), q.stride(1), total_q, km.data_ptr(), km.size(0), i32c(cu_q, "cu_seqlens_q"),
                      i32c(cu_k, "cu_seqlens_k"), i32c(cu_km, "cu_seqlens_km"), static_cast<int32_t*>(idx.data_ptr()),
                      val ? static_cast<float*>(val->data_ptr()) : nullptr, topk, total_q * topk, (int)batch, (int)h, (int)hk,
                      (int)d, (int)max_q, (int)max_k, (int)topk, (int)chunk, causal ? 1 : 0, dtype_code(q),
                      current_stream()));
  if (check_status_now()) {
    int code = 0;
    check(fmb_gate_status(&code));
  }
  return {idx, val};
}

struct Pattern {
  Tensor col_offsets, col_nnz, indices;
  OptTensor row_slots;       // where every (row, j-th chunk) pair landed in `indices`
  int64_t topk = 0;
};

// idx: (T, H, K) view with contiguous last dimension.  keep_rows: also the row-major view (only for
// lists that name a chunk at most once per row, as the lists of gate_topk do)
Pattern build_csc(const Tensor& idx, const Tensor& cu_q, int64_t max_q, int64_t ncol, bool keep_rows) {
  require_cuda(idx);
  TORCH_CHECK(idx.dim() == 3 && idx.scalar_type() == at::kInt && idx.stride(-1) == 1,
              "topk_idx must be int32 with contiguous last dimension");
  const int64_t total_q = idx.size(0), h = idx.size(1), topk = idx.size(2), batch = cu_q.numel() - 1;
  const int32_t* cu = i32c(cu_q, "cu_seqlens_q");
  c10::cuda::CUDAGuard guard(idx.device());
  Pattern p;
  p.topk = topk;
  p.col_offsets = at::empty({batch, h, ncol}, idx.options().dtype(at::kLong));
  p.col_nnz = at::empty({batch, h, ncol}, idx.options());
  p.indices = at::empty({total_q * h * topk}, idx.options());
  const size_t nbytes = fmb_build_csc_workspace_bytes((int)batch, (int)h, (int)max_q, (int)ncol);
  Tensor ws = bytes_on(idx, nbytes);
  auto* idxp = static_cast<const int32_t*>(idx.data_ptr());
  auto* co = static_cast<int64_t*>(p.col_offsets.data_ptr());
  auto* cn = static_cast<int32_t*>(p.col_nnz.data_ptr());
  auto* in = static_cast<int32_t*>(p.indices.data_ptr());
  if (keep_rows && share_lists() && p.indices.numel() > 0 && p.indices.numel() < 0xffffffffll) {
    p.row_slots = at::empty({h, total_q, topk}, idx.options());
    check(fmb_build_csc_rows(idxp, idx.stride(0), idx.stride(1), cu, co, cn, in,
                             static_cast<uint32_t*>(p.row_slots->data_ptr()), ws.data_ptr(), nbytes, (int)batch, (int)h,
                             (int)topk, total_q, (int)max_q, (int)ncol, current_stream()));
  } else {
    check(fmb_build_csc(idxp, idx.stride(0), idx.stride(1), cu, co, cn, in, ws.data_ptr(), nbytes, (int)batch, (int)h,
                        (int)topk, (int)max_q, (int)ncol, current_stream()));
  }
  return p;
}

// ---------------------------------------------------------------------------- rows of known patterns
// A pattern that a caller took from flash_topk_varlen_func and hands to flash_moba_attn_varlen_func
// is recognised by its storage, so that the attention calls on it build no lists of their own.  An
// entry lives only as long as the pattern's `indices` do (weak references); an in-place write to a
// pattern tensor changes its version and misses.  The rows hold places that follow from the sequences'
// bounds, so these are part of the key.  Inference tensors have no version, so that a write to one could not
// be seen: patterns of such tensors are not remembered.  At most kKnown entries, beside those that a captured
// graph reads: these stay as long as the pattern, which the graph's owner has to keep, does.
struct TensorId {
  const void* ptr = nullptr;
  int64_t numel = 0;
  uint32_t version = 0;
  explicit TensorId(const Tensor& t) : ptr(t.data_ptr()), numel(t.numel()), version(t._version()) {}
  TensorId() = default;
  bool operator==(const TensorId& o) const { return ptr == o.ptr && numel == o.numel && version == o.version; }
};
struct Known {
  TensorId id[4];
  c10::weak_intrusive_ptr<c10::StorageImpl> alive[4];
  Tensor row_slots;
  int64_t topk = 0;
  bool pinned = false;       // a graph reads row_slots
  Known(const Pattern& p, const Tensor& cu_q)
      : id{TensorId(p.col_offsets), TensorId(p.col_nnz), TensorId(p.indices), TensorId(cu_q)},
        alive{p.col_offsets.storage().getWeakStorageImpl(), p.col_nnz.storage().getWeakStorageImpl(),
              p.indices.storage().getWeakStorageImpl(), cu_q.storage().getWeakStorageImpl()},
        row_slots(*p.row_slots), topk(p.topk) {}
  bool expired() const { return alive[0].expired() || alive[1].expired() || alive[2].expired() || alive[3].expired(); }
};
constexpr size_t kKnown = 4;
std::mutex g_known_mu;
std::vector<Known>& known() {
  static auto* v = new std::vector<Known>();      // never destroyed: holds device memory
  return *v;
}
bool traceable(const Pattern& p, const Tensor& cu_q) {
  return !p.col_offsets.is_inference() && !p.col_nnz.is_inference() && !p.indices.is_inference() && !cu_q.is_inference();
}
void remember(const Pattern& p, const Tensor& cu_q) {
  if (!p.row_slots || !traceable(p, cu_q)) return;
  std::lock_guard<std::mutex> lock(g_known_mu);
  auto& v = known();
  v.erase(std::remove_if(v.begin(), v.end(), [](const Known& k) { return k.expired(); }), v.end());
  auto spare = [](const Known& k) { return !k.pinned; };
  if ((size_t)std::count_if(v.begin(), v.end(), spare) >= kKnown) v.erase(std::find_if(v.begin(), v.end(), spare));
  v.emplace_back(p, cu_q);
}
Pattern recall(const Tensor& co, const Tensor& cn, const Tensor& in, const Tensor& cu_q) {
  Pattern p;
  p.col_offsets = co; p.col_nnz = cn; p.indices = in;
  if (!traceable(p, cu_q)) return p;
  std::lock_guard<std::mutex> lock(g_known_mu);
  auto& v = known();
  v.erase(std::remove_if(v.begin(), v.end(), [](const Known& k) { return k.expired(); }), v.end());
  const TensorId a(co), b(cn), c(in), d(cu_q);
  for (Known& k : v)
    if (k.id[0] == a && k.id[1] == b && k.id[2] == c && k.id[3] == d) {
      k.pinned = k.pinned || capturing();
      p.row_slots = k.row_slots;
      p.topk = k.topk;
      break;
    }
  return p;
}

// ---------------------------------------------------------------------------- stages F and B
void check_pattern(const Pattern& p) {
  TORCH_CHECK(p.col_offsets.scalar_type() == at::kLong, "moba_col_offsets must have dtype torch.int64");
  TORCH_CHECK(p.col_nnz.scalar_type() == at::kInt, "moba_col_nnz must have dtype torch.int32");
  TORCH_CHECK(p.indices.scalar_type() == at::kInt, "moba_row_indices must have dtype torch.int32");
  TORCH_CHECK(p.col_offsets.is_contiguous(), "moba_col_offsets must be contiguous");
  TORCH_CHECK(p.col_nnz.is_contiguous(), "moba_col_nnz must be contiguous");
  TORCH_CHECK(p.indices.is_contiguous(), "moba_row_indices must be contiguous");
  TORCH_CHECK(p.col_offsets.dim() == 3 && p.col_offsets.sizes() == p.col_nnz.sizes(),
              "moba_col_offsets / moba_col_nnz must both be (batch, heads, ncol)");
}

// What is offered to the attention call that follows on this thread ends with this scope: an exception between the
// offer and the call must not leave it to the next call.
struct Offers {
  ~Offers() {
    fmb_attn_status_mirror(nullptr);
    fmb_attn_rows_offer(nullptr, 0, 0, 0);
    fmb_attn_key_spans(nullptr, nullptr);
  }
};

// offers the pattern builder's rows of this pattern to the attention call that follows on this thread
bool offer_rows(const Pattern& p, int64_t total_q, int64_t h) {
  if (!share_lists() || !p.row_slots || p.row_slots->numel() != total_q * h * p.topk ||
      p.indices.numel() != p.row_slots->numel())
    return false;
  // the rows may have been built on another stream; the caller, who never sees them, cannot say so
  c10::cuda::CUDACachingAllocator::recordStream(p.row_slots->storage().data_ptr(), c10::cuda::getCurrentCUDAStream());
  check(fmb_attn_rows_offer(static_cast<const uint32_t*>(p.row_slots->data_ptr()), total_q, (int)h, (int)p.topk));
  return true;
}

// Workspace for one attention call: the single-pass size if it fits the cap (FMB_WORKSPACE_GB, default
// 64 GiB), otherwise the largest pass of whole kv-head groups that does; the library then walks the
// heads in passes of that size.
using SizeFn = size_t (*)(int64_t, int, int, int, int64_t, int, int, int, int);
Tensor workspace(SizeFn query, const Tensor& q, int64_t hk, int64_t n_indices, int64_t batch, int64_t max_k, int64_t chunk,
                 size_t* nbytes) {
  const char* e = std::getenv("FMB_WORKSPACE_GB");
  const size_t cap = (size_t)((e ? std::atof(e) : 64.0) * 1073741824.0);
  const int h = (int)q.size(1), group = (int)(h / (hk > 0 ? hk : h));
  int nh = h;
  auto size = [&] {
    return query(q.size(0), h, (int)hk, (int)q.size(2), n_indices, (int)batch, (int)max_k, (int)chunk, nh);
  };
  size_t n = size();
  while (n > cap && nh > group) {
    nh = std::max(group, nh / 2 / group * group);
    n = size();
  }
  *nbytes = n;
  return bytes_on(q, n);
}

// (out (T, H, d), lse (H, T), the slot / row lists the call built if it had to build any in one pass)
std::tuple<Tensor, Tensor, OptTensor> attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Pattern& p,
                                               const Tensor& cu_q, const Tensor& cu_k, int64_t max_q, int64_t max_k,
                                               int64_t chunk, double scale, bool causal, const OptTensor& out_given,
                                               const OptTensor& k_begin, const OptTensor& k_end) {
  for (const Tensor* t : {&q, &k, &v, &p.col_offsets, &p.col_nnz, &p.indices}) require_cuda(*t);
  last_contig(q, "q");
  last_contig(k, "k");
  last_contig(v, "v");
  TORCH_CHECK(q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type(),
              "query, key and value must have the same dtype");
  check_pattern(p);
  TORCH_CHECK(chunk > 0, "lg_block_n must be positive");
  const int64_t total_q = q.size(0), h = q.size(1), d = q.size(2), hk = k.size(1), batch = cu_q.numel() - 1;
  TORCH_CHECK(p.col_offsets.size(0) == batch && p.col_offsets.size(1) == h, "pattern shape does not match (batch, heads)");
  const int64_t ncol = (max_k + chunk - 1) / chunk;
  TORCH_CHECK(p.col_offsets.size(2) == ncol, "pattern has ", p.col_offsets.size(2),
              " columns, expected ceil(max_seqlen_k/lg_block_n) = ", ncol);
  const int32_t* cuq = i32c(cu_q, "cu_seqlens_q");
  const int32_t* cuk = i32c(cu_k, "cu_seqlens_k");
  c10::cuda::CUDAGuard guard(q.device());
  Tensor out = out_given ? *out_given : at::empty_like(q);
  Tensor lse = at::empty({h, total_q}, q.options().dtype(at::kFloat));
  const int64_t n_indices = p.indices.numel();
  size_t nbytes = 0;
  Tensor ws = workspace(fmb_attn_fwd_workspace_bytes, q, hk, n_indices, batch, max_k, chunk, &nbytes);
  const bool runs = total_q > 0 && batch > 0;
  const Offers offers;
  StatusTicket ticket("attn_fwd", q, runs);
  const bool offered = offer_rows(p, total_q, h);
  if (k_begin && k_end)
    check(fmb_attn_key_spans(static_cast<const int32_t*>(k_begin->data_ptr()), static_cast<const int32_t*>(k_end->data_ptr())));
  const int rc = fmb_attn_fwd(
      q.data_ptr(), q.stride(0), q.stride(1), k.data_ptr(), k.stride(0), k.stride(1), v.data_ptr(), v.stride(0), v.stride(1),
      out.data_ptr(), out.stride(0), out.stride(1), static_cast<float*>(lse.data_ptr()),
      static_cast<const int64_t*>(p.col_offsets.data_ptr()), static_cast<const int32_t*>(p.col_nnz.data_ptr()),
      static_cast<const int32_t*>(p.indices.data_ptr()), n_indices, cuq, cuk, ws.data_ptr(), nbytes, (int)batch, (int)h, (int)hk,
      (int)d, total_q, (int)max_q, (int)max_k, (int)chunk, (float)scale, causal ? 1 : 0, dtype_code(q), current_stream());
  ticket.end(rc, ws);
  OptTensor lists;
  if (share_lists() && n_indices > 0 && runs && !offered) {
    const size_t nlist = fmb_attn_lists_bytes(total_q, (int)h, (int)hk, (int)d, n_indices, (int)batch, (int)max_k, (int)chunk);
    Tensor l = bytes_on(q, nlist);
    const int rs = fmb_attn_lists_save(ws.data_ptr(), nbytes, total_q, (int)h, (int)hk, (int)d, n_indices, (int)batch, (int)max_k,
                                       (int)chunk, l.data_ptr(), nlist, current_stream());
    if (rs == 0) lists = l;
    else if (rs != 1) check(rs);                    // 1: the call ran in several passes, nothing to keep
  }
  return {out, lse, lists};
}

// into dq, dk, dv; returns softmax_d (H, T)
Tensor attn_bwd(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
                const Tensor& dq, const Tensor& dk, const Tensor& dv, const Pattern& p, const Tensor& cu_q, const Tensor& cu_k,
                int64_t max_q, int64_t max_k, int64_t chunk, double scale, bool causal, const OptTensor& lists) {
  const std::pair<const Tensor*, const char*> all[] = {{&dout, "dout"}, {&q, "q"}, {&k, "k"}, {&v, "v"},
                                                       {&out, "out"}, {&dq, "dq"}, {&dk, "dk"}, {&dv, "dv"}};
  for (auto& [t, name] : all) {
    require_cuda(*t);
    last_contig(*t, name);
  }
  require_cuda(lse);
  check_pattern(p);
  const int64_t total_q = q.size(0), h = q.size(1), d = q.size(2), total_k = k.size(0), hk = k.size(1);
  const int64_t batch = cu_q.numel() - 1, n_indices = p.indices.numel();
  TORCH_CHECK(lse.scalar_type() == at::kFloat && lse.is_contiguous() && lse.dim() == 2 && lse.size(0) == h && lse.size(1) == total_q,
              "softmax_lse must be a contiguous float32 (heads, total_q) tensor");
  const int32_t* cuq = i32c(cu_q, "cu_seqlens_q");
  const int32_t* cuk = i32c(cu_k, "cu_seqlens_k");
  c10::cuda::CUDAGuard guard(q.device());
  Tensor softmax_d = at::empty({h, total_q}, q.options().dtype(at::kFloat));
  size_t nbytes = 0;
  Tensor ws = workspace(fmb_attn_bwd_workspace_bytes, q, hk, n_indices, batch, max_k, chunk, &nbytes);
  const bool runs = total_q > 0 && batch > 0;
  const Offers offers;
  StatusTicket ticket("attn_bwd", q, runs);
  if (!offer_rows(p, total_q, h) && lists && share_lists()) {
    const int rl = fmb_attn_lists_load(ws.data_ptr(), nbytes, total_q, (int)h, (int)hk, (int)d, n_indices, (int)batch, (int)max_k,
                                       (int)chunk, lists->data_ptr(), (size_t)lists->numel(), current_stream());
    if (rl != 0 && rl != 1) check(rl);
  }
  const int rc = fmb_attn_bwd(
      dout.data_ptr(), dout.stride(0), dout.stride(1), q.data_ptr(), q.stride(0), q.stride(1), k.data_ptr(), k.stride(0),
      k.stride(1), v.data_ptr(), v.stride(0), v.stride(1), out.data_ptr(), out.stride(0), out.stride(1),
      static_cast<const float*>(lse.data_ptr()), dq.data_ptr(), dq.stride(0), dq.stride(1), dk.data_ptr(), dk.stride(0),
      dk.stride(1), dv.data_ptr(), dv.stride(0), dv.stride(1), static_cast<float*>(softmax_d.data_ptr()),
      static_cast<const int64_t*>(p.col_offsets.data_ptr()), static_cast<const int32_t*>(p.col_nnz.data_ptr()),
      static_cast<const int32_t*>(p.indices.data_ptr()), n_indices, cuq, cuk, ws.data_ptr(), nbytes, (int)batch, (int)h, (int)hk,
      (int)d, total_q, total_k, (int)max_q, (int)max_k, (int)chunk, (float)scale, causal ? 1 : 0, dtype_code(q),
      current_stream());
  ticket.end(rc, ws);
  return softmax_d;
}

// ---------------------------------------------------------------------------- autograd node
// Head dimension the kernels run at: 64, 128 or 256; anything else is zero-padded up to the next of
// them (zero columns change neither the scores nor the first d outputs).  Above 256: rejected by the
// library with its message.
int64_t padded_head_dim(int64_t d) {
  for (int64_t built : {64, 128, 256})
    if (d <= built) return built;
  return (d + 7) / 8 * 8;
}
Tensor pad_to(const Tensor& t, int64_t d) {
  return t.size(2) == d ? fix_last_stride(t) : at::constant_pad_nd(t, {0, d - t.size(2)}, 0);
}

struct AttnCall {
  Pattern p;
  Tensor cu_q, cu_k;
  int64_t max_q, max_k, chunk;
  double scale;
  bool causal;
};

class MobaAttention : public torch::autograd::Function<MobaAttention> {
 public:
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& q0, const Tensor& k0,
                                                const Tensor& v0, const std::shared_ptr<AttnCall>& c, bool keep) {
    const int64_t d_og = q0.size(2), d = padded_head_dim(d_og);
    Tensor q = pad_to(q0, d), k = pad_to(k0, d), v = pad_to(v0, d);
    auto [out, lse, lists] =
        attn_fwd(q, k, v, c->p, c->cu_q, c->cu_k, c->max_q, c->max_k, c->chunk, c->scale, c->causal, {}, {}, {});
    Tensor shown = d == d_og ? out : out.narrow(2, 0, d_og);
    ctx->set_materialize_grads(false);               // no zeros made up for the log-sum-exps' gradient
    if (keep) {
      ctx->save_for_backward({q, k, v, out, lse, c->cu_q, c->cu_k, c->p.col_offsets, c->p.col_nnz, c->p.indices});
      auto& s = ctx->saved_data;
      // Which of the two there is depends on what else has been built meanwhile, so they are not saved tensors: a
      // recomputation has to save what the first pass saved
      if (c->p.row_slots) s["row_slots"] = *c->p.row_slots;
      if (lists) s["lists"] = *lists;
      s["geo"] = c10::List<int64_t>({c->max_q, c->max_k, c->chunk, c->p.topk, (int64_t)c->causal, d_og});
      s["scale"] = c->scale;
    }
    return {shown, lse};
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list g) {
    auto saved = ctx->get_saved_variables();
    const auto geo = ctx->saved_data["geo"].toIntVector();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2];
    Pattern p;
    p.col_offsets = saved[7]; p.col_nnz = saved[8]; p.indices = saved[9];
    p.topk = geo[3];
    OptTensor lists;
    if (auto it = ctx->saved_data.find("row_slots"); it != ctx->saved_data.end()) p.row_slots = it->second.toTensor();
    if (auto it = ctx->saved_data.find("lists"); it != ctx->saved_data.end()) lists = it->second.toTensor();
    const int64_t d_og = geo[5], d = q.size(2);
    Tensor dout = g[0].defined() ? pad_to(g[0], d) : at::zeros_like(saved[3]);
    Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
    attn_bwd(dout, q, k, v, saved[3], saved[4], dq, dk, dv, p, saved[5], saved[6], geo[0], geo[1], geo[2],
             ctx->saved_data["scale"].toDouble(), geo[4] != 0, lists);
    if (d != d_og) {
      dq = dq.narrow(2, 0, d_og);
      dk = dk.narrow(2, 0, d_og);
      dv = dv.narrow(2, 0, d_og);
    }
    return {dq, dk, dv, Tensor(), Tensor()};
  }
};

// attention over a pattern, recorded for autograd: (out, lse)
std::tuple<Tensor, Tensor> attention(const Tensor& q, const Tensor& k, const Tensor& v, Pattern p, const Tensor& cu_q,
                                     const Tensor& cu_k, int64_t max_q, int64_t max_k, int64_t chunk,
                                     std::optional<double> scale, bool causal) {
  TORCH_CHECK(q.dim() == 3 && k.dim() == 3 && v.dim() == 3, "q, k and v must have shape (tokens, heads, head_dim)");
  auto c = std::make_shared<AttnCall>();
  c->p = std::move(p);
  c->cu_q = cu_q; c->cu_k = cu_k; c->max_q = max_q; c->max_k = max_k; c->chunk = chunk; c->causal = causal;
  c->scale = scale ? *scale : 1.0 / std::sqrt((double)q.size(2));
  const bool keep = at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad());
  auto r = MobaAttention::apply(q, k, v, c, keep);
  return {r[0], r[1]};
}

// ---------------------------------------------------------------------------- public compositions
Pattern pattern_from_centroids(const Tensor& q, const Tensor& km, const Tensor& cu_q, const Tensor& cu_k, const Tensor& cu_km,
                               int64_t max_q, int64_t max_k, int64_t topk, int64_t chunk, bool causal) {
  TORCH_CHECK(chunk > 0, "moba_chunk_size must be positive");
  auto [idx, val] = gate_topk(q, km, cu_q, cu_k, cu_km, max_q, max_k, topk, chunk, causal, false);
  return build_csc(idx.permute({1, 0, 2}), cu_q, max_q, (max_k + chunk - 1) / chunk, true);
}

Pattern moba_pattern(const Tensor& q0, const Tensor& k0, const Tensor& cu_q, const Tensor& cu_k, int64_t max_q, int64_t max_k,
                     int64_t topk, int64_t chunk, bool causal) {
  at::NoGradGuard no_grad;
  TORCH_CHECK(q0.dim() == 3 && k0.dim() == 3, "q and k must have shape (tokens, heads, head_dim)");
  const int64_t d = padded_head_dim(q0.size(2));
  Tensor q = pad_to(q0, d), k = pad_to(k0, d);
  auto [km, cu_km] = mean_pool(k, cu_k, max_k, chunk);
  return pattern_from_centroids(q, km, cu_q, cu_k, cu_km, max_q, max_k, topk, chunk, causal);
}

// A call with few query rows and no derivatives to record: one launch for gating and attention
// (fmb_decode_fwd); undefined where the general path is to run, which also refuses what cannot be (forward-mode
// derivatives: the autograd node has none).
Tensor try_decode(const Tensor& q0, const Tensor& k0, const Tensor& v0, const OptTensor& km0, const OptTensor& cu_km0,
                  const Tensor& cu_q, const Tensor& cu_k, int64_t max_k, int64_t topk, int64_t chunk, bool causal) {
  if (at::GradMode::is_enabled() && (q0.requires_grad() || k0.requires_grad() || v0.requires_grad())) return {};
  for (const Tensor* t : {&q0, &k0, &v0})
    if (t->dim() != 3 || t->_fw_grad(/*level=*/0).defined()) return {};
  if (q0.size(2) % 8 != 0 || k0.size(2) != q0.size(2) || v0.sizes() != k0.sizes()) return {};
  const int64_t total_q = q0.size(0), h = q0.size(1), d = q0.size(2), hk = k0.size(1), batch = cu_q.numel() - 1;
  if (!fmb_decode_preferred(total_q, k0.size(0), (int)batch, (int)h, (int)hk, (int)d, (int)max_k, (int)topk, (int)chunk)) return {};
  at::NoGradGuard no_grad;
  Tensor q = fix_last_stride(q0), k = fix_last_stride(k0), v = fix_last_stride(v0), km, cu_km;
  for (const Tensor* t : {(const Tensor*)&q, (const Tensor*)&k, (const Tensor*)&v, &cu_q, &cu_k}) require_cuda(*t);
  TORCH_CHECK(q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type(),
              "query, key and value must have the same dtype");
  if (km0) {
    km = km0->contiguous();
    cu_km = *cu_km0;
    TORCH_CHECK(km.dim() == 3 && km.size(1) == hk && km.size(2) == d && km.scalar_type() == q.scalar_type(),
                "the centroids must have the keys' heads, head_dim and dtype");
  } else {
    std::tie(km, cu_km) = mean_pool(k, cu_k, max_k, chunk);
  }
  c10::cuda::CUDAGuard guard(q.device());
  Tensor out = at::empty_like(q);
  check(fmb_decode_fwd(q.data_ptr(), q.stride(0), q.stride(1), k.data_ptr(), k.stride(0), k.stride(1), v.data_ptr(), v.stride(0),
                       v.stride(1), km.data_ptr(), out.data_ptr(), out.stride(0), out.stride(1), i32c(cu_q, "cu_seqlens_q"),
                       i32c(cu_k, "cu_seqlens_k"), i32c(cu_km, "cu_seqlens_km"), (int)batch, (int)h, (int)hk, (int)d, total_q,
                       (int)max_k, (int)topk, (int)chunk, (float)(1.0 / std::sqrt((double)d)), causal ? 1 : 0, dtype_code(q),
                       current_stream()));
  return out;
}

using Triple = std::tuple<Tensor, Tensor, Tensor>;
Triple shown(const Pattern& p, const Tensor& cu_q) {
  remember(p, cu_q);
  return {p.col_offsets, p.col_nnz, p.indices};
}

Triple py_topk_varlen(const Tensor& q, const Tensor& k, const Tensor& cu_q, const Tensor& cu_k, int64_t max_q, int64_t max_k,
                      int64_t topk, int64_t chunk, bool causal) {
  return shown(moba_pattern(q, k, cu_q, cu_k, max_q, max_k, topk, chunk, causal), cu_q);
}
Triple py_fused_topk(const Tensor& q, const Tensor& km, const Tensor& cu_q, const Tensor& cu_k, const Tensor& cu_km, int64_t max_q,
                     int64_t max_k, int64_t topk, int64_t chunk, bool causal) {
  at::NoGradGuard no_grad;
  return shown(pattern_from_centroids(fix_last_stride(q), km.contiguous(), cu_q, cu_k, cu_km, max_q, max_k, topk, chunk, causal), cu_q);
}
Triple py_build_csc(const Tensor& idx, const Tensor& cu_q, int64_t max_q, int64_t ncol, bool keep_rows) {
  return shown(build_csc(idx, cu_q, max_q, ncol, keep_rows), cu_q);
}
std::tuple<Tensor, Tensor> py_attn_varlen(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu_q,
                                          const Tensor& cu_k, int64_t max_q, int64_t max_k, const Tensor& co, const Tensor& cn,
                                          const Tensor& in, int64_t chunk, std::optional<double> scale, bool causal) {
  return attention(q, k, v, recall(co.contiguous(), cn.contiguous(), in.contiguous(), cu_q), cu_q, cu_k, max_q, max_k, chunk, scale,
                   causal);
}
Tensor py_moba_varlen(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu_q, const Tensor& cu_k, int64_t max_q,
                      int64_t max_k, int64_t chunk, int64_t topk, bool causal) {
  if (Tensor out = try_decode(q, k, v, {}, {}, cu_q, cu_k, max_k, topk, chunk, causal); out.defined()) return out;
  Pattern p = moba_pattern(q, k, cu_q, cu_k, max_q, max_k, topk, chunk, causal);
  return std::get<0>(attention(q, k, v, std::move(p), cu_q, cu_k, max_q, max_k, chunk, std::nullopt, causal));
}
Tensor py_moba_cached(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& km, const Tensor& cu_km, const Tensor& cu_q,
                      const Tensor& cu_k, int64_t max_q, int64_t max_k, int64_t topk, int64_t chunk) {
  if (Tensor out = try_decode(q, k, v, km, cu_km, cu_q, cu_k, max_k, topk, chunk, true); out.defined()) return out;
  Pattern p;
  {
    at::NoGradGuard no_grad;
    p = pattern_from_centroids(fix_last_stride(q), km, cu_q, cu_k, cu_km, max_q, max_k, topk, chunk, true);
  }
  return std::get<0>(attention(q, k, v, std::move(p), cu_q, cu_k, max_q, max_k, chunk, std::nullopt, true));
}
std::tuple<Tensor, Tensor, OptTensor> py_attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& co,
                                                  const Tensor& cn, const Tensor& in, const Tensor& cu_q, const Tensor& cu_k,
                                                  int64_t max_q, int64_t max_k, int64_t chunk, double scale, bool causal,
                                                  const OptTensor& out, const OptTensor& k_begin, const OptTensor& k_end) {
  return attn_fwd(q, k, v, recall(co, cn, in, cu_q), cu_q, cu_k, max_q, max_k, chunk, scale, causal, out, k_begin, k_end);
}
Tensor py_attn_bwd(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
                   const Tensor& dq, const Tensor& dk, const Tensor& dv, const Tensor& co, const Tensor& cn, const Tensor& in,
                   const Tensor& cu_q, const Tensor& cu_k, int64_t max_q, int64_t max_k, int64_t chunk, double scale, bool causal,
                   const OptTensor& lists) {
  return attn_bwd(dout, q, k, v, out, lse, dq, dk, dv, recall(co, cn, in, cu_q), cu_q, cu_k, max_q, max_k, chunk, scale, causal, lists);
}

}  // namespace

PYBIND11_MODULE(_fmb_torch, m) {
  m.def("mean_pool", torch::wrap_pybind_function_no_gil(mean_pool));
  m.def("gate_topk", torch::wrap_pybind_function_no_gil(gate_topk));
  m.def("build_csc", torch::wrap_pybind_function_no_gil(py_build_csc));
  m.def("attn_fwd", torch::wrap_pybind_function_no_gil(py_attn_fwd));
  m.def("attn_bwd", torch::wrap_pybind_function_no_gil(py_attn_bwd));
  m.def("topk_varlen", torch::wrap_pybind_function_no_gil(py_topk_varlen));
  m.def("fused_topk", torch::wrap_pybind_function_no_gil(py_fused_topk));
  m.def("attn_varlen", torch::wrap_pybind_function_no_gil(py_attn_varlen));
  m.def("moba_varlen", torch::wrap_pybind_function_no_gil(py_moba_varlen));
  m.def("moba_cached", torch::wrap_pybind_function_no_gil(py_moba_cached));
  m.def("check_pending_status", torch::wrap_pybind_function_no_gil(check_pending_status));
}
