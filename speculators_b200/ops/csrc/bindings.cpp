// Torch operator registration for the sm_100a kernels of this package.
// Every op validates device / dtype / layout, then launches on the current stream.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/library.h>

#include "attention_params.h"
#include "ep_a2a.h"
#include "gemm_split.h"
#include <ATen/ATen.h>

#include <algorithm>
#include <deque>
#include <mutex>

namespace sb200 {
int rmsnorm_bwd_partial_rows(int rows, int H, bool with_dx);
void launch_add_rmsnorm_fwd(const void*, const void*, const void*, void*, void*, int, int, float, cudaStream_t);
void launch_rmsnorm_fwd(const void*, const void*, const int64_t*, void*, float*, int, int, int64_t,
                        int64_t, float, int64_t, int, const int*, cudaStream_t);
struct BoundsRecord {
  int site;
  long long index;
  long long limit;
};
int read_bounds_norm(BoundsRecord*);
int read_bounds_ep(BoundsRecord*);
void launch_rmsnorm_bwd(const void*, int64_t, const void*, int64_t, const void*, int64_t, const void*, const float*, const void*, int64_t, void*, int64_t,
                        float*, void*, int, int, int, int, const int*, cudaStream_t);
void launch_heads_fwd(const void*, int64_t, const void* const*, const int*, void*, float*, int, int, float, const int64_t*, const float*, const float*, int64_t,
                      int, int, const int*, cudaStream_t);
int heads_bwd_groups(int, int);
int64_t repeated_part_floats(int, int, int);
void launch_heads_bwd(const void* const*, const int64_t*, const int*, const void*, int64_t, const void* const*, const float*, float* const*, void* const*,
                      const int*, const int*, void*, int64_t, int, int, float*, const int64_t*, const float*, const float*, int64_t, int, int, const int*,
                      cudaStream_t);
void launch_repeated_rows_sum(const void*, int64_t, int, int, float*, void*, int64_t, cudaStream_t);
void launch_document_interval(const int64_t*, int, int, int*, int*, cudaStream_t);
void launch_select_anchors(const bool*, const float*, int, int, int, int, int64_t*, bool*, cudaStream_t);
void launch_anchor_spec(const int64_t*, const int*, int, const int64_t*, int, int, int, int, int*, int*, int*, cudaStream_t);
void launch_anchor_slots(const int64_t*, const bool*, const int64_t*, const int64_t*, const bool*, int, int, int, int64_t, int, int64_t*, int64_t*, int64_t*,
                         int64_t*, bool*, cudaStream_t);
void launch_compact(const bool*, int, int64_t*, int*, cudaStream_t);
void launch_cod_step(const int64_t*, const int64_t*, int, const bool*, int, int, int, unsigned char*, int64_t*, int64_t*, int64_t*, int64_t*, int*, cudaStream_t);
void launch_peagle_spec(const int64_t*, const int64_t*, const bool*, const int64_t*, const int*, int, int, int, int, int*, int*, int*, int*, cudaStream_t);
void launch_step_rows(const uint8_t*, const int64_t*, const int64_t*, const int* const*, int, int, int, int64_t*, int*, int*, int64_t*, int64_t*, uint8_t*, uint8_t*,
                      int*, int* const*, int*, cudaStream_t);
void launch_take_rows(int, const void* const*, const int64_t*, const int*, void* const*, const int64_t*, const int*, int, cudaStream_t);
void launch_put_rows(int, const void* const*, const int64_t*, const int*, void* const*, const int*, int, cudaStream_t);
int embedding_bwd_partial_rows(int);
void launch_embedding_bwd(const int64_t*, const int64_t*, const void*, int64_t, int, int, int64_t, int64_t, void*, int, float*, cudaStream_t);
void launch_swiglu_fwd(const void*, void*, int64_t, int, const int*, cudaStream_t);
void launch_swiglu_bwd(const void*, const void*, void*, int64_t, int, const int*, cudaStream_t);
void launch_rope_merge(const void* const*, const int64_t*, const int*, const int*, void*, int64_t, const int64_t*, const float*, const float*, int64_t, int, int,
                       int, float, const int*, cudaStream_t);
void launch_gate_mul_fwd(const void*, const void*, void*, int, int, int, int64_t, int, cudaStream_t);
void launch_gate_mul_bwd(const void*, const void*, const void*, void*, void*, int, int, int, int64_t, int, int64_t, cudaStream_t);
int launch_topk_rows(const float*, int, int, int, int64_t*, cudaStream_t);
int moe_plan_blocks(int);
int launch_moe_plan(const int64_t*, int, int, int, int*, int*, int*, int*, int*, const int*, int, cudaStream_t);
void launch_moe_gather(const void*, int64_t, const int*, const int*, int, void*, int, int, cudaStream_t);
void launch_moe_gather_bwd(const void*, const int*, int, void*, int, int, const int*, cudaStream_t);
void launch_moe_combine(const void*, const int*, const void*, int, const void*, const void*, const void*, void*, int, int, const int*, cudaStream_t);
void launch_moe_combine_bwd(const void*, const void*, const int*, const int*, const void*, int, void*, void*, const void*, const void*, void*, void*, int, int, int,
                            const int*, cudaStream_t);
int launch_gemm_grouped_swiglu(const void*, const void*, void*, void*, int, int, int, int64_t, int64_t, const int*, const int*, int, int*, cudaStream_t);
void launch_rope(void*, const int64_t*, const float*, const float*, int64_t, int, int, int, int64_t,
                 int64_t, float, const int*, cudaStream_t);
int launch_loss_fwd(int, const void*, const void*, const uint8_t*, const uint8_t*, const int64_t*, float*, float*, int*,
                    int*, int, int, int64_t, int64_t, int, const int*, float*, cudaStream_t);
int launch_loss_bwd(int, const void*, const void*, const float*, const float*, const float*, void*, int, int, int,
                    int64_t, int64_t, int64_t, int, const int*, const int*, cudaStream_t);
int64_t launch_count();
int launch_gemm_tn_tcgen05(const void*, const void*, void*, const void*, int, int, int, int64_t, int64_t, int64_t, int64_t, int,
                           int*, int, const int*, SplitSpace*, cudaStream_t);
int launch_gemm_tcgen05(const void*, const void*, void*, const void*, int, int, int, int64_t, int64_t, int64_t, int64_t, int, int, int,
                        int*, int, const int*, SplitSpace*, cudaStream_t);
int launch_gemm_parts(int, const void* const*, const void* const*, const int*, const int64_t*, const int64_t*, const int* const*, void*, int, int, int64_t, int, int*,
                      SplitSpace*, cudaStream_t);
int launch_gemm_grouped_parts(int, const void* const*, const void* const*, const int*, const int64_t*, const int64_t*, const int* const*, void*, int, int, int,
                              const int*, int, int*, cudaStream_t);
int launch_gemm_stack(const void*, const void*, void*, const void*, int, int, int, int, int, int, float, float, int, float, int, int*, SplitSpace*,
                      cudaStream_t);
void launch_moe_group_plan(const int*, int, int*, int*, cudaStream_t);
int launch_gemm_grouped(const void*, const void*, void*, int, int, int, int64_t, int64_t, int64_t, int, int, int, const int*, const int*, int, int*,
                        cudaStream_t);
int lmhead_stat_words();
int lmhead_tiles_n(int);
int launch_lmhead_logits_stats(const void*, const void*, void*, const void*, int, int, int, int64_t, int64_t, int64_t, int64_t, int, int, float*,
                               int*, cudaStream_t);
int launch_lmhead_combine(const float*, const void*, const uint8_t*, float*, float*, int*, int*, int, int, int64_t, int, cudaStream_t);
int sumsq_num_partials();
int peer_malloc(int64_t, void**);
int peer_free(void*);
int peer_export(void*, unsigned char*);
int peer_import(const unsigned char*, void**);
int peer_close(void*);
int fused_optim_ctl_words();
int fused_optim_num_partials();
int launch_fused_sharded_adamw(int, int, int64_t, const void* const*, void* const*, void* const*, const void*, void*, float*, float*,
                               float*, float*, float*, const float*, int*, uint32_t, cudaStream_t);
int launch_gemm_swiglu(const void*, const void*, void*, void*, int, int, int, int64_t, int64_t, int64_t, int64_t, int*, const int*, cudaStream_t);
int launch_gemm_scatter(const void*, const void*, void* const*, int, int, int, int, int, int64_t, int64_t, int*, cudaStream_t);
int tp_allreduce_ctl_words();
int launch_tp_reduce_broadcast(int, int, int, int, const void*, void* const*, void*, const void*, void* const*, int, int*, uint32_t, cudaStream_t);
int hs_ring_ctl_words_per_slot();
int launch_hs_push(const void*, int64_t, void*, uint32_t*, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t*, int*, cudaStream_t);
int launch_hs_pop(void*, int64_t, const void*, uint32_t*, uint32_t, uint32_t, uint32_t*, int*, cudaStream_t);
void launch_step_tail(const float*, const int*, const int*, const uint8_t*, uint8_t*, int, float, float, float*, float*, const float*, float*, const int*,
                      cudaStream_t);
void launch_sumsq(const void*, int, int64_t, float*, float*, int, cudaStream_t);
void launch_set_hyper(float*, const float*, cudaStream_t);
void launch_adamw(float*, float*, float*, const void*, int, void*, int64_t, const float*,
                  const float*, cudaStream_t);
void launch_muon_momentum(const void*, int, float*, void*, const int64_t*, const int*, int, const int*, int, const float*, const float*, float, int, float*,
                          float*, cudaStream_t);
void launch_muon_apply(float*, const void*, void*, const int64_t*, const int*, int, const float*, const float*, float, float, cudaStream_t);
int muon_chunk_elements();
}  // namespace sb200

namespace {

using at::Tensor;

inline cudaStream_t cur_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

void check_rows(const Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
  TORCH_CHECK(t.scalar_type() == at::kBFloat16, name, " must be bfloat16");
  TORCH_CHECK(t.dim() == 2 && t.stride(1) == 1, name, " must be 2-D with unit inner stride");
  TORCH_CHECK(t.stride(0) % 8 == 0 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0, name,
              " rows must be 16-byte aligned");
}

// Operands that plain operators would have refused to combine.
void check_same_device(const Tensor& t, std::initializer_list<const Tensor*> others) {
  for (const Tensor* o : others) TORCH_CHECK(o->device() == t.device(), "expected tensors on one device, got ", t.device(), " and ", o->device());
}

// rows_used (optional int32[1] on the device): rows past it are left alone.
const int* used_rows(const c10::optional<Tensor>& rows_used) {
  if (!rows_used.has_value()) return nullptr;
  TORCH_CHECK(rows_used->is_cuda() && rows_used->scalar_type() == at::kInt && rows_used->numel() >= 1);
  return rows_used->data_ptr<int>();
}
const uint8_t* row_flags(const c10::optional<Tensor>& t, int64_t rows) {
  if (!t.has_value()) return nullptr;
  TORCH_CHECK((t->scalar_type() == at::kBool || t->scalar_type() == at::kByte) && t->is_contiguous() && t->numel() >= rows, "bool / uint8 row flags expected");
  return reinterpret_cast<const uint8_t*>(t->data_ptr());
}

// ---- memory of GEMMs that divide tiles ---------------------------------------------------------------------
// Partial sums come from the caching allocator, for the launch alone.  Counters and flags have to be zero when the kernel starts,
// and a launch of a captured graph finds them used at its next replay: they come in slabs of kSlots launches that one memset
// zeroes, on the launch's stream and - under capture - as a node of the graph, in whose memory the slab then is.  A slot
// serves one launch.  The slab in use is kept per stream and capture (the last kSlabs of them, 600 KB each); one that is
// dropped goes back to the allocator in its stream's order, behind the launches that use it.
struct SyncSlabs {
  static constexpr int kSlots = 64, kSlabs = 32;
  struct Slab {
    int device;
    cudaStream_t stream;
    unsigned long long capture;  // 0: none
    Tensor memory;
    int used;
  };
  std::mutex mutex;
  std::deque<Slab> slabs;  // the least recently made first
  static SyncSlabs& instance() {
    static SyncSlabs* all = new SyncSlabs;  // outlives the threads and the driver: never destroyed
    return *all;
  }
  int* slot(const Tensor& near, cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    if (cudaStreamGetCaptureInfo(stream, &status, &id) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    if (status != cudaStreamCaptureStatusActive) id = 0;
    const int ints = (sb200::gemm_split_sync_ints() + 31) / 32 * 32, device = near.get_device();
    std::lock_guard<std::mutex> lock(mutex);
    auto it = std::find_if(slabs.begin(), slabs.end(), [&](const Slab& s) { return s.device == device && s.stream == stream; });
    if (it != slabs.end() && (it->capture != id || it->used == kSlots)) {
      slabs.erase(it);
      it = slabs.end();
    }
    if (it == slabs.end()) {
      Slab s{device, stream, id, at::empty({(int64_t)kSlots * ints}, near.options().dtype(at::kInt)), 0};
      if (cudaMemsetAsync(s.memory.data_ptr(), 0, s.memory.nbytes(), stream) != cudaSuccess) return nullptr;
      if (slabs.size() == kSlabs) slabs.pop_front();
      slabs.push_back(std::move(s));
      it = slabs.end() - 1;
    }
    return it->memory.data_ptr<int>() + (int64_t)it->used++ * ints;
  }
};
struct TorchSplitSpace : sb200::SplitSpace {
  const Tensor& near;
  Tensor partial;
  explicit TorchSplitSpace(const Tensor& t) : near(t) {}
  bool get(float** sums, int** sync) override {
    *sync = SyncSlabs::instance().slot(near, cur_stream());
    if (*sync == nullptr) return false;
    partial = at::empty({sb200::gemm_split_floats()}, near.options().dtype(at::kFloat));
    *sums = partial.data_ptr<float>();
    return true;
  }
};

void norm_fwd(const Tensor& x, const Tensor& w, const c10::optional<Tensor>& row_index, Tensor y,
              c10::optional<Tensor> rstd, double eps, bool centred, const c10::optional<Tensor>& live) {
  check_rows(x, "x");
  check_rows(y, "y");
  const int H = (int)y.size(1);
  const int rows = (int)y.size(0);
  TORCH_CHECK(x.size(1) == H && w.numel() == H && w.is_contiguous() &&
                  w.scalar_type() == at::kBFloat16,
              "rmsnorm: shape/dtype mismatch");
  TORCH_CHECK(H % 8 == 0 && H <= 32768, "rmsnorm: H must be a multiple of 8 and <= 32768");
  const int64_t* idx = nullptr;
  if (row_index.has_value()) {
    TORCH_CHECK(row_index->scalar_type() == at::kLong && row_index->is_contiguous() &&
                    row_index->numel() == rows,
                "rmsnorm: row_index must be int64[rows]");
    idx = row_index->data_ptr<int64_t>();
  } else {
    TORCH_CHECK(x.size(0) == rows, "rmsnorm: row count mismatch");
  }
  float* rs = nullptr;
  if (rstd.has_value()) {
    TORCH_CHECK(rstd->scalar_type() == at::kFloat && rstd->numel() == rows && rstd->is_contiguous());
    rs = rstd->data_ptr<float>();
  }
  c10::cuda::CUDAGuard guard(x.device());
  sb200::launch_rmsnorm_fwd(x.data_ptr(), w.data_ptr(), idx, y.data_ptr(), rs, rows, H, x.stride(0),
                            y.stride(0), (float)eps, x.size(0), centred ? 1 : 0, used_rows(live), cur_stream());
}
// -> (x + add, its norm); contiguous bf16 [rows, H]
std::tuple<Tensor, Tensor> add_rmsnorm_fwd(const Tensor& x, const Tensor& add, const Tensor& w, double eps) {
  for (const Tensor* t : std::initializer_list<const Tensor*>{&x, &add})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->dim() == 2 && t->is_contiguous() && (reinterpret_cast<uintptr_t>(t->data_ptr()) & 15) == 0,
                "add_rmsnorm_fwd: contiguous bf16 [rows, H] expected");
  check_same_device(x, {&add, &w});
  const int64_t H = x.size(1);
  TORCH_CHECK(add.sizes() == x.sizes() && H % 8 == 0 && H > 256 && H <= 32768, "add_rmsnorm_fwd: shapes");
  TORCH_CHECK(w.is_cuda() && w.scalar_type() == at::kBFloat16 && w.is_contiguous() && w.numel() == H && (reinterpret_cast<uintptr_t>(w.data_ptr()) & 15) == 0);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor sum = at::empty_like(x), y = at::empty_like(x);
  sb200::launch_add_rmsnorm_fwd(x.data_ptr(), add.data_ptr(), w.data_ptr(), sum.data_ptr(), y.data_ptr(), (int)x.size(0), (int)H, (float)eps, cur_stream());
  return {sum, y};
}
void rmsnorm_fwd(const Tensor& x, const Tensor& w, const c10::optional<Tensor>& row_index, Tensor y, c10::optional<Tensor> rstd, double eps,
                 const c10::optional<Tensor>& live) {
  norm_fwd(x, w, row_index, y, rstd, eps, false, live);
}

// dx = norm gradient of (dy + dy2) (+ add), dw bf16[H] (=, +=); dy2, add, dx, dw optional.  centred: the weight is 1 + w.
void rmsnorm_bwd(const Tensor& dy, const c10::optional<Tensor>& dy2, const Tensor& x, const Tensor& w, const Tensor& rstd, const c10::optional<Tensor>& add,
                 c10::optional<Tensor> dx, c10::optional<Tensor> dw, bool accumulate_dw, bool centred, const c10::optional<Tensor>& live) {
  const int64_t rows = x.size(0), H = x.size(1);
  auto rows_of = [&](const c10::optional<Tensor>& t, const char* name, int64_t& stride) -> void* {
    if (!t.has_value()) return nullptr;
    check_rows(*t, name);
    TORCH_CHECK(t->size(0) == rows && t->size(1) == H, "rmsnorm_bwd: ", name, " has another shape");
    stride = t->stride(0);
    return t->data_ptr();
  };
  int64_t sy = 0, sy2 = 0, sx = 0, sa = 0, sd = 0;
  void* py = rows_of(dy, "dy", sy);
  void* py2 = rows_of(dy2, "dy2", sy2);
  void* px = rows_of(x, "x", sx);
  void* pa = rows_of(add, "add", sa);
  void* pd = rows_of(dx, "dx", sd);
  TORCH_CHECK(H % 8 == 0 && H <= 32768 && w.numel() == H && w.scalar_type() == at::kBFloat16 && w.is_contiguous());
  TORCH_CHECK(rstd.scalar_type() == at::kFloat && rstd.numel() == rows && rstd.is_contiguous());
  c10::cuda::CUDAGuard guard(x.device());
  Tensor partial;
  if (dw.has_value()) {
    TORCH_CHECK(dw->scalar_type() == at::kBFloat16 && dw->numel() == H && dw->is_contiguous());
    partial = at::empty({sb200::rmsnorm_bwd_partial_rows((int)rows, (int)H, pd != nullptr), H}, rstd.options());
    if (rows == 0 && !accumulate_dw) dw->zero_();
  }
  sb200::launch_rmsnorm_bwd(py, sy, py2, sy2, px, sx, w.data_ptr(), rstd.data_ptr<float>(), pa, sa, pd, sd, dw.has_value() ? partial.data_ptr<float>() : nullptr,
                            dw.has_value() ? dw->data_ptr() : nullptr, (int)rows, (int)H, accumulate_dw ? 1 : 0, centred ? 1 : 0, used_rows(live), cur_stream());
}

void check_rotation(const Tensor& positions, const Tensor& cos_t, const Tensor& sin_t, int64_t tokens, int64_t hd, int64_t rot) {
  TORCH_CHECK(rot % 16 == 0 && rot <= hd && hd % 8 == 0, "rotation: rot a multiple of 16, hd of 8");
  TORCH_CHECK(positions.scalar_type() == at::kLong && positions.is_contiguous() && positions.numel() == tokens);
  TORCH_CHECK(cos_t.scalar_type() == at::kFloat && sin_t.scalar_type() == at::kFloat && cos_t.is_contiguous() && sin_t.is_contiguous() && cos_t.dim() == 2 &&
              cos_t.size(1) == rot / 2 && sin_t.sizes() == cos_t.sizes() && (reinterpret_cast<uintptr_t>(cos_t.data_ptr()) & 15) == 0 &&
              (reinterpret_cast<uintptr_t>(sin_t.data_ptr()) & 15) == 0, "rotation: aligned fp32 [positions, rot / 2] tables expected");
}
const void* head_weight(const c10::optional<Tensor>& w, int64_t heads, int64_t hd) {
  if (heads == 0) return nullptr;
  TORCH_CHECK(w.has_value() && w->scalar_type() == at::kBFloat16 && w->is_contiguous() && w->numel() == hd && (reinterpret_cast<uintptr_t>(w->data_ptr()) & 15) == 0);
  return w->data_ptr();
}

// -> (rotated normalised heads [T, (na + nb) hd], rstd [T na] then [T nb]); repeated: src holds two rows more than the
// first tokens, and the tokens after those (positions has them all) read the first of the two
std::tuple<Tensor, Tensor> heads_fwd(const Tensor& src, const c10::optional<Tensor>& w_a, int64_t na, const c10::optional<Tensor>& w_b, int64_t nb, double eps,
                                     const Tensor& positions, const Tensor& cos_t, const Tensor& sin_t, int64_t hd, int64_t rot, bool repeated,
                                     const c10::optional<Tensor>& live) {
  TORCH_CHECK(!repeated || !live.has_value(), "heads_fwd: a row count and repeated rows exclude each other");
  check_rows(src, "src");
  const int64_t T = repeated ? positions.numel() : src.size(0);
  TORCH_CHECK((hd == 64 || hd == 128 || hd == 256) && na >= 1 && nb >= 0 && src.size(1) >= (na + nb) * hd);
  TORCH_CHECK(!repeated || (src.size(0) >= 2 && T > src.size(0) - 2), "heads_fwd: two rows for the repeated tokens expected");
  check_rotation(positions, cos_t, sin_t, T, hd, rot);
  c10::cuda::CUDAGuard guard(src.device());
  Tensor out = at::empty({T, (na + nb) * hd}, src.options());
  Tensor rstd = at::empty({T * (na + nb)}, src.options().dtype(at::kFloat));
  const void* w[2] = {head_weight(w_a, na, hd), head_weight(w_b, nb, hd)};
  const int heads[2] = {(int)na, (int)nb};
  sb200::launch_heads_fwd(src.data_ptr(), src.stride(0), w, heads, out.data_ptr(), rstd.data_ptr<float>(), (int)T,
                          (int)(repeated ? src.size(0) - 2 : src.size(0)), (float)eps,
                          positions.data_ptr<int64_t>(), cos_t.data_ptr<float>(), sin_t.data_ptr<float>(), cos_t.size(0), (int)hd, (int)rot, used_rows(live), cur_stream());
  return {out, rstd};
}

// d: gradients (or None) of the a, b and plain blocks, each below and from `split` on (a whole when there is a b)
Tensor heads_bwd(const c10::List<c10::optional<Tensor>>& d, int64_t split, const Tensor& src, const Tensor& rstd, const c10::optional<Tensor>& w_a, int64_t na,
                 const c10::optional<Tensor>& w_b, int64_t nb, int64_t nv, const c10::optional<Tensor>& dw_a, bool acc_a, const c10::optional<Tensor>& dw_b,
                 bool acc_b, const Tensor& positions, const Tensor& cos_t, const Tensor& sin_t, int64_t hd, int64_t rot, bool repeated,
                 const c10::optional<Tensor>& live) {
  TORCH_CHECK(!repeated || !live.has_value(), "heads_bwd: a row count and repeated rows exclude each other");
  check_rows(src, "src");
  const int64_t T = positions.numel(), tokens = repeated ? src.size(0) - 2 : src.size(0);
  TORCH_CHECK(repeated ? (tokens >= 0 && T > tokens && split == tokens && nb > 0) : T == tokens, "heads_bwd: rows and positions do not match");
  TORCH_CHECK(d.size() == 6 && (hd == 64 || hd == 128 || hd == 256) && src.size(1) >= (na + nb + nv) * hd && split >= 0 && split <= T);
  TORCH_CHECK(rstd.scalar_type() == at::kFloat && rstd.is_contiguous() && rstd.numel() == T * (na + nb));
  check_rotation(positions, cos_t, sin_t, T, hd, rot);
  const int heads[3] = {(int)na, (int)nb, (int)nv};
  const void* ptr[6];
  int64_t stride[6];
  const int splits[3] = {(int)(nb > 0 ? T : split), (int)split, (int)split};
  std::vector<Tensor> hold;
  for (int i = 0; i < 6; ++i) {
    ptr[i] = nullptr;
    stride[i] = 0;
    const c10::optional<Tensor> g = d.get(i);
    if (!g.has_value()) continue;
    check_rows(*g, "gradient");
    TORCH_CHECK(g->size(1) == heads[i / 2] * hd && g->size(0) == (i % 2 ? T - splits[i / 2] : splits[i / 2]), "heads_bwd: gradient of another shape");
    hold.push_back(*g);
    ptr[i] = g->data_ptr();
    stride[i] = g->stride(0);
  }
  c10::cuda::CUDAGuard guard(src.device());
  Tensor out = at::empty({src.size(0), src.size(1)}, src.options());
  if (src.size(1) > (na + nb + nv) * hd || tokens == 0) out.zero_();
  const c10::optional<Tensor>* dws[2] = {&dw_a, &dw_b};
  Tensor partial[2];
  float* pp[2] = {nullptr, nullptr};
  void* pw[2] = {nullptr, nullptr};
  for (int i = 0; i < 2; ++i) {
    if (!dws[i]->has_value() || heads[i] == 0) continue;
    TORCH_CHECK((*dws[i])->scalar_type() == at::kBFloat16 && (*dws[i])->numel() == hd && (*dws[i])->is_contiguous());
    if (tokens == 0 && !(i ? acc_b : acc_a)) (*dws[i])->zero_();
    partial[i] = at::empty({sb200::heads_bwd_groups((int)tokens, heads[i]) + (repeated ? heads[i] : 0), hd}, rstd.options());
    pp[i] = partial[i].data_ptr<float>();
    pw[i] = (*dws[i])->data_ptr();
  }
  const void* w[2] = {head_weight(w_a, na, hd), head_weight(w_b, nb, hd)};
  const int acc[2] = {acc_a ? 1 : 0, acc_b ? 1 : 0};
  Tensor sums;
  if (repeated) sums = at::empty({sb200::repeated_part_floats((int)(T - tokens), (int)(na + nb + nv), (int)hd)}, rstd.options());
  sb200::launch_heads_bwd(ptr, stride, splits, src.data_ptr(), src.stride(0), w, rstd.data_ptr<float>(), pp, pw, acc, heads, out.data_ptr(), out.stride(0), (int)tokens, (int)T,
                          repeated ? sums.data_ptr<float>() : nullptr, positions.data_ptr<int64_t>(), cos_t.data_ptr<float>(), sin_t.data_ptr<float>(), cos_t.size(0), (int)hd, (int)rot, used_rows(live), cur_stream());
  return out;
}

// dst[0], dst[1] = the fp32 sum of all rows of d as a rounded row and what the rounding left
void repeated_rows_sum(const Tensor& d, Tensor dst) {
  check_rows(d, "d");
  check_rows(dst, "dst");
  TORCH_CHECK(d.size(0) >= 1 && dst.size(0) == 2 && dst.size(1) == d.size(1) && d.size(1) % 8 == 0);
  c10::cuda::CUDAGuard guard(d.device());
  Tensor part = at::empty({sb200::repeated_part_floats((int)d.size(0), (int)d.size(1), 1)}, d.options().dtype(at::kFloat));
  sb200::launch_repeated_rows_sum(d.data_ptr(), d.stride(0), (int)d.size(0), (int)d.size(1), part.data_ptr<float>(), dst.data_ptr(), dst.stride(0), cur_stream());
}

// ---- row bookkeeping -------------------------------------------------------------------------------
const int64_t* long_ptr(const Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kLong && t.is_contiguous(), name, ": contiguous int64 CUDA tensor expected");
  return t.data_ptr<int64_t>();
}
const bool* bool_ptr(const Tensor& t, int64_t n, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBool && t.is_contiguous() && t.numel() == n, name, ": contiguous bool CUDA tensor expected");
  return t.data_ptr<bool>();
}
std::tuple<Tensor, Tensor> document_interval(const Tensor& doc, int64_t window) {
  const int64_t* d = long_ptr(doc, "document_ids");
  c10::cuda::CUDAGuard guard(doc.device());
  Tensor both = at::empty({2, doc.numel()}, doc.options().dtype(at::kInt));
  Tensor lo = both.select(0, 0), hi = both.select(0, 1);
  sb200::launch_document_interval(d, (int)doc.numel(), (int)window, lo.data_ptr<int>(), hi.data_ptr<int>(), cur_stream());
  return {lo, hi};
}
// mask bool[T], keys fp32[T] in [0, 1) -> (anchors int64[slots] ascending and padded with zeros, which of them are, bool[slots])
std::tuple<Tensor, Tensor> select_anchors(const Tensor& mask, const Tensor& keys, int64_t slots, int64_t block) {
  const int64_t T = mask.numel();
  const bool* m = bool_ptr(mask, T, "mask");
  TORCH_CHECK(keys.is_cuda() && keys.scalar_type() == at::kFloat && keys.is_contiguous() && keys.numel() == T, "select_anchors: a float32 key per row expected");
  check_same_device(mask, {&keys});
  TORCH_CHECK(slots >= 0 && block > 0 && T < (int64_t(1) << 31) - 65536 && slots < (int64_t(1) << 31) - 65536);
  c10::cuda::CUDAGuard guard(mask.device());
  Tensor anchors = at::empty({slots}, mask.options().dtype(at::kLong)), picked = at::empty({slots}, mask.options());
  sb200::launch_select_anchors(m, keys.data_ptr<float>(), (int)T, (int)std::min<int64_t>(block, T), (int)slots, (int)std::min(slots, T),
                               anchors.data_ptr<int64_t>(), picked.data_ptr<bool>(), cur_stream());
  return {anchors, picked};
}
// doc_lo int32[T]: start of each row's document; window < 0: none -> lo, hi int32[n * block], extra int32[n * block, block]
std::tuple<Tensor, Tensor, Tensor> anchor_spec(const Tensor& doc, const Tensor& doc_lo, const Tensor& anchors, int64_t block, int64_t window, bool causal) {
  const int64_t T = doc.numel(), n = anchors.numel();
  const int64_t *d = long_ptr(doc, "document_ids"), *a = long_ptr(anchors, "anchors");
  TORCH_CHECK(doc_lo.is_cuda() && doc_lo.scalar_type() == at::kInt && doc_lo.is_contiguous() && doc_lo.numel() == T, "doc_lo: int32 per row expected");
  check_same_device(doc, {&doc_lo, &anchors});
  TORCH_CHECK(block > 0 && n * block * block < (int64_t(1) << 31) * 64 && n * block < (int64_t(1) << 31));
  c10::cuda::CUDAGuard guard(doc.device());
  auto opt = doc_lo.options();
  Tensor lo = at::empty({n * block}, opt), hi = at::empty({n * block}, opt), extra = at::empty({n * block, block}, opt);
  sb200::launch_anchor_spec(d, doc_lo.data_ptr<int>(), (int)T, a, (int)n, (int)block, (int)std::min<int64_t>(window, (int64_t(1) << 31) - 1), causal ? 1 : 0,
                            lo.data_ptr<int>(), hi.data_ptr<int>(), extra.data_ptr<int>(), cur_stream());
  return {lo, hi, extra};
}
// anchors as select_anchors gives them -> token, position, row, target row (int64[n * block]), counted (bool[n * block])
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> anchor_slots(const Tensor& anchors, const Tensor& picked, const Tensor& ids, const Tensor& positions,
                                                                const Tensor& mask, int64_t block, int64_t mask_token, bool from_anchor) {
  const int64_t T = mask.numel(), n = anchors.numel(), N = n * block;
  const int64_t *a = long_ptr(anchors, "anchors"), *i = long_ptr(ids, "ids"), *pos = long_ptr(positions, "positions");
  const bool *pk = bool_ptr(picked, n, "picked"), *m = bool_ptr(mask, T, "mask");
  check_same_device(anchors, {&picked, &ids, &positions, &mask});
  TORCH_CHECK(ids.numel() == T && positions.numel() == T && T > 0 && block > 0 && N < (int64_t(1) << 31));
  c10::cuda::CUDAGuard guard(anchors.device());
  Tensor of = at::empty({4, N}, anchors.options()), counts = at::empty({N}, mask.options());
  Tensor token = of.select(0, 0), position = of.select(0, 1), index = of.select(0, 2), target = of.select(0, 3);
  sb200::launch_anchor_slots(a, pk, i, pos, m, (int)T, (int)n, (int)block, mask_token, from_anchor ? 1 : 0, token.data_ptr<int64_t>(), position.data_ptr<int64_t>(),
                             index.data_ptr<int64_t>(), target.data_ptr<int64_t>(), counts.data_ptr<bool>(), cur_stream());
  return {token, position, index, target, counts};
}
// positions of the set entries -> (int64[T] of which the first count are filled, int32[1] count)
std::tuple<Tensor, Tensor> compact_rows(const Tensor& valid) {
  const bool* v = bool_ptr(valid, valid.numel(), "valid");
  c10::cuda::CUDAGuard guard(valid.device());
  Tensor list = at::empty({valid.numel()}, valid.options().dtype(at::kLong)), count = at::empty({1}, valid.options().dtype(at::kInt));
  sb200::launch_compact(v, (int)valid.numel(), list.data_ptr<int64_t>(), count.data_ptr<int>(), cur_stream());
  return {list, count};
}
// anchor / depths: int64[take] views the step fills; -> (picked int64[take], next pool int64[take], its size int32[1])
std::tuple<Tensor, Tensor, Tensor> cod_step(const Tensor& pool, const c10::optional<Tensor>& perm, int64_t take, const Tensor& valid, int64_t depth,
                                            bool filter_zero, Tensor anchor, Tensor depths) {
  const int64_t T = valid.numel();
  TORCH_CHECK(take >= 0 && take <= pool.numel() && anchor.numel() == take && depths.numel() == take && (!perm.has_value() || perm->numel() >= take));
  const bool* v = bool_ptr(valid, T, "valid");
  c10::cuda::CUDAGuard guard(valid.device());
  auto opt = valid.options();
  Tensor flags = at::empty({perm.has_value() ? T : 0}, opt.dtype(at::kByte)), picked = at::empty({take}, opt.dtype(at::kLong));
  Tensor next = at::empty({take}, opt.dtype(at::kLong)), count = at::empty({1}, opt.dtype(at::kInt));
  sb200::launch_cod_step(long_ptr(pool, "pool"), perm.has_value() ? long_ptr(*perm, "perm") : nullptr, (int)take, v, (int)T, (int)depth, filter_zero ? 1 : 0,
                         flags.data_ptr<uint8_t>(), picked.data_ptr<int64_t>(), const_cast<int64_t*>(long_ptr(anchor, "anchor")),
                         const_cast<int64_t*>(long_ptr(depths, "depths")), next.data_ptr<int64_t>(), count.data_ptr<int>(), cur_stream());
  return {picked, next, count};
}
// -> (lo, hi int32[n], extra int32[n, num_depths - 1] or empty)
std::tuple<Tensor, Tensor, Tensor> peagle_spec(const Tensor& anchor, const Tensor& depth, const c10::optional<Tensor>& row_valid, const Tensor& doc,
                                               const Tensor& doc_lo, int64_t num_depths, int64_t window) {
  const int64_t n = anchor.numel(), T = doc.numel();
  TORCH_CHECK(depth.numel() == n && doc_lo.numel() == T && doc_lo.scalar_type() == at::kInt && doc_lo.is_contiguous() && T > 0);
  c10::cuda::CUDAGuard guard(doc.device());
  auto opt = doc.options().dtype(at::kInt);
  const bool extras = num_depths > 1 && n > T;
  Tensor lo = at::empty({n}, opt), hi = at::empty({n}, opt), extra = at::empty({extras ? n : 0, num_depths - 1}, opt);
  Tensor table = extras ? at::full({num_depths, T}, -1, opt) : at::empty({0}, opt);
  sb200::launch_peagle_spec(long_ptr(anchor, "anchor_pos"), long_ptr(depth, "depth"), row_valid.has_value() ? bool_ptr(*row_valid, n, "row_valid") : nullptr,
                            long_ptr(doc, "document_ids"), doc_lo.data_ptr<int>(), (int)n, (int)T, (int)num_depths, (int)window, table.data_ptr<int>(),
                            lo.data_ptr<int>(), hi.data_ptr<int>(), extras ? extra.data_ptr<int>() : nullptr, cur_stream());
  return {lo, hi, extra};
}
// The rows a training-time-test step of S passes needs (see wanted_rows_kernel).  Without targets the second list stays unwritten.
// -> (index int64[2, T], inverse int32[2, T], count int32[2]; ids, positions int64[S, T], mask bool[S, T], prev bool[T], target_row int32[S, T],
//     intervals int32[n, 2, T] as given, extra keys int32[S (S - 1) / 2, T] flat)
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> step_rows(const Tensor& mask, const Tensor& ids, const Tensor& positions,
                                                                                                     const std::vector<Tensor>& intervals, int64_t passes, bool targets) {
  const int64_t T = positions.numel(), N = ids.numel(), S = passes;
  TORCH_CHECK(T > 0 && T < (int64_t{1} << 31) / std::max<int64_t>(S * S, 1) && S >= 1 && intervals.size() <= 2 && N >= T && mask.numel() == N &&
              mask.is_cuda() && (!targets || N == T));
  c10::cuda::CUDAGuard guard(ids.device());
  const auto l = ids.options().dtype(at::kLong), n = ids.options().dtype(at::kInt), b = ids.options().dtype(at::kBool);
  Tensor index = at::empty({2, T}, l), inverse = at::empty({2, T}, n), count = at::empty({2}, n);
  Tensor ids_out = at::empty({S, T}, l), pos_out = at::empty({S, T}, l), mask_out = at::empty({S, T}, b), prev = at::empty({T}, b);
  Tensor target_row = at::empty({targets ? S : 0, T}, n), spans = at::empty({(int64_t)intervals.size(), 2, T}, n), extra = at::empty({S * (S - 1) / 2, T}, n);
  const int* in[2] = {nullptr, nullptr};
  int* out[2] = {nullptr, nullptr};
  for (size_t k = 0; k < intervals.size(); ++k) {
    TORCH_CHECK(intervals[k].is_cuda() && intervals[k].scalar_type() == at::kInt && intervals[k].is_contiguous() && intervals[k].dim() == 2 && intervals[k].size(0) == 2 &&
                intervals[k].size(1) == T, "step_rows: intervals are contiguous int32 [2, T]");
    in[k] = intervals[k].data_ptr<int>();
    out[k] = spans.select(0, (int64_t)k).data_ptr<int>();
  }
  sb200::launch_step_rows(row_flags(mask, N), long_ptr(ids, "ids"), long_ptr(positions, "positions"), in, (int)T, (int)N, (int)S, index.data_ptr<int64_t>(),
                          inverse.data_ptr<int>(), count.data_ptr<int>(), ids_out.data_ptr<int64_t>(), pos_out.data_ptr<int64_t>(),
                          reinterpret_cast<uint8_t*>(mask_out.data_ptr()), reinterpret_cast<uint8_t*>(prev.data_ptr()), targets ? target_row.data_ptr<int>() : nullptr, out,
                          extra.data_ptr<int>(), cur_stream());
  return {index, inverse, count, ids_out, pos_out, mask_out, prev, target_row, spans, extra};
}
struct RowCopyArgs {
  const void* from[2];
  void* to[2];
  int64_t stride[2];
  int W[2];
  std::vector<Tensor> out;
};
RowCopyArgs row_copy_args(const std::vector<Tensor>& x, int64_t rows) {
  TORCH_CHECK(x.size() == 1 || x.size() == 2, "one or two matrices");
  RowCopyArgs a{};
  for (size_t i = 0; i < x.size(); ++i) {
    check_rows(x[i], "rows");
    TORCH_CHECK(x[i].size(1) % 8 == 0 && x[i].device() == x[0].device());
    a.out.push_back(at::empty({rows, x[i].size(1)}, x[i].options()));
    a.from[i] = x[i].data_ptr();
    a.to[i] = a.out[i].data_ptr();
    a.stride[i] = x[i].stride(0);
    a.W[i] = (int)x[i].size(1);
  }
  return a;
}
// out[r] = x[index[r]] for r < live, for one or two matrices (index: rows of x, not checked); put_rows is its gradient
std::vector<Tensor> take_rows(const std::vector<Tensor>& x, const Tensor& index, const c10::optional<Tensor>& live) {
  c10::cuda::CUDAGuard guard(index.device());
  RowCopyArgs a = row_copy_args(x, index.numel());
  sb200::launch_take_rows((int)x.size(), a.from, a.stride, a.W, a.to, long_ptr(index, "index"), used_rows(live), (int)index.numel(), cur_stream());
  return a.out;
}
std::vector<Tensor> put_rows(const std::vector<Tensor>& d, const Tensor& inverse) {
  TORCH_CHECK(inverse.is_cuda() && inverse.scalar_type() == at::kInt && inverse.is_contiguous());
  c10::cuda::CUDAGuard guard(inverse.device());
  RowCopyArgs a = row_copy_args(d, inverse.numel());
  sb200::launch_put_rows((int)d.size(), a.from, a.stride, a.W, a.to, inverse.data_ptr<int>(), (int)inverse.numel(), cur_stream());
  return a.out;
}
// dw rows of the ids (ascending, `order` their source rows of d) stored or added to
void embedding_bwd(const Tensor& ids, const Tensor& order, const Tensor& d, int64_t padding, Tensor dw, bool accumulate) {
  check_rows(d, "d");
  TORCH_CHECK(ids.numel() == d.size(0) && order.numel() == d.size(0) && dw.dim() == 2 && dw.is_contiguous() && dw.scalar_type() == at::kBFloat16 &&
              dw.size(1) == d.size(1) && d.size(1) % 8 == 0 && (reinterpret_cast<uintptr_t>(dw.data_ptr()) & 15) == 0);
  c10::cuda::CUDAGuard guard(d.device());
  Tensor part = at::empty({sb200::embedding_bwd_partial_rows((int)d.size(0)), d.size(1)}, d.options().dtype(at::kFloat));
  sb200::launch_embedding_bwd(long_ptr(ids, "ids"), long_ptr(order, "order"), d.data_ptr(), d.stride(0), (int)d.size(0), (int)d.size(1), dw.size(0), padding,
                              dw.data_ptr(), accumulate ? 1 : 0, part.data_ptr<float>(), cur_stream());
}

Tensor swiglu_fwd(const Tensor& gate_up, const c10::optional<Tensor>& rows_used) {
  check_rows(gate_up, "gate_up");
  TORCH_CHECK(gate_up.is_contiguous() && gate_up.size(1) % 16 == 0);
  const int64_t rows = gate_up.size(0);
  const int I = (int)(gate_up.size(1) / 2);
  c10::cuda::CUDAGuard guard(gate_up.device());
  Tensor h = at::empty({rows, I}, gate_up.options());
  sb200::launch_swiglu_fwd(gate_up.data_ptr(), h.data_ptr(), rows, I, used_rows(rows_used), cur_stream());
  return h;
}

Tensor swiglu_bwd_rows(const Tensor& dh, const Tensor& gate_up, const c10::optional<Tensor>& rows_used) {
  check_rows(gate_up, "gate_up");
  check_rows(dh, "dh");
  TORCH_CHECK(gate_up.is_contiguous() && dh.is_contiguous() && dh.size(1) * 2 == gate_up.size(1));
  c10::cuda::CUDAGuard guard(gate_up.device());
  Tensor out = at::empty_like(gate_up);
  sb200::launch_swiglu_bwd(dh.data_ptr(), gate_up.data_ptr(), out.data_ptr(), gate_up.size(0),
                           (int)dh.size(1), used_rows(rows_used), cur_stream());
  return out;
}
Tensor swiglu_bwd(const Tensor& dh, const Tensor& gate_up) { return swiglu_bwd_rows(dh, gate_up, c10::nullopt); }

// [q | k | v] gradients (2-D rows, k and v optional) side by side, rotated back where marked (q always, k with rotate_k).
Tensor rope_merge(const Tensor& q, const c10::optional<Tensor>& k, const c10::optional<Tensor>& v, bool rotate_k, const Tensor& positions, const Tensor& cos_t,
                  const Tensor& sin_t, int64_t hd, int64_t rot, double sign, const c10::optional<Tensor>& live) {
  check_rotation(positions, cos_t, sin_t, q.size(0), hd, rot);
  const Tensor* parts[3] = {&q, k.has_value() ? &*k : nullptr, v.has_value() ? &*v : nullptr};
  const void* src[3] = {nullptr, nullptr, nullptr};
  int64_t stride[3] = {0, 0, 0}, width = 0;
  int heads[3] = {0, 0, 0}, rotate[3] = {1, rotate_k ? 1 : 0, 0};
  for (int i = 0; i < 3; ++i) {
    if (parts[i] == nullptr) continue;
    check_rows(*parts[i], "rope_merge input");
    TORCH_CHECK(parts[i]->size(0) == q.size(0) && parts[i]->size(1) % hd == 0, "rope_merge: whole heads of the same rows expected");
    src[i] = parts[i]->data_ptr();
    stride[i] = parts[i]->stride(0);
    heads[i] = (int)(parts[i]->size(1) / hd);
    width += parts[i]->size(1);
  }
  c10::cuda::CUDAGuard guard(q.device());
  Tensor out = at::empty({q.size(0), width}, q.options());
  sb200::launch_rope_merge(src, stride, heads, rotate, out.data_ptr(), width, positions.data_ptr<int64_t>(), cos_t.data_ptr<float>(), sin_t.data_ptr<float>(),
                           cos_t.size(0), (int)q.size(0), (int)hd, (int)rot, (float)sign, used_rows(live), cur_stream());
  return out;
}

// ---- gated attention ---------------------------------------------------------------------------
// out: contiguous [T, heads, hd]; gate: [T, heads, hd] view with unit inner stride (a half of each head's projection).
void check_gate(const Tensor& out, const Tensor& gate, const char* name) {
  TORCH_CHECK(out.is_cuda() && out.scalar_type() == at::kBFloat16 && out.dim() == 3 && out.is_contiguous() && out.size(2) % 8 == 0);
  TORCH_CHECK(gate.is_cuda() && gate.scalar_type() == at::kBFloat16 && gate.sizes() == out.sizes() && gate.stride(2) == 1 && gate.stride(1) % 8 == 0 &&
              gate.stride(0) % 8 == 0 && (reinterpret_cast<uintptr_t>(gate.data_ptr()) & 15) == 0, name, ": strided [T, heads, hd] with aligned rows expected");
}
Tensor gate_mul_fwd(const Tensor& out, const Tensor& gate) {
  check_gate(out, gate, "gate");
  c10::cuda::CUDAGuard guard(out.device());
  Tensor y = at::empty_like(out);
  sb200::launch_gate_mul_fwd(out.data_ptr(), gate.data_ptr(), y.data_ptr(), (int)out.size(0), (int)out.size(1), (int)out.size(2), gate.stride(0),
                             (int)gate.stride(1), cur_stream());
  return y;
}
Tensor gate_mul_bwd(const Tensor& dy, const Tensor& out, const Tensor& gate, Tensor dgate) {
  check_gate(out, gate, "gate");
  check_gate(out, dgate, "dgate");
  TORCH_CHECK(dy.sizes() == out.sizes() && dy.is_contiguous() && dy.scalar_type() == at::kBFloat16 && dgate.stride(1) == gate.stride(1));
  c10::cuda::CUDAGuard guard(out.device());
  Tensor dout = at::empty_like(out);
  sb200::launch_gate_mul_bwd(dy.data_ptr(), out.data_ptr(), gate.data_ptr(), dout.data_ptr(), dgate.data_ptr(), (int)out.size(0), (int)out.size(1),
                             (int)out.size(2), gate.stride(0), (int)gate.stride(1), dgate.stride(0), cur_stream());
  return dout;
}

// ---- mixture-of-experts row movement ---------------------------------------------------------------
// columns of the k largest of every row, descending, equal ones by column: fp32 [rows, E <= 1024] -> int64 [rows, k]
Tensor topk_rows(const Tensor& p, int64_t k) {
  TORCH_CHECK(p.is_cuda() && p.scalar_type() == at::kFloat && p.dim() == 2 && p.is_contiguous() && p.size(1) <= 1024 && k >= 1 && k <= p.size(1), "topk_rows");
  c10::cuda::CUDAGuard guard(p.device());
  Tensor index = at::empty({p.size(0), k}, p.options().dtype(at::kLong));
  const int rc = sb200::launch_topk_rows(p.data_ptr<float>(), (int)p.size(0), (int)p.size(1), (int)k, index.data_ptr<int64_t>(), cur_stream());
  TORCH_CHECK(rc == 0, "topk_rows launch failed (", rc, ")");
  return index;
}
// expert int64[T, k] -> (seg int32[E + 1], 256-row tile prefix int32[E + 1], slot_row int32[T * k], row_slot int32[capacity]).
std::tuple<Tensor, Tensor, Tensor, Tensor> moe_plan(const Tensor& expert, int64_t E, int64_t capacity, int64_t k, const c10::optional<Tensor>& live) {
  TORCH_CHECK(k >= 1 && expert.numel() % k == 0, "moe_plan: k slots per token");
  TORCH_CHECK(expert.is_cuda() && expert.scalar_type() == at::kLong && expert.is_contiguous() && expert.numel() > 0);
  TORCH_CHECK(E >= 1 && E <= 1024 && capacity >= (expert.numel() + 127 * E + 127) / 128 * 128, "moe_plan: at most 1024 experts and room for every padded segment");
  c10::cuda::CUDAGuard guard(expert.device());
  auto opt = expert.options().dtype(at::kInt);
  const int n = (int)expert.numel();
  Tensor hist = at::empty({sb200::moe_plan_blocks(n), E}, opt), seg = at::empty({E + 1}, opt), tiles = at::empty({E + 1}, opt);
  Tensor slot_row = at::empty({n}, opt), row_slot = at::empty({capacity}, opt);
  const int rc = sb200::launch_moe_plan(expert.data_ptr<int64_t>(), n, (int)E, (int)capacity, hist.data_ptr<int>(), seg.data_ptr<int>(), tiles.data_ptr<int>(),
                                        slot_row.data_ptr<int>(), row_slot.data_ptr<int>(), used_rows(live), (int)k, cur_stream());
  TORCH_CHECK(rc == 0, "moe_plan launch failed (", rc, ")");
  return {seg, tiles, slot_row, row_slot};
}
const int* int_ptr(const Tensor& t, int64_t least, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kInt && t.is_contiguous() && t.numel() >= least, name, ": int32 CUDA tensor expected");
  return t.data_ptr<int>();
}
// the used row count is the last entry of seg
const int* rows_used_of(const Tensor& seg) { return int_ptr(seg, 2, "seg") + (seg.numel() - 1); }

Tensor moe_gather(const Tensor& x, const Tensor& row_slot, const Tensor& seg, int64_t k) {
  check_rows(x, "x");
  const int64_t cap = row_slot.numel(), H = x.size(1);
  TORCH_CHECK(H % 8 == 0);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor out = at::empty({cap, H}, x.options());
  sb200::launch_moe_gather(x.data_ptr(), x.stride(0), int_ptr(row_slot, 1, "row_slot"), rows_used_of(seg), (int)k, out.data_ptr(), (int)cap, (int)H, cur_stream());
  return out;
}
Tensor moe_gather_bwd(const Tensor& d_pad, const Tensor& slot_row, int64_t k, const c10::optional<Tensor>& live) {
  check_rows(d_pad, "d_pad");
  TORCH_CHECK(d_pad.is_contiguous() && d_pad.size(1) % 8 == 0 && slot_row.numel() % k == 0);
  const int64_t T = slot_row.numel() / k, H = d_pad.size(1);
  c10::cuda::CUDAGuard guard(d_pad.device());
  Tensor dx = at::empty({T, H}, d_pad.options());
  sb200::launch_moe_gather_bwd(d_pad.data_ptr(), int_ptr(slot_row, 1, "slot_row"), (int)k, dx.data_ptr(), (int)T, (int)H, used_rows(live), cur_stream());
  return dx;
}
const void* token_rows(const c10::optional<Tensor>& t, int64_t T, int64_t W, const char* name) {
  if (!t.has_value()) return nullptr;
  TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->is_contiguous() && t->numel() == T * W, name, ": contiguous bf16 [T, .] expected");
  return t->data_ptr();
}
Tensor moe_combine(const Tensor& y_pad, const Tensor& slot_row, const Tensor& p, const c10::optional<Tensor>& shared, const c10::optional<Tensor>& gate,
                   const c10::optional<Tensor>& residual, const c10::optional<Tensor>& live) {
  check_rows(y_pad, "y_pad");
  TORCH_CHECK(y_pad.is_contiguous() && p.dim() == 2 && p.is_contiguous() && p.scalar_type() == at::kBFloat16 && p.numel() == slot_row.numel());
  TORCH_CHECK(shared.has_value() == gate.has_value(), "moe_combine: the shared expert comes with its gate");
  const int64_t T = p.size(0), k = p.size(1), H = y_pad.size(1);
  c10::cuda::CUDAGuard guard(y_pad.device());
  Tensor out = at::empty({T, H}, y_pad.options());
  sb200::launch_moe_combine(y_pad.data_ptr(), int_ptr(slot_row, 1, "slot_row"), p.data_ptr(), (int)k, token_rows(shared, T, H, "shared"), token_rows(gate, T, 1, "gate"),
                            token_rows(residual, T, H, "residual"), out.data_ptr(), (int)T, (int)H, used_rows(live), cur_stream());
  return out;
}
// -> (dy_pad, dp, dshared, dgate); the last two empty without a shared expert
std::tuple<Tensor, Tensor, Tensor, Tensor> moe_combine_bwd(const Tensor& dout, const Tensor& y_pad, const Tensor& row_slot, const Tensor& seg, const Tensor& p,
                                                           const c10::optional<Tensor>& shared, const c10::optional<Tensor>& gate,
                                                           const c10::optional<Tensor>& live) {
  check_rows(y_pad, "y_pad");
  const int64_t T = p.size(0), k = p.size(1), H = y_pad.size(1), cap = row_slot.numel();
  TORCH_CHECK(y_pad.is_contiguous() && y_pad.size(0) == cap && p.is_contiguous() && p.scalar_type() == at::kBFloat16);
  c10::cuda::CUDAGuard guard(y_pad.device());
  Tensor dy_pad = at::empty_like(y_pad), dp = at::empty_like(p);
  Tensor dshared = at::empty({shared.has_value() ? T : 0, H}, y_pad.options()), dgate = at::empty({shared.has_value() ? T : 0, 1}, y_pad.options());
  sb200::launch_moe_combine_bwd(token_rows(dout, T, H, "dout"), y_pad.data_ptr(), int_ptr(row_slot, 1, "row_slot"), rows_used_of(seg), p.data_ptr(), (int)k,
                                dy_pad.data_ptr(), dp.data_ptr(), token_rows(shared, T, H, "shared"), token_rows(gate, T, 1, "gate"), dshared.data_ptr(),
                                dgate.data_ptr(), (int)T, (int)cap, (int)H, used_rows(live), cur_stream());
  return {dy_pad, dp, dshared, dgate};
}

// x: [tokens, >= heads*hd] view (row stride arbitrary); rotates the first `heads` heads in place.
void rope_(Tensor x, const Tensor& positions, const Tensor& cos_t, const Tensor& sin_t, int64_t heads,
           int64_t hd, int64_t rot, double sign, const c10::optional<Tensor>& live) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1);
  TORCH_CHECK(x.size(1) >= heads * hd && rot % 2 == 0 && rot <= hd);
  TORCH_CHECK(positions.scalar_type() == at::kLong && positions.is_contiguous() &&
              positions.numel() == x.size(0));
  TORCH_CHECK(cos_t.scalar_type() == at::kFloat && sin_t.scalar_type() == at::kFloat &&
              cos_t.is_contiguous() && sin_t.is_contiguous() && cos_t.dim() == 2 &&
              cos_t.size(1) == rot / 2 && sin_t.sizes() == cos_t.sizes());
  c10::cuda::CUDAGuard guard(x.device());
  sb200::launch_rope(x.data_ptr(), positions.data_ptr<int64_t>(), cos_t.data_ptr<float>(),
                     sin_t.data_ptr<float>(), x.size(0), (int)heads, (int)hd, (int)rot, x.stride(0),
                     cos_t.size(0), (float)sign, used_rows(live), cur_stream());
}


// int32[rows]: the row of the targets each row is compared with, -1 for none
const int* row_targets(const c10::optional<Tensor>& t, int64_t rows) {
  if (!t.has_value()) return nullptr;
  TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kInt && t->is_contiguous() && t->numel() >= rows, "int32 target rows expected");
  return t->data_ptr<int>();
}

// target_row: rows of `targets` to compare with, in place of a shift (they are not checked against its size)
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> loss_fwd_tv(int64_t op, const Tensor& logits, const Tensor& targets, const c10::optional<Tensor>& active,
                                                           const c10::optional<Tensor>& also, int64_t shift, int64_t rows,
                                                           const c10::optional<Tensor>& target_row, bool with_tv) {
  TORCH_CHECK(logits.is_cuda() && targets.is_cuda());
  TORCH_CHECK(logits.scalar_type() == at::kBFloat16 && targets.scalar_type() == at::kBFloat16);
  TORCH_CHECK(logits.dim() == 2 && targets.dim() == 2 && logits.stride(1) == 1 &&
              targets.stride(1) == 1 && logits.size(1) == targets.size(1));
  TORCH_CHECK(rows >= 0 && rows <= logits.size(0) && (target_row.has_value() || (rows + shift <= targets.size(0) && shift >= 0)));
  c10::cuda::CUDAGuard guard(logits.device());
  auto fopt = logits.options().dtype(at::kFloat);
  Tensor loss = at::empty({rows}, fopt);
  Tensor stats = at::empty({5, rows}, fopt);
  Tensor am_d = at::empty({rows}, logits.options().dtype(at::kInt));
  Tensor am_t = at::empty({rows}, logits.options().dtype(at::kInt));
  Tensor tv = at::empty({with_tv ? rows : 0}, fopt);
  const int rc = sb200::launch_loss_fwd((int)op, logits.data_ptr(), targets.data_ptr(), row_flags(active, rows), row_flags(also, rows), nullptr,
                                        loss.data_ptr<float>(), stats.data_ptr<float>(),
                                        am_d.data_ptr<int>(), am_t.data_ptr<int>(), (int)rows,
                                        (int)logits.size(1), logits.stride(0), targets.stride(0),
                                        (int)shift, row_targets(target_row, rows), with_tv ? tv.data_ptr<float>() : nullptr, cur_stream());
  TORCH_CHECK(rc == 0, "loss_fwd: unknown op ", op);
  return {loss, stats, am_d, am_t, tv};
}
std::tuple<Tensor, Tensor, Tensor, Tensor> loss_fwd_either(int64_t op, const Tensor& logits, const Tensor& targets, const c10::optional<Tensor>& active,
                                                           const c10::optional<Tensor>& also, int64_t shift, int64_t rows,
                                                           const c10::optional<Tensor>& target_row) {
  auto [loss, stats, am_d, am_t, tv] = loss_fwd_tv(op, logits, targets, active, also, shift, rows, target_row, false);
  return {loss, stats, am_d, am_t};
}
std::tuple<Tensor, Tensor, Tensor, Tensor> loss_fwd(int64_t op, const Tensor& logits, const Tensor& targets, const c10::optional<Tensor>& active, int64_t shift,
                                                    int64_t rows) {
  return loss_fwd_either(op, logits, targets, active, c10::nullopt, shift, rows, c10::nullopt);
}

// ---- grouped (mixture-of-experts) products ----------------------------------------------------
// counts int32[E] (device) -> (seg int32[E + 1], mtile_start int32[E + 1]): 128-row aligned segment offsets of the
// padded row order and the prefix sum of 256-row tiles per expert.  Nothing is read back to the host.
std::tuple<Tensor, Tensor> moe_group_plan(const Tensor& counts) {
  TORCH_CHECK(counts.is_cuda() && counts.scalar_type() == at::kInt && counts.is_contiguous() && counts.dim() == 1);
  c10::cuda::CUDAGuard guard(counts.device());
  const int64_t E = counts.numel();
  Tensor seg = at::empty({E + 1}, counts.options());
  Tensor mts = at::empty({E + 1}, counts.options());
  sb200::launch_moe_group_plan(counts.data_ptr<int>(), (int)E, seg.data_ptr<int>(), mts.data_ptr<int>(), cur_stream());
  return {seg, mts};
}

// out[R, N] = x[R, K] . w_e^T for the rows of expert e (w: [E, N, K]); with `transposed` the weight is
// [E, K, N] read in place (input gradient: out[R, N] = x[R, K] . w_e).  Rows follow the padded order of moe_group_plan.
void gemm_grouped_rows(const Tensor& x, const Tensor& w, Tensor out, bool transposed, const Tensor& seg, const Tensor& mts, Tensor status) {
  check_rows(x, "x");
  check_rows(out, "out");
  TORCH_CHECK(w.is_cuda() && w.scalar_type() == at::kBFloat16 && w.dim() == 3 && w.is_contiguous(), "w must be a contiguous bf16 [E, ., .] stack");
  const int64_t E = w.size(0), R = x.size(0), K = x.size(1);
  const int64_t N = transposed ? w.size(2) : w.size(1);
  TORCH_CHECK((transposed ? w.size(1) : w.size(2)) == K && out.size(0) == R && out.size(1) == N, "gemm_grouped_rows: shape mismatch");
  TORCH_CHECK(K % 128 == 0 && N % 256 == 0 && R % 128 == 0, "gemm_grouped_rows: K % 128, N % 256 and rows % 128 must be 0");
  TORCH_CHECK(seg.is_cuda() && seg.scalar_type() == at::kInt && seg.numel() == E + 1 && mts.scalar_type() == at::kInt && mts.numel() == E + 1);
  c10::cuda::CUDAGuard guard(x.device());
  const int rc = sb200::launch_gemm_grouped(x.data_ptr(), w.data_ptr(), out.data_ptr(), (int)R, (int)N, (int)K, x.stride(0), w.stride(1),
                                            out.stride(0), 0, 1, transposed ? 1 : 0, seg.data_ptr<int>(), mts.data_ptr<int>(), (int)E,
                                            status.data_ptr<int>(), cur_stream());
  TORCH_CHECK(rc == 0, "gemm_grouped_rows launch failed (", rc, ")");
}

// (gate_up [R, 2 I], h [R, I] = silu(gate) * up) for stacked [gate; up] experts w: [E, 2 I, K].
std::tuple<Tensor, Tensor> gemm_grouped_swiglu(const Tensor& x, const Tensor& w, const Tensor& seg, const Tensor& mts, Tensor status) {
  check_rows(x, "x");
  TORCH_CHECK(w.is_cuda() && w.scalar_type() == at::kBFloat16 && w.dim() == 3 && w.is_contiguous(), "w must be a contiguous bf16 [E, 2 I, K] stack");
  const int64_t E = w.size(0), R = x.size(0), K = x.size(1), I = w.size(1) / 2;
  TORCH_CHECK(w.size(2) == K && K % 128 == 0 && w.size(1) == 2 * I && I % 128 == 0 && R % 128 == 0, "gemm_grouped_swiglu: shape mismatch");
  TORCH_CHECK(seg.is_cuda() && seg.scalar_type() == at::kInt && seg.numel() == E + 1 && mts.scalar_type() == at::kInt && mts.numel() == E + 1);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor gate_up = at::empty({R, 2 * I}, x.options()), h = at::empty({R, I}, x.options());
  const int rc = sb200::launch_gemm_grouped_swiglu(x.data_ptr(), w.data_ptr(), gate_up.data_ptr(), h.data_ptr(), (int)R, (int)I, (int)K, x.stride(0), K,
                                                   seg.data_ptr<int>(), mts.data_ptr<int>(), (int)E, status.data_ptr<int>(), cur_stream());
  TORCH_CHECK(rc == 0, "gemm_grouped_swiglu launch failed (", rc, ")");
  return {gate_up, h};
}

// dw[e] (=, +=) dy[seg_e, :]^T . x[seg_e, :]  (dw: [E, M, N], dy: [R, M], x: [R, N]); an expert without rows gets zeros (store) / is left alone (accumulate).
void gemm_grouped_wgrad_parts(const std::vector<Tensor>& dy, const std::vector<Tensor>& x, Tensor dw, bool accumulate, const std::vector<Tensor>& seg,
                              const Tensor& mts, Tensor status) {
  TORCH_CHECK(dw.is_cuda() && dw.scalar_type() == at::kBFloat16 && dw.dim() == 3 && dw.is_contiguous());
  const int64_t E = dw.size(0), M = dw.size(1), N = dw.size(2);
  const size_t n = dy.size();
  TORCH_CHECK(n >= 1 && n <= 4 && x.size() == n && seg.size() == n, "gemm_grouped_wgrad: one to four uses");
  const void *a[4], *b[4];
  const int* sp[4];
  int K[4];
  int64_t lda[4], ldb[4];
  for (size_t i = 0; i < n; ++i) {
    check_rows(dy[i], "dy");
    check_rows(x[i], "x");
    TORCH_CHECK(dy[i].size(1) == M && x[i].size(1) == N && x[i].size(0) == dy[i].size(0) && dy[i].size(0) % 128 == 0, "gemm_grouped_wgrad: shape mismatch");
    TORCH_CHECK(seg[i].is_cuda() && seg[i].scalar_type() == at::kInt && seg[i].numel() == E + 1);
    a[i] = dy[i].data_ptr();
    b[i] = x[i].data_ptr();
    sp[i] = seg[i].data_ptr<int>();
    K[i] = (int)dy[i].size(0);
    lda[i] = dy[i].stride(0);
    ldb[i] = x[i].stride(0);
  }
  c10::cuda::CUDAGuard guard(dw.device());
  const int rc = sb200::launch_gemm_grouped_parts((int)n, a, b, K, lda, ldb, sp, dw.data_ptr(), (int)M, (int)N, accumulate ? 1 : 0, mts.data_ptr<int>(), (int)E,
                                                  status.data_ptr<int>(), cur_stream());
  TORCH_CHECK(rc == 0, "gemm_grouped_wgrad launch failed (", rc, ")");
}
void gemm_grouped_wgrad(const Tensor& dy, const Tensor& x, Tensor dw, bool accumulate, const Tensor& seg, const Tensor& mts, Tensor status) {
  gemm_grouped_wgrad_parts({dy}, {x}, dw, accumulate, {seg}, mts, status);
}

// dw (+)= sum_i dy_i^T . x_i: the weight gradient over several uses of a weight
// live: how many rows of each use count (one int32 per use, an empty tensor: all; an empty list: all of every use)
void gemm_wgrad_parts_rows(const std::vector<Tensor>& dy, const std::vector<Tensor>& x, Tensor dw, bool accumulate, Tensor status,
                           const std::vector<Tensor>& live) {
  check_rows(dw, "dw");
  const int64_t M = dw.size(0), N = dw.size(1);
  const size_t n = dy.size();
  TORCH_CHECK(n >= 1 && n <= 4 && x.size() == n && (live.empty() || live.size() == n), "gemm_wgrad_parts: one to four uses");
  const void *a[4], *b[4];
  const int* rows_of[4];
  int K[4];
  int64_t lda[4], ldb[4];
  for (size_t i = 0; i < n; ++i) {
    check_rows(dy[i], "dy");
    check_rows(x[i], "x");
    TORCH_CHECK(dy[i].size(1) == M && x[i].size(1) == N && x[i].size(0) == dy[i].size(0) && dy[i].size(0) > 0, "gemm_wgrad_parts: shape mismatch");
    rows_of[i] = live.empty() || live[i].numel() == 0 ? nullptr : used_rows(live[i]);
    a[i] = dy[i].data_ptr();
    b[i] = x[i].data_ptr();
    K[i] = (int)dy[i].size(0);
    lda[i] = dy[i].stride(0);
    ldb[i] = x[i].stride(0);
  }
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 1);
  c10::cuda::CUDAGuard guard(dw.device());
  TorchSplitSpace space(dw);
  const int rc = sb200::launch_gemm_parts((int)n, a, b, K, lda, ldb, rows_of, dw.data_ptr(), (int)M, (int)N, dw.stride(0), accumulate ? 1 : 0, status.data_ptr<int>(),
                                          &space, cur_stream());
  TORCH_CHECK(rc == 0, "gemm_wgrad_parts launch failed (", rc, ")");
}

void gemm_wgrad_parts(const std::vector<Tensor>& dy, const std::vector<Tensor>& x, Tensor dw, bool accumulate, Tensor status) {
  gemm_wgrad_parts_rows(dy, x, dw, accumulate, status, {});
}

// lm_head product fused with the row loss: logits = x @ w^T on the tcgen05 kernel whose epilogue also
// reduces every (row, 256-column tile) of the logits and of targets[row + shift] to online-softmax
// records; a second kernel merges them into the outputs of loss_fwd.  op 0 (KL) or 3 (CE on the argmax).
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> lmhead_loss_fwd(int64_t op, const Tensor& x, const Tensor& w, const Tensor& targets,
                                                                   const c10::optional<Tensor>& active, int64_t shift, int64_t rows,
                                                                   Tensor status) {
  check_rows(x, "x");
  check_rows(w, "w");
  check_rows(targets, "targets");
  TORCH_CHECK(op == 0 || op == 3, "lmhead_loss_fwd: op 0 (kl) or 3 (ce)");
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  TORCH_CHECK(w.size(1) == K && targets.size(1) == N && N % 8 == 0, "lmhead_loss_fwd: shape mismatch");
  TORCH_CHECK(rows >= 0 && rows <= M && shift >= 0 && rows + shift <= targets.size(0));
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 1);
  c10::cuda::CUDAGuard guard(x.device());
  auto fopt = x.options().dtype(at::kFloat);
  const int tiles_n = sb200::lmhead_tiles_n((int)N);
  Tensor logits = at::empty({M, N}, x.options());
  Tensor partial = at::empty({M, tiles_n, sb200::lmhead_stat_words()}, fopt);
  Tensor loss = at::empty({rows}, fopt);
  Tensor stats = at::empty({5, rows}, fopt);
  Tensor am_d = at::empty({rows}, x.options().dtype(at::kInt));
  Tensor am_t = at::empty({rows}, x.options().dtype(at::kInt));
  const uint8_t* act = nullptr;
  if (active.has_value()) {
    TORCH_CHECK((active->scalar_type() == at::kBool || active->scalar_type() == at::kByte) && active->is_contiguous() &&
                active->numel() == rows);
    act = reinterpret_cast<const uint8_t*>(active->data_ptr());
  }
  int rc = sb200::launch_lmhead_logits_stats(x.data_ptr(), w.data_ptr(), logits.data_ptr(), targets.data_ptr(), (int)M, (int)N, (int)K,
                                             x.stride(0), w.stride(0), logits.stride(0), targets.stride(0), (int)targets.size(0),
                                             (int)shift, partial.data_ptr<float>(), status.data_ptr<int>(), cur_stream());
  TORCH_CHECK(rc == 0, "lmhead_loss_fwd: GEMM launch failed (", rc, ")");
  rc = sb200::launch_lmhead_combine(partial.data_ptr<float>(), logits.data_ptr(), act, loss.data_ptr<float>(), stats.data_ptr<float>(),
                                    am_d.data_ptr<int>(), am_t.data_ptr<int>(), (int)rows, tiles_n, logits.stride(0), (int)op, cur_stream());
  TORCH_CHECK(rc == 0, "lmhead_loss_fwd: combine launch failed (", rc, ")");
  return {logits, loss, stats, am_d, am_t};
}

// Token cross-entropy: labels int64[rows]; rows with keep == 0 cost nothing and get loss 0.
std::tuple<Tensor, Tensor> ce_label_fwd(const Tensor& logits, const Tensor& labels, const c10::optional<Tensor>& keep) {
  TORCH_CHECK(logits.is_cuda() && logits.scalar_type() == at::kBFloat16 && logits.dim() == 2 && logits.stride(1) == 1);
  const int64_t rows = logits.size(0);
  TORCH_CHECK(labels.scalar_type() == at::kLong && labels.is_contiguous() && labels.numel() == rows);
  c10::cuda::CUDAGuard guard(logits.device());
  auto fopt = logits.options().dtype(at::kFloat);
  Tensor loss = at::empty({rows}, fopt);
  Tensor stats = at::empty({5, rows}, fopt);
  const uint8_t* act = nullptr;
  if (keep.has_value()) {
    TORCH_CHECK((keep->scalar_type() == at::kBool || keep->scalar_type() == at::kByte) && keep->is_contiguous() && keep->numel() == rows);
    act = reinterpret_cast<const uint8_t*>(keep->data_ptr());
  }
  const int rc = sb200::launch_loss_fwd(3, logits.data_ptr(), nullptr, act, nullptr, labels.data_ptr<int64_t>(), loss.data_ptr<float>(),
                                        stats.data_ptr<float>(), nullptr, nullptr, (int)rows, (int)logits.size(1),
                                        logits.stride(0), logits.stride(0), 0, nullptr, nullptr, cur_stream());
  TORCH_CHECK(rc == 0, "ce_label_fwd failed (", rc, ")");
  return {loss, stats};
}

Tensor loss_bwd_scaled(int64_t op, const Tensor& logits, const Tensor& targets, const Tensor& grad_out, const c10::optional<Tensor>& grad_scale,
                       const Tensor& stats, int64_t shift, int64_t rows, const c10::optional<Tensor>& target_row, const c10::optional<Tensor>& live) {
  TORCH_CHECK(!grad_scale.has_value() || (grad_scale->is_cuda() && grad_scale->scalar_type() == at::kFloat && grad_scale->numel() == 1));
  TORCH_CHECK(grad_out.scalar_type() == at::kFloat && grad_out.is_contiguous() &&
              grad_out.numel() == rows);
  TORCH_CHECK(stats.scalar_type() == at::kFloat && stats.is_contiguous() && stats.size(0) == 5 &&
              stats.size(1) == rows);
  c10::cuda::CUDAGuard guard(logits.device());
  Tensor d = at::empty({logits.size(0), logits.size(1)}, logits.options());
  const int rc = sb200::launch_loss_bwd(
      (int)op, logits.data_ptr(), targets.data_ptr(), grad_out.data_ptr<float>(),
      grad_scale.has_value() ? grad_scale->data_ptr<float>() : nullptr, stats.data_ptr<float>(), d.data_ptr(), (int)rows, (int)logits.size(0), (int)logits.size(1),
      logits.stride(0), targets.stride(0), d.stride(0), (int)shift, row_targets(target_row, rows), used_rows(live), cur_stream());
  TORCH_CHECK(rc == 0, "loss_bwd: unknown op ", op);
  return d;
}
Tensor loss_bwd(int64_t op, const Tensor& logits, const Tensor& targets, const Tensor& grad_out, const Tensor& stats, int64_t shift, int64_t rows) {
  return loss_bwd_scaled(op, logits, targets, grad_out, c10::nullopt, stats, shift, rows, c10::nullopt, c10::nullopt);
}

void sumsq(const Tensor& g, Tensor out, bool accumulate) {
  TORCH_CHECK(g.is_cuda() && g.is_contiguous() && out.scalar_type() == at::kFloat && out.numel() >= 1);
  TORCH_CHECK(g.scalar_type() == at::kBFloat16 || g.scalar_type() == at::kFloat);
  c10::cuda::CUDAGuard guard(g.device());
  Tensor partial = at::empty({sb200::sumsq_num_partials()}, out.options());
  sb200::launch_sumsq(g.data_ptr(), g.scalar_type() == at::kBFloat16, g.numel(),
                      partial.data_ptr<float>(), out.data_ptr<float>(), accumulate, cur_stream());
}

// Muon, both element-wise halves, for every matrix of a table in one launch.
//   table int64[M, 3]: offset in the flat gradient / weight buffers, elements, offset in the state buffers (offsets multiples of 8)
//   chunks int32[C, 2]: matrix and chunk of muon_chunk_elements() elements inside it; first_chunk int32[M + 1]
void check_muon_table(const Tensor& table, const Tensor& chunks) {
  TORCH_CHECK(table.is_cuda() && table.scalar_type() == at::kLong && table.dim() == 2 && table.size(1) == 3 && table.is_contiguous());
  TORCH_CHECK(chunks.is_cuda() && chunks.scalar_type() == at::kInt && chunks.dim() == 2 && chunks.size(1) == 2 && chunks.is_contiguous());
}
bool aligned16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }

// buf <- momentum update of the clipped gradient, out <- bf16 (nesterov) update over its Frobenius norm (inv_norm[M] <- its inverse).
void muon_momentum(const Tensor& grad, Tensor buf, Tensor out, const Tensor& table, const Tensor& chunks, const Tensor& first_chunk, const Tensor& hyper,
                   const Tensor& norm_sq, double momentum, bool nesterov, Tensor inv_norm) {
  check_muon_table(table, chunks);
  TORCH_CHECK(grad.is_cuda() && grad.is_contiguous() && (grad.scalar_type() == at::kBFloat16 || grad.scalar_type() == at::kFloat));
  TORCH_CHECK(buf.is_cuda() && buf.scalar_type() == at::kFloat && buf.is_contiguous());
  TORCH_CHECK(out.is_cuda() && out.scalar_type() == at::kBFloat16 && out.is_contiguous() && out.numel() == buf.numel());
  TORCH_CHECK(aligned16(grad) && aligned16(buf) && aligned16(out), "muon_momentum: buffers must be 16-byte aligned");
  TORCH_CHECK(first_chunk.is_cuda() && first_chunk.scalar_type() == at::kInt && first_chunk.numel() == table.size(0) + 1);
  TORCH_CHECK(hyper.is_cuda() && hyper.scalar_type() == at::kFloat && hyper.numel() >= 9);
  TORCH_CHECK(norm_sq.is_cuda() && norm_sq.scalar_type() == at::kFloat && norm_sq.numel() >= 1);
  TORCH_CHECK(inv_norm.is_cuda() && inv_norm.scalar_type() == at::kFloat && inv_norm.numel() >= table.size(0));
  c10::cuda::CUDAGuard guard(buf.device());
  Tensor partial = at::empty({chunks.size(0)}, inv_norm.options());
  sb200::launch_muon_momentum(grad.data_ptr(), grad.scalar_type() == at::kBFloat16, buf.data_ptr<float>(), out.data_ptr(), table.data_ptr<int64_t>(),
                              chunks.data_ptr<int>(), (int)chunks.size(0), first_chunk.data_ptr<int>(), (int)table.size(0), hyper.data_ptr<float>(),
                              norm_sq.data_ptr<float>(), (float)momentum, nesterov ? 1 : 0, partial.data_ptr<float>(), inv_norm.data_ptr<float>(), cur_stream());
}

// master <- master * (1 - lr * wd) - lr * adjust[matrix] * update, w16 <- bf16(master); lr = hyper[0] * lr_ratio.
void muon_apply(Tensor master, const Tensor& update, Tensor w16, const Tensor& table, const Tensor& chunks, const Tensor& adjust, const Tensor& hyper,
                double lr_ratio, double weight_decay) {
  check_muon_table(table, chunks);
  TORCH_CHECK(master.is_cuda() && master.scalar_type() == at::kFloat && master.is_contiguous());
  TORCH_CHECK(update.is_cuda() && update.scalar_type() == at::kBFloat16 && update.is_contiguous() && update.numel() == master.numel());
  TORCH_CHECK(w16.is_cuda() && w16.scalar_type() == at::kBFloat16 && w16.is_contiguous());
  TORCH_CHECK(aligned16(master) && aligned16(update) && aligned16(w16), "muon_apply: buffers must be 16-byte aligned");
  TORCH_CHECK(adjust.is_cuda() && adjust.scalar_type() == at::kFloat && adjust.is_contiguous() && adjust.numel() == table.size(0));
  TORCH_CHECK(hyper.is_cuda() && hyper.scalar_type() == at::kFloat && hyper.numel() >= 9);
  c10::cuda::CUDAGuard guard(master.device());
  sb200::launch_muon_apply(master.data_ptr<float>(), update.data_ptr(), w16.data_ptr(), table.data_ptr<int64_t>(), chunks.data_ptr<int>(), (int)chunks.size(0),
                           adjust.data_ptr<float>(), hyper.data_ptr<float>(), (float)lr_ratio, (float)weight_decay, cur_stream());
}

int64_t muon_chunk_elements_binding() { return sb200::muon_chunk_elements(); }

// hyper (fp32[16], CUDA) <- vals (<= 16 host doubles), passed as kernel arguments.
void set_hyper(Tensor hyper, std::vector<double> vals) {
  TORCH_CHECK(hyper.is_cuda() && hyper.scalar_type() == at::kFloat && hyper.numel() >= 16 && hyper.is_contiguous());
  TORCH_CHECK(vals.size() <= 16);
  float host[16] = {0};
  for (size_t i = 0; i < vals.size(); ++i) host[i] = (float)vals[i];
  c10::cuda::CUDAGuard guard(hyper.device());
  sb200::launch_set_hyper(hyper.data_ptr<float>(), host, at::cuda::getCurrentCUDAStream());
}

void adamw(Tensor master, Tensor m, Tensor v, const Tensor& grad, c10::optional<Tensor> w16,
           const Tensor& hyper, const c10::optional<Tensor>& norm_sq) {
  const int64_t n = master.numel();
  TORCH_CHECK(master.is_cuda() && master.scalar_type() == at::kFloat && master.is_contiguous());
  TORCH_CHECK(m.scalar_type() == at::kFloat && v.scalar_type() == at::kFloat && m.numel() == n &&
              v.numel() == n && m.is_contiguous() && v.is_contiguous());
  TORCH_CHECK(grad.numel() == n && grad.is_contiguous() &&
              (grad.scalar_type() == at::kBFloat16 || grad.scalar_type() == at::kFloat));
  TORCH_CHECK(hyper.scalar_type() == at::kFloat && hyper.numel() >= 9 && hyper.is_cuda());
  void* w = nullptr;
  if (w16.has_value()) {
    TORCH_CHECK(w16->scalar_type() == at::kBFloat16 && w16->numel() == n && w16->is_contiguous());
    w = w16->data_ptr();
  }
  const float* ns = nullptr;
  if (norm_sq.has_value()) {
    TORCH_CHECK(norm_sq->scalar_type() == at::kFloat && norm_sq->is_cuda());
    ns = norm_sq->data_ptr<float>();
  }
  c10::cuda::CUDAGuard guard(master.device());
  sb200::launch_adamw(master.data_ptr<float>(), m.data_ptr<float>(), v.data_ptr<float>(),
                      grad.data_ptr(), grad.scalar_type() == at::kBFloat16, w, n,
                      hyper.data_ptr<float>(), ns, cur_stream());
}

int64_t launch_count() { return sb200::launch_count(); }

// ---- peer memory + fused sharded optimizer -------------------------------------------------
int64_t peer_alloc(int64_t nbytes) {
  void* p = nullptr;
  TORCH_CHECK(sb200::peer_malloc(nbytes, &p) == 0, "peer_alloc: cudaMalloc of ", nbytes, " bytes failed");
  return reinterpret_cast<int64_t>(p);
}
void peer_release(int64_t ptr) { sb200::peer_free(reinterpret_cast<void*>(ptr)); }
Tensor peer_handle(int64_t ptr) {
  Tensor h = at::empty({64}, at::TensorOptions().dtype(at::kByte));
  TORCH_CHECK(sb200::peer_export(reinterpret_cast<void*>(ptr), h.data_ptr<uint8_t>()) == 0, "peer_handle: cudaIpcGetMemHandle failed");
  return h;
}
int64_t peer_open(const Tensor& handle) {
  TORCH_CHECK(handle.device().is_cpu() && handle.scalar_type() == at::kByte && handle.numel() == 64 && handle.is_contiguous());
  void* p = nullptr;
  TORCH_CHECK(sb200::peer_import(handle.data_ptr<uint8_t>(), &p) == 0, "peer_open: cudaIpcOpenMemHandle failed");
  return reinterpret_cast<int64_t>(p);
}
void peer_close(int64_t ptr) { sb200::peer_close(reinterpret_cast<void*>(ptr)); }
// Non-owning tensor over raw device memory (the caller keeps the allocation alive).
Tensor peer_tensor(int64_t ptr, int64_t numel, at::ScalarType dtype, int64_t device) {
  auto opts = at::TensorOptions().dtype(dtype).device(at::kCUDA, (c10::DeviceIndex)device);
  return at::from_blob(reinterpret_cast<void*>(ptr), {numel}, opts);
}
int64_t fused_optim_ctl_words() { return sb200::fused_optim_ctl_words(); }

// ---- tail of a training-time-test pass --------------------------------------------------------
// row_loss fp32[rows], pred / target int32[rows], mask uint8[rows] (0 / non-0), prev uint8 or bool [rows] (updated in place).
// Returns (out fp32[4] = loss, correct, total, cond_total; weight fp32[rows] = d loss / d row_loss).
// -> (out float[5]: loss, correct, total, cond_total, 1; weight float[rows]; earlier + loss)
std::tuple<Tensor, Tensor, Tensor> step_tail(const Tensor& row_loss, const Tensor& pred, const Tensor& target, const Tensor& mask, Tensor prev,
                                             double decay, double eps, const c10::optional<Tensor>& earlier, const c10::optional<Tensor>& target_row) {
  TORCH_CHECK(!earlier.has_value() || (earlier->is_cuda() && earlier->scalar_type() == at::kFloat && earlier->numel() == 1));
  const int64_t rows = row_loss.numel();
  TORCH_CHECK(row_loss.is_cuda() && row_loss.scalar_type() == at::kFloat && row_loss.is_contiguous());
  TORCH_CHECK(pred.scalar_type() == at::kInt && target.scalar_type() == at::kInt && pred.is_contiguous() && target.is_contiguous());
  TORCH_CHECK(pred.numel() >= rows && target.numel() >= rows && mask.numel() >= rows && prev.numel() >= rows);
  TORCH_CHECK((mask.scalar_type() == at::kByte || mask.scalar_type() == at::kBool) && mask.is_contiguous());
  TORCH_CHECK((prev.scalar_type() == at::kByte || prev.scalar_type() == at::kBool) && prev.is_contiguous());
  c10::cuda::CUDAGuard guard(row_loss.device());
  Tensor out = at::empty({5}, row_loss.options()), total = at::empty({}, row_loss.options());
  Tensor weight = at::empty({rows}, row_loss.options());
  sb200::launch_step_tail(row_loss.data_ptr<float>(), pred.data_ptr<int>(), target.data_ptr<int>(),
                          static_cast<const uint8_t*>(mask.data_ptr()), static_cast<uint8_t*>(prev.data_ptr()), (int)rows, (float)decay,
                          (float)eps, out.data_ptr<float>(), weight.data_ptr<float>(), earlier.has_value() ? earlier->data_ptr<float>() : nullptr,
                           total.data_ptr<float>(), row_targets(target_row, rows), cur_stream());
  return {out, weight, total};
}

// ---- hidden-state ring (device-to-device hand-off) -----------------------------------------
int64_t hs_ring_ctl_words() { return sb200::hs_ring_ctl_words_per_slot(); }

// src: contiguous CUDA tensor (payload, size a multiple of 16 bytes); slot_data / slot_ctl: device addresses
// of the slot in the consumer's memory as mapped into this process; scratch: int32[2] zeros on this device.
void hs_push(const Tensor& src, int64_t slot_data, int64_t slot_ctl, int64_t seq, int64_t n_slots, int64_t rows, int64_t width,
             int64_t spin_limit, Tensor scratch, Tensor status) {
  TORCH_CHECK(src.is_cuda() && src.is_contiguous() && scratch.is_cuda() && status.is_cuda());
  TORCH_CHECK(scratch.scalar_type() == at::kInt && scratch.numel() >= 2 && status.scalar_type() == at::kInt && status.numel() >= 1);
  c10::cuda::CUDAGuard guard(src.device());
  const int rc = sb200::launch_hs_push(src.data_ptr(), (int64_t)src.nbytes(), reinterpret_cast<void*>(slot_data),
                                       reinterpret_cast<uint32_t*>(slot_ctl), (uint32_t)seq, (uint32_t)n_slots, (uint32_t)rows, (uint32_t)width,
                                       (uint32_t)spin_limit, reinterpret_cast<uint32_t*>(scratch.data_ptr<int>()), status.data_ptr<int>(),
                                       cur_stream());
  TORCH_CHECK(rc == 0, "hs_push: bad arguments or launch failure (", rc, ")");
}

void hs_pop(Tensor dst, int64_t slot_data, int64_t slot_ctl, int64_t seq, int64_t spin_limit, Tensor scratch, Tensor status) {
  TORCH_CHECK(dst.is_cuda() && dst.is_contiguous() && scratch.is_cuda() && status.is_cuda());
  TORCH_CHECK(scratch.scalar_type() == at::kInt && scratch.numel() >= 4 && status.scalar_type() == at::kInt && status.numel() >= 1);
  c10::cuda::CUDAGuard guard(dst.device());
  const int rc = sb200::launch_hs_pop(dst.data_ptr(), (int64_t)dst.nbytes(), reinterpret_cast<const void*>(slot_data),
                                      reinterpret_cast<uint32_t*>(slot_ctl), (uint32_t)seq, (uint32_t)spin_limit,
                                      reinterpret_cast<uint32_t*>(scratch.data_ptr<int>()), status.data_ptr<int>(), cur_stream());
  TORCH_CHECK(rc == 0, "hs_pop: bad arguments or launch failure (", rc, ")");
}

// g_ptrs / w_ptrs / ctl_ptrs: int64 CPU tensors [world] of device addresses valid on this rank.
// g_mc / w_mc: multicast (NVSwitch) addresses of the gradient / weight buffers, 0 = use the per-peer addresses.
void fused_sharded_adamw(int64_t world, int64_t rank, int64_t shard, const Tensor& g_ptrs, const Tensor& w_ptrs, const Tensor& ctl_ptrs,
                         int64_t g_mc, int64_t w_mc, Tensor master, Tensor m, Tensor v, Tensor gred, const Tensor& hyper, Tensor status, int64_t spin_limit) {
  // validated before the fixed-size pointer arrays below are filled
  TORCH_CHECK(world >= 1 && world <= 8 && rank >= 0 && rank < world && shard > 0 && shard % 8 == 0,
              "fused_sharded_adamw: need 1 <= world <= 8, 0 <= rank < world and a positive shard that is a multiple of 8");
  TORCH_CHECK(spin_limit > 0 && spin_limit <= 0xFFFFFFF0LL, "fused_sharded_adamw: spin_limit out of range");
  TORCH_CHECK(g_ptrs.device().is_cpu() && g_ptrs.scalar_type() == at::kLong && g_ptrs.numel() == world);
  TORCH_CHECK(w_ptrs.device().is_cpu() && w_ptrs.scalar_type() == at::kLong && w_ptrs.numel() == world);
  TORCH_CHECK(ctl_ptrs.device().is_cpu() && ctl_ptrs.scalar_type() == at::kLong && ctl_ptrs.numel() == world);
  for (const Tensor* t : {&master, &m, &v, &gred})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == shard, "shard buffers must be fp32[shard]");
  TORCH_CHECK(hyper.is_cuda() && hyper.scalar_type() == at::kFloat && hyper.numel() >= 9);
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt);
  c10::cuda::CUDAGuard guard(master.device());
  const void* g[8];
  void* w[8];
  void* c[8];
  for (int q = 0; q < world; ++q) {
    g[q] = reinterpret_cast<const void*>(g_ptrs.data_ptr<int64_t>()[q]);
    w[q] = reinterpret_cast<void*>(w_ptrs.data_ptr<int64_t>()[q]);
    c[q] = reinterpret_cast<void*>(ctl_ptrs.data_ptr<int64_t>()[q]);
  }
  Tensor partial = at::empty({sb200::fused_optim_num_partials()}, master.options());
  const int rc = sb200::launch_fused_sharded_adamw((int)world, (int)rank, shard, g, w, c, reinterpret_cast<const void*>(g_mc),
                                                   reinterpret_cast<void*>(w_mc), master.data_ptr<float>(), m.data_ptr<float>(),
                                                   v.data_ptr<float>(), gred.data_ptr<float>(), partial.data_ptr<float>(),
                                                   hyper.data_ptr<float>(), status.data_ptr<int>(), (uint32_t)spin_limit, cur_stream());
  TORCH_CHECK(rc == 0, "fused_sharded_adamw launch failed (", rc, ")");
}

// ---- gated MLP: gate | up product with the activation in the GEMM epilogue ------------------------
// w: [2 I, K], gate rows first.  Returns (gate_up [M, 2 I], h [M, I] = silu(gate) * up).
std::tuple<Tensor, Tensor> gemm_swiglu(const Tensor& x, const Tensor& w, Tensor status, const c10::optional<Tensor>& live) {
  check_rows(x, "x");
  check_rows(w, "w");
  const int64_t M = x.size(0), K = x.size(1), I = w.size(0) / 2;
  TORCH_CHECK(w.size(1) == K && w.size(0) == 2 * I && I % 128 == 0, "gemm_swiglu: w must be [2 I, K] with I a multiple of 128");
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 1);
  c10::cuda::CUDAGuard guard(x.device());
  Tensor gate_up = at::empty({M, 2 * I}, x.options());
  Tensor h = at::empty({M, I}, x.options());
  const int rc = sb200::launch_gemm_swiglu(x.data_ptr(), w.data_ptr(), gate_up.data_ptr(), h.data_ptr(), (int)M, (int)I, (int)K, x.stride(0), w.stride(0),
                                           2 * I, I, status.data_ptr<int>(), used_rows(live), cur_stream());
  TORCH_CHECK(rc == 0, "gemm_swiglu launch failed (", rc, ")");
  return {gate_up, h};
}

// ---- row-parallel product of a tensor-parallel layer ------------------------------------------
// partial = x[M, K] . w[N, K]^T; the tile columns owned by rank o (N / world columns each, a multiple of 256) are stored
// into slot `rank` of stage_ptrs[o] ([world][M][N / world] on rank o; int64 CPU tensor of addresses valid on this device).
void gemm_scatter(const Tensor& x, const Tensor& w, const Tensor& stage_ptrs, int64_t rank, Tensor status) {
  check_rows(x, "x");
  check_rows(w, "w");
  const int64_t world = stage_ptrs.numel(), M = x.size(0), K = x.size(1), N = w.size(0);
  TORCH_CHECK(world >= 1 && world <= 8 && rank >= 0 && rank < world, "gemm_scatter: need 1 <= world <= 8 and 0 <= rank < world");
  TORCH_CHECK(stage_ptrs.device().is_cpu() && stage_ptrs.scalar_type() == at::kLong);
  TORCH_CHECK(w.size(1) == K && N % world == 0 && (N / world) % 256 == 0, "gemm_scatter: N / world must be a multiple of 256");
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 1);
  c10::cuda::CUDAGuard guard(x.device());
  void* stage[8];
  for (int q = 0; q < world; ++q) stage[q] = reinterpret_cast<void*>(stage_ptrs.data_ptr<int64_t>()[q]);
  const int rc = sb200::launch_gemm_scatter(x.data_ptr(), w.data_ptr(), stage, (int)world, (int)rank, (int)M, (int)N, (int)K, x.stride(0),
                                            w.stride(0), status.data_ptr<int>(), cur_stream());
  TORCH_CHECK(rc == 0, "gemm_scatter launch failed (", rc, ")");
}

int64_t tp_allreduce_ctl_words() { return sb200::tp_allreduce_ctl_words(); }

// Reduces this rank's column slice of the staged partial products (stage: local [world, rows, cols]), adds the residual's
// slice (local [rows, world * cols], optional) and writes the slice into every rank's output (out_ptrs / out_mc).
void tp_reduce_broadcast(const Tensor& stage, const Tensor& out_ptrs, int64_t out_mc, const c10::optional<Tensor>& residual,
                         const Tensor& ctl_ptrs, int64_t rank, bool barrier, Tensor status, int64_t spin_limit) {
  TORCH_CHECK(stage.is_cuda() && stage.scalar_type() == at::kBFloat16 && stage.dim() == 3 && stage.is_contiguous(), "stage must be bf16 [world, rows, cols]");
  const int64_t world = stage.size(0), rows = stage.size(1), cols = stage.size(2);
  TORCH_CHECK(world >= 1 && world <= 8 && rank >= 0 && rank < world && cols % 8 == 0, "tp_reduce_broadcast: need 1 <= world <= 8 and cols % 8 == 0");
  TORCH_CHECK(spin_limit > 0 && spin_limit <= 0xFFFFFFF0LL, "tp_reduce_broadcast: spin_limit out of range");
  TORCH_CHECK(out_ptrs.device().is_cpu() && out_ptrs.scalar_type() == at::kLong && out_ptrs.numel() == world);
  TORCH_CHECK(ctl_ptrs.device().is_cpu() && ctl_ptrs.scalar_type() == at::kLong && ctl_ptrs.numel() == world);
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 1);
  const void* res = nullptr;
  if (residual.has_value()) {
    TORCH_CHECK(residual->is_cuda() && residual->scalar_type() == at::kBFloat16 && residual->is_contiguous() && residual->numel() == rows * world * cols &&
                (reinterpret_cast<uintptr_t>(residual->data_ptr()) & 15) == 0, "residual must be contiguous bf16 [rows, world * cols]");
    res = residual->data_ptr();
  }
  c10::cuda::CUDAGuard guard(stage.device());
  void* out[8];
  void* ctl[8];
  for (int q = 0; q < world; ++q) {
    out[q] = reinterpret_cast<void*>(out_ptrs.data_ptr<int64_t>()[q]);
    ctl[q] = reinterpret_cast<void*>(ctl_ptrs.data_ptr<int64_t>()[q]);
    TORCH_CHECK((reinterpret_cast<uintptr_t>(out[q]) & 15) == 0 && ctl[q] != nullptr, "tp_reduce_broadcast: misaligned output / missing control block");
  }
  const int rc = sb200::launch_tp_reduce_broadcast((int)world, (int)rank, (int)rows, (int)cols, stage.data_ptr(), out, reinterpret_cast<void*>(out_mc), res,
                                                   ctl, barrier ? 1 : 0, status.data_ptr<int>(), (uint32_t)spin_limit, cur_stream());
  TORCH_CHECK(rc == 0, "tp_reduce_broadcast launch failed (", rc, ")");
}

// ---- debug build: index checks -------------------------------------------------------------
bool checked_build() {
#ifdef SB200_CHECK_BOUNDS
  return true;
#else
  return false;
#endif
}
// One row (site, index, limit) per module with index checks; site 0 = nothing recorded since
// the last call.  Reading clears the records.  Always zeros in the normal build.
Tensor bounds_report() {
  Tensor out = at::zeros({2, 3}, at::TensorOptions().dtype(at::kLong));
  sb200::BoundsRecord rec[2];
  TORCH_CHECK(sb200::read_bounds_norm(&rec[0]) == 0 && sb200::read_bounds_ep(&rec[1]) == 0, "bounds_report: reading the device records failed");
  for (int i = 0; i < 2; ++i) {
    out[i][0] = (int64_t)rec[i].site;
    out[i][1] = (int64_t)rec[i].index;
    out[i][2] = (int64_t)rec[i].limit;
  }
  return out;
}

// ---- expert-parallel token exchange --------------------------------------------------------
// *_ptrs: int64 CPU tensors [world] with the address of one buffer on every rank as mapped here.
sb200::EpPeers ep_peers(const Tensor& ptrs, int64_t world) {
  TORCH_CHECK(ptrs.device().is_cpu() && ptrs.scalar_type() == at::kLong && ptrs.numel() == world && world >= 1 && world <= 16);
  sb200::EpPeers out{};
  for (int q = 0; q < world; ++q) out.ptr[q] = (unsigned long long)ptrs.data_ptr<int64_t>()[q];
  return out;
}
void check_slots(const Tensor& t, int64_t n, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kInt && t.is_contiguous() && t.numel() == n, name, ": int32 CUDA [", n, "] expected");
}

void ep_push(const Tensor& src, const Tensor& src_row, const Tensor& dst_rank, const Tensor& dst_pos, const c10::optional<Tensor>& scale,
             const Tensor& dst_ptrs, int64_t capacity, Tensor counter, const Tensor& flag_ptrs, int64_t rank, int64_t world,
             int64_t seq) {
  check_rows(src, "src");
  TORCH_CHECK(src.is_contiguous() && src.size(1) % 8 == 0, "src rows must be contiguous with a multiple of 8 columns");
  const int64_t n = src_row.numel();
  check_slots(src_row, n, "src_row");
  check_slots(dst_rank, n, "dst_rank");
  check_slots(dst_pos, n, "dst_pos");
  if (scale.has_value()) TORCH_CHECK(scale->is_cuda() && scale->scalar_type() == at::kFloat && scale->is_contiguous() && scale->numel() == n);
  TORCH_CHECK(counter.is_cuda() && counter.scalar_type() == at::kInt && counter.numel() >= 1);
  c10::cuda::CUDAGuard guard(src.device());
  const sb200::EpPeers dstp = ep_peers(dst_ptrs, world), flg = ep_peers(flag_ptrs, world);
  const int rc = sb200::launch_ep_push((const __nv_bfloat16*)src.data_ptr(), src_row.data_ptr<int>(), dst_rank.data_ptr<int>(),
                                       dst_pos.data_ptr<int>(), scale.has_value() ? scale->data_ptr<float>() : nullptr, (int)n,
                                       (int)src.size(1), (int)src.size(0), (int)capacity, dstp,
                                       reinterpret_cast<unsigned int*>(counter.data_ptr<int>()), flg, (int)rank, (int)world, (uint32_t)seq,
                                       cur_stream());
  TORCH_CHECK(rc == 0, "ep_push launch failed (", rc, ")");
}

void ep_signal(const Tensor& flag_ptrs, int64_t rank, int64_t world, int64_t seq, const Tensor& on_device_of) {
  c10::cuda::CUDAGuard guard(on_device_of.device());
  const int rc = sb200::launch_ep_signal(ep_peers(flag_ptrs, world), (int)rank, (int)world, (uint32_t)seq, cur_stream());
  TORCH_CHECK(rc == 0, "ep_signal launch failed (", rc, ")");
}

void ep_wait(const Tensor& flags_local, int64_t world, int64_t seq, int64_t spin_limit, Tensor status) {
  TORCH_CHECK(flags_local.is_cuda() && flags_local.scalar_type() == at::kInt && flags_local.is_contiguous() && flags_local.numel() >= world);
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 1);
  c10::cuda::CUDAGuard guard(flags_local.device());
  const int rc = sb200::launch_ep_wait(reinterpret_cast<const uint32_t*>(flags_local.data_ptr<int>()), (int)world, (uint32_t)seq,
                                       (uint32_t)spin_limit, status.data_ptr<int>(), cur_stream());
  TORCH_CHECK(rc == 0, "ep_wait launch failed (", rc, ")");
}

void ep_pull(const Tensor& src_ptrs, int64_t capacity, const Tensor& src_rank, const Tensor& src_pos, const c10::optional<Tensor>& weight,
             int64_t world, Tensor out, int64_t k, c10::optional<Tensor> rows_out) {
  check_rows(out, "out");
  TORCH_CHECK(out.is_contiguous() && out.size(1) % 8 == 0);
  const int64_t n = out.size(0) * k;
  check_slots(src_rank, n, "src_rank");
  check_slots(src_pos, n, "src_pos");
  if (weight.has_value()) TORCH_CHECK(weight->is_cuda() && weight->scalar_type() == at::kFloat && weight->is_contiguous() && weight->numel() == n);
  if (rows_out.has_value())
    TORCH_CHECK(rows_out->is_cuda() && rows_out->scalar_type() == at::kBFloat16 && rows_out->is_contiguous() &&
                rows_out->numel() == n * out.size(1), "rows_out: bf16 [T*k, H] expected");
  c10::cuda::CUDAGuard guard(out.device());
  const int rc = sb200::launch_ep_pull(ep_peers(src_ptrs, world), src_rank.data_ptr<int>(), src_pos.data_ptr<int>(),
                                       weight.has_value() ? weight->data_ptr<float>() : nullptr, (int)out.size(0), (int)k, (int)out.size(1),
                                       (int)world, (int)capacity, (__nv_bfloat16*)out.data_ptr(),
                                       rows_out.has_value() ? (__nv_bfloat16*)rows_out->data_ptr() : nullptr, cur_stream());
  TORCH_CHECK(rc == 0, "ep_pull launch failed (", rc, ")");
}

// ---- tcgen05 GEMM ------------------------------------------------------------------------
// out[M,N] = a[M,K] @ b[N,K]^T; epilogue 0 = store, 1 = out += result, 2 = result + residual.
// `status` (int32[1], device) receives a non-zero code if a bounded wait in the kernel ran out.
// variant: 0 = choose; see launch_gemm_impl.
void gemm_tn_variant(const Tensor& a, const Tensor& b, Tensor out, const c10::optional<Tensor>& residual, int64_t epilogue, Tensor status,
                     int64_t variant, const c10::optional<Tensor>& live) {
  TORCH_CHECK(a.is_cuda() && b.is_cuda() && out.is_cuda() && status.is_cuda());
  TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16 && out.scalar_type() == at::kBFloat16);
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && out.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1 && out.stride(1) == 1);
  TORCH_CHECK(a.size(1) == b.size(1) && out.size(0) == a.size(0) && out.size(1) == b.size(0), "gemm_tn: shape mismatch");
  TORCH_CHECK(status.scalar_type() == at::kInt && status.numel() >= 1);
  const void* res = nullptr;
  int64_t ldr = 0;
  if (residual.has_value()) {
    TORCH_CHECK(residual->scalar_type() == at::kBFloat16 && residual->dim() == 2 && residual->stride(1) == 1 &&
                residual->size(0) == out.size(0) && residual->size(1) == out.size(1));
    res = residual->data_ptr();
    ldr = residual->stride(0);
  }
  TORCH_CHECK(epilogue != 2 || res != nullptr, "gemm_tn: epilogue 2 needs a residual");
  c10::cuda::CUDAGuard guard(a.device());
  TorchSplitSpace space(a);
  const int rc = sb200::launch_gemm_tn_tcgen05(a.data_ptr(), b.data_ptr(), out.data_ptr(), res, (int)a.size(0), (int)b.size(0),
                                               (int)a.size(1), a.stride(0), b.stride(0), out.stride(0), ldr, (int)epilogue,
                                               status.data_ptr<int>(), (int)variant, used_rows(live), variant == 6 ? &space : nullptr, cur_stream());
  TORCH_CHECK(rc == 0, "gemm_tn launch failed (", rc, ")");
}

void gemm_tn(const Tensor& a, const Tensor& b, Tensor out, const c10::optional<Tensor>& residual, int64_t epilogue, Tensor status,
             const c10::optional<Tensor>& live) {
  gemm_tn_variant(a, b, out, residual, epilogue, status, 0, live);
}

// out[M,N] (=, +=) op(a) @ op(b)^T with either operand stored transposed:
//   a_mn false: a is [M, K];  true: a is [K, M] (the product uses a^T, read in place)
//   b_mn false: b is [N, K];  true: b is [K, N]
// dgrad of a linear layer: gemm(dy[T,out], w[out,in], dx, b_mn = true);
// wgrad: gemm(dy[T,out], x[T,in], dw[out,in], a_mn = b_mn = true, epilogue 1 to accumulate).
// live (device int32): how many rows of the activations count - the rows of a and out, or with both operands transposed the sum's
void gemm_variant(const Tensor& a, const Tensor& b, Tensor out, int64_t epilogue, bool a_mn, bool b_mn, Tensor status, int64_t variant,
                  const c10::optional<Tensor>& live) {
  TORCH_CHECK(a.is_cuda() && b.is_cuda() && out.is_cuda() && status.is_cuda());
  TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16 && out.scalar_type() == at::kBFloat16);
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && out.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1 && out.stride(1) == 1);
  TORCH_CHECK(epilogue == 0 || epilogue == 1, "gemm: epilogue 0 (store) or 1 (accumulate)");
  const int64_t M = a_mn ? a.size(1) : a.size(0), K = a_mn ? a.size(0) : a.size(1);
  const int64_t N = b_mn ? b.size(1) : b.size(0), Kb = b_mn ? b.size(0) : b.size(1);
  TORCH_CHECK(K == Kb && out.size(0) == M && out.size(1) == N, "gemm: shape mismatch");
  TORCH_CHECK(status.scalar_type() == at::kInt && status.numel() >= 1);
  c10::cuda::CUDAGuard guard(a.device());
  TorchSplitSpace space(a);
  const int rc = sb200::launch_gemm_tcgen05(a.data_ptr(), b.data_ptr(), out.data_ptr(), nullptr, (int)M, (int)N, (int)K, a.stride(0),
                                            b.stride(0), out.stride(0), 0, (int)epilogue, a_mn ? 1 : 0, b_mn ? 1 : 0,
                                            status.data_ptr<int>(), (int)variant, used_rows(live), variant == 0 || variant == 6 ? &space : nullptr, cur_stream());
  TORCH_CHECK(rc == 0, "gemm launch failed (", rc, ")");
}

void gemm(const Tensor& a, const Tensor& b, Tensor out, int64_t epilogue, bool a_mn, bool b_mn, Tensor status, const c10::optional<Tensor>& live) {
  gemm_variant(a, b, out, epilogue, a_mn, b_mn, status, 0, live);
}

// Stacks of products: out[z] = alpha op(a[z]) @ op(b[z])^T (+ beta addend[z]), rounded as separate bf16 passes would round; with a
// `diagonal` (+ diagonal I), in fp32 and rounded once.
// Operands as in gemm, each a dense [batch, ., .] stack; symmetric: the caller knows that the products are.
void gemm_stack(const Tensor& a, const Tensor& b, Tensor out, const c10::optional<Tensor>& addend, bool a_mn, bool b_mn, double alpha, double beta,
                bool symmetric, Tensor status, c10::optional<double> diagonal) {
  for (const Tensor* t : std::initializer_list<const Tensor*>{&a, &b, &out})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->dim() == 3 && t->is_contiguous(), "gemm_stack: contiguous bf16 [batch, rows, cols] expected");
  const int64_t B = a.size(0), M = a_mn ? a.size(2) : a.size(1), K = a_mn ? a.size(1) : a.size(2), N = b_mn ? b.size(2) : b.size(1);
  TORCH_CHECK(b.size(0) == B && out.size(0) == B && (b_mn ? b.size(1) : b.size(2)) == K && out.size(1) == M && out.size(2) == N, "gemm_stack: shape mismatch");
  TORCH_CHECK(!symmetric || M == N, "gemm_stack: a symmetric product is square");
  if (addend.has_value())
    TORCH_CHECK(addend->is_cuda() && addend->scalar_type() == at::kBFloat16 && addend->is_contiguous() && addend->sizes() == out.sizes(), "gemm_stack: addend");
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 1);
  c10::cuda::CUDAGuard guard(a.device());
  TorchSplitSpace space(a);
  const int rc = sb200::launch_gemm_stack(a.data_ptr(), b.data_ptr(), out.data_ptr(), addend.has_value() ? addend->data_ptr() : nullptr, (int)B, (int)M, (int)N,
                                          (int)K, a_mn ? 1 : 0, b_mn ? 1 : 0, (float)alpha, (float)beta,
                                          diagonal.has_value() ? 1 : 0, (float)diagonal.value_or(0.0), symmetric ? 1 : 0, status.data_ptr<int>(), &space, cur_stream());
  TORCH_CHECK(rc == 0, "gemm_stack launch failed (", rc, ")");
}

// ---- masked attention ------------------------------------------------------------------
void check_heads(const Tensor& t, const char* name, int64_t hd) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 3, name, ": bf16 CUDA [T, heads, hd] expected");
  TORCH_CHECK(t.size(2) == hd && t.stride(2) == 1 && t.stride(1) == hd, name, ": heads must be contiguous");
  TORCH_CHECK(t.stride(0) % 8 == 0 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0, name, ": rows must be 16-byte aligned");
}

sb200::AttnParams make_params(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& lo, const Tensor& hi,
                              const c10::optional<Tensor>& ke, const c10::optional<Tensor>& ve,
                              const c10::optional<Tensor>& ext_idx, double scale) {
  const int64_t hd = q.size(2);
  check_heads(q, "q", hd);
  check_heads(k, "k", hd);
  check_heads(v, "v", hd);
  TORCH_CHECK(hd == 64 || hd == 128 || hd == 256, "attention: head_dim must be 64, 128 or 256");
  TORCH_CHECK(k.size(0) == v.size(0) && k.size(1) == v.size(1) && q.size(1) % k.size(1) == 0);
  TORCH_CHECK(lo.scalar_type() == at::kInt && hi.scalar_type() == at::kInt && lo.is_contiguous() && hi.is_contiguous() &&
              lo.numel() == q.size(0) && hi.numel() == q.size(0), "lo/hi must be int32[Tq]");
  sb200::AttnParams p{};
  p.q = (const __nv_bfloat16*)q.data_ptr();
  p.k = (const __nv_bfloat16*)k.data_ptr();
  p.v = (const __nv_bfloat16*)v.data_ptr();
  p.lo = lo.data_ptr<int>();
  p.hi = hi.data_ptr<int>();
  p.Tq = (int)q.size(0);
  p.Tc = (int)k.size(0);
  p.nh = (int)q.size(1);
  p.nkv = (int)k.size(1);
  p.q_rs = q.stride(0);
  p.k_rs = k.stride(0);
  p.v_rs = v.stride(0);
  p.scale = (float)scale;
  if (ext_idx.has_value() && ext_idx->numel() > 0) {
    TORCH_CHECK(ke.has_value() && ve.has_value(), "extra keys need k_ext and v_ext");
    check_heads(*ke, "k_ext", hd);
    check_heads(*ve, "v_ext", hd);
    TORCH_CHECK(ke->size(0) == ve->size(0) && ke->size(1) == p.nkv && ve->size(1) == p.nkv);
    TORCH_CHECK(ext_idx->scalar_type() == at::kInt && ext_idx->is_contiguous() && ext_idx->dim() == 2 && ext_idx->size(0) == p.Tq);
    p.ke = (const __nv_bfloat16*)ke->data_ptr();
    p.ve = (const __nv_bfloat16*)ve->data_ptr();
    p.ext_idx = ext_idx->data_ptr<int>();
    p.Te = (int)ke->size(0);
    p.E = (int)ext_idx->size(1);
    p.ke_rs = ke->stride(0);
    p.ve_rs = ve->stride(0);
  }
  return p;
}

// Block-structured extras (tcgen05 kernels): the extra keys of row r are the rows of its block of `block` rows in
// k_ext / v_ext (only up to r with `causal`); the per-row index list is then not used.
void use_block_extras(sb200::AttnParams& p, const Tensor& q, int64_t block, bool causal) {
  if (block <= 0) return;
  TORCH_CHECK(p.ke != nullptr && p.ve != nullptr, "block-structured extras need k_ext and v_ext");
  TORCH_CHECK(128 % block == 0, "block-structured extras: the block size must divide 128");
  TORCH_CHECK(p.Te >= p.Tq, "block-structured extras: k_ext / v_ext hold one row per query row");
  p.E = 0;
  p.ext_idx = nullptr;
  p.ext_block = (int)block;
  p.ext_causal = causal ? 1 : 0;
  (void)q;
}

std::tuple<Tensor, Tensor> attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& lo, const Tensor& hi,
                                    const c10::optional<Tensor>& ke, const c10::optional<Tensor>& ve,
                                    const c10::optional<Tensor>& ext_idx, double scale) {
  sb200::AttnParams p = make_params(q, k, v, lo, hi, ke, ve, ext_idx, scale);
  c10::cuda::CUDAGuard guard(q.device());
  Tensor out = at::empty({q.size(0), q.size(1), q.size(2)}, q.options());
  Tensor lse2 = at::empty({q.size(1), q.size(0)}, q.options().dtype(at::kFloat));
  p.out = (__nv_bfloat16*)out.data_ptr();
  p.o_rs = out.stride(0);
  p.lse2 = lse2.data_ptr<float>();
  const int rc = sb200::launch_attn_fwd(p, (int)q.size(2), cur_stream());
  TORCH_CHECK(rc == 0, "attn_fwd launch failed (", rc, ")");
  return {out, lse2};
}

// Forward on the tcgen05 tensor cores (head_dim 64 or 128, or 256 without extra keys).  `status` (int32[1], device) receives a
// non-zero code if a bounded wait in the kernel ran out.
std::tuple<Tensor, Tensor> attn_fwd_tc(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& lo, const Tensor& hi,
                                       const c10::optional<Tensor>& ke, const c10::optional<Tensor>& ve,
                                       const c10::optional<Tensor>& ext_idx, double scale, Tensor status, int64_t ext_block,
                                       bool ext_causal) {
  sb200::AttnParams p = make_params(q, k, v, lo, hi, ke, ve, ext_idx, scale);
  use_block_extras(p, q, ext_block, ext_causal);
  TORCH_CHECK(q.size(2) == 64 || q.size(2) == 128 || (q.size(2) == 256 && p.E == 0 && p.ext_block == 0), "attn_fwd_tc: head_dim must be 64 or 128, or 256 without extra keys");
  TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 1);
  c10::cuda::CUDAGuard guard(q.device());
  Tensor out = at::empty({q.size(0), q.size(1), q.size(2)}, q.options());
  Tensor lse2 = at::empty({q.size(1), q.size(0)}, q.options().dtype(at::kFloat));
  p.out = (__nv_bfloat16*)out.data_ptr();
  p.o_rs = out.stride(0);
  p.lse2 = lse2.data_ptr<float>();
  const int rc = q.size(2) == 256 ? sb200::launch_attn_fwd_wide_tc(p, status.data_ptr<int>(), cur_stream())
                                  : sb200::launch_attn_fwd_tc(p, (int)q.size(2), status.data_ptr<int>(), cur_stream());
  TORCH_CHECK(rc == 0, "attn_fwd_tc launch failed (", rc, ")");
  return {out, lse2};
}

// A decoder layer's forward without a gradient: norm, projection, head norms and rotation, attention, projection, sum and norm,
// gated MLP, sum (and the next layer's norm, given its weight).  Called one by one from Python its nine launches take 200 us of
// the host, more than they take on the device up to some 1000 rows of a narrow decoder; from here about 40.
// -> (result, its norm if w_next), or nothing where the operands are not what the kernels take (the caller's modules then do).
std::vector<Tensor> decoder_layer_fwd(const Tensor& h, const c10::optional<Tensor>& normed, const Tensor& w_in, const Tensor& w_qkv, const c10::optional<Tensor>& w_q,
                                      const c10::optional<Tensor>& w_k, const Tensor& w_o, const Tensor& w_post, const Tensor& w_gate_up, const Tensor& w_down,
                                      const c10::optional<Tensor>& w_next, const Tensor& positions, const Tensor& cos_t, const Tensor& sin_t, const Tensor& lo,
                                      const Tensor& hi, int64_t nh, int64_t nkv, int64_t hd, int64_t rot, double eps_in, double eps_heads, double eps_post,
                                      double eps_next, double scale, bool tensor_cores, const Tensor& status) {
  auto dense = [&](const Tensor& t, std::initializer_list<int64_t> shape) {
    return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.device() == h.device() && t.sizes() == c10::IntArrayRef(shape) && t.is_contiguous() &&
           (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
  };
  if (h.dim() != 2 || w_down.dim() != 2 || nh <= 0 || nkv <= 0) return {};
  const int64_t T = h.size(0), H = h.size(1), I = w_down.size(1), nq = nh * hd, nk = nkv * hd;
  const bool heads = w_q.has_value();
  if (T <= 0 || H % 8 || H <= 256 || H > 32768 || I % 128 || nh % nkv || (hd != 64 && hd != 128 && hd != 256) || rot > hd || rot % (heads ? 16 : 2)) return {};
  if (!dense(h, {T, H}) || (normed.has_value() && !dense(*normed, {T, H})) || !dense(w_in, {H}) || !dense(w_qkv, {nq + 2 * nk, H}) || !dense(w_o, {H, nq}) ||
      !dense(w_post, {H}) || !dense(w_gate_up, {2 * I, H}) || !dense(w_down, {H, I}) || (w_next.has_value() && !dense(*w_next, {H})))
    return {};
  if (heads && (!w_k.has_value() || !dense(*w_q, {hd}) || !dense(*w_k, {hd}))) return {};
  if (positions.scalar_type() != at::kLong || !positions.is_contiguous() || positions.numel() != T) return {};
  for (const Tensor* t : std::initializer_list<const Tensor*>{&positions, &cos_t, &sin_t, &lo, &hi})
    if (t->device() != h.device()) return {};
  c10::cuda::CUDAGuard guard(h.device());
  const c10::optional<Tensor> none;
  auto product = [&](const Tensor& x, const Tensor& w) {
    Tensor out = at::empty({T, w.size(0)}, h.options());
    gemm_tn(x, w, out, none, 0, status, none);
    return out;
  };
  Tensor x;
  if (normed.has_value()) x = *normed;
  else norm_fwd(h, w_in, none, x = at::empty_like(h), none, eps_in, false, none);
  const Tensor qkv = product(x, w_qkv);
  Tensor qk = qkv;
  if (heads) qk = std::get<0>(heads_fwd(qkv, w_q, nh, w_k, nkv, eps_heads, positions, cos_t, sin_t, hd, rot, false, none));
  else rope_(qkv, positions, cos_t, sin_t, nh + nkv, hd, rot, 1.0, none);
  const Tensor q = qk.narrow(1, 0, nq).unflatten(1, {nh, hd}), k = qk.narrow(1, nq, nk).unflatten(1, {nkv, hd}), v = qkv.narrow(1, nq + nk, nk).unflatten(1, {nkv, hd});
  Tensor out = std::get<0>(tensor_cores ? attn_fwd_tc(q, k, v, lo, hi, none, none, none, scale, status, 0, false) : attn_fwd(q, k, v, lo, hi, none, none, none, scale));
  auto [mid, mid_normed] = add_rmsnorm_fwd(h, product(out.view({T, nq}), w_o), w_post, eps_post);
  const Tensor down = product(std::get<1>(gemm_swiglu(mid_normed, w_gate_up, status, none)), w_down);
  if (!w_next.has_value()) return {mid + down};
  auto [next, next_normed] = add_rmsnorm_fwd(mid, down, *w_next, eps_next);
  return {next, next_normed};
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> attn_bwd(
    const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse2,
    const Tensor& lo, const Tensor& hi, const c10::optional<Tensor>& ke, const c10::optional<Tensor>& ve,
    const c10::optional<Tensor>& ext_idx, double scale, int64_t impl, const c10::optional<Tensor>& status, int64_t ext_block,
    bool ext_causal) {
  // impl 0: mma.sync kernels; 1: tcgen05 kernels (head_dim 64 or 128, or 256 without extra keys; `status` receives a code if a bounded wait ran out)
  sb200::AttnParams p = make_params(q, k, v, lo, hi, ke, ve, ext_idx, scale);
  TORCH_CHECK(ext_block <= 0 || impl == 1, "block-structured extras run on the tcgen05 kernels only");
  use_block_extras(p, q, ext_block, ext_causal);
  const int64_t hd = q.size(2);
  if (impl == 1) {
    TORCH_CHECK(hd == 64 || hd == 128 || (hd == 256 && p.E == 0 && p.ext_block == 0), "attn_bwd: the tcgen05 kernels need head_dim 64 or 128, or 256 without extra keys");
    TORCH_CHECK(status.has_value() && status->is_cuda() && status->scalar_type() == at::kInt && status->numel() >= 1);
  }
  check_heads(dout, "dout", hd);
  check_heads(out, "out", hd);
  TORCH_CHECK(dout.size(0) == q.size(0) && dout.size(1) == q.size(1) && out.sizes() == dout.sizes());
  TORCH_CHECK(lse2.scalar_type() == at::kFloat && lse2.is_contiguous() && lse2.numel() == q.size(0) * q.size(1));
  c10::cuda::CUDAGuard guard(q.device());
  Tensor dq = at::empty({q.size(0), q.size(1), hd}, q.options());
  Tensor dk = at::empty({k.size(0), k.size(1), hd}, q.options());
  Tensor dv = at::empty({k.size(0), k.size(1), hd}, q.options());
  Tensor delta = at::empty({q.size(1), q.size(0)}, lse2.options());
  Tensor dke, dve;
  if (p.ext_block > 0) {
    const Tensor both = at::empty({2, p.Te, p.nkv, hd}, q.options());
    dke = both.select(0, 0);
    dve = both.select(0, 1);
    p.dke16 = (__nv_bfloat16*)dke.data_ptr();
    p.dve16 = (__nv_bfloat16*)dve.data_ptr();
  } else if (p.E > 0) {
    const Tensor both = at::zeros({2, p.Te, p.nkv, hd}, lse2.options());
    dke = both.select(0, 0);
    dve = both.select(0, 1);
    p.dke = dke.data_ptr<float>();
    p.dve = dve.data_ptr<float>();
  } else {
    dke = at::empty({0}, lse2.options());
    dve = at::empty({0}, lse2.options());
  }
  Tensor dkv_part;
  if (p.nh > p.nkv) {  // grouped queries: per-head fp32 partials, summed in head order afterwards
    dkv_part = at::empty({p.nh / p.nkv, 2, k.size(0), k.size(1), hd}, lse2.options());
    p.dkv_part = dkv_part.data_ptr<float>();
  }
  const int n_tiles = (p.Tc + sb200::kAttnKeyTile - 1) / sb200::kAttnKeyTile;
  Tensor qmin = at::empty({n_tiles}, lo.options());
  Tensor qmax = at::empty({n_tiles}, lo.options());
  p.out = (__nv_bfloat16*)out.data_ptr();
  p.o_rs = out.stride(0);
  p.lse2 = lse2.data_ptr<float>();
  p.dout = (const __nv_bfloat16*)dout.data_ptr();
  p.do_rs = dout.stride(0);
  p.delta = delta.data_ptr<float>();
  p.dq = (__nv_bfloat16*)dq.data_ptr();
  p.dq_rs = dq.stride(0);
  p.dk = (__nv_bfloat16*)dk.data_ptr();
  p.dv = (__nv_bfloat16*)dv.data_ptr();
  p.tile_qmin = qmin.data_ptr<int>();
  p.tile_qmax = qmax.data_ptr<int>();
  const int rc = impl == 1 && hd == 256 ? sb200::launch_attn_bwd_wide_tc(p, qmin.data_ptr<int>(), qmax.data_ptr<int>(), status->data_ptr<int>(), cur_stream())
                 : impl == 1 ? sb200::launch_attn_bwd_tc(p, (int)hd, qmin.data_ptr<int>(), qmax.data_ptr<int>(), status->data_ptr<int>(), cur_stream())
                           : sb200::launch_attn_bwd(p, (int)hd, qmin.data_ptr<int>(), qmax.data_ptr<int>(), cur_stream());
  TORCH_CHECK(rc == 0, "attn_bwd launch failed (", rc, ")");
  if (p.E > 0) {  // both gradients of the extra keys in the inputs' type with one conversion
    const Tensor both = at::as_strided(dke, {2, p.Te, p.nkv, hd}, {(int64_t)p.Te * p.nkv * hd, p.nkv * hd, hd, 1}).to(q.scalar_type());
    dke = both.select(0, 0);
    dve = both.select(0, 1);
  }
  return {dq, dk, dv, dke, dve};
}

}  // namespace

TORCH_LIBRARY(sb200, m) {
  // a trailing `live` (int32[1] on the device): how many of the rows are in use
  m.def("add_rmsnorm_fwd", &add_rmsnorm_fwd);
  m.def("decoder_layer_fwd(Tensor h, Tensor? normed, Tensor w_in, Tensor w_qkv, Tensor? w_q, Tensor? w_k, Tensor w_o, Tensor w_post, Tensor w_gate_up, "
        "Tensor w_down, Tensor? w_next, Tensor positions, Tensor cos_t, Tensor sin_t, Tensor lo, Tensor hi, int nh, int nkv, int hd, int rot, float eps_in, "
        "float eps_heads, float eps_post, float eps_next, float scale, bool tensor_cores, Tensor status) -> Tensor[]", &decoder_layer_fwd);
  m.def("rmsnorm_fwd(Tensor x, Tensor w, Tensor? row_index, Tensor y, Tensor? rstd, float eps, Tensor? live=None) -> ()", &rmsnorm_fwd);
  m.def("norm_fwd(Tensor x, Tensor w, Tensor? row_index, Tensor y, Tensor? rstd, float eps, bool centred, Tensor? live=None) -> ()", &norm_fwd);
  m.def("rmsnorm_bwd(Tensor dy, Tensor? dy2, Tensor x, Tensor w, Tensor rstd, Tensor? add, Tensor? dx, Tensor? dw, bool accumulate_dw, bool centred, "
        "Tensor? live=None) -> ()", &rmsnorm_bwd);
  m.def("step_rows", &step_rows);
  m.def("take_rows", &take_rows);
  m.def("put_rows", &put_rows);
  m.def("swiglu_fwd(Tensor gate_up, Tensor? rows_used=None) -> Tensor", &swiglu_fwd);
  m.def("swiglu_bwd", &swiglu_bwd);
  m.def("swiglu_bwd_rows", &swiglu_bwd_rows);
  m.def("heads_fwd(Tensor src, Tensor? w_a, int na, Tensor? w_b, int nb, float eps, Tensor positions, Tensor cos, Tensor sin, int hd, int rot, bool repeated, "
        "Tensor? live=None) -> (Tensor, Tensor)", &heads_fwd);
  m.def("heads_bwd(Tensor?[] d, int split, Tensor src, Tensor rstd, Tensor? w_a, int na, Tensor? w_b, int nb, int nv, Tensor? dw_a, bool acc_a, Tensor? dw_b, "
        "bool acc_b, Tensor positions, Tensor cos, Tensor sin, int hd, int rot, bool repeated, Tensor? live=None) -> Tensor", &heads_bwd);
  m.def("rope_merge(Tensor q, Tensor? k, Tensor? v, bool rotate_k, Tensor positions, Tensor cos, Tensor sin, int hd, int rot, float sign, Tensor? live=None) -> "
        "Tensor", &rope_merge);
  m.def("loss_fwd_either(int op, Tensor logits, Tensor targets, Tensor? active, Tensor? also, int shift, int rows, Tensor? target_row=None) -> "
        "(Tensor, Tensor, Tensor, Tensor)", &loss_fwd_either);
  m.def("loss_fwd_tv(int op, Tensor logits, Tensor targets, Tensor? active, Tensor? also, int shift, int rows, Tensor? target_row, bool with_tv) -> "
        "(Tensor, Tensor, Tensor, Tensor, Tensor)", &loss_fwd_tv);
  m.def("loss_bwd_scaled(int op, Tensor logits, Tensor targets, Tensor grad_out, Tensor? grad_scale, Tensor stats, int shift, int rows, "
        "Tensor? target_row=None, Tensor? live=None) -> Tensor", &loss_bwd_scaled);
  m.def("repeated_rows_sum", &repeated_rows_sum);
  m.def("document_interval", &document_interval);
  m.def("select_anchors", &select_anchors);
  m.def("anchor_spec", &anchor_spec);
  m.def("anchor_slots", &anchor_slots);
  m.def("compact_rows", &compact_rows);
  m.def("cod_step", &cod_step);
  m.def("peagle_spec", &peagle_spec);
  m.def("embedding_bwd", &embedding_bwd);
  m.def("gate_mul_fwd", &gate_mul_fwd);
  m.def("gate_mul_bwd", &gate_mul_bwd);
  m.def("topk_rows", &topk_rows);
  m.def("moe_plan(Tensor expert, int E, int capacity, int k=1, Tensor? live=None) -> (Tensor, Tensor, Tensor, Tensor)", &moe_plan);
  m.def("moe_gather", &moe_gather);
  m.def("moe_gather_bwd(Tensor d_pad, Tensor slot_row, int k, Tensor? live=None) -> Tensor", &moe_gather_bwd);
  m.def("moe_combine(Tensor y_pad, Tensor slot_row, Tensor p, Tensor? shared, Tensor? gate, Tensor? residual, Tensor? live=None) -> Tensor", &moe_combine);
  m.def("moe_combine_bwd(Tensor dout, Tensor y_pad, Tensor row_slot, Tensor seg, Tensor p, Tensor? shared, Tensor? gate, Tensor? live=None) -> "
        "(Tensor, Tensor, Tensor, Tensor)", &moe_combine_bwd);
  m.def("gemm_grouped_swiglu", &gemm_grouped_swiglu);
  m.def("rope_(Tensor x, Tensor positions, Tensor cos, Tensor sin, int heads, int hd, int rot, float sign, Tensor? live=None) -> ()", &rope_);
  m.def("loss_fwd", &loss_fwd);
  m.def("loss_bwd", &loss_bwd);
  m.def("ce_label_fwd", &ce_label_fwd);
  m.def("sumsq", &sumsq);
  m.def("adamw", &adamw);
  m.def("muon_momentum", &muon_momentum);
  m.def("muon_apply", &muon_apply);
  m.def("muon_chunk_elements", &muon_chunk_elements_binding);
  m.def("set_hyper", &set_hyper);
  m.def("launch_count", &launch_count);
  m.def("peer_alloc", &peer_alloc);
  m.def("peer_release", &peer_release);
  m.def("peer_handle", &peer_handle);
  m.def("peer_open", &peer_open);
  m.def("peer_close", &peer_close);
  m.def("peer_tensor", &peer_tensor);
  m.def("fused_optim_ctl_words", &fused_optim_ctl_words);
  m.def("fused_sharded_adamw", &fused_sharded_adamw);
  m.def("gemm_swiglu(Tensor x, Tensor w, Tensor status, Tensor? live=None) -> (Tensor, Tensor)", &gemm_swiglu);
  m.def("gemm_scatter", &gemm_scatter);
  m.def("tp_allreduce_ctl_words", &tp_allreduce_ctl_words);
  m.def("tp_reduce_broadcast", &tp_reduce_broadcast);
  m.def("step_tail(Tensor row_loss, Tensor pred, Tensor target, Tensor mask, Tensor prev, float decay, float eps, Tensor? earlier, Tensor? target_row=None) -> "
        "(Tensor, Tensor, Tensor)", &step_tail);
  m.def("checked_build", &checked_build);
  m.def("bounds_report", &bounds_report);
  m.def("ep_push", &ep_push);
  m.def("ep_signal", &ep_signal);
  m.def("ep_wait", &ep_wait);
  m.def("ep_pull", &ep_pull);
  m.def("hs_ring_ctl_words", &hs_ring_ctl_words);
  m.def("hs_push", &hs_push);
  m.def("hs_pop", &hs_pop);
  m.def("gemm_tn(Tensor a, Tensor b, Tensor out, Tensor? residual, int epilogue, Tensor status, Tensor? live=None) -> ()", &gemm_tn);
  m.def("gemm(Tensor a, Tensor b, Tensor out, int epilogue, bool a_mn, bool b_mn, Tensor status, Tensor? live=None) -> ()", &gemm);
  m.def("gemm_variant(Tensor a, Tensor b, Tensor out, int epilogue, bool a_mn, bool b_mn, Tensor status, int variant, Tensor? live=None) -> ()", &gemm_variant);
  m.def("gemm_stack(Tensor a, Tensor b, Tensor out, Tensor? addend, bool a_mn, bool b_mn, float alpha, float beta, bool symmetric, Tensor status, "
        "float? diagonal=None) -> ()", &gemm_stack);
  m.def("lmhead_loss_fwd", &lmhead_loss_fwd);
  m.def("moe_group_plan", &moe_group_plan);
  m.def("gemm_grouped_rows", &gemm_grouped_rows);
  m.def("gemm_grouped_wgrad", &gemm_grouped_wgrad);
  m.def("gemm_wgrad_parts", &gemm_wgrad_parts);
  m.def("gemm_wgrad_parts_rows", &gemm_wgrad_parts_rows);
  m.def("gemm_grouped_wgrad_parts", &gemm_grouped_wgrad_parts);
  m.def("gemm_tn_variant(Tensor a, Tensor b, Tensor out, Tensor? residual, int epilogue, Tensor status, int variant, Tensor? live=None) -> ()", &gemm_tn_variant);
  m.def("attn_fwd", &attn_fwd);
  m.def("attn_fwd_tc", &attn_fwd_tc);
  m.def("attn_bwd", &attn_bwd);
}
