// Host path of the public classes: argument checks, output allocation, autograd and the calls into
// the C-ABI library (include/bsp.h), as one native module (torch_blocksparse_b200/_ops).
//
// Why native: at small sizes a call is bound by the host, not by the kernel.  With the autograd
// functions in Python and 40-argument ctypes calls a forward took 44 us and a forward + backward
// 150-190 us of host time around 9 and 33 us of kernels (one sequence of 1024 tokens, 12 heads).
// Each operation object below holds what does not change between calls (the layout's tables on one
// device, block, mode), so that a call from Python passes little more than the tensors.
//
// Semantics follow the reference's autograd functions:
//   MatMul      torch_blocksparse/matmul.py:299-364, 460-552, 558-606
//   Softmax     torch_blocksparse/softmax.py:253-326 (in place; rpe and masks get no gradient)
//   Attention   torch_blocksparse/deepspeedsparseselfattention.py:135-166
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/types.h>
#include <ATen/ops/constant_pad_nd.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>

#include "bsp.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int kMaxSoftmaxRow = 32768;

// ---- errors and arguments ----------------------------------------------------------------------
[[noreturn]] void raise_status(int rc) {
  const char* msg = bsp_last_error();
  switch (rc) {
    case BSP_ERR_INVALID: TORCH_CHECK_VALUE(false, msg);
    case BSP_ERR_UNSUPPORTED: TORCH_CHECK_NOT_IMPLEMENTED(false, msg);
    default: TORCH_CHECK(false, msg);
  }
  TORCH_CHECK(false, msg);
}
void check(int rc) { if (rc != BSP_OK) raise_status(rc); }

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return BSP_F32;
    case at::kHalf: return BSP_F16;
    case at::kBFloat16: return BSP_BF16;
    default: TORCH_CHECK_VALUE(false, "unsupported dtype ", t.scalar_type(), " (float32, float16 and bfloat16 are)");
  }
}

void require_cuda(const Tensor& t) {
  TORCH_CHECK(t.is_cuda(), "torch_blocksparse_b200 runs on CUDA tensors only (got a ", t.device(), " tensor)");
}

// Everything a call reads has to lie on one device, and a pointer has to be of the type it is read as.
void require_same(const Tensor& t, const Tensor& ref, const char* what) {
  TORCH_CHECK(t.device() == ref.device(), what, " is on ", t.device(), ", the call runs on ", ref.device());
  TORCH_CHECK_VALUE(t.scalar_type() == ref.scalar_type(), what, " must be ", ref.scalar_type(), " (got ", t.scalar_type(), ")");
}

// Whether a call on these tensors goes through autograd: one of them needs a gradient (a bias or a
// mask too, although it receives none: the result can then be differentiated), or carries a
// forward-mode tangent, which the functions below refuse (passing them by would drop it silently).
bool needs_grad(const Tensor& t) { return t.requires_grad(); }
bool needs_grad(const OptTensor& t) { return t && t->requires_grad(); }
bool has_tangent(const Tensor& t) { return t._fw_grad(0).defined(); }
bool has_tangent(const OptTensor& t) { return t && has_tangent(*t); }
template <typename... Ts> bool recorded(const Ts&... t) {
  return (at::GradMode::is_enabled() && (needs_grad(t) || ...)) || (has_tangent(t) || ...);
}
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
int64_t vec_of(const Tensor& t) { return 16 / static_cast<int64_t>(t.element_size()); }
bool aligned16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15) == 0; }

// Wall time of one launch (bench=True), in seconds, and what the reference calls it.
struct Times : torch::CustomClassHolder {
  double c = -1, da = -1, db = -1;
};
class Timer {
 public:
  Timer(double* out, const Tensor& ref) : out_(out) {
    if (!out_) return;
    stream_ = static_cast<cudaStream_t>(stream_of(ref));
    TORCH_CHECK(cudaEventCreate(&t0_) == cudaSuccess && cudaEventCreate(&t1_) == cudaSuccess, "cannot create a timing event");
    cudaEventRecord(t0_, stream_);
  }
  void stop() {
    if (!out_) return;
    cudaEventRecord(t1_, stream_);
    cudaEventSynchronize(t1_);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, t0_, t1_);
    *out_ = ms * 1e-3;
    int status = 0;
    check(bsp_device_status(&status));   // this path synchronises anyway: a bounded wait that expired raises here
  }
  ~Timer() { if (t0_) cudaEventDestroy(t0_); if (t1_) cudaEventDestroy(t1_); }

 private:
  double* out_;
  cudaStream_t stream_ = nullptr;
  cudaEvent_t t0_ = nullptr, t1_ = nullptr;
};

// ---- MatMul ------------------------------------------------------------------------------------
struct MatMulOp : torch::CustomClassHolder {
  Tensor hdr, meta;                        // header (host) and tables (device) of the layout
  int64_t H, Mb, Nb, nnz, block;
  char mode[4];
  bool trans_a, trans_b;
  const int32_t* h() const { return hdr.const_data_ptr<int32_t>(); }
  const int32_t* d() const { return meta.const_data_ptr<int32_t>(); }
};

// A [Z, H, R, C] operand as the kernels address it: one unit inner stride, every other stride a
// multiple of 16 bytes, aligned base; anything else is copied.
struct Dense {
  Tensor t;
  int64_t s[4];
};
Dense prep_dense(const Tensor& x) {
  const int64_t vec = vec_of(x);
  Dense d{x, {x.stride(0), x.stride(1), x.stride(2), x.stride(3)}};
  if (x.size(0) == 1) d.s[0] = 0;          // strides of size-1 dimensions carry no meaning
  if (x.size(1) == 1) d.s[1] = 0;
  if (x.size(2) == 1) d.s[2] = x.size(3);
  if (x.size(3) == 1) d.s[3] = 1;
  bool ok = d.s[3] == 1 || d.s[2] == 1;
  if (ok) {
    const int64_t other = d.s[3] == 1 ? d.s[2] : d.s[3];
    ok = d.s[0] % vec == 0 && d.s[1] % vec == 0 && (other == 1 || other % vec == 0) && aligned16(x);
  }
  if (!ok) {
    d.t = x.contiguous();
    for (int i = 0; i < 4; ++i) d.s[i] = d.t.stride(i);
  }
  return d;
}
bool block_format(const Tensor& x, int64_t block) {
  return x.stride(3) == 1 && x.stride(2) == block && x.stride(1) == block * block && aligned16(x) &&
         (x.size(0) == 1 || x.stride(0) % vec_of(x) == 0);
}
Tensor prep_sparse(const Tensor& x, int64_t block) { return block_format(x, block) ? x : x.contiguous(); }
// Whether batch entries of a block-format tensor share memory (an expanded tensor, the gradient of a
// sum over the batch): such a tensor can be read, but not written in place.
bool shares_batch(const Tensor& x, int64_t block) {
  return x.size(0) > 1 && x.size(1) > 0 && x.stride(0) < x.size(1) * block * block;
}

// `any_k`: the reduction size need not be a multiple of 16 (both operands must be k-strided then).
Tensor sdd(const MatMulOp& p, Tensor a, Tensor b, bool ta, bool tb, bool tc, double* time, bool any_k = false) {
  if (tc) {
    std::swap(a, b);
    const bool t = ta;
    ta = !tb;
    tb = !t;
  }
  const Dense A = prep_dense(a), B = prep_dense(b);
  const int64_t Z = a.size(0), K = a.size(ta ? 2 : 3), M = a.size(ta ? 3 : 2), N = b.size(tb ? 2 : 3);
  TORCH_CHECK_VALUE(any_k || K % 16 == 0, "Reduction size for SDD must be a multiple of 16");
  TORCH_CHECK_VALUE(b.size(0) == Z && b.size(1) == a.size(1) && a.size(1) == p.H && b.size(tb ? 3 : 2) == K &&
                        M == p.Mb * p.block && N == p.Nb * p.block,
                    "sdd: operand shapes ", a.sizes(), ", ", b.sizes(), " do not match layout [", p.H, ", ", p.Mb, ", ", p.Nb,
                    "] with block ", p.block);
  Tensor c = at::empty({Z, p.nnz, p.block, p.block}, a.options());
  Timer timer(time, c);
  check(bsp_sdd(A.t.const_data_ptr(), B.t.const_data_ptr(), c.mutable_data_ptr(), dtype_code(a), p.block, Z, p.H, K,
                A.s[0], A.s[1], A.s[ta ? 3 : 2], A.s[ta ? 2 : 3], B.s[0], B.s[1], B.s[tb ? 3 : 2], B.s[tb ? 2 : 3],
                c.stride(0), p.h(), p.d(), stream_of(c)));
  timer.stop();
  return c;
}

// The dense operand of dsd / dds, whose free dimension is `dim`.  A width that is no multiple of 16
// bytes is read where it lies if the reduction side is contiguous and the rest can be addressed (a
// width of one has no stride of its own); along the free side rows would end inside a 16-byte piece:
// those operands are padded with zeros, and the result is cut back to the caller's size.
Dense prep_free(const Tensor& x, int64_t dim) {
  const int64_t vec = vec_of(x), red = 5 - dim, pad = (vec - x.size(dim) % vec) % vec;
  if (pad == 0) return prep_dense(x);
  if (x.stride(red) == 1) {
    Dense d{x, {x.size(0) == 1 ? 0 : x.stride(0), x.size(1) == 1 ? 0 : x.stride(1), x.stride(2), x.stride(3)}};
    if (x.size(dim) == 1) d.s[dim] = x.size(red);
    if (d.s[dim] != 1 && d.s[dim] % vec == 0 && d.s[0] % vec == 0 && d.s[1] % vec == 0 && aligned16(x)) return d;
  }
  return prep_dense(dim == 3 ? at::constant_pad_nd(x, {0, pad}) : at::constant_pad_nd(x, {0, 0, 0, pad}));
}
// The result of dsd / dds, [Z, H, rows, cols], for kernels that compute `n` entries of the free
// dimension of which the caller sees `keep`.  Rows along a free dimension are a multiple of 16 bytes apart.
struct Out {
  Tensor c;
  int64_t free_dim, keep;
  Tensor cut() const { return c.size(free_dim) == keep ? c : c.narrow(free_dim, 0, keep); }
};
Out make_out(const Tensor& like, int64_t Z, int64_t H, int64_t rows, int64_t cols, int64_t free_dim, int64_t keep, int64_t vec) {
  if (free_dim == 3) cols = (cols + vec - 1) / vec * vec;
  return {at::empty({Z, H, rows, cols}, like.options()), free_dim, keep};
}

Tensor dsd(const MatMulOp& p, const Tensor& a, const Tensor& b0, bool ta, bool tb, bool tc, double* time) {
  const int64_t vec = vec_of(b0), fd = tb ? 2 : 3;
  const Tensor s = prep_sparse(a, p.block);
  const Dense B = prep_free(b0, fd);
  const Tensor& b = B.t;
  const int64_t Z = b.size(0), H = b.size(1), M = p.block * (ta ? p.Nb : p.Mb), N = b.size(fd);
  TORCH_CHECK_VALUE(a.size(0) == Z && a.size(1) == p.nnz && a.size(2) == p.block && a.size(3) == p.block && H == p.H &&
                        b.size(tb ? 3 : 2) == p.block * (ta ? p.Mb : p.Nb),
                    "dsd: operand shapes ", a.sizes(), ", ", b.sizes(), " do not match layout [", p.H, ", ", p.Mb, ", ", p.Nb,
                    "] with block ", p.block);
  const Out o = make_out(a, Z, H, tc ? N : M, tc ? M : N, tc ? 2 : 3, b0.size(fd), vec);
  const Tensor& c = o.c;
  Timer timer(time, c);
  check(bsp_dsd(s.const_data_ptr(), B.t.const_data_ptr(), c.mutable_data_ptr(), dtype_code(a), p.block, Z, H, N, s.stride(0), ta,
                B.s[0], B.s[1], B.s[tb ? 3 : 2], B.s[tb ? 2 : 3], c.stride(0), c.stride(1), c.stride(tc ? 3 : 2),
                c.stride(tc ? 2 : 3), p.h(), p.d(), stream_of(c)));
  timer.stop();
  return o.cut();
}

Tensor dds(const MatMulOp& p, const Tensor& a0, const Tensor& b, bool ta, bool tb, bool tc, double* time) {
  const int64_t vec = vec_of(a0), fd = ta ? 3 : 2;
  const Tensor s = prep_sparse(b, p.block);
  const Dense A = prep_free(a0, fd);
  const Tensor& a = A.t;
  const int64_t Z = a.size(0), H = a.size(1), M = a.size(fd), N = p.block * (tb ? p.Mb : p.Nb);
  TORCH_CHECK_VALUE(b.size(0) == Z && b.size(1) == p.nnz && b.size(2) == p.block && b.size(3) == p.block && H == p.H &&
                        a.size(ta ? 2 : 3) == p.block * (tb ? p.Nb : p.Mb),
                    "dds: operand shapes ", a.sizes(), ", ", b.sizes(), " do not match layout [", p.H, ", ", p.Mb, ", ", p.Nb,
                    "] with block ", p.block);
  const Out o = make_out(a, Z, H, tc ? N : M, tc ? M : N, tc ? 3 : 2, a0.size(fd), vec);
  const Tensor& c = o.c;
  Timer timer(time, c);
  check(bsp_dds(A.t.const_data_ptr(), s.const_data_ptr(), c.mutable_data_ptr(), dtype_code(a), p.block, Z, H, M, A.s[0], A.s[1],
                A.s[ta ? 3 : 2], A.s[ta ? 2 : 3], s.stride(0), tb, c.stride(0), c.stride(1), c.stride(tc ? 3 : 2),
                c.stride(tc ? 2 : 3), p.h(), p.d(), stream_of(c)));
  timer.stop();
  return o.cut();
}

// The product of mode c a b ('s' one of them) of the operands in this order; the third letter follows from the first two.
Tensor product(char c, char a, const MatMulOp& p, const Tensor& x, const Tensor& y, bool tx, bool ty, bool tc, double* time) {
  if (c == 's') return sdd(p, x, y, tx, ty, tc, time);
  return a == 's' ? dsd(p, x, y, tx, ty, tc, time) : dds(p, x, y, tx, ty, tc, time);
}

struct MatMulFn : torch::autograd::Function<MatMulFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& a, const Tensor& b, const c10::intrusive_ptr<MatMulOp>& p,
                        const c10::intrusive_ptr<Times>& times) {
    ctx->save_for_backward({a, b});
    ctx->saved_data["p"] = c10::IValue::make_capsule(p);
    if (times) ctx->saved_data["t"] = c10::IValue::make_capsule(times);
    return product(p->mode[0], p->mode[1], *p, a, b, p->trans_a, p->trans_b, false, times ? &times->c : nullptr);
  }
  // da through mode[1] mode[0] mode[2], db through mode[2] mode[1] mode[0] (matmul.py:587-606)
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const auto p = c10::static_intrusive_pointer_cast<MatMulOp>(ctx->saved_data["p"].toCapsule());
    const auto t = ctx->saved_data.find("t");
    const auto times = t == ctx->saved_data.end() ? nullptr : c10::static_intrusive_pointer_cast<Times>(t->second.toCapsule());
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &a = saved[0], &b = saved[1], &dc = grads[0];
    const c10::cuda::CUDAGuard guard(a.device());
    const char* m = p->mode;
    variable_list out(4);
    if (ctx->needs_input_grad(0))
      out[0] = product(m[1], m[0], *p, dc, b, false, !p->trans_b, p->trans_a, times ? &times->da : nullptr);
    if (ctx->needs_input_grad(1))
      out[1] = product(m[2], m[1], *p, a, dc, !p->trans_a, false, p->trans_b, times ? &times->db : nullptr);
    return out;
  }
};

// Leading dimensions of size 1 up to `dims` (matmul.py:663-668).
Tensor pad_shape(Tensor x, int64_t dims) {
  while (x.dim() < dims) x = x.unsqueeze(0);
  return x;
}

Tensor matmul_call(const c10::intrusive_ptr<MatMulOp>& p, const Tensor& a0, const Tensor& b0, const c10::intrusive_ptr<Times>& times) {
  // (the block format has three dimensions in the reference's reading; a batch of one is added)
  const Tensor a = pad_shape(a0, 4), b = pad_shape(b0, 4);
  TORCH_CHECK_VALUE(a.scalar_type() == b.scalar_type(), "operands must have the same dtype (got ", a.scalar_type(), " and ",
                    b.scalar_type(), ")");
  require_cuda(a);
  require_cuda(b);
  require_same(b, a, "the second operand");
  const c10::cuda::CUDAGuard guard(a.device());
  if (recorded(a, b)) return MatMulFn::apply(a, b, p, times);
  return product(p->mode[0], p->mode[1], *p, a, b, p->trans_a, p->trans_b, false, times ? &times->c : nullptr);
}

// y = x . W for x [..., in_features] and the nonzero blocks of W ([in, out], one head): the dds
// product on the rows of x, without copies for rows of any number; the weight's gradient reduces
// over the rows (torch_blocksparse/matmul.py:693-709).
struct LinearFn : torch::autograd::Function<LinearFn> {
  static Tensor run(const MatMulOp& p, const Tensor& x, const Tensor& w, double* time) {
    std::vector<int64_t> shape = x.sizes().vec();
    const Tensor y = dds(p, x.reshape({1, 1, -1, x.size(-1)}), w.unsqueeze(0), false, p.trans_b, false, time);
    shape.back() = y.size(3);
    return y.view(shape);
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const c10::intrusive_ptr<MatMulOp>& p,
                        double* time) {
    ctx->save_for_backward({x, w});
    ctx->saved_data["p"] = c10::IValue::make_capsule(p);
    return run(*p, x, w, time);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const auto p = c10::static_intrusive_pointer_cast<MatMulOp>(ctx->saved_data["p"].toCapsule());
    const variable_list s = ctx->get_saved_variables();
    const c10::cuda::CUDAGuard guard(s[0].device());
    const Tensor x = s[0].reshape({1, 1, -1, s[0].size(-1)}), w = s[1].unsqueeze(0);
    const Tensor dy = grads[0].reshape({1, 1, -1, grads[0].size(-1)});
    variable_list out(4);
    if (ctx->needs_input_grad(0)) out[0] = dds(*p, dy, w, false, !p->trans_b, false, nullptr).view(s[0].sizes());
    if (ctx->needs_input_grad(1)) {
      // (the kernels read x and dy k-strided here, so any number of rows; other strides are copied)
      const bool strided = x.stride(3) == 1 && dy.stride(3) == 1;
      out[1] = sdd(*p, strided ? x : x.contiguous(), strided ? dy : dy.contiguous(), true, false, p->trans_b, nullptr, true).squeeze(0);
    }
    return out;
  }
};

Tensor linear_call(const c10::intrusive_ptr<MatMulOp>& p, const Tensor& x, const Tensor& w0, const c10::intrusive_ptr<Times>& times) {
  require_cuda(x);
  require_cuda(w0);
  TORCH_CHECK_VALUE(p->mode[0] == 'd' && p->mode[1] == 'd' && !p->trans_a, "Linear: its product is x . W, mode 'dds' with x as it is");
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor w = w0.scalar_type() == x.scalar_type() ? w0 : w0.to(x.scalar_type());
  require_same(w, x, "the weight");
  double* time = times ? &times->c : nullptr;
  if (recorded(x, w)) return LinearFn::apply(x, w, p, time);
  return LinearFn::run(*p, x, w, time);
}

// ---- rpe and masks -----------------------------------------------------------------------------
// The optional inputs of Softmax and of the attention as C arguments; `keep` holds the tensors the
// pointers belong to (copies, where the caller's layout could not be read).
struct Masks {
  const void *rpe = nullptr, *kpm = nullptr, *am = nullptr;
  int64_t rpe_sz = 0, rpe_sh = 0, rpe_sr = 0, kpm_sz = 0, am_sr = 0;
  int kpm_mul = 0, am_mul = 0;
};

void set_rpe(Masks& m, OptTensor& rpe, int64_t Z, int64_t H, int64_t M, int64_t N) {
  if (!rpe) return;
  if (rpe->dim() == 3) rpe = rpe->unsqueeze(0);
  TORCH_CHECK_VALUE(rpe->dim() == 4 && rpe->size(1) == H && rpe->size(2) == M && rpe->size(3) == N &&
                        (rpe->size(0) == 1 || rpe->size(0) == Z),
                    "rpe must be [Z, ", H, ", ", M, ", ", N, "] (got ", rpe->sizes(), ")");
  if (rpe->stride(3) != 1 && rpe->size(3) != 1) rpe = rpe->contiguous();
  m.rpe = rpe->const_data_ptr();
  m.rpe_sz = rpe->size(0) == 1 ? 0 : rpe->stride(0);
  m.rpe_sh = rpe->stride(1);
  m.rpe_sr = rpe->stride(2);
}
void set_kpm(Masks& m, OptTensor& kpm, int64_t Z, int64_t N) {
  if (!kpm) return;
  TORCH_CHECK_VALUE(kpm->dim() == 2 && kpm->size(1) == N && (kpm->size(0) == 1 || kpm->size(0) == Z),
                    "key_padding_mask must be [Z, ", N, "] (got ", kpm->sizes(), ")");
  if (kpm->stride(1) != 1) kpm = kpm->contiguous();
  m.kpm = kpm->const_data_ptr();
  m.kpm_sz = kpm->size(0) == 1 ? 0 : kpm->stride(0);
}
void set_am(Masks& m, OptTensor& am, int64_t M, int64_t N) {
  if (!am) return;
  TORCH_CHECK_VALUE(am->dim() == 2 && am->size(0) == M && am->size(1) == N, "attn_mask must be [", M, ", ", N, "] (got ",
                    am->sizes(), ")");
  if (am->stride(1) != 1) am = am->contiguous();
  m.am = am->const_data_ptr();
  m.am_sr = am->stride(0);
}
void check_masks(const OptTensor& rpe, const OptTensor& kpm, const OptTensor& am, const Tensor& x) {
  const at::ScalarType t = x.scalar_type();
  TORCH_CHECK_VALUE(!rpe || rpe->scalar_type() == t, "relative position embedding must be ", t);
  TORCH_CHECK_VALUE(!am || am->scalar_type() == t, "Attention mask must be ", t);
  TORCH_CHECK_VALUE(!kpm || kpm->scalar_type() == t, "Key padding mask must be ", t);
  if (rpe) require_same(*rpe, x, "relative position embedding");
  if (kpm) require_same(*kpm, x, "key_padding_mask");
  if (am) require_same(*am, x, "attn_mask");
}

// ---- Softmax -----------------------------------------------------------------------------------
struct SoftmaxOp : torch::CustomClassHolder {
  Tensor lut;
  int64_t maxlut, H, Mb, Nb, block;
};

void softmax_fwd(const SoftmaxOp& p, const Tensor& x, double scale, OptTensor rpe, OptTensor kpm, OptTensor am, bool kpm_mul,
                 bool am_mul, double* time) {
  TORCH_CHECK_NOT_IMPLEMENTED(p.maxlut * p.block < kMaxSoftmaxRow, "Reductions larger than 32768 elements are not yet implemented");
  TORCH_CHECK_VALUE(x.dim() == 4 && x.size(2) == p.block && x.size(3) == p.block &&
                        x.size(1) * 4 + 2 * p.H * p.Mb == p.lut.numel(),
                    "x of shape ", x.sizes(), " is not a block-format tensor for this layout");
  const int64_t Z = x.size(0), M = p.Mb * p.block, N = p.Nb * p.block;
  TORCH_CHECK(!block_format(x, p.block) || !shares_batch(x, p.block),
              "softmax: batch entries of x refer to the same memory, which the result would overwrite; clone() the tensor first");
  const Tensor work = prep_sparse(x, p.block);
  Masks m;
  set_rpe(m, rpe, Z, p.H, M, N);
  set_kpm(m, kpm, Z, N);
  set_am(m, am, M, N);
  Timer timer(time, x);
  check(bsp_softmax_fwd(work.mutable_data_ptr(), dtype_code(x), Z, work.stride(0), p.block, p.H, p.Mb,
                        p.lut.const_data_ptr<int32_t>(), p.maxlut, static_cast<float>(scale), m.rpe, m.rpe_sz, m.rpe_sh, m.rpe_sr,
                        m.kpm, m.kpm_sz, kpm_mul, m.am, m.am_sr, am_mul, stream_of(x)));
  timer.stop();
  if (!work.is_same(x)) x.copy_(work);
}

struct SoftmaxFn : torch::autograd::Function<SoftmaxFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const c10::intrusive_ptr<SoftmaxOp>& p, double scale,
                        const OptTensor& rpe, const OptTensor& kpm, const OptTensor& am, bool kpm_mul, bool am_mul, double* time) {
    softmax_fwd(*p, x, scale, rpe, kpm, am, kpm_mul, am_mul, time);
    ctx->mark_dirty({x});
    ctx->save_for_backward({x});
    ctx->saved_data["p"] = c10::IValue::make_capsule(p);
    ctx->saved_data["scale"] = scale;
    return x;
  }
  // The incoming gradient is overwritten and returned (softmax.py:325-326).
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const auto p = c10::static_intrusive_pointer_cast<SoftmaxOp>(ctx->saved_data["p"].toCapsule());
    const Tensor y = ctx->get_saved_variables()[0];
    const c10::cuda::CUDAGuard guard(y.device());
    Tensor dx = prep_sparse(grads[0], p->block);
    if (shares_batch(dx, p->block)) dx = dx.clone(at::MemoryFormat::Contiguous);
    const Tensor yy = prep_sparse(y, p->block);
    check(bsp_softmax_bwd(yy.const_data_ptr(), dx.mutable_data_ptr(), dtype_code(y), y.size(0), yy.stride(0), dx.stride(0), p->block,
                          p->H, p->Mb, p->lut.const_data_ptr<int32_t>(), p->maxlut,
                          static_cast<float>(ctx->saved_data["scale"].toDouble()), stream_of(y)));
    variable_list out(9);
    out[0] = dx;
    return out;
  }
};

bool mode_flag(const std::string& mode, const char* name) {
  TORCH_CHECK_VALUE(mode == "add" || mode == "mul", name, " must be 'add' or 'mul'");
  return mode == "mul";
}

Tensor softmax_call(const c10::intrusive_ptr<SoftmaxOp>& p, const Tensor& x, double scale, const OptTensor& rpe,
                    const OptTensor& kpm, const OptTensor& am, const std::string& kpm_mode, const std::string& am_mode,
                    const c10::intrusive_ptr<Times>& times) {
  check_masks(rpe, kpm, am, x);
  require_cuda(x);
  const bool kpm_mul = mode_flag(kpm_mode, "key_padding_mask_mode"), am_mul = mode_flag(am_mode, "attn_mask_mode");
  const c10::cuda::CUDAGuard guard(x.device());
  double* time = times ? &times->c : nullptr;
  if (recorded(x, rpe, kpm, am))
    return SoftmaxFn::apply(x, p, scale, rpe, kpm, am, kpm_mul, am_mul, time);
  {
    const at::AutoDispatchBelowADInplaceOrView below;
    softmax_fwd(*p, x, scale, rpe, kpm, am, kpm_mul, am_mul, time);
  }
  if (!x.is_inference()) x.unsafeGetTensorImpl()->bump_version();
  return x;
}

// ---- attention ---------------------------------------------------------------------------------
struct AttentionOp : torch::CustomClassHolder {
  Tensor hdr, meta;                        // header (host) and tables (device) of the layout
  Tensor thdr, tiles;                      // the same of the tcgen05 tile lists; undefined: none
  int64_t H, nb, block;
};

// What a backward needs besides the saved tensors.
struct AttentionCall : torch::CustomClassHolder {
  c10::intrusive_ptr<AttentionOp> p;
  double scale;
  bool has_rpe, has_kpm, has_am, kpm_mul, use_tiles;
  int am_mul;
};

// [Z, H, L, D] operand with unit stride on D and strides that are multiples of 16 bytes.
Tensor rows(const Tensor& x) {
  const bool ok = x.stride(3) == 1 && aligned16(x) && x.stride(0) % 8 == 0 && x.stride(1) % 8 == 0 && x.stride(2) % 8 == 0;
  return ok ? x : x.contiguous();
}

// Head dimensions other than 64 and 128 are taken only by the kernels that read through tensor maps:
// whatever such a map cannot describe (a broadcast operand, a mask off the 16-byte grid) is copied.
Tensor rows_for(const Tensor& x) {
  Tensor r = rows(x);
  const int64_t D = r.size(3);
  if (D == 64 || D == 128) return r;
  const bool broadcast = (r.stride(0) == 0 && r.size(0) > 1) || (r.stride(1) == 0 && r.size(1) > 1) || r.stride(2) == 0;
  return broadcast ? r.contiguous() : r;
}

// Checks the operands of an attention call and brings them into a form the kernels can address.
struct AttentionOperands {
  Tensor q, k, v;
  OptTensor rpe, kpm, am;
};
AttentionOperands attention_operands(const Tensor& q, const Tensor& k, const Tensor& v, OptTensor rpe, OptTensor kpm, OptTensor am) {
  TORCH_CHECK_VALUE(q.dim() == 4 && k.sizes() == q.sizes() && v.sizes() == q.sizes(), "query, key and value must be [Z, H, L, D] (got ",
                    q.sizes(), ", ", k.sizes(), ", ", v.sizes(), ")");
  require_same(k, q, "the key");
  require_same(v, q, "the value");
  check_masks(rpe, kpm, am, q);
  require_cuda(q);
  const int64_t D = q.size(3);
  if (D != 64 && D != 128) {
    if (rpe && rpe->dim() >= 3 && !(aligned16(*rpe) && rpe->stride(-1) == 1 && rpe->stride(-2) % 8 == 0 && rpe->stride(-2) > 0 &&
                 rpe->stride(-3) % 8 == 0 && rpe->stride(-3) > 0 && (rpe->dim() < 4 || rpe->stride(0) % 8 == 0)))
      rpe = rpe->clone(at::MemoryFormat::Contiguous);
    if (kpm && kpm->dim() == 2 && !(aligned16(*kpm) && kpm->stride(0) % 8 == 0)) kpm = kpm->clone(at::MemoryFormat::Contiguous);
    if (am && am->dim() == 2 && !(aligned16(*am) && am->stride(0) % 8 == 0 && am->stride(0) > 0)) am = am->clone(at::MemoryFormat::Contiguous);
  }
  return {rows_for(q), rows_for(k), rows_for(v), rpe, kpm, am};
}

struct AttentionFn : torch::autograd::Function<AttentionFn> {
  static Tensor run(const AttentionCall& c, const Tensor& q, const Tensor& k, const Tensor& v, Masks& m, bool seq_first, Tensor* lse) {
    const int64_t Z = q.size(0), H = q.size(1), L = q.size(2), D = q.size(3);
    // seq_first: the result in [L, Z, H * D] memory order, handed to the kernel through its strides
    Tensor o = seq_first ? at::empty({L, Z, H, D}, q.options()).permute({1, 2, 0, 3}) : at::empty({Z, H, L, D}, q.options());
    *lse = at::empty({Z, H, L}, q.options().dtype(at::kFloat));
    const AttentionOp& p = *c.p;
    const bool t = c.use_tiles && p.tiles.defined();
    check(bsp_attn_fwd(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), o.mutable_data_ptr(), lse->mutable_data_ptr<float>(),
                       dtype_code(q), p.block, Z, H, L, D, q.stride(0), q.stride(1), q.stride(2), k.stride(0), k.stride(1), k.stride(2),
                       v.stride(0), v.stride(1), v.stride(2), o.stride(0), o.stride(1), o.stride(2),
                       p.hdr.const_data_ptr<int32_t>(), p.meta.const_data_ptr<int32_t>(),
                       t ? p.thdr.const_data_ptr<int32_t>() : nullptr, t ? p.tiles.const_data_ptr<int32_t>() : nullptr,
                       static_cast<float>(c.scale), m.rpe, m.rpe_sz, m.rpe_sh, m.rpe_sr, m.kpm, m.kpm_sz, m.kpm_mul, m.am, m.am_sr,
                       m.am_mul, stream_of(q)));
    return o;
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v,
                        const c10::intrusive_ptr<AttentionCall>& c, Masks& m, const OptTensor& rpe, const OptTensor& kpm,
                        const OptTensor& am, bool seq_first) {
    Tensor lse;
    Tensor o = run(*c, q, k, v, m, seq_first, &lse);
    variable_list keep = {q, k, v, o, lse};
    if (rpe) keep.push_back(*rpe);
    if (kpm) keep.push_back(*kpm);
    if (am) keep.push_back(*am);
    ctx->save_for_backward(std::move(keep));
    ctx->saved_data["c"] = c10::IValue::make_capsule(c);
    return o;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const auto c = c10::static_intrusive_pointer_cast<AttentionCall>(ctx->saved_data["c"].toCapsule());
    const variable_list s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k = s[1], &v = s[2], &o = s[3], &lse = s[4];
    const c10::cuda::CUDAGuard guard(q.device());
    const int64_t Z = q.size(0), H = q.size(1), L = q.size(2), D = q.size(3);
    Masks m;
    size_t at = 5;
    OptTensor rpe, kpm, am;
    if (c->has_rpe) set_rpe(m, rpe = s[at++], Z, H, L, L);
    if (c->has_kpm) set_kpm(m, kpm = s[at++], Z, L);
    if (c->has_am) set_am(m, am = s[at++], L, L);
    m.kpm_mul = c->kpm_mul;
    m.am_mul = c->am_mul;
    const Tensor dout = rows_for(grads[0]);
    const Tensor dq = at::empty({Z, H, L, D}, q.options()), dk = at::empty({Z, H, L, D}, q.options()),
                 dv = at::empty({Z, H, L, D}, q.options()), delta = at::empty({Z, H, L}, lse.options());
    const AttentionOp& p = *c->p;
    const bool t = c->use_tiles && p.tiles.defined();
    check(bsp_attn_bwd(q.const_data_ptr(), k.const_data_ptr(), v.const_data_ptr(), o.const_data_ptr(), dout.const_data_ptr(),
                       lse.const_data_ptr<float>(), delta.mutable_data_ptr<float>(), dq.mutable_data_ptr(), dk.mutable_data_ptr(),
                       dv.mutable_data_ptr(), dtype_code(q), p.block, Z, H, L, D, q.stride(0), q.stride(1), q.stride(2), k.stride(0),
                       k.stride(1), k.stride(2), v.stride(0), v.stride(1), v.stride(2), o.stride(0), o.stride(1), o.stride(2),
                       dout.stride(0), dout.stride(1), dout.stride(2), p.hdr.const_data_ptr<int32_t>(),
                       p.meta.const_data_ptr<int32_t>(), t ? p.thdr.const_data_ptr<int32_t>() : nullptr,
                       t ? p.tiles.const_data_ptr<int32_t>() : nullptr, static_cast<float>(c->scale), m.rpe, m.rpe_sz, m.rpe_sh,
                       m.rpe_sr, m.kpm, m.kpm_sz, m.kpm_mul, m.am, m.am_sr, m.am_mul, stream_of(q)));
    variable_list out(9);
    out[0] = dq;
    out[1] = dk;
    out[2] = dv;
    return out;
  }
};

Tensor attention_call(const c10::intrusive_ptr<AttentionOp>& p, const Tensor& q0, const Tensor& k0, const Tensor& v0, double scale,
                      const OptTensor& rpe0, const OptTensor& kpm0, const OptTensor& am0, bool kpm_mul, int am_mul, bool use_tiles,
                      bool seq_first) {
  auto [q, k, v, rpe, kpm, am] = attention_operands(q0, k0, v0, rpe0, kpm0, am0);
  const int64_t Z = q.size(0), H = q.size(1), L = q.size(2);
  TORCH_CHECK_VALUE(p->H == H && p->nb * p->block == L, "layout [", p->H, ", ", p->nb, ", ", p->nb, "] with block ", p->block,
                    " does not fit operands of shape ", q.sizes());
  const c10::cuda::CUDAGuard guard(q.device());
  Masks m;
  set_rpe(m, rpe, Z, H, L, L);
  set_kpm(m, kpm, Z, L);
  set_am(m, am, L, L);
  m.kpm_mul = kpm_mul;
  m.am_mul = am_mul;
  auto c = c10::make_intrusive<AttentionCall>();
  c->p = p;
  c->scale = scale;
  c->has_rpe = rpe.has_value();
  c->has_kpm = kpm.has_value();
  c->has_am = am.has_value();
  c->kpm_mul = kpm_mul;
  c->am_mul = am_mul;
  c->use_tiles = use_tiles;
  if (recorded(q, k, v, rpe, kpm, am))
    return AttentionFn::apply(q, k, v, c, m, rpe, kpm, am, seq_first);
  Tensor lse;
  return AttentionFn::run(*c, q, k, v, m, seq_first, &lse);
}

// The checks of the attention wrapper on its three operands and the key as [Z, H, L, D]: a key given
// as [.., D, L] is viewed back (deepspeedsparseselfattention.py:119-123, 139-141).
Tensor attention_key(const Tensor& q, const Tensor& k0, const Tensor& v) {
  const Tensor k = k0.size(2) != q.size(2) ? k0.permute({0, 1, 3, 2}) : k0;
  TORCH_CHECK_NOT_IMPLEMENTED(q.sizes() == k.sizes() && k.sizes() == v.sizes(), "only self-attention is supported for now");
  return k;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  namespace py = pybind11;
  py::class_<Times, c10::intrusive_ptr<Times>>(m, "Times")
      .def(py::init([] { return c10::make_intrusive<Times>(); }))
      .def_readonly("c", &Times::c).def_readonly("da", &Times::da).def_readonly("db", &Times::db);
  py::class_<MatMulOp, c10::intrusive_ptr<MatMulOp>>(m, "MatMulOp")
      .def(py::init([](Tensor hdr, Tensor meta, int64_t block, const std::string& mode, bool ta, bool tb) {
        auto p = c10::make_intrusive<MatMulOp>();
        const int32_t* h = hdr.const_data_ptr<int32_t>();
        p->H = h[1]; p->Mb = h[2]; p->Nb = h[3]; p->nnz = h[4];
        p->hdr = hdr; p->meta = meta; p->block = block; p->trans_a = ta; p->trans_b = tb;
        TORCH_CHECK_VALUE(mode.size() == 3, "mode must be sdd, dsd or dds");
        std::copy(mode.begin(), mode.end(), p->mode);
        p->mode[3] = 0;
        return p;
      }))
      .def("__call__", &matmul_call, py::arg("a"), py::arg("b"), py::arg("times") = c10::intrusive_ptr<Times>(),
           py::call_guard<py::gil_scoped_release>())
      .def("linear", &linear_call, py::call_guard<py::gil_scoped_release>());
  py::class_<SoftmaxOp, c10::intrusive_ptr<SoftmaxOp>>(m, "SoftmaxOp")
      .def(py::init([](Tensor lut, int64_t maxlut, int64_t H, int64_t Mb, int64_t Nb, int64_t block) {
        auto p = c10::make_intrusive<SoftmaxOp>();
        p->lut = lut; p->maxlut = maxlut; p->H = H; p->Mb = Mb; p->Nb = Nb; p->block = block;
        return p;
      }))
      .def("__call__", &softmax_call, py::call_guard<py::gil_scoped_release>());
  py::class_<AttentionOp, c10::intrusive_ptr<AttentionOp>>(m, "AttentionOp")
      .def(py::init([](Tensor hdr, Tensor meta, OptTensor thdr, OptTensor tiles, int64_t block) {
        auto p = c10::make_intrusive<AttentionOp>();
        const int32_t* h = hdr.const_data_ptr<int32_t>();
        TORCH_CHECK_VALUE(h[2] == h[3], "an attention layout must be [heads, L/block, L/block]");
        p->H = h[1]; p->nb = h[2];
        p->hdr = hdr; p->meta = meta; p->block = block;
        if (tiles) { p->thdr = *thdr; p->tiles = *tiles; }
        return p;
      }))
      .def("__call__", &attention_call, py::call_guard<py::gil_scoped_release>());
  m.def("attention_key", &attention_key);
  m.def("attention_operands", [](const Tensor& q, const Tensor& k, const Tensor& v, OptTensor rpe, OptTensor kpm, OptTensor am) {
    AttentionOperands o = attention_operands(q, k, v, rpe, kpm, am);
    return std::make_tuple(o.q, o.k, o.v, o.rpe, o.kpm, o.am);
  });
  m.def("attention_gradient", &rows_for);
}
