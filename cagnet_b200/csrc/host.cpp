// Native host path: the calls of one multiply and of one single-process training epoch, queued from C++.
//
// An epoch of a small graph is a dozen kernels of 2 - 10 us; queued one by one from Python, through autograd and the
// optimizer's own kernels, it took 750 us of host time (2.7 K vertices: 0.77 ms for 0.17 ms of kernels).  Here the same
// sequence is one call: buffers from PyTorch's caching allocator, kernels of libcagnet_b200.so on the current stream.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <array>
#include <vector>

#include "../../include/cagnet_b200.h"

namespace py = pybind11;

namespace {

void check(int status, const char* what) {
  if (status != CAGNET_OK)
    throw std::runtime_error(std::string("cagnet_b200 ") + what + " failed with status " + std::to_string(status) + ": " +
                             cagnet_last_error_string());
}

[[noreturn]] void refuse(const std::string& text) { throw std::runtime_error("cagnet_b200: " + text); }

std::string shape_text(const at::Tensor& t) {
  std::string s = "(";
  for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
  return s + ")";
}

// Leading dimension of a row-major fp32 matrix on the device.
int64_t ld_of(const at::Tensor& t, const char* name) {
  if (!t.is_cuda()) refuse(std::string(name) + " must be a CUDA tensor (there is no CPU path)");
  if (t.scalar_type() != at::kFloat || t.dim() != 2) refuse(std::string(name) + " must be a 2-D float32 tensor");
  const int64_t rows = t.size(0), cols = t.size(1);
  if (cols > 1 && t.stride(1) != 1) refuse(std::string(name) + " must be row-major (unit column stride)");
  if (rows > 1) {
    if (t.stride(0) < cols) refuse(std::string(name) + " has overlapping rows");
    return t.stride(0);
  }
  return std::max<int64_t>(cols, 1);
}

int64_t pad_ld(int64_t f) { return f <= 64 ? (f + 3) / 4 * 4 : (f + 31) / 32 * 32; }

at::Tensor bytes_buffer(const at::TensorOptions& o, size_t bytes) {
  return at::empty({static_cast<int64_t>((std::max<size_t>(bytes, 16) + 3) / 4)}, o);
}

// Scratch memory of one call: from one allocation of `room` bytes as long as that lasts, which saves a small epoch's host
// some 20 trips to the allocator, from allocations of their own beyond.  Everything goes back when the call returns.
class Scratch {
 public:
  Scratch(const at::TensorOptions& o, size_t room) : options_(o), left_(room) {
    if (room) next_ = static_cast<char*>(keep(room));
  }
  void* bytes(size_t n, at::Tensor* owner = nullptr) {
    n = (std::max<size_t>(n, 16) + 511) / 512 * 512;
    if (n <= left_) {
      char* p = next_;
      next_ += n;
      left_ -= n;
      return p;
    }
    if (!owner) return keep(n);
    *owner = bytes_buffer(options_, n);        // released with its matrix
    return owner->data_ptr();
  }

 private:
  void* keep(size_t n) {
    kept_.push_back(bytes_buffer(options_, n));
    return kept_.back().data_ptr();
  }
  at::TensorOptions options_;
  std::vector<at::Tensor> kept_;
  char* next_ = nullptr;
  size_t left_;
};

// A scratch matrix, rows padded as ops.empty_padded pads them.
struct Buffer {
  at::Tensor owner;
  float* data = nullptr;
  int64_t ld = 0;
  Buffer() = default;
  Buffer(Scratch& s, int64_t n, int64_t f) : ld(pad_ld(f)) {
    data = static_cast<float*>(s.bytes(static_cast<size_t>(std::max<int64_t>(n, 1)) * ld * 4, &owner));
  }
  explicit Buffer(const at::Tensor& t) : owner(t), data(t.data_ptr<float>()), ld(t.stride(0)) {}
  float* p() const { return data; }
};

int64_t multiply(const cagnet_block* b, const float* B, int64_t ldb, float* C, int64_t ldc, int32_t f, float beta, Scratch& scratch,
                 void* stream) {
  const size_t bytes = cagnet_spmm_block_workspace_bytes(b, B, ldb, f);
  at::Tensor owner;
  void* ws = bytes ? scratch.bytes(bytes, &owner) : nullptr;
  check(cagnet_spmm_block_f32(b, B, ldb, C, ldc, f, beta, ws, bytes, stream), "spmm");
  return cagnet_spmm_block_launches(b, ldb, f);
}

int64_t spmm(uintptr_t block, int64_t device, const at::Tensor& B, const at::Tensor& C, double beta) {
  const auto* b = reinterpret_cast<const cagnet_block*>(block);
  const int64_t ldb = ld_of(B, "B"), ldc = ld_of(C, "C");
  if (B.size(0) != b->m || C.size(0) != b->n || B.size(1) != C.size(1))
    refuse("spmm shape mismatch: A " + std::to_string(b->n) + "x" + std::to_string(b->m) + ", B " + shape_text(B) + ", C " + shape_text(C));
  if (B.get_device() != device || C.get_device() != device) refuse("spmm operands on different devices");
  if (B.size(1) > INT32_MAX) refuse("spmm is too wide");
  c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
  Scratch scratch(C.options().requires_grad(false), 0);
  return multiply(b, B.data_ptr<float>(), ldb, C.data_ptr<float>(), ldc, static_cast<int32_t>(B.size(1)), static_cast<float>(beta),
                  scratch, c10::cuda::getCurrentCUDAStream().stream());
}

// C += A.B with A as COO: the verdict of the index check is read back while the (guarded) product is already queued.
int64_t spmm_coo(const at::Tensor& rows, const at::Tensor& cols, const at::Tensor& vals, int64_t n, int64_t m, const at::Tensor& B,
                 const at::Tensor& C, bool validate) {
  const int64_t ldb = ld_of(B, "B"), ldc = ld_of(C, "C"), nnz = vals.numel();
  for (const at::Tensor* t : {&rows, &cols, &vals}) {
    if (!t->is_cuda() || !t->is_contiguous() || t->dim() != 1 || t->numel() != nnz || t->scalar_type() != (t == &vals ? at::kFloat : at::kInt))
      refuse("spmm_gpu needs 1-D contiguous int32 indices and float32 values of one length on the device");
    if (t->get_device() != C.get_device()) refuse("spmm operands on different devices");
  }
  if (B.size(0) != m || C.size(0) != n || B.size(1) != C.size(1))
    refuse("spmm shape mismatch: A " + std::to_string(n) + "x" + std::to_string(m) + ", B " + shape_text(B) + ", C " + shape_text(C));
  if (B.get_device() != C.get_device()) refuse("spmm operands on different devices");
  const int32_t f = static_cast<int32_t>(B.size(1));
  c10::cuda::CUDAGuard guard(C.device());
  cudaStream_t s = c10::cuda::getCurrentCUDAStream().stream();
  const auto o = C.options().requires_grad(false);
  // what a call waits on: one pinned word and one event per host thread and device
  struct Verdict {
    int32_t* word = nullptr;
    cudaEvent_t done = nullptr;
  };
  static thread_local std::array<Verdict, 64> verdicts;
  Verdict& v = verdicts[static_cast<size_t>(C.get_device()) % verdicts.size()];
  at::Tensor status;
  if (validate) {
    if (!v.word) {
      if (cudaHostAlloc(reinterpret_cast<void**>(&v.word), sizeof(int32_t), cudaHostAllocDefault) != cudaSuccess ||
          cudaEventCreateWithFlags(&v.done, cudaEventDisableTiming) != cudaSuccess)
        refuse("spmm_gpu: cannot allocate a pinned word");
    }
    status = at::empty({1}, o.dtype(at::kInt));
    check(cagnet_check_coo_i32(rows.data_ptr<int>(), cols.data_ptr<int>(), static_cast<int32_t>(n), static_cast<int32_t>(m), nnz,
                               status.data_ptr<int>(), s), "check_coo");
    if (cudaMemcpyAsync(v.word, status.data_ptr<int>(), sizeof(int32_t), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaEventRecord(v.done, s) != cudaSuccess)
      refuse(std::string("spmm_gpu: ") + cudaGetErrorString(cudaGetLastError()));
  }
  const size_t bytes = cagnet_spmm_coo_workspace_bytes(static_cast<int32_t>(m), nnz, B.data_ptr<float>(), ldb, f);
  at::Tensor ws = bytes_buffer(o, bytes);
  check(cagnet_spmm_coo_f32(rows.data_ptr<int>(), cols.data_ptr<int>(), vals.data_ptr<float>(), static_cast<int32_t>(n),
                            static_cast<int32_t>(m), nnz, B.data_ptr<float>(), ldb, C.data_ptr<float>(), ldc, f,
                            validate ? status.data_ptr<int>() : nullptr, ws.data_ptr(), ws.numel() * 4, s), "spmm_gpu");
  if (validate) {
    cudaError_t e;
    {
      py::gil_scoped_release release;
      e = cudaEventSynchronize(v.done);
    }
    if (e != cudaSuccess) refuse(std::string("spmm_gpu: ") + cudaGetErrorString(e));
    static const char* const reasons[] = {"row indices not sorted", "column index out of range", "row index out of range"};
    if (*v.word) refuse(std::string("malformed sparse block: ") + (*v.word >= 3 && *v.word <= 5 ? reasons[*v.word - 3] : "?"));
  }
  return 2 + (validate ? 1 : 0);
}

// State of torch.optim.Adam over both weights; the step counts are the optimizer's own (fp32 on the host) and are advanced.
struct Adam {
  at::Tensor m1, v1, step1, m2, v2, step2;
  double lr, beta1, beta2, eps;
};

// One epoch of the two-layer model on one process: out = act2((A h) W2), h = act1((A x) W1) -- or A (h W), where
// `min_width` and the layer's widths ask for it --, masked NLL, gradients of both weights (dist1d.GCNFunc,
// dist1d.MaskedNLL), and Adam when its state is given.  `hook(begin, layer_block, width)` brackets every sparse product.
py::tuple epoch(uintptr_t fwd, uintptr_t bwd, const at::Tensor& x, const at::Tensor& w1, const at::Tensor& w2,
                const at::Tensor& y, const at::Tensor& mask, int64_t count, int64_t cls_lo, int64_t cls_hi, bool activations,
                bool min_width, std::optional<Adam> adam, py::object hook) {
  const auto* A = reinterpret_cast<const cagnet_block*>(fwd);
  const auto* At = reinterpret_cast<const cagnet_block*>(bwd);
  const int64_t ldx = ld_of(x, "x"), n = A->n;
  ld_of(w1, "weight1");
  ld_of(w2, "weight2");
  const int32_t f = static_cast<int32_t>(w1.size(0)), h = static_cast<int32_t>(w1.size(1)), c = static_cast<int32_t>(w2.size(1));
  if (x.size(1) != f || w2.size(0) != h || x.size(0) != n || A->m != n || At->n != n || At->m != n || !w1.is_contiguous() ||
      !w2.is_contiguous())
    refuse("epoch: shapes of the operands do not fit");
  if (y.scalar_type() != at::kLong || !y.is_cuda() || !y.is_contiguous() || y.numel() != n || !mask.is_cuda() || mask.numel() != n ||
      !mask.is_contiguous() || (mask.scalar_type() != at::kBool && mask.scalar_type() != at::kByte))
    refuse("epoch: int64 labels and a bool mask on the device are needed");
  c10::cuda::CUDAGuard guard(x.device());
  void* s = c10::cuda::getCurrentCUDAStream().stream();
  const auto o = x.options().requires_grad(false);
  int64_t launches = 0;
  // One allocation for what a small epoch needs: its matrices (eight at most) and about as much again for workspaces.
  const int64_t floats = n * (pad_ld(f) + 4 * pad_ld(h) + 3 * pad_ld(c));
  const bool small = floats <= (8 << 20);
  Scratch scratch(o, small ? static_cast<size_t>(floats) * 8 + (4 << 20) : 0);
  auto product = [&](const cagnet_block* b, const float* B, int64_t ldb, const Buffer& C, int32_t width) {
    if (!hook.is_none()) hook(true, b == At && b != A, width);
    launches += multiply(b, B, ldb, C.p(), C.ld, width, 0.f, scratch, s);
    if (!hook.is_none()) hook(false, b == At && b != A, width);
  };
  auto gemm = [&](const float* X, int64_t ld, const at::Tensor& W, bool transposed, const Buffer& Z, int32_t K, int32_t N, int epi,
                  const float* aux, int64_t ldaux) {
    check(cagnet_gemm_nn_f32(X, ld, W.data_ptr<float>(), W.size(1), transposed, Z.p(), Z.ld, n, K, N, epi, aux, ldaux, s), "gemm_nn");
    ++launches;
  };
  // out = act(Z W) with the activation fused where the product's epilogue has it; log-softmax of up to 256 columns comes with the
  // loss (below)
  auto dense_layer = [&](const float* X, int64_t ld, const at::Tensor& W, const Buffer& Z, int32_t K, int32_t N, bool last) {
    if (!activations) return gemm(X, ld, W, false, Z, K, N, CAGNET_EPI_NONE, nullptr, 0);
    if (!last) return gemm(X, ld, W, false, Z, K, N, CAGNET_EPI_RELU, nullptr, 0);
    gemm(X, ld, W, false, Z, K, N, CAGNET_EPI_NONE, nullptr, 0);
    check(cagnet_log_softmax_fwd_f32(Z.p(), Z.ld, Z.p(), Z.ld, n, N, s), "log_softmax");
    ++launches;
  };
  // weight gradients as partial sums; a small epoch's wait for each other and go in one launch
  std::array<cagnet_tn_sum, 2> sums;
  std::array<cagnet_tn_product, 2> waiting = {};
  auto tn = [&](int layer, const float* H, int64_t ldh, const Buffer& G, int32_t K, int32_t N) {
    const size_t bytes = cagnet_gemm_tn_workspace_bytes(n, K, N);
    void* ws = scratch.bytes(bytes);
    if (small) {
      waiting[layer] = {H, G.p(), ldh, G.ld, K, N, ws, bytes};
      return;
    }
    check(cagnet_gemm_tn_partials_f32(H, ldh, G.p(), G.ld, n, K, N, ws, bytes, &sums[layer], s), "gemm_tn");
    ++launches;
  };
  const float* X = x.data_ptr<float>();
  const bool narrow1 = min_width && h < f, widen1 = min_width && h > f, narrow2 = min_width && c < h, widen2 = min_width && c > h;

  // ---- forward
  Buffer H(scratch, n, h), agg1, agg2;
  if (narrow1) {
    Buffer hw(scratch, n, h);
    gemm(X, ldx, w1, false, hw, f, h, CAGNET_EPI_NONE, nullptr, 0);
    product(A, hw.p(), hw.ld, H, h);
    if (activations) {
      check(cagnet_relu_fwd_f32(H.p(), H.ld, H.p(), H.ld, n, h, s), "relu");
      ++launches;
    }
  } else {
    Buffer z(scratch, n, f);
    product(A, X, ldx, z, f);
    dense_layer(z.p(), z.ld, w1, H, f, h, false);
    if (widen1) agg1 = z;
  }
  at::Tensor loss = at::empty({}, o);
  const size_t loss_bytes = cagnet_nll_workspace_bytes(n);
  float* loss_ws = static_cast<float*>(scratch.bytes(loss_bytes));
  Buffer dz(scratch, n, c);
  int32_t parts = 0;
  const auto* mask8 = static_cast<const uint8_t*>(mask.data_ptr());
  bool loss_done = false;
  const at::Tensor out_t = at::empty({std::max<int64_t>(n, 1), pad_ld(c)}, o);
  const Buffer out(out_t);
  if (narrow2) {
    Buffer hw(scratch, n, c);
    gemm(H.p(), H.ld, w2, false, hw, h, c, CAGNET_EPI_NONE, nullptr, 0);
    product(A, hw.p(), hw.ld, out, c);
    if (activations && c <= 256) {
      check(cagnet_log_softmax_nll_f32(out.p(), out.ld, n, c, y.data_ptr<int64_t>(), mask8, static_cast<int32_t>(cls_lo),
                                       static_cast<int32_t>(cls_hi), static_cast<float>(count), out.p(), out.ld, dz.p(), dz.ld, &parts,
                                       loss_ws, loss_bytes, s), "log_softmax_nll");
      ++launches;
      loss_done = true;
    } else if (activations) {
      check(cagnet_log_softmax_fwd_f32(out.p(), out.ld, out.p(), out.ld, n, c, s), "log_softmax");
      ++launches;
    }
  } else {
    Buffer z(scratch, n, h);
    product(A, H.p(), H.ld, z, h);
    if (activations && c <= 256) {                  // with the loss and its gradient
      int32_t kernels = 0;
      check(cagnet_gemm_nll_f32(z.p(), z.ld, w2.data_ptr<float>(), c, n, h, c, y.data_ptr<int64_t>(), mask8, static_cast<int32_t>(cls_lo),
                                static_cast<int32_t>(cls_hi), static_cast<float>(count), out.p(), out.ld, dz.p(), dz.ld, &parts, &kernels,
                                loss_ws, loss_bytes, s), "gemm_nll");
      launches += kernels;
      loss_done = true;
    } else {
      dense_layer(z.p(), z.ld, w2, out, h, c, true);
    }
    if (widen2) agg2 = z;
  }

  // ---- loss, and its gradient before the second activation
  if (activations && !loss_done) {
    check(cagnet_nll_softmax_bwd_f32(out.p(), out.ld, y.data_ptr<int64_t>(), mask8, n, c, static_cast<int32_t>(cls_lo),
                                     static_cast<int32_t>(cls_hi), static_cast<float>(count), dz.p(), dz.ld, &parts,
                                     loss_ws, loss_bytes, s), "nll_softmax_bwd");
    ++launches;
  } else if (!activations) {
    check(cagnet_nll_masked_f32(out.p(), out.ld, y.data_ptr<int64_t>(), mask8, n, c, static_cast<int32_t>(cls_lo),
                                static_cast<int32_t>(cls_hi), static_cast<float>(count), 1.f, loss.data_ptr<float>(), dz.p(), dz.ld,
                                loss_ws, loss_bytes, s), "nll_masked");
    launches += 2;
  }

  // ---- backward: second layer
  Buffer dh(scratch, n, h), ag1, ag2;         // dh: gradient before the first activation
  const int mask_epi = activations ? CAGNET_EPI_RELU_MASK : CAGNET_EPI_NONE;
  if (widen2) {
    Buffer dzw(scratch, n, h);
    gemm(dz.p(), dz.ld, w2, true, dzw, c, h, CAGNET_EPI_NONE, nullptr, 0);
    product(At, dzw.p(), dzw.ld, dh, h);
    if (activations) {
      check(cagnet_relu_bwd_f32(H.p(), H.ld, dh.p(), dh.ld, dh.p(), dh.ld, n, h, s), "relu_bwd");
      ++launches;
    }
    tn(1, agg2.p(), agg2.ld, dz, h, c);
  } else {
    ag2 = Buffer(scratch, n, c);
    product(At, dz.p(), dz.ld, ag2, c);
    gemm(ag2.p(), ag2.ld, w2, true, dh, c, h, mask_epi, H.p(), H.ld);
    tn(1, H.p(), H.ld, ag2, h, c);
    if (!small) ag2 = Buffer();
  }
  // ---- backward: first layer
  if (widen1) {
    tn(0, agg1.p(), agg1.ld, dh, f, h);
  } else {
    ag1 = Buffer(scratch, n, h);
    product(At, dh.p(), dh.ld, ag1, h);
    tn(0, X, ldx, ag1, f, h);
  }
  if (small) {
    int32_t kernels = 0;
    check(cagnet_gemm_tn_partials2_f32(waiting.data(), sums.data(), n, &kernels, s), "gemm_tn");
    launches += kernels;
  }
  // ---- gradients from their partial sums, Adam, loss
  at::Tensor g1 = at::empty({f, h}, o), g2 = at::empty({h, c}, o);
  std::array<float*, 6> a = {};
  int64_t step = 1;
  if (adam) {
    float *t1 = adam->step1.data_ptr<float>(), *t2 = adam->step2.data_ptr<float>();
    step = static_cast<int64_t>(*t1) + 1;
    a = {w1.data_ptr<float>(), adam->m1.data_ptr<float>(), adam->v1.data_ptr<float>(),
         w2.data_ptr<float>(), adam->m2.data_ptr<float>(), adam->v2.data_ptr<float>()};
    *t1 += 1.f;
    *t2 += 1.f;
    adam->step1.unsafeGetTensorImpl()->bump_version();
    adam->step2.unsafeGetTensorImpl()->bump_version();
  }
  check(cagnet_epoch_tail_f32(&sums[0], g1.data_ptr<float>(), a[0], a[1], a[2], &sums[1], g2.data_ptr<float>(), a[3], a[4], a[5],
                              adam ? adam->lr : 0., adam ? adam->beta1 : 0., adam ? adam->beta2 : 0., adam ? adam->eps : 0., step,
                              loss_ws, parts, static_cast<float>(count), activations ? loss.data_ptr<float>() : nullptr, s), "epoch_tail");
  ++launches;
  return py::make_tuple(out_t.narrow(1, 0, c).narrow(0, 0, n), loss, g1, g2, launches);
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  m.def("spmm", &spmm);
  m.def("spmm_coo", &spmm_coo);
  py::class_<Adam>(m, "Adam").def(py::init([](at::Tensor m1, at::Tensor v1, at::Tensor step1, at::Tensor m2, at::Tensor v2,
                                              at::Tensor step2, double lr, double beta1, double beta2, double eps) {
    return Adam{m1, v1, step1, m2, v2, step2, lr, beta1, beta2, eps};
  }));
  m.def("epoch", &epoch);
}
