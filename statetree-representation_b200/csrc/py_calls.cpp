// The host path of a module call in native code: TreeLinear products and lists of them (q / k / v, gate / up) for inputs that need
// no conversion.  What Python does for such a call (checks, the output and its views, pointer arrays, the ctypes call) takes 15 to
// 30 us, several times a small product's time on the GPU; this takes 3 to 5.
//
// Nothing is kept between calls but the addresses of the kernel library's entry points.  A call that is not of the plain form
// (another device or type, a bias, rows that are not contiguous or not 16-byte aligned) returns None and takes the general path in
// linear.py, which also raises its errors.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/utils/pybind.h>

#include <cstdint>
#include <stdexcept>
#include <vector>

namespace py = pybind11;

namespace {
using Gemv = int (*)(const void*, const int32_t*, const uint32_t*, const uint32_t*, const void*, void*, float*, int64_t, int64_t,
                     int64_t, void*, int64_t, int32_t*, void*);
using Gemm = int (*)(const void*, const int32_t*, const uint32_t*, const void*, void*, float*, int64_t, int64_t, int64_t, void*,
                     int64_t, int32_t*, void*);
using GemvList = int (*)(int64_t, const void* const*, const int32_t* const*, const uint32_t* const*, const uint32_t* const*,
                         const void*, void* const*, float* const*, int64_t, const int64_t*, int64_t, void*, int64_t, void*);
using GemmList = int (*)(int64_t, const void* const*, const int32_t* const*, const uint32_t* const*, const void*, void* const*,
                         float* const*, int64_t, const int64_t*, int64_t, int32_t*, void*);
using LastError = const char* (*)();

struct Library {
  Gemv gemv;
  Gemm gemm;
  GemvList gemv_list;
  GemmList gemm_list;
  LastError last_error;
};

// rows of x if it can be read as it is: BF16 [..., N] on `device`, contiguous, 16-byte aligned, at least one row; else 0
int64_t plain_rows(const at::Tensor& x, int64_t N, const at::Device& device) {
  if (x.scalar_type() != at::kBFloat16 || x.device() != device || x.dim() < 1 || x.size(-1) != N || x.numel() == 0 ||
      x.layout() != at::kStrided || !x.is_contiguous() || x.is_conj() || x.is_neg())
    return 0;
  return (reinterpret_cast<uintptr_t>(x.const_data_ptr()) & 15u) == 0 ? x.numel() / N : 0;
}

void check(const Library& lib, int rc) {
  if (rc != 0) throw std::runtime_error(lib.last_error());
}

std::vector<int64_t> out_sizes(const at::Tensor& x, int64_t M) {
  auto s = x.sizes().vec();
  s.back() = M;
  return s;
}

// Library.of(addresses): the entry points of the loaded kernel library
Library library(uint64_t gemv, uint64_t gemm, uint64_t gemv_list, uint64_t gemm_list, uint64_t last_error) {
  return Library{reinterpret_cast<Gemv>(gemv), reinterpret_cast<Gemm>(gemm), reinterpret_cast<GemvList>(gemv_list),
                 reinterpret_cast<GemmList>(gemm_list), reinterpret_cast<LastError>(last_error)};
}

// x W^T for one tree: the GEMV (use_gemm false) or the tcgen05 GEMM
py::object linear(const Library& lib, bool use_gemm, const at::Tensor& tree, const at::Tensor& eo, const at::Tensor& el,
                  const at::Tensor& eb, const at::Tensor& x, const at::Tensor& ws, const at::Tensor& cnt) {
  const int64_t M = tree.size(0) * 16, N = tree.size(1) * 64, B = plain_rows(x, N, tree.device());
  if (B == 0) return py::none();
  at::Tensor y;
  int rc;
  {
    py::gil_scoped_release nogil;
    const c10::cuda::CUDAGuard guard(tree.device());
    y = at::empty(out_sizes(x, M), x.options().requires_grad(false));
    void* stream = c10::cuda::getCurrentCUDAStream(tree.device().index()).stream();
    const int64_t ws_bytes = ws.numel() * (int64_t)ws.element_size();
    auto i32 = [](const at::Tensor& t) { return reinterpret_cast<const int32_t*>(t.const_data_ptr()); };
    auto u32 = [](const at::Tensor& t) { return reinterpret_cast<const uint32_t*>(t.const_data_ptr()); };
    int32_t* const c = reinterpret_cast<int32_t*>(cnt.data_ptr());
    rc = use_gemm ? lib.gemm(tree.const_data_ptr(), i32(eo), u32(el), x.const_data_ptr(), y.data_ptr(), nullptr, B, M, N,
                             ws.data_ptr(), ws_bytes, c, stream)
                  : lib.gemv(tree.const_data_ptr(), i32(eo), u32(eb), u32(el), x.const_data_ptr(), y.data_ptr(), nullptr, B, M, N,
                             ws.data_ptr(), ws_bytes, c, stream);
  }
  check(lib, rc);
  return py::cast(y);
}

// the same for one to four trees that share their columns; tables = (eo, el, eb) of each.  ws (GEMV) or cnt (GEMM)
py::object linear_list(const Library& lib, bool use_gemm, const std::vector<at::Tensor>& trees,
                       const std::vector<std::vector<at::Tensor>>& tables, const at::Tensor& x, const at::Tensor& scratch) {
  constexpr int MAX = 4;
  const int n = (int)trees.size();
  if (n < 1 || n > MAX || tables.size() != trees.size()) return py::none();
  const at::Device device = trees[0].device();
  const int64_t N = trees[0].size(1) * 64, B = plain_rows(x, N, device);
  if (B == 0) return py::none();
  std::vector<at::Tensor> ys;
  int rc;
  {
    py::gil_scoped_release nogil;
    const c10::cuda::CUDAGuard guard(device);
    const void* T[MAX];
    const int32_t* EO[MAX];
    const uint32_t *EL[MAX], *EB[MAX];
    void* Y[MAX];
    int64_t M[MAX], total = 0;
    for (int i = 0; i < n; ++i) total += M[i] = trees[i].size(0) * 16;
    at::Tensor flat = at::empty({B * total}, x.options().requires_grad(false));
    int64_t at_row = 0;
    for (int i = 0; i < n; ++i) {                                // one allocation, a contiguous [.., M] block per tree
      auto sizes = out_sizes(x, M[i]);
      std::vector<int64_t> strides(sizes.size());
      int64_t step = 1;
      for (int d = (int)sizes.size() - 1; d >= 0; --d) { strides[d] = step; step *= sizes[d]; }
      ys.push_back(flat.as_strided(sizes, strides, B * at_row));
      at_row += M[i];
      T[i] = trees[i].const_data_ptr();
      EO[i] = reinterpret_cast<const int32_t*>(tables[i][0].const_data_ptr());
      EL[i] = reinterpret_cast<const uint32_t*>(tables[i][1].const_data_ptr());
      EB[i] = reinterpret_cast<const uint32_t*>(tables[i][2].const_data_ptr());
      Y[i] = ys[i].data_ptr();
    }
    void* stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    rc = use_gemm ? lib.gemm_list(n, T, EO, EL, x.const_data_ptr(), Y, nullptr, B, M, N, reinterpret_cast<int32_t*>(scratch.data_ptr()),
                                  stream)
                  : lib.gemv_list(n, T, EO, EB, EL, x.const_data_ptr(), Y, nullptr, B, M, N, scratch.data_ptr(),
                                  scratch.numel() * (int64_t)scratch.element_size(), stream);
  }
  check(lib, rc);
  return py::cast(ys);
}
}  // namespace

PYBIND11_MODULE(_calls, m) {
  py::class_<Library>(m, "Library");
  m.def("library", &library);
  m.def("linear", &linear);
  m.def("linear_list", &linear_list);
}
