// The host path of a module call in native code: TreeLinear products and lists of them (q / k / v, gate / up) for inputs that need
// no conversion, and the launches of a matrix's conversion and its check.  What Python does for such a product (checks, the output
// and its views, pointer arrays, the ctypes call) takes 15 to 30 us, several times a small product's time on the GPU; this takes
// 3 to 5.
//
// Nothing is kept between calls but the addresses of the kernel library's entry points.  A call that is not of the plain form
// (another device or type, a bias, rows that are not contiguous or not 16-byte aligned) returns None and takes the general path in
// linear.py, which also raises its errors.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/version.h>

#include <cstdint>
#include <map>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/statetree_b200.h"

namespace py = pybind11;

namespace {
// the entry points of the loaded kernel library, with the types of the header that this file was compiled with
struct Library {
  decltype(&st_gemv) gemv;
  decltype(&st_gemm) gemm;
  decltype(&st_gemv_list) gemv_list;
  decltype(&st_gemm_list) gemm_list;
  decltype(&st_last_error) last_error;
  decltype(&st_encode) encode;
  decltype(&st_encode_offsets_workspace_bytes) offsets_bytes;
  decltype(&st_encode_offsets) offsets;
  decltype(&st_encode_lists) lists;
  decltype(&st_dec_check) dec_check;
  decltype(&st_lists_check) lists_check;
};

// rows of x if it can be read as it is: BF16 [..., N] on `device`, contiguous, 16-byte aligned, at least one row; else 0
int64_t plain_rows(const at::Tensor& x, int64_t N, const at::Device& device) {
  if (x.scalar_type() != at::kBFloat16 || x.device() != device || x.dim() < 1 || x.size(-1) != N || x.numel() == 0 ||
      x.layout() != at::kStrided || !x.is_contiguous() || x.is_conj() || x.is_neg())
    return 0;
  return (reinterpret_cast<uintptr_t>(x.const_data_ptr()) & 15u) == 0 ? x.numel() / N : 0;
}

bool on(const at::Device& device, const at::Tensor& a, const at::Tensor& b, const at::Tensor& c) {
  return a.device() == device && b.device() == device && c.device() == device;
}

void check(const Library& lib, int rc) {
  if (rc != 0) throw std::runtime_error(lib.last_error());
}

std::vector<int64_t> out_sizes(const at::Tensor& x, int64_t M) {
  auto s = x.sizes().vec();
  s.back() = M;
  return s;
}

// binds the entry points: their addresses by name
Library library(const std::map<std::string, uint64_t>& address) {
  Library lib;
  auto bind = [&](auto& entry, const char* name) {
    entry = reinterpret_cast<std::remove_reference_t<decltype(entry)>>(address.at(name));
  };
  bind(lib.gemv, "st_gemv");
  bind(lib.gemm, "st_gemm");
  bind(lib.gemv_list, "st_gemv_list");
  bind(lib.gemm_list, "st_gemm_list");
  bind(lib.last_error, "st_last_error");
  bind(lib.encode, "st_encode");
  bind(lib.offsets_bytes, "st_encode_offsets_workspace_bytes");
  bind(lib.offsets, "st_encode_offsets");
  bind(lib.lists, "st_encode_lists");
  bind(lib.dec_check, "st_dec_check");
  bind(lib.lists_check, "st_lists_check");
  return lib;
}

// x W^T for one tree: the GEMV (use_gemm false) or the tcgen05 GEMM
py::object linear(const Library& lib, bool use_gemm, const at::Tensor& tree, const at::Tensor& eo, const at::Tensor& el,
                  const at::Tensor& eb, const at::Tensor& x, const at::Tensor& ws, const at::Tensor& cnt) {
  const int64_t M = tree.size(0) * 16, N = tree.size(1) * 64, B = plain_rows(x, N, tree.device());
  if (B == 0 || !on(tree.device(), eo, el, eb)) return py::none();
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
  for (int i = 0; i < n; ++i)
    if (trees[i].device() != device || trees[i].size(1) * 64 != N || tables[i].size() != 3 ||
        !on(device, tables[i][0], tables[i][1], tables[i][2]))
      return py::none();
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

// W [M, N] BF16 on a GPU, contiguous, 16-byte aligned -> (tree, rows, cols, bits, eo, el, eb): the format's parts and the kernels'
// side tables.  The lists' length depends on the data, so the stream is synchronised once, before they are made; the kernel that
// fills them may still run when the call returns.
py::tuple encode(const Library& lib, const at::Tensor& W) {
  TORCH_CHECK(W.is_cuda() && W.dim() == 2 && W.scalar_type() == at::kBFloat16 && W.is_contiguous(),
              "encode: a contiguous BF16 matrix on a GPU");
  const int64_t M = W.size(0), N = W.size(1);
  TORCH_CHECK(M > 0 && N > 0 && M % 16 == 0 && N % 64 == 0, "encode: rows must be a multiple of 16, columns of 64");
  const int64_t NG = N / 64, nrec = M / 16 * NG;
  at::Tensor tree, rows, cols, bits, eo, el, eb;
  {
    py::gil_scoped_release nogil;
    const c10::cuda::CUDAGuard guard(W.device());
    void* stream = c10::cuda::getCurrentCUDAStream(W.device().index()).stream();
    const auto u8 = W.options().requires_grad(false).dtype(at::kByte), i32 = u8.dtype(at::kInt);
    auto ip = [](const at::Tensor& t) { return reinterpret_cast<int32_t*>(t.data_ptr()); };
    auto up = [](const at::Tensor& t) { return reinterpret_cast<uint32_t*>(t.data_ptr()); };
    tree = at::empty({M / 16, NG, 1552}, u8);
    eo = at::empty({nrec + 1}, i32);
    eb = at::empty({M / 16 * ((NG + 7) / 8), 16}, i32);
    const int64_t need = lib.offsets_bytes(M, N);
    at::Tensor rowcnt = at::empty({M * NG}, u8), reccnt = at::empty({nrec + 1}, i32), roff = at::empty({M * NG}, i32),
               ws = at::empty({need}, u8);
    uint8_t* const rc = reinterpret_cast<uint8_t*>(rowcnt.data_ptr());
    check(lib, lib.encode(W.const_data_ptr(), M, N, tree.data_ptr(), rc, ip(reccnt), stream));
    check(lib, lib.offsets(rc, ip(reccnt), M, N, ip(roff), ip(eo), ws.data_ptr(), need, stream));
    const int64_t n = eo.select(0, nrec).item<int32_t>();         // (synchronises)
    rows = at::empty({n}, i32);
    cols = at::empty({n}, i32);
    bits = at::empty({n}, i32.dtype(at::kShort));
    el = n ? at::empty({n}, i32) : at::zeros({1}, i32);
    void* const spare = el.data_ptr();                            // (no escapes: empty tensors have no address; nothing is written)
    check(lib, lib.lists(W.const_data_ptr(), M, N, rc, ip(roff), ip(eo), up(el), up(eb),
                         reinterpret_cast<int32_t*>(n ? rows.data_ptr() : spare), reinterpret_cast<int32_t*>(n ? cols.data_ptr() : spare),
                         reinterpret_cast<int16_t*>(n ? bits.data_ptr() : spare), stream));
  }
  return py::make_tuple(tree, rows, cols, bits, eo, el, eb);
}

// launches the check of a tree against W (contiguous, 16-byte aligned) and of the stored lists and eb, if there are any (an empty
// vector: none): an int32 count of what is wrong, on the GPU
at::Tensor check_start(const Library& lib, const at::Tensor& tree, const at::Tensor& eo, const at::Tensor& el, const at::Tensor& W,
                       const std::vector<at::Tensor>& stored) {
  TORCH_CHECK(W.is_cuda() && W.dim() == 2 && W.scalar_type() == at::kBFloat16 && W.is_contiguous(),
              "dec_check: a contiguous BF16 matrix on a GPU");
  TORCH_CHECK(tree.is_cuda() && tree.dim() == 3 && tree.size(0) * 16 == W.size(0) && tree.size(1) * 64 == W.size(1),
              "dec_check: the tree is not one of this matrix");
  TORCH_CHECK(eo.is_cuda() && el.is_cuda() && (stored.empty() || stored.size() == 4), "dec_check: tables");
  py::gil_scoped_release nogil;
  const int64_t M = W.size(0), N = W.size(1);
  const c10::cuda::CUDAGuard guard(W.device());
  void* stream = c10::cuda::getCurrentCUDAStream(W.device().index()).stream();
  at::Tensor bad = at::zeros({1}, W.options().requires_grad(false).dtype(at::kInt));
  auto i32 = [](const at::Tensor& t) { return reinterpret_cast<const int32_t*>(t.const_data_ptr()); };
  auto u32 = [](const at::Tensor& t) { return reinterpret_cast<const uint32_t*>(t.const_data_ptr()); };
  int32_t* const b = reinterpret_cast<int32_t*>(bad.data_ptr());
  check(lib, lib.dec_check(tree.const_data_ptr(), i32(eo), u32(el), M, N, W.const_data_ptr(), b, stream));
  if (!stored.empty()) {
    for (const at::Tensor& t : stored) TORCH_CHECK(t.is_cuda(), "dec_check: tables");
    const int64_t n = stored[0].numel();
    TORCH_CHECK(stored[1].numel() == n && stored[2].numel() == n, "dec_check: lists of different lengths");
    check(lib, lib.lists_check(i32(stored[0]), i32(stored[1]), reinterpret_cast<const int16_t*>(stored[2].const_data_ptr()), n, i32(eo),
                               u32(el), u32(stored[3]), M, N, W.const_data_ptr(), b, stream));
  }
  return bad;
}
}  // namespace

PYBIND11_MODULE(_calls, m) {
  m.attr("ABI") = ST_ABI_VERSION;                // what this file was compiled against (compared when it is loaded)
  m.attr("TORCH") = TORCH_VERSION;
  py::class_<Library>(m, "Library");
  m.def("library", &library);
  m.def("linear", &linear);
  m.def("linear_list", &linear_list);
  m.def("encode", &encode);
  m.def("check_start", &check_start);
}
