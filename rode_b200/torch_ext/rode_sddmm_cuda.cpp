// Torch binding `rode_sddmm_cuda`: the Python entry of the RoDe SDDMM path.
//
// Mirrors the module the reference builds from RoDe_SDDMM/rode_sddmm_cuda.cu (functions
// `preprocess` :54-131 and `sddmm_forward` :136-249, module definition :254-278): same
// function names, argument order, checks and return shapes.  It contains no kernels; it
// turns tensors into pointers and calls the C ABI of librode_b200.so.
//
// Differences from the reference binding:
//   * preprocess runs the row decomposition on the GPU.  A CPU row_offsets tensor (the
//     reference's calling convention) is copied to the current CUDA device, decomposed
//     there, and the results are returned as CPU tensors; a CUDA row_offsets tensor gives
//     CUDA results without any host round trip except the two counts.
//   * sddmm_forward launches on torch's current stream, where block and residue part run side by
//     side as programmatic dependents, instead of creating, synchronising and destroying two
//     streams per call (RoDe_SDDMM/rode_sddmm_cuda.cu:203-246); it does not block the host.
//   * k_version may be any multiple of 4 up to 256.
//   * covers_values (default false) says that row_offsets runs from 0 to the number of values, so that the result
//     need not be zero-filled first.
//   * ordered (default false) gives the call scratch memory in which it orders the segments by their columns; order_verdict
//     and *_order_pays say whether that helps.
//   * sddmm_operands_fit checks both dense operands in one call.
//   * spmm_forward and hot_columns are new: the reference has no Python entry for SpMM.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <tuple>

#include "rode_b200.h"

namespace {

#define RODE_CHECK_CUDA(x) TORCH_CHECK((x).device().is_cuda(), #x " must be a CUDA tensor")
#define RODE_CHECK_CONTIGUOUS(x) TORCH_CHECK((x).is_contiguous(), #x " must be contiguous")
#define RODE_CHECK_INPUT(x) \
    RODE_CHECK_CUDA(x);     \
    RODE_CHECK_CONTIGUOUS(x)
#define RODE_CHECK_FLOAT(x) TORCH_CHECK((x).dtype() == torch::kFloat32, #x " must be float32")
#define RODE_CHECK_INT(x) TORCH_CHECK((x).dtype() == torch::kInt32, #x " must be int32")

// A fresh CUDA tensor straight from the allocator: a small call's time is host work, and the dispatcher's part
// of torch::empty is a fifth of it.
torch::Tensor empty_cuda(at::IntArrayRef sizes, at::ScalarType dtype, const c10::Device &device) {
    return at::detail::empty_cuda(sizes, dtype, device, c10::nullopt);
}

void check_status(int status) { TORCH_CHECK(status == RODE_OK, "rode_b200: ", rode_last_error()); }

std::tuple<torch::Tensor, torch::Tensor, torch::Tensor, int, int> py_preprocess(torch::Tensor row_offsets, int nnz,
                                                                                 int seg_length, int k_block,
                                                                                 int vec_len) {
    TORCH_CHECK(row_offsets.dtype() == torch::kInt32, "row_offsets must be int32");
    TORCH_CHECK(row_offsets.dim() == 1 && row_offsets.size(0) >= 1, "row_offsets must have m + 1 entries");
    TORCH_CHECK(at::cuda::is_available(), "rode_b200 needs a CUDA device; there is no CPU path");
    const bool on_host = row_offsets.device().is_cpu();
    torch::Tensor rp = (on_host ? row_offsets.to(torch::kCUDA) : row_offsets).contiguous();
    const c10::cuda::CUDAGuard guard(rp.device());
    const int m = static_cast<int>(rp.size(0)) - 1;

    long long cap = 0;
    check_status(rode_preprocess_capacity(seg_length, vec_len, m, nnz, &cap));
    size_t ws_bytes = 0;
    check_status(rode_preprocess_workspace_bytes(m, &ws_bytes));
    auto opts = torch::TensorOptions().dtype(torch::kInt32).device(rp.device());
    torch::Tensor blk = torch::empty({std::max<long long>(cap, 1)}, opts);
    torch::Tensor st = torch::empty({cap + 1}, opts);
    torch::Tensor res = torch::empty({std::max(m, 1)}, opts);
    torch::Tensor counts = torch::empty({2}, opts);
    torch::Tensor ws = torch::empty({static_cast<long long>(ws_bytes)}, opts.dtype(torch::kUInt8));
    auto stream = at::cuda::getCurrentCUDAStream(rp.device().index());
    check_status(rode_preprocess(seg_length, k_block, vec_len, m, rp.data_ptr<int>(), blk.data_ptr<int>(),
                                 st.data_ptr<int>(), res.data_ptr<int>(), counts.data_ptr<int>(),
                                 counts.data_ptr<int>() + 1, ws.data_ptr(), ws_bytes, stream.stream()));
    torch::Tensor counts_host = counts.cpu();  // synchronises the stream
    const int n_blk = counts_host.data_ptr<int>()[0];
    const int n_res = counts_host.data_ptr<int>()[1];
    // Shapes as the reference returns them: [max(n_blk,1)], [n_blk + 1], [max(n_res,1)].
    blk = blk.narrow(0, 0, std::max(n_blk, 1));
    st = st.narrow(0, 0, n_blk + 1);
    res = res.narrow(0, 0, std::max(n_res, 1));
    if (on_host) return std::make_tuple(blk.cpu(), st.cpu(), res.cpu(), n_blk, n_res);
    return std::make_tuple(blk.contiguous(), st.contiguous(), res.contiguous(), n_blk, n_res);
}

// Both dense operands are as sddmm_forward takes them: float32, row-major, of these shapes, where `values` is.  (One call in the
// place of a dozen attributes of two tensors, which cost a small call from Python a microsecond; who gets false finds out
// what is wrong in his own time.)
bool py_sddmm_operands_fit(const torch::Tensor &lhs, const torch::Tensor &rhs, const torch::Tensor &values, int64_t m, int64_t n,
                           int64_t k) {
    const auto fits = [&](const torch::Tensor &t, int64_t rows) {
        return t.dim() == 2 && t.size(0) == rows && t.size(1) == k && t.scalar_type() == torch::kFloat32 &&
               t.device() == values.device() && t.is_contiguous();
    };
    return fits(lhs, m) && fits(rhs, n);
}

torch::Tensor py_sddmm_forward(const torch::Tensor &block_indices, const torch::Tensor &residue_indices,
                                 const torch::Tensor &st_offsets, int m1, int m2, const torch::Tensor &row_offsets, const torch::Tensor &column_indices,
                                 const torch::Tensor &values, int m, int n, const torch::Tensor &lhs_matrix,
                                 const torch::Tensor &rhs_matrix, int k_version, bool covers_values, bool ordered) {
    RODE_CHECK_INPUT(block_indices);
    RODE_CHECK_INPUT(residue_indices);
    RODE_CHECK_INPUT(st_offsets);
    RODE_CHECK_INPUT(row_offsets);
    RODE_CHECK_INPUT(column_indices);
    RODE_CHECK_INPUT(values);
    RODE_CHECK_INPUT(lhs_matrix);
    RODE_CHECK_INPUT(rhs_matrix);
    RODE_CHECK_INT(block_indices);
    RODE_CHECK_INT(residue_indices);
    RODE_CHECK_INT(st_offsets);
    RODE_CHECK_INT(row_offsets);
    RODE_CHECK_INT(column_indices);
    RODE_CHECK_FLOAT(values);
    RODE_CHECK_FLOAT(lhs_matrix);
    RODE_CHECK_FLOAT(rhs_matrix);

    const int k = static_cast<int>(lhs_matrix.size(1));
    TORCH_CHECK(k_version > 0 && k_version % 4 == 0 && k_version <= 256,
                "k_version must be a multiple of 4, at most 256");
    TORCH_CHECK(k == k_version, "k dimension must match k_version");
    TORCH_CHECK(lhs_matrix.size(0) == m, "lhs_matrix rows must equal m");
    TORCH_CHECK(rhs_matrix.size(0) == n, "rhs_matrix rows must equal n");
    TORCH_CHECK(rhs_matrix.size(1) == k, "rhs_matrix cols must equal k");
    TORCH_CHECK(row_offsets.size(0) == m + 1, "row_offsets must have m + 1 entries");

    const c10::cuda::CUDAGuard guard(values.device());
    if (m1 == 0 && m2 == 0) return torch::zeros({values.size(0)}, values.options());
    // Entries outside [row_offsets[0], row_offsets[m]) belong to no row (a row pointer cut out of a larger one, padding
    // behind the last row) and are zero, as the reference returns them; the kernels write all others.
    torch::Tensor out = covers_values ? empty_cuda({values.size(0)}, torch::kFloat32, values.device())
                                      : torch::zeros({values.size(0)}, values.options());
    const cudaStream_t s = at::cuda::getCurrentCUDAStream(values.device().index()).stream();
    size_t ws_bytes = 0;
    torch::Tensor ws;
    if (ordered) {
        check_status(rode_sddmm_workspace_bytes(m1, k, values.size(0), &ws_bytes));
        ws = empty_cuda({static_cast<long long>(ws_bytes)}, torch::kUInt8, values.device());
    }
    check_status(rode_sddmm_f32_ordered(m, m1, m2, n, k, values.size(0), block_indices.data_ptr<int>(),
                                        residue_indices.data_ptr<int>(), st_offsets.data_ptr<int>(), row_offsets.data_ptr<int>(),
                                        column_indices.data_ptr<int>(), values.data_ptr<float>(), lhs_matrix.data_ptr<float>(),
                                        rhs_matrix.data_ptr<float>(), out.data_ptr<float>(), ordered ? ws.data_ptr() : nullptr,
                                        ws_bytes, s, s));
    return out;
}

// What rode_order_verdict says of the columns, -1 where the sizes are out of its range.  Reads the verdict back.
int py_order_verdict(const torch::Tensor &block_indices, int m1, const torch::Tensor &row_offsets,
                     const torch::Tensor &column_indices, int n) {
    RODE_CHECK_INPUT(block_indices);
    RODE_CHECK_INPUT(row_offsets);
    RODE_CHECK_INPUT(column_indices);
    RODE_CHECK_INT(block_indices);
    RODE_CHECK_INT(row_offsets);
    RODE_CHECK_INT(column_indices);
    const c10::cuda::CUDAGuard guard(column_indices.device());
    const long long nnz = column_indices.numel();
    int in_range = 0;
    check_status(rode_order_verdict(m1, n, nnz, nullptr, nullptr, nullptr, &in_range, nullptr, nullptr));
    if (!in_range) return -1;
    torch::Tensor verdict = torch::empty({1}, column_indices.options());
    check_status(rode_order_verdict(m1, n, nnz, row_offsets.data_ptr<int>(), column_indices.data_ptr<int>(),
                                    block_indices.data_ptr<int>(), &in_range, verdict.data_ptr<int>(),
                                    at::cuda::getCurrentCUDAStream(column_indices.device().index()).stream()));
    return verdict.item<int>();
}

// Popularity bitmap of the columns for spmm_forward's `hot_columns` argument (rode_hot_columns),
// or None when the library finds that marks would not help.  Reads the flag word back.
c10::optional<torch::Tensor> py_hot_columns(const torch::Tensor &column_indices, int n_cols, int64_t dense_row_bytes,
                                            int64_t budget_bytes) {
    RODE_CHECK_INPUT(column_indices);
    RODE_CHECK_INT(column_indices);
    TORCH_CHECK(n_cols >= 0 && dense_row_bytes > 0 && budget_bytes >= 0, "bad size argument");
    const c10::cuda::CUDAGuard guard(column_indices.device());
    size_t words = 0, ws_bytes = 0;
    check_status(rode_hot_columns_words(n_cols, &words));
    check_status(rode_hot_columns_workspace_bytes(n_cols, &ws_bytes));
    auto opts = column_indices.options();
    torch::Tensor bitmap = torch::empty({static_cast<long long>(words)}, opts);
    torch::Tensor ws = torch::empty({static_cast<long long>(ws_bytes)}, opts.dtype(torch::kUInt8));
    auto stream = at::cuda::getCurrentCUDAStream(column_indices.device().index());
    check_status(rode_hot_columns(column_indices.numel(), n_cols, column_indices.data_ptr<int>(),
                                  static_cast<size_t>(dense_row_bytes), static_cast<size_t>(budget_bytes),
                                  reinterpret_cast<unsigned *>(bitmap.data_ptr<int>()), ws.data_ptr(), ws_bytes,
                                  stream.stream()));
    const bool useful = bitmap[static_cast<long long>(words) - 1].item<int>() != 0;
    if (!useful) return c10::nullopt;
    return bitmap;
}

torch::Tensor py_spmm_forward(const torch::Tensor &block_indices, const torch::Tensor &residue_indices,
                                const torch::Tensor &st_offsets, int m1, int m2, const torch::Tensor &row_offsets, const torch::Tensor &column_indices,
                                const torch::Tensor &values, int m, int k, const torch::Tensor &dense,
                                const c10::optional<torch::Tensor> &hot_columns, bool ordered) {
    RODE_CHECK_INPUT(block_indices);
    RODE_CHECK_INPUT(residue_indices);
    RODE_CHECK_INPUT(st_offsets);
    RODE_CHECK_INPUT(row_offsets);
    RODE_CHECK_INPUT(column_indices);
    RODE_CHECK_INPUT(values);
    RODE_CHECK_INPUT(dense);
    RODE_CHECK_INT(block_indices);
    RODE_CHECK_INT(residue_indices);
    RODE_CHECK_INT(st_offsets);
    RODE_CHECK_INT(row_offsets);
    RODE_CHECK_INT(column_indices);
    TORCH_CHECK(values.dtype() == torch::kFloat32 || values.dtype() == torch::kFloat64,
                "values must be float32 or float64");
    TORCH_CHECK(dense.dtype() == values.dtype(), "dense must have the dtype of values");
    TORCH_CHECK(dense.dim() == 2 && dense.size(0) == k, "dense must be [k, n]");
    TORCH_CHECK(row_offsets.size(0) == m + 1, "row_offsets must have m + 1 entries");
    const int n = static_cast<int>(dense.size(1));

    const c10::cuda::CUDAGuard guard(values.device());
    if (m1 == 0 && m2 == 0) return torch::zeros({m, n}, dense.options());
    torch::Tensor out = empty_cuda({m, n}, dense.scalar_type(), dense.device());  // every row is written
    // Without segments the workspace holds the claim counters of the persistent residue kernel only, which starts at 16
    // waves of 32 warps per SM with 32 rows each over at most two column tiles: 1.2 million rows on 148 SMs.
    size_t ws_bytes = 0;
    torch::Tensor ws;
    void *ws_ptr = nullptr;
    if (m1 > 0 || m >= 1 << 19) {
        check_status((ordered ? rode_spmm_ordered_workspace_bytes : rode_spmm_workspace_bytes)(
            m1, n, static_cast<int>(dense.element_size()), &ws_bytes));
        ws = empty_cuda({static_cast<long long>(ws_bytes)}, torch::kUInt8, dense.device());
        ws_ptr = ws.data_ptr();
    }
    const unsigned *hot = nullptr;
    if (hot_columns.has_value()) {
        RODE_CHECK_INPUT(*hot_columns);
        RODE_CHECK_INT(*hot_columns);
        TORCH_CHECK(hot_columns->numel() == (static_cast<long long>(k) + 31) / 32 + 1,
                    "hot_columns must come from hot_columns() for this matrix");
        hot = reinterpret_cast<const unsigned *>(hot_columns->data_ptr<int>());
    }
    const cudaStream_t s = at::cuda::getCurrentCUDAStream(values.device().index()).stream();
    if (ordered) {
        const auto call = [&](auto *entry, auto *type) {
            using T = std::remove_pointer_t<decltype(type)>;
            check_status(entry(m, m1, k, n, values.size(0), values.data_ptr<T>(), column_indices.data_ptr<int>(),
                               row_offsets.data_ptr<int>(), block_indices.data_ptr<int>(), st_offsets.data_ptr<int>(),
                               dense.data_ptr<T>(), out.data_ptr<T>(), ws_ptr, ws_bytes, s, s));
        };
        if (dense.dtype() == torch::kFloat32)
            call(&rode_spmm_f32_ordered, static_cast<float *>(nullptr));
        else
            call(&rode_spmm_f64_ordered, static_cast<double *>(nullptr));
        return out;
    }
    if (dense.dtype() == torch::kFloat32)
        check_status(rode_spmm_f32_all(m, m1, k, n, values.size(0), values.data_ptr<float>(), column_indices.data_ptr<int>(),
                                       row_offsets.data_ptr<int>(), block_indices.data_ptr<int>(),
                                       st_offsets.data_ptr<int>(), dense.data_ptr<float>(), out.data_ptr<float>(),
                                       ws_ptr, ws_bytes, hot, s, s));
    else
        check_status(rode_spmm_f64_all(m, m1, k, n, values.size(0), values.data_ptr<double>(), column_indices.data_ptr<int>(),
                                       row_offsets.data_ptr<int>(), block_indices.data_ptr<int>(),
                                       st_offsets.data_ptr<int>(), dense.data_ptr<double>(), out.data_ptr<double>(),
                                       ws_ptr, ws_bytes, hot, s, s));
    return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("preprocess", &py_preprocess, "RoDe CSR row decomposition (GPU)", py::arg("row_offsets"), py::arg("nnz"),
          py::arg("seg_length"), py::arg("k_block"), py::arg("vec_len"));
    m.def("sddmm_forward", &py_sddmm_forward, "RoDe SDDMM forward (CUDA)", py::arg("block_indices"),
          py::arg("residue_indices"), py::arg("st_offsets"), py::arg("m1"), py::arg("m2"), py::arg("row_offsets"),
          py::arg("column_indices"), py::arg("values"), py::arg("m"), py::arg("n"), py::arg("lhs_matrix"),
          py::arg("rhs_matrix"), py::arg("k_version"), py::arg("covers_values") = false, py::arg("ordered") = false);
    m.def("sddmm_operands_fit", &py_sddmm_operands_fit, py::arg("lhs"), py::arg("rhs"), py::arg("values"), py::arg("m"),
          py::arg("n"), py::arg("k"));
    m.def("order_verdict", &py_order_verdict, "What an order of the segments by their columns can give (CUDA)",
          py::arg("block_indices"), py::arg("m1"), py::arg("row_offsets"), py::arg("column_indices"), py::arg("n"));
    m.def("spmm_order_pays", &rode_spmm_order_pays, py::arg("verdict"), py::arg("m1"), py::arg("k"), py::arg("n"),
          py::arg("nnz"), py::arg("elem_size"));
    m.def("sddmm_order_pays", &rode_sddmm_order_pays, py::arg("verdict"), py::arg("m"), py::arg("m1"), py::arg("n"), py::arg("k"),
          py::arg("nnz"));
    m.def("spmm_forward", &py_spmm_forward, "RoDe SpMM forward (CUDA)", py::arg("block_indices"),
          py::arg("residue_indices"), py::arg("st_offsets"), py::arg("m1"), py::arg("m2"), py::arg("row_offsets"),
          py::arg("column_indices"), py::arg("values"), py::arg("m"), py::arg("k"), py::arg("dense"),
          py::arg("hot_columns") = py::none(), py::arg("ordered") = false);
    m.def("hot_columns", &py_hot_columns, "Column popularity bitmap for spmm_forward, or None (CUDA)",
          py::arg("column_indices"), py::arg("n_cols"), py::arg("dense_row_bytes"), py::arg("budget_bytes") = 0);
}
