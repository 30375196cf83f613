// The eager host path of the public ops: operand checks, allocations, launches and the autograd nodes of
// gemm_fp8, grouped_gemm_fp8 and the quantise / dequantise ops, in C++ over the C ABI of ptb.h.
//
// Why native: a small forward (256 x 512 x 1024 blockwise) keeps the GPU busy for 16 us, and the Python form of the
// same call -- an autograd.Function, a ctypes call and four torch.empty per kernel, a device context each --
// took 81 us of host time.  Here a kernel costs its launch (2 - 3 us) and half a microsecond per allocation, and a
// backward pass runs in the autograd engine without taking the interpreter lock.
//
// The arithmetic schedule is that of the Python autograd Functions (pytorch/ops/gemm_fp8.py, grouped_gemm_fp8.py);
// what differs is only which companions are made: operand copies that exist for a gradient nobody asked for (inference,
// frozen weights) are not computed.  Every entry returns None when an argument is not the plain case handled
// here, and the Python form -- with its checks, its error messages and its per-kernel instrumentation -- takes over.
#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <pybind11/pybind11.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <stdexcept>
#include <string>

#include "ptb.h"

namespace py = pybind11;
using at::ScalarType;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

constexpr int kMxGranularity = 4; // ScalingGranularity.MX_BLOCKWISE
constexpr int64_t kBlk = 128, kMxBlk = 32;

std::atomic<int64_t> g_calls{0}; // C-ABI calls that enqueued work from here
std::atomic<bool> g_check_status{false}; // debug: wait for the device after every GEMM and read the status word
std::atomic<bool> g_recording{false};    // per-kernel times are being recorded
PyObject *g_error_class = nullptr, *g_timed_region = nullptr;

struct PtbFail : std::runtime_error {
    using std::runtime_error::runtime_error;
};

void check(int rc, const char *what) {
    if (rc != 0) throw PtbFail(std::string(what) + " failed with status " + std::to_string(rc) + ": " + ptb_last_error());
}

// One C-ABI call.  While per-kernel times are recorded -- a backward pass may meet that although its forward pass did not --
// the recorder's own context manager brackets it with events.
template <typename F> void run(const char *what, F &&f) {
    int rc;
    if (g_recording.load(std::memory_order_relaxed)) {
        py::gil_scoped_acquire gil;
        py::object region = py::handle(g_timed_region)(what);
        region.attr("__enter__")();
        rc = f();
        region.attr("__exit__")(py::none(), py::none(), py::none());
    } else {
        rc = f();
    }
    check(rc, what);
    g_calls.fetch_add(1, std::memory_order_relaxed);
}

template <typename F> void run_gemm(const char *what, cudaStream_t st, F &&f) {
    run(what, f);
    if (!g_check_status.load(std::memory_order_relaxed)) return;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return;
    cudaDeviceSynchronize();
    int code = 0;
    check(ptb_gemm_status(&code, 1), "ptb_gemm_status");
    if (code != 0)
        throw PtbFail(std::string(what) + ": a device-side wait ran out (status " + std::to_string(code) +
                      "); the output is incomplete");
}

#define PTB_RUN(fn, ...) run(#fn, [&] { return fn(__VA_ARGS__); })
#define PTB_RUN_GEMM(fn, ...) run_gemm(#fn, c.st, [&] { return fn(__VA_ARGS__); })

int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }
int64_t round_up(int64_t a, int64_t b) { return cdiv(a, b) * b; }

int code_of(ScalarType t) {
    switch (t) {
    case ScalarType::Float: return PTB_F32;
    case ScalarType::Half: return PTB_F16;
    case ScalarType::BFloat16: return PTB_BF16;
    case ScalarType::Float8_e4m3fn: return PTB_E4M3;
    case ScalarType::Float8_e5m2: return PTB_E5M2;
    default: return -1;
    }
}
bool is_hp(ScalarType t) { const int c = code_of(t); return c >= PTB_F32 && c <= PTB_BF16; }
bool is_16bit(ScalarType t) { return t == ScalarType::Half || t == ScalarType::BFloat16; }
bool is_fp8(ScalarType t) { const int c = code_of(t); return c == PTB_E4M3 || c == PTB_E5M2; }

// One call's device and stream: everything is allocated and enqueued there.
struct Call {
    c10::cuda::OptionalCUDAGuard guard;
    at::Device dev;
    cudaStream_t st;
    explicit Call(const Tensor &t) : dev(t.device()) {
        guard.set_device(dev);
        st = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    }
    Tensor empty(at::IntArrayRef shape, ScalarType dt) const {
        return at::detail::empty_cuda(shape, dt, dev, std::nullopt);
    }
};

// An FP8 copy with its inverse scales: element (row, k-block) of the scales is s[row * sm + kb * sk] (group * sg).
struct Quant {
    Tensor q, s;
    int64_t sm = 0, sk = 0, sg = 0;
    const float *scale() const { return s.const_data_ptr<float>(); }
};

// ---- quantise -------------------------------------------------------------------------------------------------
Quant quant_tensorwise(const Call &c, const Tensor &x, ScalarType dt) {
    Quant r{c.empty(x.sizes(), dt), c.empty({}, ScalarType::Float)};
    Tensor ws = c.empty({PTB_TENSORWISE_WS_BYTES}, ScalarType::Byte);
    PTB_RUN(ptb_quant_fp8_tensorwise, x.const_data_ptr(), code_of(x.scalar_type()), x.numel(), r.q.mutable_data_ptr(),
            code_of(dt), r.s.mutable_data_ptr<float>(), ws.mutable_data_ptr(), c.st);
    return r;
}

Quant quant_rowwise(const Call &c, const Tensor &x, ScalarType dt, int64_t axis) {
    axis = axis < 0 ? axis + x.dim() : axis;
    int64_t B = 1, N = 1;
    auto sshape = x.sizes().vec();
    for (int64_t i = 0; i < axis; ++i) B *= sshape[i];
    for (int64_t i = axis + 1; i < x.dim(); ++i) N *= sshape[i];
    const int64_t M = sshape[axis];
    sshape[axis] = 1;
    Quant r{c.empty(x.sizes(), dt), c.empty(sshape, ScalarType::Float)};
    r.sm = 1;
    Tensor ws;
    if (N > 1) ws = c.empty({B * N}, ScalarType::Float);
    PTB_RUN(ptb_quant_fp8_rowwise, x.const_data_ptr(), code_of(x.scalar_type()), B, M, N, r.q.mutable_data_ptr(), code_of(dt),
            r.s.mutable_data_ptr<float>(), N > 1 ? ws.mutable_data_ptr() : nullptr, c.st);
    return r;
}

Tensor dequant_rowwise(const Call &c, const Tensor &q, const Tensor &s, ScalarType dt, int64_t axis) {
    axis = axis < 0 ? axis + q.dim() : axis;
    int64_t B = 1, N = 1;
    for (int64_t i = 0; i < axis; ++i) B *= q.size(i);
    for (int64_t i = axis + 1; i < q.dim(); ++i) N *= q.size(i);
    Tensor out = c.empty(q.sizes(), dt);
    PTB_RUN(ptb_dequant_fp8_rowwise, q.const_data_ptr(), code_of(q.scalar_type()), B, q.size(axis), N,
            s.const_data_ptr<float>(), out.mutable_data_ptr(), code_of(dt), c.st);
    return out;
}

// The other-direction companion of a rowwise copy: the dequantised values (rounded to the operand's own type)
// quantised along `axis`.
Quant requant_rowwise(const Call &c, const Quant &r, ScalarType hp, int64_t have_axis, int64_t axis) {
    const int64_t nd = r.q.dim(), N = r.q.size(nd - 1);
    if (have_axis != nd - 1 || axis != nd - 2 || N == 1 || r.q.numel() == 0)
        return quant_rowwise(c, dequant_rowwise(c, r.q, r.s, hp, have_axis), r.q.scalar_type(), axis);
    const int64_t M = r.q.size(axis), B = r.q.numel() / (M * N);
    auto sshape  = r.q.sizes().vec();
    sshape[axis] = 1;
    Quant o{c.empty(r.q.sizes(), r.q.scalar_type()), c.empty(sshape, ScalarType::Float)};
    o.sm      = 1;
    Tensor ws = c.empty({B * N}, ScalarType::Float);
    PTB_RUN(ptb_requant_fp8_rowwise, r.q.const_data_ptr(), code_of(r.q.scalar_type()), r.scale(), code_of(hp), B, M, N,
            o.q.mutable_data_ptr(), o.s.mutable_data_ptr<float>(), ws.mutable_data_ptr(), c.st);
    return o;
}

Quant quant_block_rows(const Call &c, const Tensor &x, ScalarType dt) {
    const int64_t M = x.size(0), N = x.size(1), nb = cdiv(N, kBlk);
    Quant r{c.empty({M, N}, dt), c.empty({M, nb}, ScalarType::Float), nb, 1};
    PTB_RUN(ptb_quant_fp8_block1d, x.const_data_ptr(), code_of(x.scalar_type()), M, N, 1, r.q.mutable_data_ptr(), code_of(dt),
            r.s.mutable_data_ptr<float>(), c.st);
    return r;
}

Quant quant_block_cols(const Call &c, const Tensor &x, ScalarType dt) {
    const int64_t M = x.size(0), N = x.size(1);
    Quant r{c.empty({M, N}, dt), c.empty({cdiv(M, kBlk), N}, ScalarType::Float), 1, N};
    PTB_RUN(ptb_quant_fp8_block1d, x.const_data_ptr(), code_of(x.scalar_type()), M, N, 0, r.q.mutable_data_ptr(), code_of(dt),
            r.s.mutable_data_ptr<float>(), c.st);
    return r;
}

std::pair<Quant, Quant> quant_block_dual(const Call &c, const Tensor &x, ScalarType dt) {
    const int64_t M = x.size(0), N = x.size(1), nb = cdiv(N, kBlk);
    Quant row{c.empty({M, N}, dt), c.empty({M, nb}, ScalarType::Float), nb, 1};
    Quant col{c.empty({M, N}, dt), c.empty({cdiv(M, kBlk), N}, ScalarType::Float), 1, N};
    PTB_RUN(ptb_quant_fp8_block1d_dual, x.const_data_ptr(), code_of(x.scalar_type()), M, N, row.q.mutable_data_ptr(),
            row.s.mutable_data_ptr<float>(), col.q.mutable_data_ptr(), col.s.mutable_data_ptr<float>(), code_of(dt), c.st);
    return {row, col};
}

// 128x128 tiles of [M, N] or [G, M, N]
Quant quant_block_tiles(const Call &c, const Tensor &w, ScalarType dt) {
    const bool batched = w.dim() == 3;
    const int64_t B = batched ? w.size(0) : 1, M = w.size(-2), N = w.size(-1), mb = cdiv(M, kBlk), nb = cdiv(N, kBlk);
    Quant r{c.empty(w.sizes(), dt), batched ? c.empty({B, mb, nb}, ScalarType::Float) : c.empty({mb, nb}, ScalarType::Float),
            nb, 1, mb * nb};
    PTB_RUN(ptb_quant_fp8_block2d, w.const_data_ptr(), code_of(w.scalar_type()), B, M, N, r.q.mutable_data_ptr(), code_of(dt),
            r.s.mutable_data_ptr<float>(), c.st);
    return r;
}

// [M, N] or [G, M, N] -> {row copy, transposed column copy}; a direction that is not wanted stays undefined
std::pair<Quant, Quant> quant_mx(const Call &c, const Tensor &x, ScalarType dt, bool want_row, bool want_col, bool row_2d,
                                 bool col_2d) {
    const bool batched = x.dim() == 3;
    const int64_t G = batched ? x.size(0) : 1, M = x.size(-2), N = x.size(-1);
    const int64_t Mp = round_up(M, kBlk), Np = round_up(N, kBlk);
    auto make = [&](int64_t rows, int64_t cols, ScalarType t) {
        return batched ? c.empty({G, rows, cols}, t) : c.empty({rows, cols}, t);
    };
    Quant row, col;
    if (want_row) row = {make(M, Np, dt), make(M, Np / kMxBlk, ScalarType::Byte)};
    if (want_col) col = {make(N, Mp, dt), make(N, Mp / kMxBlk, ScalarType::Byte)};
    PTB_RUN(ptb_quant_mxfp8, x.const_data_ptr(), code_of(x.scalar_type()), G, M, N,
            want_row ? row.q.mutable_data_ptr() : nullptr, want_row ? row.s.mutable_data_ptr() : nullptr,
            want_col ? col.q.mutable_data_ptr() : nullptr, want_col ? col.s.mutable_data_ptr() : nullptr, row_2d, col_2d,
            code_of(dt), c.st);
    return {row, col};
}

// ---- dense GEMM -------------------------------------------------------------------------------------------------
// op(A) . op(B); trans_c gives the transposed product by exchanging the operands.
Tensor gemm(const Call &c, const Quant &a, bool ta, const Quant &b, bool tb, ScalarType out_dt, bool trans_c, int gran,
            bool b_tiles) {
    if (trans_c) return gemm(c, b, !tb, a, !ta, out_dt, false, gran, b_tiles);
    const int64_t M = a.q.size(ta ? 1 : 0), K = a.q.size(ta ? 0 : 1), N = b.q.size(tb ? 0 : 1);
    Tensor out = c.empty({M, N}, out_dt);
    int64_t asm_ = a.sm, ask = a.sk, bsn = b.sm, bsk = b.sk;
    if (gran == PTB_BLOCKWISE && b_tiles && !tb) std::swap(bsn, bsk); // tile scales are stored like the matrix: [K/128, N/128]
    PTB_RUN_GEMM(ptb_gemm_fp8, a.q.const_data_ptr(), code_of(a.q.scalar_type()), ta, a.q.size(1), b.q.const_data_ptr(),
                 code_of(b.q.scalar_type()), tb, b.q.size(1), out.mutable_data_ptr(), code_of(out_dt), N, M, N, K, gran,
                 a.scale(), asm_, ask, b.scale(), bsn, bsk, b_tiles, 0, c.st);
    return out;
}

Tensor gemm_mx(const Call &c, const Quant &a, const Quant &b, ScalarType out_dt) {
    const int64_t M = a.q.size(0), K = a.q.size(1), N = b.q.size(0);
    Tensor out = c.empty({M, N}, out_dt);
    PTB_RUN_GEMM(ptb_gemm_mxfp8, a.q.const_data_ptr(), code_of(a.q.scalar_type()), K, a.s.const_data_ptr(), a.s.size(1),
                 b.q.const_data_ptr(), code_of(b.q.scalar_type()), K, b.s.const_data_ptr(), b.s.size(1), out.mutable_data_ptr(),
                 code_of(out_dt), N, M, N, K, 0, c.st);
    return out;
}

struct DenseSpec {
    bool ta, tb;
    ScalarType out, fwd, bwd;
    int gran;
};

struct Saved { // what backward needs: the wgrad-direction copy of a and the dgrad-direction copy of b
    Quant a, b;
};

// `cached`: b arrives quantised (its scales in b_scale), in the forward direction only.
Tensor dense_forward(const Tensor &a_in, const Tensor &b_in, const Tensor *b_scale, const DenseSpec &d, bool need_a, bool need_b,
                     Saved *save) {
    Call c(a_in);
    const Tensor a = a_in.contiguous(), b = b_in.contiguous();
    Quant qb;
    if (b_scale) {
        qb = {b, b_scale->contiguous()};
        if (d.gran == PTB_ROWWISE) qb.sm = 1;
        if (d.gran == PTB_BLOCKWISE) { qb.sm = qb.s.size(1); qb.sk = 1; }
    }
    switch (d.gran) {
    case PTB_TENSORWISE: {
        const Quant qa = quant_tensorwise(c, a, d.fwd);
        if (!b_scale) qb = quant_tensorwise(c, b, d.fwd);
        if (need_b) save->a = qa;
        if (need_a) save->b = qb;
        return gemm(c, qa, d.ta, qb, d.tb, d.out, false, d.gran, false);
    }
    case PTB_ROWWISE: {
        const int64_t b_axis = d.tb ? 1 : 0;
        const Quant qa = quant_rowwise(c, a, d.fwd, 1);
        if (!b_scale) qb = quant_rowwise(c, b, d.fwd, b_axis);
        if (need_b) save->a = requant_rowwise(c, qa, a.scalar_type(), 1, 0);
        if (need_a) save->b = requant_rowwise(c, qb, b.scalar_type(), b_axis, 1 - b_axis);
        return gemm(c, qa, false, qb, d.tb, d.out, false, d.gran, false);
    }
    case PTB_BLOCKWISE: {
        Quant qa;
        if (need_b) std::tie(qa, save->a) = quant_block_dual(c, a, d.fwd);
        else qa = quant_block_rows(c, a, d.fwd);
        if (!b_scale) qb = quant_block_tiles(c, b, d.fwd);
        if (need_a) save->b = qb;
        return gemm(c, qa, false, qb, d.tb, d.out, false, d.gran, true);
    }
    default: {
        auto [a_row, a_col] = quant_mx(c, a, d.fwd, true, need_b, false, false);
        Quant b_col;
        if (!b_scale) std::tie(qb, b_col) = quant_mx(c, b, d.fwd, true, need_a, true, true);
        if (need_b) save->a = a_col;
        if (need_a) save->b = b_col;
        return gemm_mx(c, a_row, qb, d.out);
    }
    }
}

std::pair<Tensor, Tensor> dense_backward(const Tensor &grad, const Saved &s, const DenseSpec &d, bool need_a, bool need_b) {
    Call c(grad);
    const Tensor g = grad.contiguous();
    Tensor da, db;
    switch (d.gran) {
    case PTB_TENSORWISE: {
        const Quant qg = quant_tensorwise(c, g, d.bwd);
        if (need_a) da = gemm(c, qg, false, s.b, !d.tb, d.out, d.ta, d.gran, false);
        if (need_b) db = gemm(c, s.a, !d.ta, qg, false, d.out, d.tb, d.gran, false);
        break;
    }
    case PTB_ROWWISE:
        if (need_a) da = gemm(c, quant_rowwise(c, g, d.bwd, 1), false, s.b, !d.tb, d.out, false, d.gran, false);
        if (need_b) db = gemm(c, s.a, true, quant_rowwise(c, g, d.bwd, 0), false, d.out, d.tb, d.gran, false);
        break;
    case PTB_BLOCKWISE: {
        Quant g_row, g_col;
        if (need_a && need_b) std::tie(g_row, g_col) = quant_block_dual(c, g, d.bwd);
        else if (need_a) g_row = quant_block_rows(c, g, d.bwd);
        else if (need_b) g_col = quant_block_cols(c, g, d.bwd);
        if (need_a) da = gemm(c, g_row, false, s.b, !d.tb, d.out, false, d.gran, true);
        if (need_b) db = gemm(c, s.a, true, g_col, false, d.out, d.tb, d.gran, false);
        break;
    }
    default: {
        auto [g_row, g_col] = quant_mx(c, g, d.bwd, need_a, need_b, false, false);
        if (need_a) da = gemm_mx(c, g_row, s.b, d.out);
        if (need_b) db = gemm_mx(c, g_col, s.a, d.out);
    }
    }
    return {da, db};
}

// ---- grouped GEMM ------------------------------------------------------------------------------------------------
struct GroupedSpec {
    bool tb;
    ScalarType out, fwd, bwd;
    int gran, num_sms;
};

// Where each group's rows lie: unpadded offsets, and for the blockwise and MX wgrad the 128-row padded layout.
struct Layout {
    Tensor offs, padded, table;
};

Tensor group_offsets(const Call &c, const Tensor &lens) {
    Tensor offs = c.empty({lens.numel() + 1}, ScalarType::Long);
    PTB_RUN(ptb_group_offs, lens.const_data_ptr<int64_t>(), lens.numel(), offs.mutable_data_ptr<int64_t>(), c.st);
    return offs;
}

// row copy with transposed scales [N/128, M], segment-padded column copy
std::pair<Quant, Quant> quant_segments(const Call &c, const Tensor &x, ScalarType dt, const Tensor &lens, Layout &l) {
    const int64_t M = x.size(0), N = x.size(1), G = lens.numel(), Mp = M + G * kBlk;
    Quant row{c.empty({M, N}, dt), c.empty({cdiv(N, kBlk), M}, ScalarType::Float), 1, M};
    Quant col{c.empty({Mp, N}, dt), c.empty({cdiv(Mp, kBlk), N}, ScalarType::Float), 1, N};
    Tensor pads = c.empty({2 * G + 1}, ScalarType::Long);
    Tensor table = c.empty({cdiv(Mp, kBlk), 2}, ScalarType::Int);
    int64_t *p = pads.mutable_data_ptr<int64_t>();
    PTB_RUN(ptb_quant_fp8_segment_row_col, x.const_data_ptr(), code_of(x.scalar_type()), M, N, G,
            lens.const_data_ptr<int64_t>(), l.offs.const_data_ptr<int64_t>(), row.q.mutable_data_ptr(),
            col.q.mutable_data_ptr(), row.s.mutable_data_ptr<float>(), col.s.mutable_data_ptr<float>(), p + G + 1, p,
            table.mutable_data_ptr(), code_of(dt), c.st);
    l.padded = pads; // first G + 1 words: the padded offsets
    return {row, col};
}

std::pair<Quant, Quant> quant_mx_groups(const Call &c, const Tensor &x, ScalarType dt, int64_t G, Layout &l) {
    const int64_t M = x.size(0), N = x.size(1), Np = round_up(N, kBlk), Mc = round_up(M + G * kBlk, kBlk);
    Quant row{c.empty({M, Np}, dt), c.empty({M, Np / kMxBlk}, ScalarType::Byte)};
    Quant col{c.empty({N, Mc}, dt), c.empty({N, Mc / kMxBlk}, ScalarType::Byte)};
    Tensor pads = c.empty({4 * G + 2}, ScalarType::Long);
    Tensor table = c.empty({Mc / kBlk * 4}, ScalarType::Int);
    int64_t *p = pads.mutable_data_ptr<int64_t>(); // column offsets first: they are what wgrad reads
    PTB_RUN(ptb_quant_mxfp8_grouped, x.const_data_ptr(), code_of(x.scalar_type()), M, N, l.offs.const_data_ptr<int64_t>(), G, 1,
            row.q.mutable_data_ptr(), row.s.mutable_data_ptr(), col.q.mutable_data_ptr(), col.s.mutable_data_ptr(), p + G + 1,
            p + 2 * G + 1, p + 3 * G + 2, p, table.mutable_data_ptr(), 0, 0, code_of(dt), c.st);
    l.padded = pads;
    return {row, col};
}

Tensor grouped_gemm(const Call &c, const Quant &a, const Quant &b, bool tb, const Tensor &offs, const GroupedSpec &d) {
    const int64_t M = a.q.size(0), K = a.q.size(1), G = b.q.size(0), N = b.q.size(tb ? 1 : 2);
    Tensor out = c.empty({M, N}, d.out);
    int64_t bsg = b.sg, bsn = b.sm, bsk = b.sk;
    if (d.gran == PTB_BLOCKWISE && !tb) std::swap(bsn, bsk);
    if (d.gran == PTB_ROWWISE) bsg = N;
    PTB_RUN_GEMM(ptb_grouped_gemm_fp8, a.q.const_data_ptr(), code_of(a.q.scalar_type()), K, b.q.const_data_ptr(),
                 code_of(b.q.scalar_type()), tb, out.mutable_data_ptr(), code_of(d.out), N, offs.const_data_ptr<int64_t>(), G,
                 M, N, K, d.gran, a.scale(), a.sm, a.sk, b.scale(), bsg, bsn, bsk, d.num_sms, c.st);
    return out;
}

// out[g] = lhs_g^T . rhs_g
Tensor grouped_wgrad(const Call &c, const Quant &lhs, const Quant &rhs, const Tensor &offs, int64_t G, const GroupedSpec &d) {
    const int64_t rows = lhs.q.size(0), OM = lhs.q.size(1), ON = rhs.q.size(1);
    Tensor out = c.empty({G, OM, ON}, d.out);
    PTB_RUN_GEMM(ptb_grouped_gemm_fp8_variable_k, lhs.q.const_data_ptr(), code_of(lhs.q.scalar_type()), OM,
                 rhs.q.const_data_ptr(), code_of(rhs.q.scalar_type()), ON, out.mutable_data_ptr(), code_of(d.out),
                 offs.const_data_ptr<int64_t>(), G, rows, OM, ON, d.gran, lhs.scale(), rhs.scale(), d.num_sms, c.st);
    return out;
}

Tensor grouped_gemm_mx(const Call &c, const Quant &a, const Quant &b, const Tensor &offs, const GroupedSpec &d) {
    const int64_t M = a.q.size(0), K = a.q.size(1), G = b.q.size(0), N = b.q.size(1);
    Tensor out = c.empty({M, N}, d.out);
    PTB_RUN_GEMM(ptb_grouped_gemm_mxfp8, a.q.const_data_ptr(), code_of(a.q.scalar_type()), K, a.s.const_data_ptr(), a.s.size(1),
                 b.q.const_data_ptr(), code_of(b.q.scalar_type()), b.s.const_data_ptr(), out.mutable_data_ptr(), code_of(d.out),
                 N, offs.const_data_ptr<int64_t>(), G, M, N, K, d.num_sms, c.st);
    return out;
}

Tensor grouped_wgrad_mx(const Call &c, const Quant &lhs, const Quant &rhs, const Tensor &offs, int64_t G, const GroupedSpec &d) {
    const int64_t OM = lhs.q.size(0), ON = rhs.q.size(0), rows = lhs.q.size(1);
    Tensor out = c.empty({G, OM, ON}, d.out);
    PTB_RUN_GEMM(ptb_grouped_gemm_mxfp8_variable_k, lhs.q.const_data_ptr(), code_of(lhs.q.scalar_type()), rows,
                 lhs.s.const_data_ptr(), lhs.s.size(1), rhs.q.const_data_ptr(), code_of(rhs.q.scalar_type()), rows,
                 rhs.s.const_data_ptr(), rhs.s.size(1), out.mutable_data_ptr(), code_of(d.out), offs.const_data_ptr<int64_t>(),
                 G, rows, OM, ON, d.num_sms, c.st);
    return out;
}

Tensor grouped_forward(const Tensor &a_in, const Tensor &b_in, const Tensor *b_scale, const Tensor &lens, const Tensor *offs,
                       const GroupedSpec &d, bool need_a, bool need_b, Saved *save, Layout *l) {
    Call c(a_in);
    const Tensor a = a_in.contiguous(), b = b_in.contiguous();
    const int64_t G = b.size(0);
    l->offs = offs ? offs->contiguous() : group_offsets(c, lens);
    Quant qb;
    if (b_scale) {
        qb = {b, b_scale->contiguous()};
        if (d.gran == PTB_ROWWISE) qb.sm = 1;
        if (d.gran == PTB_BLOCKWISE) { qb.sm = qb.s.size(2); qb.sk = 1; qb.sg = qb.s.size(1) * qb.s.size(2); }
    }
    switch (d.gran) {
    case PTB_TENSORWISE: {
        const Quant qa = quant_tensorwise(c, a, d.fwd);
        if (!b_scale) qb = quant_tensorwise(c, b, d.fwd);
        if (need_b) save->a = qa;
        if (need_a) save->b = qb;
        return grouped_gemm(c, qa, qb, d.tb, l->offs, d);
    }
    case PTB_ROWWISE: {
        const int64_t b_axis = d.tb ? 2 : 1;
        const Quant qa = quant_rowwise(c, a, d.fwd, 1);
        if (!b_scale) qb = quant_rowwise(c, b, d.fwd, b_axis);
        if (need_b) save->a = requant_rowwise(c, qa, a.scalar_type(), 1, 0);
        if (need_a) save->b = requant_rowwise(c, qb, b.scalar_type(), b_axis, 3 - b_axis);
        return grouped_gemm(c, qa, qb, d.tb, l->offs, d);
    }
    case PTB_BLOCKWISE: {
        Quant qa;
        if (need_b) std::tie(qa, save->a) = quant_segments(c, a, d.fwd, lens, *l);
        else qa = quant_block_rows(c, a, d.fwd); // rows past the last group are quantised too and never read
        if (!b_scale) qb = quant_block_tiles(c, b, d.fwd);
        if (need_a) save->b = qb;
        return grouped_gemm(c, qa, qb, d.tb, l->offs, d);
    }
    default: {
        Quant qa, b_col;
        if (need_b) std::tie(qa, save->a) = quant_mx_groups(c, a, d.fwd, G, *l);
        else qa = quant_mx(c, a, d.fwd, true, false, false, false).first;
        if (!b_scale) std::tie(qb, b_col) = quant_mx(c, b, d.fwd, true, need_a, true, true);
        if (need_a) save->b = b_col;
        return grouped_gemm_mx(c, qa, qb, l->offs, d);
    }
    }
}

std::pair<Tensor, Tensor> grouped_backward(const Tensor &grad, const Tensor &lens, const Saved &s, Layout &l, const GroupedSpec &d,
                                           bool need_a, bool need_b) {
    Call c(grad);
    const Tensor g = grad.contiguous();
    const int64_t G = l.offs.numel() - 1;
    Tensor da, db;
    // grad_b has b's layout: [G, N, K] = g^T . a, or [G, K, N] = a^T . g
    auto wgrad = [&](const Quant &ga, const Tensor &offs) {
        return d.tb ? grouped_wgrad(c, ga, s.a, offs, G, d) : grouped_wgrad(c, s.a, ga, offs, G, d);
    };
    switch (d.gran) {
    case PTB_TENSORWISE: {
        const Quant qg = quant_tensorwise(c, g, d.bwd);
        if (need_a) da = grouped_gemm(c, qg, s.b, !d.tb, l.offs, d);
        if (need_b) db = wgrad(qg, l.offs);
        break;
    }
    case PTB_ROWWISE:
        if (need_a) da = grouped_gemm(c, quant_rowwise(c, g, d.bwd, 1), s.b, !d.tb, l.offs, d);
        if (need_b) db = wgrad(quant_rowwise(c, g, d.bwd, 0), l.offs);
        break;
    case PTB_BLOCKWISE: {
        Quant g_row, g_col;
        if (need_b) std::tie(g_row, g_col) = quant_segments(c, g, d.bwd, lens, l);
        else g_row = quant_block_rows(c, g, d.bwd);
        if (need_a) da = grouped_gemm(c, g_row, s.b, !d.tb, l.offs, d);
        if (need_b) db = wgrad(g_col, l.padded.narrow(0, 0, G + 1));
        break;
    }
    default: {
        Quant g_row, g_col;
        if (need_b) std::tie(g_row, g_col) = quant_mx_groups(c, g, d.bwd, G, l);
        else g_row = quant_mx(c, g, d.bwd, true, false, false, false).first;
        if (need_a) da = grouped_gemm_mx(c, g_row, s.b, l.offs, d);
        if (need_b) db = grouped_wgrad_mx(c, g_col, s.a, l.padded.narrow(0, 0, G + 1), G, d);
    }
    }
    return {da, db};
}

// ---- autograd nodes ------------------------------------------------------------------------------------------------
// A failure inside backward surfaces as the same Python class as one inside forward.
template <typename F> auto in_backward(F &&f) -> decltype(f()) {
    try {
        return f();
    } catch (const PtbFail &e) {
        pybind11::gil_scoped_acquire gil;
        PyErr_SetString(g_error_class, e.what());
        python_error err;
        err.persist();
        throw std::move(err);
    }
}

void put(AutogradContext *ctx, const char *key, int64_t v) { ctx->saved_data[key] = v; }
int64_t take(AutogradContext *ctx, const char *key) { return ctx->saved_data[key].toInt(); }

// The strides of a saved copy are functions of its shape, kind and direction; they travel as plain integers.
void put_quant(AutogradContext *ctx, const char *key, const Quant &q) {
    ctx->saved_data[key] = std::vector<int64_t>{q.sm, q.sk, q.sg};
}
Quant take_quant(AutogradContext *ctx, const char *key, const Tensor &q, const Tensor &s) {
    const auto v = ctx->saved_data[key].toIntVector();
    return {q, s, v[0], v[1], v[2]};
}

struct DenseFn : public torch::autograd::Function<DenseFn> {
    static Tensor forward(AutogradContext *ctx, const Tensor &a, const Tensor &b, bool need_a, bool need_b, const DenseSpec &d) {
        Saved s;
        Tensor out = dense_forward(a, b, nullptr, d, need_a, need_b, &s);
        ctx->save_for_backward({s.a.q, s.a.s, s.b.q, s.b.s});
        put_quant(ctx, "a", s.a);
        put_quant(ctx, "b", s.b);
        put(ctx, "spec", (int64_t) d.gran | (int64_t) d.ta << 8 | (int64_t) d.tb << 9);
        put(ctx, "out", (int64_t) d.out);
        put(ctx, "bwd", (int64_t) d.bwd);
        return out;
    }
    static variable_list backward(AutogradContext *ctx, const variable_list &grads) {
        return in_backward([&] {
            const auto sv = ctx->get_saved_variables();
            const int64_t spec = take(ctx, "spec");
            DenseSpec d{(bool) (spec >> 8 & 1), (bool) (spec >> 9 & 1), (ScalarType) take(ctx, "out"), ScalarType::Float8_e4m3fn,
                        (ScalarType) take(ctx, "bwd"), (int) (spec & 255)};
            const Saved s{take_quant(ctx, "a", sv[0], sv[1]), take_quant(ctx, "b", sv[2], sv[3])};
            auto [da, db] = dense_backward(grads[0], s, d, s.b.q.defined() && ctx->needs_input_grad(0),
                                           s.a.q.defined() && ctx->needs_input_grad(1));
            return variable_list{da, db, Tensor(), Tensor(), Tensor()};
        });
    }
};

struct GroupedFn : public torch::autograd::Function<GroupedFn> {
    static Tensor forward(AutogradContext *ctx, const Tensor &a, const Tensor &b, const Tensor &lens,
                          const std::optional<Tensor> &offs, bool need_a, bool need_b, const GroupedSpec &d) {
        Saved s;
        Layout l;
        Tensor out = grouped_forward(a, b, nullptr, lens, offs ? &*offs : nullptr, d, need_a, need_b, &s, &l);
        ctx->save_for_backward({s.a.q, s.a.s, s.b.q, s.b.s, lens, l.offs});
        put_quant(ctx, "a", s.a);
        put_quant(ctx, "b", s.b);
        put(ctx, "spec", (int64_t) d.gran | (int64_t) d.tb << 9 | (int64_t) d.num_sms << 16);
        put(ctx, "out", (int64_t) d.out);
        put(ctx, "bwd", (int64_t) d.bwd);
        return out;
    }
    static variable_list backward(AutogradContext *ctx, const variable_list &grads) {
        return in_backward([&] {
            const auto sv = ctx->get_saved_variables();
            const int64_t spec = take(ctx, "spec");
            GroupedSpec d{(bool) (spec >> 9 & 1), (ScalarType) take(ctx, "out"), ScalarType::Float8_e4m3fn, (ScalarType) take(ctx, "bwd"),
                          (int) (spec & 255), (int) (spec >> 16)};
            const Saved s{take_quant(ctx, "a", sv[0], sv[1]), take_quant(ctx, "b", sv[2], sv[3])};
            Layout l{sv[5]};
            auto [da, db] = grouped_backward(grads[0], sv[4], s, l, d, s.b.q.defined() && ctx->needs_input_grad(0),
                                             s.a.q.defined() && ctx->needs_input_grad(1));
            return variable_list{da, db, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
        });
    }
};

// ---- Python entries ------------------------------------------------------------------------------------------------
template <typename F> py::object guarded(F &&f) {
    try {
        return f();
    } catch (const PtbFail &e) {
        PyErr_SetString(g_error_class, e.what());
        throw py::error_already_set();
    }
}

// The ops have no forward-mode derivative.  A tangent needs neither grad mode nor requires_grad, so a call that brings one
// looks like inference: the Python form raises, here the tangent would be dropped.
bool has_tangent(const Tensor &t) { return t._fw_grad(/*level=*/0).defined(); }

// torch.jit.trace records the Python form as an op that runs again on new inputs; a call from here would leave nothing in the
// trace but its output, as a constant.
bool traced() { return at::tracer::impl::is_dispatch_enabled(); }

bool plain_cuda(const Tensor &t) { return t.device().is_cuda() && t.layout() == at::kStrided && t.numel() > 0; }

// The scales of a weight [.., rows, cols] quantised ahead of time: as the kernels read them, and as many.  Anything else -- another
// type, a reshaped payload with the scales of its former shape -- is for the Python form, which converts or refuses.
bool scales_fit(const Tensor &w, const Tensor &s, int gran, bool tb) {
    if (s.device() != w.device() || s.layout() != at::kStrided) return false;
    const int64_t nd = w.dim();
    if (gran == kMxGranularity) {
        if ((s.scalar_type() != ScalarType::Float8_e8m0fnu && s.scalar_type() != ScalarType::Byte) || s.dim() != nd) return false;
        return s.sizes().slice(0, nd - 1) == w.sizes().slice(0, nd - 1) && s.size(-1) * kMxBlk == w.size(-1);
    }
    if (s.scalar_type() != ScalarType::Float) return false;
    if (gran == PTB_TENSORWISE) return s.numel() == 1;
    if (gran == PTB_ROWWISE) return s.numel() == (nd == 3 ? w.size(0) : 1) * w.size(tb ? -2 : -1);
    return s.dim() == nd && (nd == 2 || s.size(0) == w.size(0)) && s.size(-2) == cdiv(w.size(-2), kBlk) && s.size(-1) == cdiv(w.size(-1), kBlk);
}

py::object py_gemm_fp8(const Tensor &a, const Tensor &b, const std::optional<Tensor> &b_scale, bool ta, bool tb, ScalarType out,
                       int gran, ScalarType fwd, ScalarType bwd) {
    if (traced() || has_tangent(a) || has_tangent(b)) return py::none();
    if (!plain_cuda(a) || !plain_cuda(b) || a.device() != b.device() || a.dim() != 2 || b.dim() != 2 || !is_hp(a.scalar_type()) ||
        !is_hp(out) || a.size(ta ? 0 : 1) != b.size(tb ? 1 : 0))
        return py::none();
    if (b_scale ? !is_fp8(b.scalar_type()) || !scales_fit(b, *b_scale, gran, tb) : !is_hp(b.scalar_type())) return py::none();
    if (gran != PTB_TENSORWISE && ta) return py::none();
    if (gran == kMxGranularity && (!tb || a.size(1) % kMxBlk || b.size(0) % kMxBlk || !is_16bit(a.scalar_type()) || !is_16bit(out) ||
                                   (!b_scale && !is_16bit(b.scalar_type()))))
        return py::none();
    const DenseSpec d{ta, tb, out, fwd, bwd, gran};
    return guarded([&]() -> py::object {
        const bool grad = at::GradMode::is_enabled() && (a.requires_grad() || b.requires_grad());
        if (!grad) {
            at::AutoDispatchBelowADInplaceOrView no_autograd;
            return py::cast(dense_forward(a, b, b_scale ? &*b_scale : nullptr, d, false, false, nullptr));
        }
        if (b_scale) return py::none();
        return py::cast(DenseFn::apply(a, b, a.requires_grad(), b.requires_grad(), d));
    });
}

py::object py_grouped_gemm_fp8(const Tensor &a, const Tensor &b, const std::optional<Tensor> &b_scale, const Tensor &lens,
                               const std::optional<Tensor> &offs, bool tb, ScalarType out, int gran, ScalarType fwd, ScalarType bwd,
                               int num_sms) {
    if (traced() || has_tangent(a) || has_tangent(b)) return py::none();
    if (!plain_cuda(a) || !plain_cuda(b) || !plain_cuda(lens) || a.device() != b.device() || a.device() != lens.device() ||
        a.dim() != 2 || b.dim() != 3 || !is_hp(a.scalar_type()) || !is_16bit(out) || a.size(1) != b.size(tb ? 2 : 1) ||
        lens.dim() != 1 || lens.scalar_type() != ScalarType::Long || lens.size(0) != b.size(0) || !lens.is_contiguous())
        return py::none();
    if (offs && (!plain_cuda(*offs) || offs->device() != a.device() || offs->scalar_type() != ScalarType::Long ||
                 offs->numel() != b.size(0) + 1))
        return py::none();
    if (b_scale ? !is_fp8(b.scalar_type()) || !scales_fit(b, *b_scale, gran, tb) : !is_hp(b.scalar_type())) return py::none();
    if (gran == kMxGranularity && (!tb || a.size(1) % kMxBlk || b.size(1) % kMxBlk || !is_16bit(a.scalar_type()) ||
                                   (!b_scale && !is_16bit(b.scalar_type()))))
        return py::none();
    const GroupedSpec d{tb, out, fwd, bwd, gran, num_sms};
    return guarded([&]() -> py::object {
        const bool grad = at::GradMode::is_enabled() && (a.requires_grad() || b.requires_grad());
        if (!grad) {
            at::AutoDispatchBelowADInplaceOrView no_autograd;
            Layout l;
            return py::cast(grouped_forward(a, b, b_scale ? &*b_scale : nullptr, lens, offs ? &*offs : nullptr, d, false, false,
                                            nullptr, &l));
        }
        if (b_scale) return py::none();
        return py::cast(GroupedFn::apply(a, b, lens, offs, a.requires_grad(), b.requires_grad(), d));
    });
}

bool quantisable(const Tensor &x) {
    return plain_cuda(x) && is_hp(x.scalar_type()) && x.is_contiguous() && !(at::GradMode::is_enabled() && x.requires_grad());
}

// kind: the granularity; BLOCKWISE with tiles = 128x128 scales.  -> (q, scale_inv)
py::object py_quantize(const Tensor &x, ScalarType dt, int gran, int64_t axis, bool tiles) {
    if (traced() || !quantisable(x) || !is_fp8(dt)) return py::none();
    const int64_t nd = x.dim();
    if (gran == PTB_ROWWISE && (nd == 0 || axis < 0 || axis >= nd)) return py::none();
    if (gran == PTB_BLOCKWISE && (tiles ? nd != 2 && nd != 3 : nd != 2 || axis < 0 || axis > 1)) return py::none();
    if (gran == kMxGranularity &&
        ((nd != 2 && nd != 3) || !is_16bit(x.scalar_type()) || x.size(-1) % kMxBlk || (axis != nd - 1 && axis != nd - 2)))
        return py::none();
    return guarded([&]() -> py::object {
        Call c(x);
        Quant r;
        switch (gran) {
        case PTB_TENSORWISE: r = quant_tensorwise(c, x, dt); break;
        case PTB_ROWWISE: r = quant_rowwise(c, x, dt, axis); break;
        case PTB_BLOCKWISE:
            r = tiles ? quant_block_tiles(c, x, dt) : axis == 1 ? quant_block_rows(c, x, dt) : quant_block_cols(c, x, dt);
            break;
        default: {
            const bool row = axis == nd - 1;
            auto both = quant_mx(c, x, dt, row, !row, tiles, tiles);
            r = row ? both.first : both.second;
            r.s = r.s.view(ScalarType::Float8_e8m0fnu);
        }
        }
        return py::make_tuple(r.q, r.s);
    });
}

// -> (row copy, row scales, column copy, column scales)
py::object py_quantize_dual(const Tensor &x, ScalarType dt, int gran, bool row_2d, bool col_2d) {
    if (traced() || !quantisable(x) || !is_fp8(dt)) return py::none();
    const int64_t nd = x.dim();
    if (gran == PTB_BLOCKWISE ? nd != 2 : (nd != 2 && nd != 3) || !is_16bit(x.scalar_type()) || x.size(-1) % kMxBlk) return py::none();
    return guarded([&]() -> py::object {
        Call c(x);
        auto [row, col] = gran == PTB_BLOCKWISE ? quant_block_dual(c, x, dt) : quant_mx(c, x, dt, true, true, row_2d, col_2d);
        if (gran != PTB_BLOCKWISE) {
            row.s = row.s.view(ScalarType::Float8_e8m0fnu);
            col.s = col.s.view(ScalarType::Float8_e8m0fnu);
        }
        return py::make_tuple(row.q, row.s, col.q, col.s);
    });
}

py::object py_dequantize(const Tensor &q, const Tensor &s, ScalarType out_dt, int gran, int64_t axis, bool tiles) {
    if (traced() || !plain_cuda(q) || !plain_cuda(s) || q.device() != s.device() || !is_fp8(q.scalar_type()) || !is_hp(out_dt) ||
        !q.is_contiguous() || !s.is_contiguous())
        return py::none();
    const int64_t nd = q.dim();
    const bool f32 = s.scalar_type() == ScalarType::Float;
    const bool e8m0 = s.scalar_type() == ScalarType::Float8_e8m0fnu || s.scalar_type() == ScalarType::Byte;
    if (gran == kMxGranularity ? nd != 2 || axis < 0 || axis > 1 || q.size(1) % kMxBlk || s.dim() != 2 || !e8m0 : !f32)
        return py::none();
    if (gran == PTB_ROWWISE && (nd == 0 || axis < 0 || axis >= nd)) return py::none();
    if (gran == PTB_BLOCKWISE && (tiles ? nd != 2 && nd != 3 : nd != 2 || axis < 0 || axis > 1)) return py::none();
    return guarded([&]() -> py::object {
        Call c(q);
        const int qc = code_of(q.scalar_type()), oc = code_of(out_dt);
        if (gran == PTB_ROWWISE) return py::cast(dequant_rowwise(c, q, s, out_dt, axis));
        const bool flip = gran == kMxGranularity && axis == 0; // the transposed copy comes back untransposed
        Tensor out = flip ? c.empty({q.size(1), q.size(0)}, out_dt) : c.empty(q.sizes(), out_dt);
        void *o = out.mutable_data_ptr();
        switch (gran) {
        case PTB_TENSORWISE:
            PTB_RUN(ptb_dequant_fp8_tensorwise, q.const_data_ptr(), qc, q.numel(), s.const_data_ptr<float>(), o, oc, c.st);
            break;
        case PTB_BLOCKWISE:
            if (tiles)
                PTB_RUN(ptb_dequant_fp8_block2d, q.const_data_ptr(), qc, nd == 3 ? q.size(0) : 1, q.size(-2), q.size(-1),
                        s.const_data_ptr<float>(), o, oc, c.st);
            else
                PTB_RUN(ptb_dequant_fp8_block1d, q.const_data_ptr(), qc, q.size(0), q.size(1), axis == 1,
                        s.const_data_ptr<float>(), o, oc, c.st);
            break;
        default:
            PTB_RUN(ptb_dequant_mxfp8, q.const_data_ptr(), qc, q.size(0), q.size(1), s.const_data_ptr(), flip, o, oc, c.st);
        }
        return py::cast(out);
    });
}

} // namespace

PYBIND11_MODULE(ptb_torch, m) {
    m.doc() = "native host path of the FP8 ops";
    m.def("setup", [](py::object error_class, py::object timed_region) {
        g_error_class  = error_class.release().ptr(); // both kept for the life of the process
        g_timed_region = timed_region.release().ptr();
    });
    m.def("set_check_status", [](bool on) { g_check_status = on; });
    m.def("set_recording", [](bool on) { g_recording = on; });
    m.def("calls", [] { return g_calls.load(std::memory_order_relaxed); });
    m.def("gemm_fp8", &py_gemm_fp8);
    m.def("grouped_gemm_fp8", &py_grouped_gemm_fp8);
    m.def("quantize", &py_quantize);
    m.def("quantize_dual", &py_quantize_dual);
    m.def("dequantize", &py_dequantize);
}
