// Python bindings of the native library (module soap_tp_b200._C).
//
// The reference exposes two pybind11 modules that take raw integer addresses plus leading dimensions
// and release the GIL (src/soap_tp/csrc/slate_bindings.cpp:317-389, elpa_bindings.cpp:200-236).  The
// same calling convention is used here: tensors are passed as data_ptr() integers with explicit
// pitches, the CUDA stream as its integer handle.  Nothing here allocates device memory.
#include <pybind11/pybind11.h>
#include <pybind11/stl.h>

#include <array>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "comm.h"
#include "elementwise.h"
#include "gemm.h"
#include "gemm_half.h"
#include "jacobi.h"
#include "qr.h"
#include "tridiag.h"

namespace py = pybind11;
using namespace soapb200;

namespace {
template <class T>
T* ptr(uint64_t address) {
  return reinterpret_cast<T*>(static_cast<uintptr_t>(address));
}
cudaStream_t stream_of(uint64_t handle) { return reinterpret_cast<cudaStream_t>(static_cast<uintptr_t>(handle)); }

// A flat list of integers (addresses, pitches, sizes) read in order: a call with one list costs the interpreter a third of one
// with as many arguments.
class Arguments {
 public:
  explicit Arguments(const std::vector<int64_t>& values) : values_(values) {}
  int64_t next() {
    if (at_ >= values_.size()) throw std::invalid_argument("too few integers for this call");
    return values_[at_++];
  }
  template <typename T>
  T* pointer() { return ptr<T>(static_cast<uint64_t>(next())); }
  cudaStream_t stream() { return stream_of(static_cast<uint64_t>(next())); }
  // scaled fp16 planes: h, l, pitch, scale, then scratch of the largest magnitudes or the stride of the scales
  HalfTarget target() {
    HalfTarget t{};
    t.h = pointer<uint16_t>(); t.l = pointer<uint16_t>(); t.ld = next(); t.scale = pointer<float>(); t.largest = pointer<uint32_t>();
    return t;
  }
  HalfOperand operand() {
    HalfOperand o{};
    o.h = pointer<uint16_t>(); o.l = pointer<uint16_t>(); o.ld = next(); o.scale = pointer<float>(); o.scale_stride = next();
    return o;
  }
  // the mixed form: tf32 values, pitch, interleaved bf16 plane, pitch
  SplitTarget mixed() {
    SplitTarget t{};
    t.hi = pointer<float>(); t.ldo = next(); t.hl = pointer<uint16_t>(); t.ld16 = next();
    return t;
  }
  bool done() const { return at_ == values_.size(); }
  void finish() const {
    if (!done()) throw std::invalid_argument("too many integers for this call");
  }

 private:
  const std::vector<int64_t>& values_;
  size_t at_ = 0;
};
}  // namespace

// The planes of a basis in both orientations (one of them may be absent), handed over once with the basis itself.
struct BasisOperands {
  HalfOperand plain{}, turned{};
  const float* src;
  int64_t s_i, s_j;
  CUtensorMap maps[2][2];

  BasisOperands(int size, const std::vector<int64_t>& values) {
    Arguments in(values);
    int i = 0;
    for (HalfOperand* o : {&plain, &turned}) {
      *o = in.operand();
      if (o->h && size > 0) {      // (nothing reads the planes of an empty basis, and there is no map of them)
        half_maps(maps[i], o->h, o->l, o->ld, size, size);
        o->maps = maps[i];
      }
      ++i;
    }
    src = in.pointer<float>(); s_i = in.next(); s_j = in.next();
    in.finish();
  }
  BasisOperands(const BasisOperands&) = delete;              // (the operands point into the object)
  BasisOperands& operator=(const BasisOperands&) = delete;
};

// The scratch of rotations of one shape, handed over once: planes, the decision on the range, and the mixed form of everything.
struct RotationScratch {
  Rotation rotation{};       // without the matrix and its bases
  HalfOperand update{};
  SplitTarget mixed_update{};
  CUtensorMap source_maps[2], middle_maps[2], update_maps[2], basis_maps[4][2];      // mixed; bases: left, its transpose, right, ...
  CUtensorMap x_maps[2], xt_maps[2], half_middle_maps[2], half_update_maps[2];       // fp16 pairs

  RotationScratch(int rows, int cols, const std::vector<int64_t>& values) {
    Arguments in(values);
    Rotation& r = rotation;
    r.rows = rows; r.cols = cols;
    r.x = in.target(); r.xt = in.target();
    half_maps(x_maps, r.x.h, r.x.l, r.x.ld, rows, cols);
    r.x_maps = x_maps;
    if (r.xt.h) {
      half_maps(xt_maps, r.xt.h, r.xt.l, r.xt.ld, cols, rows);
      r.xt_maps = xt_maps;
    }
    r.middle = in.operand();
    half_maps(half_middle_maps, r.middle.h, r.middle.l, r.middle.ld, cols, rows);
    r.middle.maps = half_middle_maps;
    r.guard.wide = in.pointer<int>(); r.guard.nearest = static_cast<int>(in.next());
    r.guard.mixed = in.mixed();
    r.mixed_middle = in.mixed();
    for (int side = 0; side < 2; ++side) {
      WideBasis& basis = r.guard.bases[side];
      basis.plain = in.mixed();
      basis.turned = in.mixed();
      basis.size = side ? cols : rows;
      mixed_maps(basis_maps[2 * side], basis.plain, basis.size, basis.size);
      mixed_maps(basis_maps[2 * side + 1], basis.turned, basis.size, basis.size);
    }
    mixed_maps(source_maps, r.guard.mixed, rows, cols);
    mixed_maps(middle_maps, r.mixed_middle, cols, rows);
    r.mixed_source = source_maps;
    r.middle.mixed = middle_maps;
    if (!in.done()) {
      update = in.operand();
      mixed_update = in.mixed();
      mixed_maps(update_maps, mixed_update, rows, cols);
      update.mixed = update_maps;
      half_maps(half_update_maps, update.h, update.l, update.ld, rows, cols);
      update.maps = half_update_maps;
    }
    in.finish();
  }
  RotationScratch(const RotationScratch&) = delete;          // (the operands point into the object)
  RotationScratch& operator=(const RotationScratch&) = delete;

  // The rotation of a matrix by its bases.
  Rotation of(Arguments& in, const BasisOperands& left, const BasisOperands& right) const {
    Rotation r = rotation;
    r.source = in.pointer<void>(); r.source_type = static_cast<int>(in.next()); r.s_i = in.next(); r.s_j = in.next();
    r.left = left.plain; r.left_turned = left.turned; r.right = right.plain; r.right_turned = right.turned;
    HalfOperand* const planes[] = {&r.left, &r.left_turned, &r.right, &r.right_turned};
    for (int i = 0; i < 4; ++i) planes[i]->mixed = basis_maps[i];
    for (int side = 0; side < 2; ++side) {
      const BasisOperands& from = side ? right : left;
      WideBasis& basis = r.guard.bases[side];
      basis.src = from.src; basis.s_i = from.s_i; basis.s_j = from.s_j;
    }
    return r;
  }
};

namespace {
// An ordinary step's operands, results and scalars (beta, beta1, beta2, eps, 1 / bias 1, 1 / sqrt(bias 2)).
SteadyStep step_of(const RotationScratch& scratch, const BasisOperands& left, const BasisOperands& right, Arguments& in,
                   const std::array<double, 6>& scalars) {
  SteadyStep s{};
  s.rotation = scratch.of(in, left, right);
  s.update = scratch.update;
  s.mixed_update = scratch.mixed_update;
  s.momentum = in.pointer<float>(); s.ldm = in.next();
  s.variance = in.pointer<float>(); s.ldv = in.next();
  s.out = in.pointer<float>();
  s.left_gram = in.pointer<float>(); s.ld_left = in.next();
  s.right_gram = in.pointer<float>(); s.ld_right = in.next();
  s.beta = scalars[0];
  s.beta1 = static_cast<float>(scalars[1]); s.beta2 = static_cast<float>(scalars[2]); s.eps = static_cast<float>(scalars[3]);
  s.inv_bc1 = static_cast<float>(scalars[4]); s.inv_sqrt_bc2 = static_cast<float>(scalars[5]);
  return s;
}
}  // namespace

PYBIND11_MODULE(_C, m) {
  m.doc() = "sm_100a kernels of soap_tp_b200";
  m.def("compiled_gpu_backend", [] { return "cuda"; });
  m.def("compiled_arch", [] { return "sm_100a"; });

  m.def(
      "gemm_tf32x3",
      [](uint64_t a_hi, uint64_t a_lo, int64_t lda, uint64_t b_hi, uint64_t b_lo, int64_t ldb, int M, int N, int K,
         int mode, int symmetric, int force_narrow, float alpha, float beta, uint64_t C, int64_t ldc, uint64_t Chi,
         uint64_t Clo, int64_t ldp, uint64_t mom, uint64_t var, int64_t ldm, int64_t ldv, float beta1, float beta2,
         float eps, float inv_bc1, float inv_sqrt_bc2, int k_splits, int64_t split_stride, uint64_t status,
         uint64_t stream, int batches, int a_k_step, int a_row_step, int b_k_step, int b_row_step,
         int64_t c_batch_stride, int64_t a_k_total, int64_t a_rows_total, int64_t b_k_total, int64_t b_rows_total,
         uint64_t remap, uint64_t C2hi, uint64_t C2lo, int64_t ld2, int m_limit, int o1_row_start, int tri_nb,
         int tri_pr, int tri_Pr, int tri_pc, int tri_Pc, int tri_m0, int tri_n0, uint64_t a_hl, int64_t lda16,
         uint64_t b_hl, int64_t ldb16, uint64_t Chl, int64_t ldp16, uint64_t push_table, int64_t push_ld,
         int64_t push_ld16, int push_nb, int push_Pr, int push_Pc, int push_pr, int push_pc, int push_mixed, int b_exact) {
        GemmOperands ops{};
        ops.a_hi = ptr<const float>(a_hi); ops.a_lo = ptr<const float>(a_lo); ops.lda = lda;
        ops.b_hi = ptr<const float>(b_hi); ops.b_lo = ptr<const float>(b_lo); ops.ldb = ldb;
        GemmProblem prob{};
        prob.M = M; prob.N = N; prob.K = K;
        prob.mode = mode; prob.symmetric = symmetric; prob.force_narrow = force_narrow; prob.b_exact = b_exact;
        prob.alpha = alpha; prob.beta = beta;
        prob.C = ptr<float>(C); prob.ldc = ldc;
        prob.Chi = ptr<float>(Chi); prob.Clo = ptr<float>(Clo); prob.ldp = ldp;
        prob.mom = ptr<float>(mom); prob.var = ptr<float>(var); prob.ldm = ldm; prob.ldv = ldv;
        prob.beta1 = beta1; prob.beta2 = beta2; prob.eps = eps;
        prob.inv_bc1 = inv_bc1; prob.inv_sqrt_bc2 = inv_sqrt_bc2;
        prob.k_splits = k_splits; prob.split_stride = split_stride;
        prob.batches = batches;
        prob.a_k_step = a_k_step; prob.a_row_step = a_row_step; prob.b_k_step = b_k_step; prob.b_row_step = b_row_step;
        prob.c_batch_stride = c_batch_stride;
        ops.a_k_total = a_k_total; ops.a_rows_total = a_rows_total; ops.b_k_total = b_k_total; ops.b_rows_total = b_rows_total;
        prob.remap = ptr<const int>(remap); prob.C2hi = ptr<float>(C2hi); prob.C2lo = ptr<float>(C2lo);
        prob.ld2 = ld2; prob.m_limit = m_limit; prob.o1_row_start = o1_row_start;
        prob.tri_nb = tri_nb > 0 ? tri_nb : 1; prob.tri_pr = tri_pr; prob.tri_Pr = tri_Pr > 0 ? tri_Pr : 1;
        prob.tri_pc = tri_pc; prob.tri_Pc = tri_Pc > 0 ? tri_Pc : 1; prob.tri_m0 = tri_m0; prob.tri_n0 = tri_n0;
        ops.a_hl = ptr<const uint16_t>(a_hl); ops.lda16 = lda16;
        ops.b_hl = ptr<const uint16_t>(b_hl); ops.ldb16 = ldb16;
        prob.Chl = ptr<uint16_t>(Chl); prob.ldp16 = ldp16;
        prob.push_table = ptr<const uint64_t>(push_table); prob.push_ld = push_ld; prob.push_ld16 = push_ld16;
        prob.push_nb = push_nb; prob.push_Pr = push_Pr; prob.push_Pc = push_Pc; prob.push_pr = push_pr;
        prob.push_pc = push_pc; prob.push_mixed = push_mixed;
        py::gil_scoped_release release;
        gemm_tf32x3(ops, prob, ptr<int>(status), stream_of(stream));
      },
      py::arg("a_hi"), py::arg("a_lo"), py::arg("lda"), py::arg("b_hi"), py::arg("b_lo"), py::arg("ldb"), py::arg("M"),
      py::arg("N"), py::arg("K"), py::arg("mode"), py::arg("symmetric"), py::arg("force_narrow"), py::arg("alpha"),
      py::arg("beta"), py::arg("C"), py::arg("ldc"), py::arg("Chi"), py::arg("Clo"), py::arg("ldp"), py::arg("mom"),
      py::arg("var"), py::arg("ldm"), py::arg("ldv"), py::arg("beta1"), py::arg("beta2"), py::arg("eps"),
      py::arg("inv_bc1"), py::arg("inv_sqrt_bc2"), py::arg("k_splits"), py::arg("split_stride"), py::arg("status"),
      py::arg("stream"), py::arg("batches") = 1, py::arg("a_k_step") = 0, py::arg("a_row_step") = 0,
      py::arg("b_k_step") = 0, py::arg("b_row_step") = 0, py::arg("c_batch_stride") = 0, py::arg("a_k_total") = 0,
      py::arg("a_rows_total") = 0, py::arg("b_k_total") = 0, py::arg("b_rows_total") = 0, py::arg("remap") = 0,
      py::arg("C2hi") = 0, py::arg("C2lo") = 0, py::arg("ld2") = 0, py::arg("m_limit") = 0, py::arg("o1_row_start") = 0, py::arg("tri_nb") = 1, py::arg("tri_pr") = 0,
      py::arg("tri_Pr") = 1, py::arg("tri_pc") = 0, py::arg("tri_Pc") = 1, py::arg("tri_m0") = 0, py::arg("tri_n0") = 0,
      py::arg("a_hl") = 0, py::arg("lda16") = 0, py::arg("b_hl") = 0, py::arg("ldb16") = 0, py::arg("Chl") = 0,
      py::arg("ldp16") = 0, py::arg("push_table") = 0, py::arg("push_ld") = 0, py::arg("push_ld16") = 0,
      py::arg("push_nb") = 1, py::arg("push_Pr") = 1, py::arg("push_Pc") = 1, py::arg("push_pr") = 0,
      py::arg("push_pc") = 0, py::arg("push_mixed") = 0, py::arg("b_exact") = 0,
      "3xTF32 tcgen05 GEMM acc[m,n] = sum_k Za[k,m] Zb[k,n] with fused epilogue");

  m.def("gemm_use_cta_pairs", [](bool on) { gemm_use_cta_pairs(on); },
        "Large plain GEMMs on CTA pairs (cta_group::2, default) or on single CTAs");

  m.def("gemm_half",
        [](uint64_t a_h, uint64_t a_l, int64_t lda, uint64_t a_scale, int64_t a_stride, uint64_t b_h, uint64_t b_l, int64_t ldb,
           uint64_t b_scale, int64_t b_stride, int M, int N, int K, int mode, int symmetric, int tiles, float alpha, float beta,
           uint64_t C, int64_t ldc, uint64_t Ch, uint64_t Cl, int64_t ldp, uint64_t Cscale, int64_t ldscale, uint64_t mom,
           int64_t ldm, uint64_t var, int64_t ldv, float beta1, float beta2, float eps, float inv_bc1, float inv_sqrt_bc2,
           uint64_t status, uint64_t stream) {
          const HalfOperand a{ptr<const uint16_t>(a_h), ptr<const uint16_t>(a_l), lda, ptr<const float>(a_scale), a_stride};
          const HalfOperand b{ptr<const uint16_t>(b_h), ptr<const uint16_t>(b_l), ldb, ptr<const float>(b_scale), b_stride};
          HalfProblem p{};
          p.M = M; p.N = N; p.K = K; p.mode = mode; p.symmetric = symmetric; p.tiles = tiles;
          p.alpha = alpha; p.beta = beta; p.C = ptr<float>(C); p.ldc = ldc;
          p.Ch = ptr<uint16_t>(Ch); p.Cl = ptr<uint16_t>(Cl); p.ldp = ldp; p.Cscale = ptr<float>(Cscale); p.ldscale = ldscale;
          p.mom = ptr<float>(mom); p.ldm = ldm; p.var = ptr<float>(var); p.ldv = ldv;
          p.beta1 = beta1; p.beta2 = beta2; p.eps = eps; p.inv_bc1 = inv_bc1; p.inv_sqrt_bc2 = inv_sqrt_bc2;
          gemm_half(a, b, p, ptr<int>(status), stream_of(stream));
        },
        "acc[m,n] = sum_k Za[k,m] Zb[k,n] from scaled fp16 planes, with fused epilogue (gemm_half.h)");

  m.def("half_on_pairs", &half_on_pairs, "Whether an M x N product of fp16 pairs runs on CTA pairs by default");

  m.def("half_planes",
        [](uint64_t src, int source_type, int64_t s_i, int64_t s_j, int rows, int cols, uint64_t ph, uint64_t pl, int64_t pld,
           uint64_t pscale, uint64_t plargest, uint64_t th, uint64_t tl, int64_t tld, uint64_t tscale, uint64_t tlargest,
           uint64_t stream) {
          half_planes(ptr<const void>(src), source_type, s_i, s_j, rows, cols,
                      HalfTarget{ptr<uint16_t>(ph), ptr<uint16_t>(pl), pld, ptr<float>(pscale), ptr<uint32_t>(plargest)},
                      HalfTarget{ptr<uint16_t>(th), ptr<uint16_t>(tl), tld, ptr<float>(tscale), ptr<uint32_t>(tlargest)},
                      RangeGuard{}, stream_of(stream));
        },
        "Scaled fp16 operand planes of a matrix in one or both orientations (gemm_half.h)");

  py::class_<RotationScratch>(m, "RotationScratch", "Scratch planes of rotations of one shape, as addresses (see Arguments)")
      .def(py::init<int, int, const std::vector<int64_t>&>());
  py::class_<BasisOperands>(m, "BasisOperands", "Planes of a basis in both orientations, and the basis, as addresses")
      .def(py::init<int, const std::vector<int64_t>&>());
  // A plain product of classic planes.  Integers: hi, lo, pitch of both operands; M, N, K, mode, symmetric, force_narrow; result, its
  // pitch; hi, lo, pitch of the result's planes; splits and the distance of their results; the status word and the stream.
  m.def("gemm_planes", [](const std::vector<int64_t>& v, float alpha, float beta) {
    Arguments in(v);
    GemmOperands ops{};
    ops.a_hi = in.pointer<const float>(); ops.a_lo = in.pointer<const float>(); ops.lda = in.next();
    ops.b_hi = in.pointer<const float>(); ops.b_lo = in.pointer<const float>(); ops.ldb = in.next();
    GemmProblem prob{};
    prob.M = static_cast<int>(in.next()); prob.N = static_cast<int>(in.next()); prob.K = static_cast<int>(in.next());
    prob.mode = static_cast<int>(in.next()); prob.symmetric = static_cast<int>(in.next()); prob.force_narrow = static_cast<int>(in.next());
    prob.C = in.pointer<float>(); prob.ldc = in.next();
    prob.Chi = in.pointer<float>(); prob.Clo = in.pointer<float>(); prob.ldp = in.next();
    prob.k_splits = static_cast<int>(in.next()); prob.split_stride = in.next();
    prob.alpha = alpha; prob.beta = beta;
    int* status = in.pointer<int>();
    cudaStream_t stream = in.stream();
    in.finish();
    py::gil_scoped_release release;
    gemm_tf32x3(ops, prob, status, stream);
  });

  // Integers: the matrix (RotationScratch::of), the moments and results in the order of SteadyStep; then of the call: the phases, the
  // status word, the stream and the stream of the averages.
  m.def("steady_step", [](const RotationScratch& scratch, const BasisOperands& left, const BasisOperands& right,
                          const std::vector<int64_t>& v, const std::array<double, 6>& scalars, int phases, uint64_t status, uint64_t stream,
                          uint64_t side) {
    Arguments in(v);
    SteadyStep s = step_of(scratch, left, right, in, scalars);
    in.finish();
    s.phases = phases;
    s.side = stream_of(side);
    py::gil_scoped_release release;
    steady_step(s, ptr<int>(status), stream_of(stream));
  }, "The launches of one ordinary single-GPU step, or some of its phases (gemm_half.h, SteadyStep)");
  m.def("steady_step_shares", &steady_step_shares, "Whether steps of such matrices can share launches");
  m.def("averages_share", &averages_share, "Whether both averages of a step run in one launch");
  m.attr("STEP_GROUP") = kHalfGroup;
  m.def("steady_steps", [](const std::vector<std::tuple<const RotationScratch*, const BasisOperands*, const BasisOperands*,
                                                        std::vector<int64_t>, std::array<double, 6>>>& steps,
                           uint64_t status, uint64_t stream, uint64_t side) {
    std::vector<SteadyStep> all;
    for (const auto& [scratch, left, right, v, scalars] : steps) {
      if (!scratch || !left || !right) throw std::invalid_argument("steady_steps: no scratch or bases");
      Arguments in(v);
      all.push_back(step_of(*scratch, *left, *right, in, scalars));
      in.finish();
      all.back().phases = kStepPlanes | kStepForward | kStepBackward | kStepAverages;
      all.back().side = stream_of(side);
    }
    py::gil_scoped_release release;
    steady_steps(all.data(), static_cast<int>(all.size()), ptr<int>(status), stream_of(stream));
  }, "Ordinary steps of several small parameters in shared launches");
  m.attr("STEP_PLANES") = kStepPlanes;
  m.attr("STEP_FORWARD") = kStepForward;
  m.attr("STEP_BACKWARD") = kStepBackward;
  m.attr("STEP_AVERAGES") = kStepAverages;
  // Integers: the matrix, then direction, result, its pitch, the status word and the stream.
  m.def("rotate_half", [](const RotationScratch& scratch, const BasisOperands& left, const BasisOperands& right, const std::vector<int64_t>& v) {
    Arguments in(v);
    const Rotation r = scratch.of(in, left, right);
    const bool turned = in.next() != 0;
    float* out = in.pointer<float>();
    const int64_t ldc = in.next();
    int* status = in.pointer<int>();
    cudaStream_t stream = in.stream();
    in.finish();
    py::gil_scoped_release release;
    rotate_half(r, turned, out, ldc, status, stream);
  }, "A matrix rotated by two bases on scaled fp16 planes, or on their mixed form where its range asks for it (gemm_half.h)");

  m.def("read_status", [](uint64_t word, uint64_t pinned, uint64_t stream) {
    const cudaError_t err = cudaMemcpyAsync(ptr<void>(pinned), ptr<const void>(word), sizeof(int), cudaMemcpyDeviceToHost, stream_of(stream));
    if (err != cudaSuccess) throw std::runtime_error(std::string("read_status: ") + cudaGetErrorString(err));
  }, "Copies a device's status word into pinned host memory");

  m.def("gemm_simt",
        [](uint64_t A, int64_t a_sk, int64_t a_sm, uint64_t B, int64_t b_sk, int64_t b_sn, uint64_t C, int64_t c_sm,
           int64_t c_sn, int M, int N, int K, float alpha, float beta, uint64_t stream) {
          py::gil_scoped_release release;
          gemm_simt(ptr<const float>(A), a_sk, a_sm, ptr<const float>(B), b_sk, b_sn, ptr<float>(C), c_sm, c_sn, M, N,
                    K, alpha, beta, stream_of(stream));
        });

  m.def("adam_update",
        [](uint64_t g, int64_t ldg, uint64_t mo, int64_t ldm, uint64_t v, int64_t ldv, uint64_t u, int64_t ldu, int rows,
           int cols, float beta1, float beta2, float eps, float inv_bc1, float inv_sqrt_bc2, uint64_t stream) {
          adam_update(ptr<const float>(g), ldg, ptr<float>(mo), ldm, ptr<float>(v), ldv, ptr<float>(u), ldu, rows, cols,
                      beta1, beta2, eps, inv_bc1, inv_sqrt_bc2, stream_of(stream));
        });

  // One orientation of an fp32 matrix: (i, j) of the operand at src[i * s_i + j * s_j].
  m.def("split_planes",
        [](uint64_t src, int64_t s_i, int64_t s_j, uint64_t hi, uint64_t lo, int64_t ldo, int rows, int cols,
           float scale, int nearest, uint64_t stream, uint64_t hl, int64_t ld16) {
          split_planes(ptr<const void>(src), 0, s_i, s_j, rows, cols,
                       SplitTarget{ptr<float>(hi), ptr<float>(lo), ldo, ptr<uint16_t>(hl), ld16}, SplitTarget{}, scale, nearest,
                       stream_of(stream));
        },
        py::arg("src"), py::arg("s_i"), py::arg("s_j"), py::arg("hi"), py::arg("lo"), py::arg("ldo"), py::arg("rows"),
        py::arg("cols"), py::arg("scale"), py::arg("nearest"), py::arg("stream"), py::arg("hl") = 0, py::arg("ld16") = 0);
  // One or both orientations (hi, lo, pitch, interleaved plane, its pitch each) of an fp32 or bf16 matrix.
  m.def("split_planes_both",
        [](uint64_t src, int source_type, int64_t s_i, int64_t s_j, int rows, int cols, uint64_t phi, uint64_t plo, int64_t pld,
           uint64_t phl, int64_t pld16, uint64_t thi, uint64_t tlo, int64_t tld, uint64_t thl, int64_t tld16, int nearest,
           uint64_t stream) {
          split_planes(ptr<const void>(src), source_type, s_i, s_j, rows, cols,
                       SplitTarget{ptr<float>(phi), ptr<float>(plo), pld, ptr<uint16_t>(phl), pld16},
                       SplitTarget{ptr<float>(thi), ptr<float>(tlo), tld, ptr<uint16_t>(thl), tld16}, 1.0f, nearest,
                       stream_of(stream));
        });

  // (parameter, update, elements) each
  m.def("apply_updates", [](const std::vector<std::tuple<uint64_t, uint64_t, int64_t>>& all, int type, float keep, float lr, uint64_t stream) {
    std::vector<UpdateJob> jobs;
    for (const auto& [p, update, n] : all) jobs.push_back(UpdateJob{ptr<void>(p), ptr<const float>(update), n});
    return apply_updates(jobs.data(), static_cast<int>(jobs.size()), type, keep, lr, stream_of(stream));
  }, "Returns the launches that it took");
  m.def("adamw_update", [](uint64_t p, int type, uint64_t gradient, uint64_t mo, uint64_t v, int64_t n, float beta1_rest,
                           float beta2, float beta2_rest, float bias1, float bias2, float eps, float keep, float lr,
                           uint64_t stream) {
    adamw_update(ptr<void>(p), type, ptr<const void>(gradient), ptr<float>(mo), ptr<float>(v), n, beta1_rest, beta2, beta2_rest,
                 bias1, bias2, eps, keep, lr, stream_of(stream));
  });

  m.def("column_dot",
        [](uint64_t a, int64_t lda, uint64_t b, int64_t ldb, uint64_t out, int rows, int cols, uint64_t stream) {
          column_dot(ptr<const float>(a), lda, ptr<const float>(b), ldb, ptr<float>(out), rows, cols, stream_of(stream));
        });

  m.def("order_by_estimate", [](uint64_t table, int64_t ld, int parts, int n, uint64_t order, uint64_t stream) {
    order_by_estimate(ptr<const float>(table), ld, parts, n, ptr<int64_t>(order), stream_of(stream));
  });
  m.attr("ORDER_MAX_LENGTH") = kOrderMaxLength;

  m.def("gather2d",
        [](uint64_t src, int64_t s_i, int64_t s_j, uint64_t dst, int64_t d_i, int64_t d_j, uint64_t row_map,
           uint64_t col_map, int rows, int cols, uint64_t stream) {
          gather2d(ptr<const float>(src), s_i, s_j, ptr<float>(dst), d_i, d_j, ptr<const int64_t>(row_map),
                   ptr<const int64_t>(col_map), rows, cols, stream_of(stream));
        });

  m.def("jacobi_small",
        [](uint64_t s_hi, uint64_t s_lo, int64_t lds, int batches, uint64_t u_hi, uint64_t u_lo, int64_t ldu,
           uint64_t offdiag, float scale, int max_sweeps, float tolerance, uint64_t stream) {
          jacobi_small(ptr<const float>(s_hi), ptr<const float>(s_lo), lds, batches, ptr<float>(u_hi), ptr<float>(u_lo), ldu,
                       ptr<float>(offdiag), scale, max_sweeps, tolerance, stream_of(stream));
        });
  m.def("qr_panel",
        [](uint64_t p_hi, uint64_t p_lo, int64_t ldp, int r, int b, uint64_t v_hi, uint64_t v_lo, int64_t ldv,
           uint64_t vt_hi, uint64_t vt_lo, int64_t ldvt, uint64_t tau, uint64_t t_hi, uint64_t t_lo, uint64_t tt_hi,
           uint64_t tt_lo, int64_t ldt, uint64_t exchange, uint64_t status, uint64_t stream, uint64_t trace, int debug_skip) {
          qr_panel(ptr<const float>(p_hi), ptr<const float>(p_lo), ldp, r, b, ptr<float>(v_hi), ptr<float>(v_lo), ldv,
                   ptr<float>(vt_hi), ptr<float>(vt_lo), ldvt, ptr<float>(tau), ptr<float>(t_hi), ptr<float>(t_lo),
                   ptr<float>(tt_hi), ptr<float>(tt_lo), ldt, ptr<float>(exchange), ptr<int>(status), stream_of(stream),
                   ptr<long long>(trace), debug_skip);
        },
        py::arg("p_hi"), py::arg("p_lo"), py::arg("ldp"), py::arg("r"), py::arg("b"), py::arg("v_hi"), py::arg("v_lo"),
        py::arg("ldv"), py::arg("vt_hi"), py::arg("vt_lo"), py::arg("ldvt"), py::arg("tau"), py::arg("t_hi"),
        py::arg("t_lo"), py::arg("tt_hi"), py::arg("tt_lo"), py::arg("ldt"), py::arg("exchange"), py::arg("status"),
        py::arg("stream"), py::arg("trace") = 0, py::arg("debug_skip") = 0);
  m.def("qr_panel_pairs",
        [](uint64_t p_hi, uint64_t p_lo, int64_t ldp, int r, int b, uint64_t v_hi, uint64_t v_lo, int64_t ldv,
           uint64_t vt_hi, uint64_t vt_lo, int64_t ldvt, uint64_t tau, uint64_t t_hi, uint64_t t_lo, uint64_t tt_hi,
           uint64_t tt_lo, int64_t ldt, uint64_t exchange, uint64_t status, uint64_t stream, int rows_per_cta,
           uint64_t steps_taken) {
          qr_panel_pairs(ptr<const float>(p_hi), ptr<const float>(p_lo), ldp, r, b, ptr<float>(v_hi), ptr<float>(v_lo),
                         ldv, ptr<float>(vt_hi), ptr<float>(vt_lo), ldvt, ptr<float>(tau), ptr<float>(t_hi),
                         ptr<float>(t_lo), ptr<float>(tt_hi), ptr<float>(tt_lo), ldt, ptr<float>(exchange),
                         ptr<int>(status), stream_of(stream), rows_per_cta, ptr<long long>(steps_taken));
        },
        py::arg("p_hi"), py::arg("p_lo"), py::arg("ldp"), py::arg("r"), py::arg("b"), py::arg("v_hi"), py::arg("v_lo"),
        py::arg("ldv"), py::arg("vt_hi"), py::arg("vt_lo"), py::arg("ldvt"), py::arg("tau"), py::arg("t_hi"),
        py::arg("t_lo"), py::arg("tt_hi"), py::arg("tt_lo"), py::arg("ldt"), py::arg("exchange"), py::arg("status"),
        py::arg("stream"), py::arg("rows_per_cta") = 256, py::arg("steps_taken") = 0);
  m.def("sum_partials_to_planes",
        [](uint64_t partials, int splits, int64_t stride, int64_t ld, uint64_t hi, uint64_t lo, int64_t ldp, int rows,
           int cols, uint64_t stream) {
          sum_partials_to_planes(ptr<const float>(partials), splits, stride, ld, ptr<float>(hi), ptr<float>(lo), ldp, rows,
                                 cols, stream_of(stream));
        });
  m.def("identity_planes", [](uint64_t hi, uint64_t lo, int64_t ldp, int rows, int cols, uint64_t stream, int first_col) {
    identity_planes(ptr<float>(hi), ptr<float>(lo), ldp, rows, cols, stream_of(stream), first_col);
  }, py::arg("hi"), py::arg("lo"), py::arg("ldp"), py::arg("rows"), py::arg("cols"), py::arg("stream"), py::arg("first_col") = 0);
  m.def("planes_sum", [](uint64_t hi, uint64_t lo, int64_t ldp, uint64_t out, int64_t ldo, int depth, int cols, uint64_t stream) {
    planes_sum(ptr<const float>(hi), ptr<const float>(lo), ldp, ptr<float>(out), ldo, depth, cols, stream_of(stream));
  });
  m.def("sytrd_panel",
        [](uint64_t A, int64_t lda, int n, int j0, int nb, uint64_t vw, uint64_t x, uint64_t y, uint64_t partial, uint64_t d,
           uint64_t e, uint64_t tau, uint64_t za_hi, uint64_t za_lo, uint64_t zb_hi, uint64_t zb_lo, uint64_t v_hi,
           uint64_t v_lo, int64_t ldv, uint64_t vt_hi, uint64_t vt_lo, int64_t ldvt, uint64_t t_hi, uint64_t t_lo,
           uint64_t tt_hi, uint64_t tt_lo, int64_t ldt, uint64_t barrier, uint64_t status, int last, uint64_t stream) {
          SytrdPanelArgs args{ptr<float>(A), lda, n, j0, nb, ptr<float>(vw), ptr<float>(x), ptr<float>(y), ptr<float>(partial),
                              ptr<double>(d), ptr<double>(e), ptr<float>(tau), ptr<float>(za_hi), ptr<float>(za_lo),
                              ptr<float>(zb_hi), ptr<float>(zb_lo), ptr<float>(v_hi), ptr<float>(v_lo), ldv, ptr<float>(vt_hi),
                              ptr<float>(vt_lo), ldvt, ptr<float>(t_hi), ptr<float>(t_lo), ptr<float>(tt_hi), ptr<float>(tt_lo),
                              ldt, ptr<unsigned int>(barrier), ptr<int>(status), last};
          sytrd_panel(args, stream_of(stream));
        });
  m.def("tridiagonal_bisect", [](uint64_t d, uint64_t e, int n, double lo, double hi, double pivmin, uint64_t lambda, uint64_t stream) {
    tridiagonal_bisect(ptr<const double>(d), ptr<const double>(e), n, lo, hi, pivmin, ptr<double>(lambda), stream_of(stream));
  });
  m.def("tridiagonal_vectors", [](uint64_t d, uint64_t e, int n, uint64_t lambda, double pivmin, uint64_t lplus, uint64_t dplus,
                                  uint64_t uminus, uint64_t z, uint64_t stream) {
    tridiagonal_vectors(ptr<const double>(d), ptr<const double>(e), n, ptr<const double>(lambda), pivmin, ptr<double>(lplus),
                        ptr<double>(dplus), ptr<double>(uminus), ptr<float>(z), stream_of(stream));
  });
  m.attr("TRIDIAG_PANEL") = kTridiagPanel;
  m.attr("QR_PANEL_WIDTH") = kQrPanelWidth;
  m.attr("QR_ROWS_PER_CTA") = kQrRowsPerCta;
  m.attr("QR_MAX_ROWS") = kQrMaxRows;

  register_comm(m);
}
