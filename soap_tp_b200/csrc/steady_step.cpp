// Rotations and ordinary optimizer steps on one GPU as single native calls: engine/local.py's pipeline.
// A step of a small matrix is bound by the host; with each launch a call of its own from the interpreter a 256 x 512 step took
// 182 us, issued from here 118 us.
//
// The four products of the rotation chain depend on one another and each ends in a wave of tiles that leaves SMs idle; the
// Gram averages depend on the gradient only.  So the averages run on a stream beside it and fill what the chain leaves free.
// The chain stays on the caller's stream: its first product then overlaps the tail of the operand planes, which an event
// between streams does not allow.  Device time of a step, everything on one stream / the chain beside / the averages beside:
// 256 x 512 126 / 92 / 85 us, 512 x 1376 175 / 158 / 121 us, 1000 x 1501 198 / 198 / 148 us, 2048 x 5504 1388 / 1352 / 1186 us,
// 4096 x 4096 1900 / 1863 / 1748 us, 8192 x 8192 within the runs' spread.
#include <optional>
#include <stdexcept>

#include "gemm.h"
#include "gemm_half.h"
#include "launch_util.h"

namespace soapb200 {

namespace {
HalfOperand operand(const HalfTarget& t) { return HalfOperand{t.h, t.l, t.ld, t.scale, 0}; }

// A second stream that is forked from `home` and joined to it again when the scope ends, by whatever way.
class Fork {
 public:
  Fork(cudaStream_t home, cudaStream_t side) : home_(home), side_(side) {
    event_.record(home);
    event_.hold(side);
  }
  ~Fork() {
    try {
      event_.record(side_);
      event_.hold(home_);
    } catch (const std::exception&) {      // the error of the step itself is the one to report
    }
  }
  Fork(const Fork&) = delete;
  Fork& operator=(const Fork&) = delete;

 private:
  ScopedEvent event_;
  const cudaStream_t home_, side_;
};
}  // namespace

namespace {
// T = X^T Q (cols x rows), or U^T Q (the same shape): the first product of a rotation.
void first_product(const Rotation& r, const HalfOperand& source, bool settled, const HalfOperand& basis, int* status,
                   cudaStream_t stream) {
  HalfProblem p{};
  p.M = r.cols; p.N = r.rows; p.K = r.rows;
  p.mode = kEpiSplit;
  p.alpha = 1.0f;
  p.Ch = const_cast<uint16_t*>(r.middle.h); p.Cl = const_cast<uint16_t*>(r.middle.l); p.ldp = r.middle.ld;
  p.Cscale = const_cast<float*>(r.middle.scale); p.ldscale = r.middle.scale_stride;
  p.wide = r.guard.wide; p.settled = settled; p.mixed = r.mixed_middle;
  gemm_half(source, basis, p, status, stream);
}

HalfOperand source_of(const Rotation& r) {
  HalfOperand x = operand(r.x);
  x.mixed = r.mixed_source;
  return x;
}

HalfProblem second_product(const Rotation& r) {
  HalfProblem p{};
  p.M = r.rows; p.N = r.cols; p.K = r.cols;
  p.alpha = 1.0f;
  p.wide = r.guard.wide; p.settled = 1;      // (the planes were made two kernels ago)
  return p;
}

void make_planes(const Rotation& r, cudaStream_t stream) {
  half_planes(r.source, r.source_type, r.s_i, r.s_j, r.rows, r.cols, r.x, r.xt, r.guard, stream);
}
}  // namespace

void rotate_half(const Rotation& r, bool turned, float* out, int64_t ldc, int* status, cudaStream_t stream) {
  if (r.rows <= 0 || r.cols <= 0) return;
  make_planes(r, stream);
  first_product(r, source_of(r), false, turned ? r.left_turned : r.left, status, stream);
  HalfProblem store = second_product(r);
  store.mode = kEpiStore;
  store.C = out; store.ldc = ldc;
  gemm_half(r.middle, turned ? r.right_turned : r.right, store, status, stream);
}

void steady_step(const SteadyStep& s, int* status, cudaStream_t stream) {
  const Rotation& r = s.rotation;
  if (r.rows <= 0 || r.cols <= 0) throw std::invalid_argument("steady_step: empty matrix");
  if (s.phases & kStepPlanes) make_planes(r, stream);
  const bool averages = s.phases & kStepAverages, rotations = s.phases & (kStepForward | kStepBackward);
  const cudaStream_t side = averages && rotations ? s.side : stream;
  std::optional<Fork> fork;
  if (side != stream) fork.emplace(stream, side);

  if (s.phases & kStepForward) {
    first_product(r, source_of(r), false, r.left, status, stream);          // T = X^T Q_L
    HalfProblem adam = second_product(r);                                   // Y = T^T Q_R, Adam(Y) -> U
    adam.mode = kEpiAdam;
    adam.Ch = const_cast<uint16_t*>(s.update.h); adam.Cl = const_cast<uint16_t*>(s.update.l); adam.ldp = s.update.ld;
    adam.Cscale = const_cast<float*>(s.update.scale); adam.ldscale = s.update.scale_stride;
    adam.mixed = s.mixed_update;
    adam.mom = s.momentum; adam.ldm = s.ldm; adam.var = s.variance; adam.ldv = s.ldv;
    adam.beta1 = s.beta1; adam.beta2 = s.beta2; adam.eps = s.eps; adam.inv_bc1 = s.inv_bc1; adam.inv_sqrt_bc2 = s.inv_sqrt_bc2;
    gemm_half(r.middle, r.right, adam, status, stream);
  }
  if (s.phases & kStepBackward) {
    first_product(r, s.update, true, r.left_turned, status, stream);        // T2 = U^T Q_L^T
    HalfProblem out = second_product(r);                                    // T2^T Q_R^T
    out.mode = kEpiRowMajor;
    out.C = s.out; out.ldc = r.cols;
    gemm_half(r.middle, r.right_turned, out, status, stream);
  }
  if (averages) {
    // Products of a vector of G with another one: what counts is their error against the vectors' own sizes, which the pairs
    // keep in every range (2^-23 of an element, 2^-39 of its vector's largest).
    const HalfOperand x = operand(r.x), xt = operand(r.xt);
    HalfProblem gram{};              // L = beta L + (1 - beta) G G^T, R likewise
    gram.mode = kEpiStore;
    gram.symmetric = 1;
    gram.alpha = static_cast<float>(1.0 - s.beta);
    gram.beta = static_cast<float>(s.beta);
    gram.M = gram.N = r.rows; gram.K = r.cols;
    gram.C = s.left_gram; gram.ldc = s.ld_left;
    gemm_half(xt, xt, gram, status, side);
    gram.M = gram.N = r.cols; gram.K = r.rows;
    gram.C = s.right_gram; gram.ldc = s.ld_right;
    gemm_half(x, x, gram, status, side);
  }
}

}  // namespace soapb200
