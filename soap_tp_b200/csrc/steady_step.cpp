// Rotations and ordinary optimizer steps on one GPU as single native calls: engine/local.py's pipeline.
// A step of a small matrix is bound by the host; with each launch a call of its own from the interpreter a 256 x 512 step took
// 182 us, issued from here 118 us.
//
// The four products of the rotation chain depend on one another and each ends in a wave of tiles that leaves SMs idle; the
// Gram averages depend on the gradient only.  So the averages run on a stream beside it and fill what the chain leaves free.
// The chain stays on the caller's stream: its first product then overlaps the tail of the operand planes, which an event
// between streams does not allow.  Device time of a step, everything on one stream / the chain beside / the averages beside:
// 256 x 512 126 / 92 / 85 us, 512 x 1376 175 / 158 / 121 us, 1000 x 1501 198 / 198 / 148 us, 2048 x 5504 1388 / 1352 / 1186 us,
// 4096 x 4096 1900 / 1863 / 1748 us, 8192 x 8192 within the runs' spread.  (As measured when they were moved.  Since then, steps one after
// another that the host has issued far ahead, everything on one stream / the averages beside: 512 x 1376 127 / 102 us, 1000 x 1501 bf16
// 155 / 132, 2048 x 5504 bf16 1172 / 1059, 4096 x 4096 bf16 1644 / 1557.)
#include <algorithm>
#include <optional>
#include <stdexcept>

#include "gemm.h"
#include "gemm_half.h"
#include "launch_util.h"

namespace soapb200 {

namespace {
HalfOperand operand(const HalfTarget& t, const CUtensorMap* maps) { return HalfOperand{t.h, t.l, t.ld, t.scale, 0, nullptr, maps}; }

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
HalfJob first_product(const Rotation& r, const HalfOperand& source, bool settled, const HalfOperand& basis) {
  HalfProblem p{};
  p.M = r.cols; p.N = r.rows; p.K = r.rows;
  p.mode = kEpiSplit;
  p.alpha = 1.0f;
  p.Ch = const_cast<uint16_t*>(r.middle.h); p.Cl = const_cast<uint16_t*>(r.middle.l); p.ldp = r.middle.ld;
  p.Cscale = const_cast<float*>(r.middle.scale); p.ldscale = r.middle.scale_stride;
  p.wide = r.guard.wide; p.settled = settled; p.mixed = r.mixed_middle;
  return HalfJob{source, basis, p};
}

HalfOperand source_of(const Rotation& r) {
  HalfOperand x = operand(r.x, r.x_maps);
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

PlanesJob planes_of(const Rotation& r) {
  return PlanesJob{r.source, r.source_type, r.s_i, r.s_j, r.rows, r.cols, r.x, r.xt, r.guard};
}

// The products of a step.
HalfJob rotated(const SteadyStep& s) {                                      // T = X^T Q_L
  const Rotation& r = s.rotation;
  return first_product(r, source_of(r), false, r.left);
}
HalfJob adam(const SteadyStep& s) {                                         // Y = T^T Q_R, Adam(Y) -> U
  const Rotation& r = s.rotation;
  HalfProblem p = second_product(r);
  p.mode = kEpiAdam;
  p.Ch = const_cast<uint16_t*>(s.update.h); p.Cl = const_cast<uint16_t*>(s.update.l); p.ldp = s.update.ld;
  p.Cscale = const_cast<float*>(s.update.scale); p.ldscale = s.update.scale_stride;
  p.mixed = s.mixed_update;
  p.mom = s.momentum; p.ldm = s.ldm; p.var = s.variance; p.ldv = s.ldv;
  p.beta1 = s.beta1; p.beta2 = s.beta2; p.eps = s.eps; p.inv_bc1 = s.inv_bc1; p.inv_sqrt_bc2 = s.inv_sqrt_bc2;
  return HalfJob{r.middle, r.right, p};
}
HalfJob turned_back(const SteadyStep& s) {                                  // T2 = U^T Q_L^T
  return first_product(s.rotation, s.update, true, s.rotation.left_turned);
}
HalfJob result(const SteadyStep& s) {                                       // T2^T Q_R^T
  const Rotation& r = s.rotation;
  HalfProblem p = second_product(r);
  p.mode = kEpiRowMajor;
  p.C = s.out; p.ldc = r.cols;
  return HalfJob{r.middle, r.right_turned, p};
}
// L = beta L + (1 - beta) G G^T, R likewise.  Products of a vector of G with another one: what counts is their error against the
// vectors' own sizes, which the pairs keep in every range (2^-23 of an element, 2^-39 of its vector's largest).
HalfJob average(const SteadyStep& s, bool left) {
  const Rotation& r = s.rotation;
  const HalfOperand x = left ? operand(r.xt, r.xt_maps) : operand(r.x, r.x_maps);
  HalfProblem p{};
  p.mode = kEpiStore;
  p.symmetric = 1;
  p.alpha = static_cast<float>(1.0 - s.beta);
  p.beta = static_cast<float>(s.beta);
  p.M = p.N = left ? r.rows : r.cols;
  p.K = left ? r.cols : r.rows;
  p.C = left ? s.left_gram : s.right_gram;
  p.ldc = left ? s.ld_left : s.ld_right;
  return HalfJob{x, x, p};
}

// The phases of one step, or of several that share their launches.
template <typename Planes, typename Launch, typename Averages>
void issue(const SteadyStep& s, cudaStream_t stream, Planes planes, Launch launch, Averages launch_averages) {
  if (s.phases & kStepPlanes) planes();
  const bool averages = s.phases & kStepAverages, rotations = s.phases & (kStepForward | kStepBackward);
  const cudaStream_t side = averages && rotations ? s.side : stream;
  std::optional<Fork> fork;
  if (side != stream) fork.emplace(stream, side);
  if (s.phases & kStepForward) {
    launch(rotated, stream);
    launch(adam, stream);
  }
  if (s.phases & kStepBackward) {
    launch(turned_back, stream);
    launch(result, stream);
  }
  if (averages) launch_averages(side);
}
}  // namespace

void rotate_half(const Rotation& r, bool turned, float* out, int64_t ldc, int* status, cudaStream_t stream) {
  if (r.rows <= 0 || r.cols <= 0) return;
  half_planes(r.source, r.source_type, r.s_i, r.s_j, r.rows, r.cols, r.x, r.xt, r.guard, stream);
  const HalfJob first = first_product(r, source_of(r), false, turned ? r.left_turned : r.left);
  gemm_half(first.a, first.b, first.problem, status, stream);
  HalfProblem store = second_product(r);
  store.mode = kEpiStore;
  store.C = out; store.ldc = ldc;
  gemm_half(r.middle, turned ? r.right_turned : r.right, store, status, stream);
}

void steady_step(const SteadyStep& s, int* status, cudaStream_t stream) {
  const Rotation& r = s.rotation;
  if (r.rows <= 0 || r.cols <= 0) throw std::invalid_argument("steady_step: empty matrix");
  issue(s, stream, [&] { half_planes(r.source, r.source_type, r.s_i, r.s_j, r.rows, r.cols, r.x, r.xt, r.guard, stream); },
        [&](auto product, cudaStream_t on) {
          const HalfJob job = product(s);
          gemm_half(job.a, job.b, job.problem, status, on);
        },
        [&](cudaStream_t side) {
          const HalfJob both[2] = {average(s, true), average(s, false)};
          if (averages_share(r.rows, r.cols)) {
            gemm_half_group(both, 2, status, side);
          } else {
            for (const HalfJob& job : both) gemm_half(job.a, job.b, job.problem, status, side);
          }
        });
}

bool averages_share(int rows, int cols) { return !half_on_pairs(rows, rows, true) && !half_on_pairs(cols, cols, true); }

bool steady_step_shares(int rows, int cols) {
  return rows > 0 && cols > 0 && !half_fills_pairs(cols, rows, false) && !half_fills_pairs(rows, cols, false) &&
         !half_fills_pairs(rows, rows, true) && !half_fills_pairs(cols, cols, true);
}

void steady_steps(const SteadyStep* steps, int count, int* status, cudaStream_t stream) {
  if (count < 1 || count > kHalfGroup) throw std::invalid_argument("steady_steps: too many steps for shared launches");
  for (int i = 0; i < count; ++i) {
    if (steps[i].rotation.rows <= 0 || steps[i].rotation.cols <= 0) throw std::invalid_argument("steady_steps: empty matrix");
    if (steps[i].phases != steps[0].phases || steps[i].side != steps[0].side)
      throw std::invalid_argument("steady_steps: steps that share launches have the same phases and streams");
  }
  issue(steps[0], stream,
        [&] {
          PlanesJob jobs[kHalfGroup];
          for (int i = 0; i < count; ++i) jobs[i] = planes_of(steps[i].rotation);
          half_planes_group(jobs, count, stream);
        },
        [&](auto product, cudaStream_t on) {
          HalfJob jobs[kHalfGroup];
          for (int i = 0; i < count; ++i) jobs[i] = product(steps[i]);
          gemm_half_group(jobs, count, status, on);
        },
        [&](cudaStream_t side) {
          HalfJob jobs[2 * kHalfGroup];
          for (int i = 0; i < 2 * count; ++i) jobs[i] = average(steps[i / 2], i % 2 == 0);
          for (int i = 0; i < 2 * count; i += kHalfGroup) gemm_half_group(jobs + i, std::min(kHalfGroup, 2 * count - i), status, side);
        });
}

}  // namespace soapb200
