// One ordinary optimizer step on one GPU as a single native call: the launches of engine/local.py's pipeline in their order.
// A step of a small matrix is bound by the host; with each launch a call of its own from the interpreter a 256 x 512 step took
// 182 us, issued from here 118 us.
//
// The four products of the rotation chain depend on one another and each ends in a wave of tiles that leaves SMs idle; the
// Gram averages depend on the gradient only.  So the chain runs on a stream of its own, of higher priority, and the averages
// fill what it leaves free: 1000 x 1501 181 -> 170 us, 2048 x 5504 1308 -> 1266 us, 4096 x 4096 1866 -> 1827 us, 8192 x 8192
// within the runs' spread.
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

void steady_step(const SteadyStep& s, int* status, cudaStream_t stream) {
  if (s.rows <= 0 || s.cols <= 0) throw std::invalid_argument("steady_step: empty matrix");
  half_planes(s.gradient, s.gradient_type, s.s_i, s.s_j, s.rows, s.cols, s.x, s.xt, stream);
  const HalfOperand x = operand(s.x), xt = operand(s.xt);
  const cudaStream_t chain = s.chain;
  const Fork rotations(stream, chain);

  HalfProblem forward{};             // T = X^T Q_L
  forward.M = s.cols; forward.N = s.rows; forward.K = s.rows;
  forward.mode = kEpiSplit;
  forward.alpha = 1.0f;
  forward.Ch = const_cast<uint16_t*>(s.middle.h); forward.Cl = const_cast<uint16_t*>(s.middle.l); forward.ldp = s.middle.ld;
  forward.Cscale = const_cast<float*>(s.middle.scale); forward.ldscale = s.middle.scale_stride;
  gemm_half(x, s.left, forward, status, chain);

  HalfProblem adam{};                // Y = T^T Q_R, Adam(Y) -> U
  adam.M = s.rows; adam.N = s.cols; adam.K = s.cols;
  adam.mode = kEpiAdam;
  adam.alpha = 1.0f;
  adam.Ch = const_cast<uint16_t*>(s.update.h); adam.Cl = const_cast<uint16_t*>(s.update.l); adam.ldp = s.update.ld;
  adam.Cscale = const_cast<float*>(s.update.scale); adam.ldscale = s.update.scale_stride;
  adam.mom = s.momentum; adam.ldm = s.ldm; adam.var = s.variance; adam.ldv = s.ldv;
  adam.beta1 = s.beta1; adam.beta2 = s.beta2; adam.eps = s.eps; adam.inv_bc1 = s.inv_bc1; adam.inv_sqrt_bc2 = s.inv_sqrt_bc2;
  gemm_half(s.middle, s.right, adam, status, chain);

  gemm_half(s.update, s.left_turned, forward, status, chain);      // T2 = U^T Q_L^T

  HalfProblem out{};                 // T2^T Q_R^T
  out.M = s.rows; out.N = s.cols; out.K = s.cols;
  out.mode = kEpiRowMajor;
  out.alpha = 1.0f;
  out.C = s.out; out.ldc = s.cols;
  gemm_half(s.middle, s.right_turned, out, status, chain);

  HalfProblem gram{};                // L = beta L + (1 - beta) G G^T, R likewise
  gram.mode = kEpiStore;
  gram.symmetric = 1;
  gram.alpha = static_cast<float>(1.0 - s.beta);
  gram.beta = static_cast<float>(s.beta);
  gram.M = gram.N = s.rows; gram.K = s.cols;
  gram.C = s.left_gram; gram.ldc = s.ld_left;
  gemm_half(xt, xt, gram, status, stream);
  gram.M = gram.N = s.cols; gram.K = s.rows;
  gram.C = s.right_gram; gram.ldc = s.ld_right;
  gemm_half(x, x, gram, status, stream);
}

}  // namespace soapb200
