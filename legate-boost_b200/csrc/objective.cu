// Weighted gradients of the boosting round: g = d loss / d raw prediction times the learning rate,
// h = second derivative floored at 1e-8, both float64 [n_rows, n_outputs].
//
// Reference behaviour restated here: LBBase._get_weighted_gradient, legateboost/legateboost.py:189-224
// (unit sample weights, no subsampling), over the objectives' transform + gradient:
// SquaredErrorObjective (objectives.py:131-135): g = pred - y, h = 1;
// LogLossObjective (objectives.py:489-512): binary p = 1 / (1 + exp(-raw)), g = p - y, h = p (1 - p);
// multi-class softmax with the row maximum taken out, g = p - onehot(label), h = p (1 - p).
// The reference runs them as a chain of array operations (about ten passes over N x K float64);
// here a row is read once and its pairs are written once.
#include "internal.h"
#include "objective.cuh"

namespace lbk {
namespace {

__global__ void __launch_bounds__(256)
  k_gradient_squared_error(const double* __restrict__ raw, const double* __restrict__ y, int64_t n, double lr,
                           double* __restrict__ g, double* __restrict__ h)
{
  AfterTheKernelBefore();
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const double2 v = GradientSquaredError(raw[i], y[i], lr);
  g[i] = v.x;
  h[i] = v.y;
}

__global__ void __launch_bounds__(256)
  k_gradient_logloss_binary(const double* __restrict__ raw, const double* __restrict__ y, int64_t n, double lr,
                            double* __restrict__ g, double* __restrict__ h)
{
  AfterTheKernelBefore();
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const double2 v = GradientLogistic(raw[i], y[i], lr);
  g[i] = v.x;
  h[i] = v.y;
}

// A block takes `rows` rows: they come in and their gradients go out as whole lines, through shared memory, and
// one thread per row makes the exponentials and their sum there.  Bound by HBM (24 bytes per value); a thread that
// reads and writes its own row of K values touches a line per value: 1M x 10: 172 us, here 71 us.
// Shared memory: exponentials [rows][K | 1] (an odd pitch), sums [rows], classes [rows].
constexpr int kSoftmaxThreads = 256;
size_t SoftmaxRowBytes(int K) { return sizeof(double) * ((K | 1) + 1) + sizeof(int); }

__global__ void __launch_bounds__(kSoftmaxThreads)
  k_gradient_softmax(const double* __restrict__ raw, const double* __restrict__ label, int64_t n_rows, int K, int rows, double lr,
                     double* __restrict__ g, double* __restrict__ h)
{
  AfterTheKernelBefore();
  extern __shared__ double s_e[];
  const int pitch    = K | 1;
  double* s_div      = s_e + rows * pitch;
  int* s_cls         = reinterpret_cast<int*>(s_div + rows);
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * rows;
  const int here     = static_cast<int>(n_rows - row0 < rows ? n_rows - row0 : rows);
  const int64_t at0  = row0 * K;
  for (int i = threadIdx.x; i < here * K; i += kSoftmaxThreads) {
    const int row = i / K;
    s_e[row * pitch + i - row * K] = raw[at0 + i];
  }
  __syncthreads();
  for (int row = threadIdx.x; row < here; row += kSoftmaxThreads) {
    double* e = s_e + row * pitch;
    double s  = e[0];
    for (int k = 1; k < K; ++k) s = fmax(s, e[k]);
    double div = 0.0;
    for (int k = 0; k < K; ++k) {
      const double v = exp(e[k] - s);
      e[k]           = v;
      div += v;
    }
    s_div[row] = div;
    s_cls[row] = static_cast<int>(label[row0 + row]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < here * K; i += kSoftmaxThreads) {
    const int row  = i / K, k = i - row * K;
    const double p = s_e[row * pitch + k] / s_div[row];
    g[at0 + i]     = (k == s_cls[row] ? p - 1.0 : p) * lr;
    h[at0 + i]     = fmax(p * (1.0 - p), 1e-8);
  }
}

// more classes than shared memory takes 32 rows of: one thread per row
__global__ void __launch_bounds__(256)
  k_gradient_softmax_wide(const double* __restrict__ raw, const double* __restrict__ label, int64_t n_rows, int K, double lr,
                          double* __restrict__ g, double* __restrict__ h)
{
  AfterTheKernelBefore();
  const int64_t row = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (row >= n_rows) return;
  const double* r = raw + row * K;
  double s        = r[0];
  for (int k = 1; k < K; ++k) s = fmax(s, r[k]);
  double div = 0.0;
  for (int k = 0; k < K; ++k) div += exp(r[k] - s);
  const int cls = static_cast<int>(label[row]);
  for (int k = 0; k < K; ++k) {
    const double p = exp(r[k] - s) / div;
    g[row * K + k] = (k == cls ? p - 1.0 : p) * lr;
    h[row * K + k] = fmax(p * (1.0 - p), 1e-8);
  }
}

}  // namespace

void Gradient(int objective, const double* raw_pred, const double* y, int64_t n_rows, int n_outputs, double learning_rate,
              double* g, double* h, cudaStream_t stream)
{
  if (n_rows == 0) return;
  const int64_t n = n_rows * n_outputs;
  if (objective == LBK_SQUARED_ERROR) {
    LaunchChained(k_gradient_squared_error, static_cast<unsigned>((n + 255) / 256), 256, 0, stream, raw_pred, y, n, learning_rate, g, h);
  } else if (n_outputs == 1) {
    LaunchChained(k_gradient_logloss_binary, static_cast<unsigned>((n + 255) / 256), 256, 0, stream, raw_pred, y, n, learning_rate, g, h);
  } else {
    const int rows = static_cast<int>(std::min<size_t>(kSoftmaxThreads, 48 * 1024 / SoftmaxRowBytes(n_outputs)) / 32 * 32);
    if (rows > 0)
      LaunchChained(k_gradient_softmax, static_cast<unsigned>((n_rows + rows - 1) / rows), kSoftmaxThreads, rows * SoftmaxRowBytes(n_outputs), stream,
        raw_pred, y, n_rows, n_outputs, rows, learning_rate, g, h);
    else
      LaunchChained(k_gradient_softmax_wide, static_cast<unsigned>((n_rows + 255) / 256), 256, 0, stream, raw_pred, y, n_rows, n_outputs,
                                                                                             learning_rate, g, h);
  }
  LBK_LAUNCH_CHECK();
}

}  // namespace lbk

extern "C" int lbk_gradient(lbk_context* ctx, int objective, const double* raw_pred, const double* y, int64_t n_rows,
                            int n_outputs, double learning_rate, double* g, double* h, void* stream_)
{
  using namespace lbk;
  return Guard(ctx, [&] {
    LBK_EXPECT(ctx != nullptr, "context is null");
    LBK_EXPECT(objective == LBK_SQUARED_ERROR || objective == LBK_LOG_LOSS, "unknown objective");
    LBK_EXPECT(n_rows >= 0 && n_outputs >= 1, "bad shape");
    if (n_rows == 0) return;
    LBK_EXPECT(raw_pred && y && g && h, "null argument");
    LBK_CUDA(cudaSetDevice(ctx->device));
    Gradient(objective, raw_pred, y, n_rows, n_outputs, learning_rate, g, h, static_cast<cudaStream_t>(stream_));
  });
}
