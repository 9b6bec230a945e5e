// (gradient * learning rate, hessian floored at 1e-8) of one element (reference: see objective.cu).
#pragma once
#include "device_utils.cuh"

namespace lbk {

__device__ inline double2 GradientSquaredError(double raw, double y, double lr) { return make_double2((raw - y) * lr, 1.0); }
__device__ inline double2 GradientLogistic(double raw, double y, double lr)
{
  const double p = 1.0 / (1.0 + exp(-raw));
  return make_double2((p - y) * lr, fmax(p * (1.0 - p), 1e-8));
}

// The pair at an element: what the arrays hold, or the gradient of the squared error at raw prediction and label, which
// costs less to make again than to write and read (GradientForm).
__device__ inline double2 GradientAt(const double* g, const double* h, int64_t at, const GradientForm& form)
{
  const double a = g[at], b = h[at];
  return form.squared_error ? GradientSquaredError(a, b, form.learning_rate) : make_double2(a, b);
}

}  // namespace lbk
