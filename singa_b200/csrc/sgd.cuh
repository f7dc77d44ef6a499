// The SGD update of one element, and the kernels that end in one.
#pragma once
#include "common.cuh"

namespace sgb {

struct SgdArgs {
  float lr, mom, damp, decay, grad_scale;
  int use_momentum, nesterov, use_decay, use_scale;
};

__device__ __forceinline__ void sgd_one(float& p, float g, float& m, const SgdArgs& a) {
  // the reference's chain, one rounding per BLAS-1 step (python/singa/opt.py):
  //   g *= 1/world ; g += decay*p ; m = m*mom ; m += (1-damp)*g ; p += -lr*m
  if (a.use_scale) g = g * a.grad_scale;
  if (a.use_decay) g = fmaf(a.decay, p, g);
  float step = g;
  if (a.use_momentum) {
    float b = m * a.mom;
    b = fmaf(1.0f - a.damp, g, b);
    m = b;
    step = a.nesterov ? fmaf(a.mom, b, g) : b;
  }
  p = fmaf(0.0f - a.lr, step, p);
}

// Checks the options and fills `a` in (sgb_sgd_update_multi_f32).
inline int sgd_args(SgdArgs* a, void* const* moments, float lr, float momentum, float dampening, float weight_decay,
                    int nesterov, float grad_scale) {
  const int use_m = momentum != 0.0f;
  if (use_m && !moments) return SGB_ERR_NULL;
  if (nesterov && (!use_m || dampening != 0.0f)) return SGB_ERR_UNSUPPORTED;
  *a = SgdArgs{lr, momentum, dampening, weight_decay, grad_scale, use_m, nesterov != 0, weight_decay != 0.0f,
               grad_scale != 1.0f};
  return SGB_OK;
}

// sgb_sgd_update_multi_f32 over gradients that are rounded to fp16 and widened
// again, where they are, on the way (multi_tensor.cu).
int sgd_round_f16_multi(void* const* params, void* const* grads, void* const* moments, const size_t* sizes, size_t count,
                        const SgdArgs& a, cudaStream_t s);

}  // namespace sgb
