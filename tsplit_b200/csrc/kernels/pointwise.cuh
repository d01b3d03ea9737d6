// The element-wise operators, shared by the one-operator kernels and the pointwise programs.
#pragma once

namespace tsb_pw {

enum { UN_COPY, UN_RELU, UN_SIGMOID, UN_TANH, UN_SQRT, UN_RSQRT, UN_NEG, UN_ADDC, UN_MULC, UN_CDIV, UN_FILL };
enum { BIN_ADD, BIN_MUL, BIN_DIV, BIN_RELU_GRAD, BIN_SUB, BIN_ADD_RELU, BIN_RELU_GRAD_OUT };

template <int OP>
__device__ __forceinline__ float un(float x, float a) {
  switch (OP) {
    case UN_COPY: return x;
    case UN_RELU: return fmaxf(x, 0.f);
    case UN_SIGMOID: return 1.f / (1.f + __expf(-x));
    case UN_TANH: return tanhf(x);
    case UN_SQRT: return sqrtf(x);
    case UN_RSQRT: return rsqrtf(x);
    case UN_NEG: return -x;
    case UN_ADDC: return x + a;
    case UN_MULC: return x * a;
    case UN_CDIV: return a / x;
    default: return a;   // UN_FILL
  }
}
template <int OP>
__device__ __forceinline__ float bin(float a, float b) {
  switch (OP) {
    case BIN_ADD: return a + b;
    case BIN_MUL: return a * b;
    case BIN_DIV: return a / b;
    case BIN_RELU_GRAD: return a > 0.f ? b : (a == 0.f ? 0.5f * b : 0.f);
    case BIN_ADD_RELU: return fmaxf(a + b, 0.f);              // residual add + ReLU in one pass
    case BIN_RELU_GRAD_OUT: return a > 0.f ? b : 0.f;         // a = the ReLU OUTPUT: gradient passes where it is positive
    default: return a - b;
  }
}

}  // namespace tsb_pw
