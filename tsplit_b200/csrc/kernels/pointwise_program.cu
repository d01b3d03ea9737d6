// A chain of element-wise operators as one launch.
//
// A training step of a recurrent network or of an attention block is full of operators that touch the same elements
// one after the other (gate sums, biases, activations, their gradients).  As kernels of their own each costs a launch
// and a round trip through memory; here an executor hands over the whole chain as a list of instructions, and a thread
// runs them on its four elements: inputs arrive by cp.async, all in flight at once, values live in shared memory (one
// 16-byte column per thread and value, so there are no bank conflicts and no barriers), and only values that somebody
// else reads are stored.  Every instruction is rounded to fp32 as the operator's own kernel does, so results are the
// same bits.  Bound by launch latency for small tensors (the 1881 element-wise launches of an LSTM step become 64) and by
// DRAM for large ones: 137 M floats times a constant plus another tensor 244 us, 396 as two kernels.
#include <cuda_runtime.h>
#include <stdint.h>
#include "launch.cuh"
#include "smem_limit.h"
#include "pointwise.cuh"

#define TSB_OK 0
#define TSB_ERR_ARG 1
#define TSB_ERR_UNSUPPORTED 2
#define TSB_ERR_LAUNCH 3

namespace {

using tsb_launch::load;

using namespace tsb_pw;

constexpr int MAX_IN = 32, MAX_INS = 64, MAX_SLOTS = 48, BINARY = 32;

struct Instr {
  unsigned char op, a, b, dst;      // op: unary code, or BINARY + binary code; a, b, dst: value slots
  float alpha;
  float4* out;                      // where the value is stored, or null
};
struct Program {
  const float* in[MAX_IN];          // loaded into slots 0 .. n_in - 1
  unsigned char kind[MAX_IN];       // 0: element by element, 1: one row, repeated, 2: one number
  Instr ins[MAX_INS];
  int n_in, n_ins;
  long long n4;                     // groups of four elements
  unsigned cols4;                   // groups of four elements in a row (inputs of kind 1)
};

template <int OP>
__device__ __forceinline__ float4 un4(float4 v, float a) {
  return make_float4(un<OP>(v.x, a), un<OP>(v.y, a), un<OP>(v.z, a), un<OP>(v.w, a));
}
template <int OP>
__device__ __forceinline__ float4 bin4(float4 a, float4 b) {
  return make_float4(bin<OP>(a.x, b.x), bin<OP>(a.y, b.y), bin<OP>(a.z, b.z), bin<OP>(a.w, b.w));
}

__global__ void __launch_bounds__(256) pointwise_program(const __grid_constant__ Program p) {
  tsb_launch::enter();
  extern __shared__ float4 slots[];
  const int T = blockDim.x;
  float4* r = slots + threadIdx.x;
  const long long i = blockIdx.x * (long long)T + threadIdx.x;
  if (i >= p.n4) return;
  const unsigned in_row = (p.n4 >> 32) == 0 ? (unsigned)i % p.cols4 : (unsigned)(i % p.cols4);
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  for (int k = 0; k < p.n_in; ++k) {
    if (p.kind[k] == 2) {
      const float v = load(p.in[k]);
      r[k * T] = make_float4(v, v, v, v);
    } else {
      const float4* src = reinterpret_cast<const float4*>(p.in[k]) + (p.kind[k] == 0 ? i : in_row);
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(r + k * T);
      asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  for (int k = 0; k < p.n_ins; ++k) {
    const Instr c = p.ins[k];
    const float4 a = r[c.a * T];
    float4 v;
    switch (c.op) {
      case UN_COPY: v = a; break;
      case UN_RELU: v = un4<UN_RELU>(a, 0.f); break;
      case UN_SIGMOID: v = un4<UN_SIGMOID>(a, 0.f); break;
      case UN_TANH: v = un4<UN_TANH>(a, 0.f); break;
      case UN_SQRT: v = un4<UN_SQRT>(a, 0.f); break;
      case UN_RSQRT: v = un4<UN_RSQRT>(a, 0.f); break;
      case UN_NEG: v = un4<UN_NEG>(a, 0.f); break;
      case UN_ADDC: v = un4<UN_ADDC>(a, c.alpha); break;
      case UN_MULC: v = un4<UN_MULC>(a, c.alpha); break;
      case UN_CDIV: v = un4<UN_CDIV>(a, c.alpha); break;
      case UN_FILL: v = make_float4(c.alpha, c.alpha, c.alpha, c.alpha); break;
      case BINARY + BIN_ADD: v = bin4<BIN_ADD>(a, r[c.b * T]); break;
      case BINARY + BIN_MUL: v = bin4<BIN_MUL>(a, r[c.b * T]); break;
      case BINARY + BIN_DIV: v = bin4<BIN_DIV>(a, r[c.b * T]); break;
      case BINARY + BIN_RELU_GRAD: v = bin4<BIN_RELU_GRAD>(a, r[c.b * T]); break;
      case BINARY + BIN_SUB: v = bin4<BIN_SUB>(a, r[c.b * T]); break;
      case BINARY + BIN_ADD_RELU: v = bin4<BIN_ADD_RELU>(a, r[c.b * T]); break;
      default: v = bin4<BIN_RELU_GRAD_OUT>(a, r[c.b * T]); break;
    }
    r[c.dst * T] = v;
    if (c.out) c.out[i] = v;
  }
}

// Up to 64 short arrays copied by one launch, a block per array (parameter gradients that an operator keeps in buffers
// of its own, handed out to their nodes).
constexpr int MAX_COPIES = 64;
struct Copies {
  const float* src[MAX_COPIES];
  float* dst[MAX_COPIES];
  int n[MAX_COPIES];
};
__global__ void __launch_bounds__(256) multi_copy(const __grid_constant__ Copies c) {
  tsb_launch::enter();
  for (int i = threadIdx.x; i < c.n[blockIdx.x]; i += blockDim.x) c.dst[blockIdx.x][i] = c.src[blockIdx.x][i];
}

int rc_of(cudaError_t e) { return e == cudaSuccess ? TSB_OK : (TSB_ERR_LAUNCH | ((int)e << 8)); }

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

}  // namespace

extern "C" {

// Runs `n_ins` instructions on `n` elements (a multiple of four).  in / kind: the inputs, kind 0 with n elements,
// 1 with `cols` (a multiple of four), 2 with one; code: op, a, b, dst of each instruction, one byte each; out: where
// its value goes, or null.  Arrays of kind 0 and 1 and the outputs are 16-byte aligned; an output is no input.
int tsb_pointwise(int n_in, const void** in, const int* kind, int n_ins, const unsigned char* code, const float* alpha,
                  void** out, int slots, long long n, long long cols, void* stream) {
  if (n_in < 0 || n_in > MAX_IN || n_ins < 1 || n_ins > MAX_INS || slots < 1 || slots > MAX_SLOTS || n_in > slots)
    return TSB_ERR_ARG;
  if (n <= 0) return TSB_OK;
  if ((n & 3) || (cols & 3) || cols < 0 || cols >= (1ll << 32)) return TSB_ERR_UNSUPPORTED;
  Program p = {};
  p.n_in = n_in; p.n_ins = n_ins; p.n4 = n / 4;
  p.cols4 = cols > 0 ? (unsigned)(cols / 4) : 1;
  for (int k = 0; k < n_in; ++k) {
    if (kind[k] < 0 || kind[k] > 2 || !in[k] || (kind[k] == 1 && cols <= 0)) return TSB_ERR_ARG;
    if (kind[k] != 2 && (reinterpret_cast<uintptr_t>(in[k]) & 15)) return TSB_ERR_UNSUPPORTED;
    p.in[k] = static_cast<const float*>(in[k]);
    p.kind[k] = (unsigned char)kind[k];
  }
  for (int k = 0; k < n_ins; ++k) {
    const unsigned char* c = code + 4 * k;
    const bool known = c[0] <= UN_FILL || (c[0] >= BINARY && c[0] <= BINARY + BIN_RELU_GRAD_OUT);
    if (!known || c[1] >= slots || c[2] >= slots || c[3] >= slots) return TSB_ERR_ARG;
    if (reinterpret_cast<uintptr_t>(out[k]) & 15) return TSB_ERR_UNSUPPORTED;
    p.ins[k] = Instr{c[0], c[1], c[2], c[3], alpha[k], static_cast<float4*>(out[k])};
  }
  // small tensors: short blocks, so that more SMs take part; large ones: a block per 256 groups (see elementwise.cu)
  const int threads = p.n4 <= 64ll * sm_count() ? 64 : 256;
  const size_t smem = (size_t)slots * threads * sizeof(float4);
  static tsb_launch::SmemLimit limit;
  const cudaError_t e = limit.raise(pointwise_program, MAX_SLOTS * 256 * (int)sizeof(float4));
  if (e != cudaSuccess) return rc_of(e);
  const long long blocks = (p.n4 + threads - 1) / threads;
  if (blocks > 0x7fffffffll) return TSB_ERR_UNSUPPORTED;
  return rc_of(tsb_launch::launch(pointwise_program, dim3((unsigned)blocks), dim3(threads), smem,
                                  static_cast<cudaStream_t>(stream), p));
}

int tsb_multi_copy(int count, const void** src, void** dst, const long long* n, void* stream) {
  if (count < 0 || count > MAX_COPIES) return TSB_ERR_ARG;
  if (count == 0) return TSB_OK;
  Copies c = {};
  for (int k = 0; k < count; ++k) {
    if (n[k] < 0 || n[k] >= (1ll << 31)) return TSB_ERR_ARG;
    c.src[k] = static_cast<const float*>(src[k]);
    c.dst[k] = static_cast<float*>(dst[k]);
    c.n[k] = (int)n[k];
  }
  return rc_of(tsb_launch::launch(multi_copy, dim3((unsigned)count), dim3(256), 0, static_cast<cudaStream_t>(stream), c));
}

}  // extern "C"
