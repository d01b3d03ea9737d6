// Kernel launches that overlap the tail of the kernel before them (programmatic dependent launch).
//
// A training step of this library is a chain of some hundred to some thousand kernels on one stream, most of them a
// few microseconds long, so the time between one kernel's last block and the next one's first instruction is a large
// part of it.  Every kernel of this folder is launched with the programmatic-serialisation attribute and begins with
// enter(): its blocks may be placed, and barriers and TMEM set up, while the previous kernel drains; they wait until that
// kernel has completed and its writes are visible.  Because every kernel waits, completion stays in stream order; a
// copy, an event or a kernel of another library in between is ordered in full as before.  Stream capture keeps the
// attribute as a programmatic edge.
//
// A kernel thus begins before its inputs are written.  Loads through the read-only path (ld.global.nc: __ldg, or what
// nvcc makes of a `const T* __restrict__` parameter) want data that nothing writes while the kernel lives, and
// may be moved above the wait or served from a line that was cached before it.  So kernels launched from here
// take the pointers they read without __restrict__ and use ordinary loads, which stay behind the wait; pointers that
// they write keep __restrict__.  A plain load costs the same (137 M floats times a constant 161.5 us through the read-only
// path and 161.9 without, the sum of two such tensors 234.3 and 235.5), but it stays behind the stores before it, so a
// kernel reads what it can before it writes (read_then_write below).
//
// Captured steps: LSTM, 2428 kernels: 6718 -> 5535 us (2.77 -> 2.28 us a kernel); a 1x7 / 7x1 convolution pair at 17 x 17:
// 292 -> 275 us; a small Transformer: 808 -> 716 us.
#pragma once
#include <cuda_runtime.h>

namespace tsb_launch {

// Wait for the kernel before this one.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Let the kernel after this one take the places that are free (it waits for this one's end in wait_previous).
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// A kernel of few blocks allows it as soon as it runs itself.  A larger one leaves it to its blocks' ends: blocks that
// are placed while some SMs are still busy crowd on the others, and a grid that should spread over the chip runs
// unbalanced (ResNet-50, batch 32, 8650 us before: all kernels allowing 8594 us, up to 100 blocks 8617, up to 32 or 16
// 8455; the LSTM step is 5680 us when its one-block products do not, and 5525 us for any of the limits).
constexpr unsigned FEW_BLOCKS = 32;
__device__ __forceinline__ void enter() {
  wait_previous();
  if (gridDim.x * gridDim.y * gridDim.z <= FEW_BLOCKS) allow_next();
}

// An ordinary (coherent) load of data that an earlier kernel may have written.
template <class T>
__device__ __forceinline__ T load(const T* p) { return *p; }

// The same of 16 bytes that no kernel reads again soon (an activation until its backward pass, a gradient for good): L2
// gives up their lines before others, so that what was just written, which the next kernel reads, is still there.  A
// ResNet-50 step at batch 32, whose tensors are up to 103 MB with 126 MB of L2: batch-norm apply passes 1360 -> 1280 us,
// residual additions 293 -> 255, convolutions that read what they leave 490 -> 450.  Not for a pass that another one
// follows over the same data (the gradient's column sums read x before the apply pass does: 690 -> 750 us), nor for the
// overlapping windows of filters and pools (3 x 3 forward convolutions 150 -> 164 us).
__device__ __forceinline__ float4 load_last(const float4* p) {
  float4 v;
  asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}

// A thread's elements i, i + step, ... below end, U at a time: what they read (get), then what they write (put).  In a
// plain loop every load waits for the store of the element before it, since ordinary loads do not pass stores.  (The rest
// one by one: with guarded or halved batches for it the whole loop got slower, soft-max over 4096 x 32000 410 us and
// 606 or 497.)
template <int U, class I, class Get, class Put>
__device__ __forceinline__ void read_then_write(I i, I end, I step, Get get, Put put) {
  for (; i + (U - 1) * step < end; i += U * step) {
    decltype(get(i)) v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = get(i + u * step);
#pragma unroll
    for (int u = 0; u < U; ++u) put(i + u * step, v[u]);
  }
  for (; i < end; i += step) put(i, get(i));
}

// cluster: blocks per cluster along x (0: no cluster).  Errors are left for cudaGetLastError, as with <<<>>>.
template <class... P, class... A>
cudaError_t launch_cluster(unsigned cluster, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                           A&&... args) {
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = cluster ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <class... P, class... A>
cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  return launch_cluster(0u, kernel, grid, block, smem, st, static_cast<A&&>(args)...);
}

}  // namespace tsb_launch
