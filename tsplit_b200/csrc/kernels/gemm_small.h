// Small matrix products, bound by latency (gemm_small.cu); the interface that gemm_tcgen05.cu dispatches to.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace tsb_small {

// An operand whose K range or row range a block reads: by TMA (`tma`; map with boxes of 32 k x `rows of a tile`, or chunks
// of 32 rows) or, where its strides allow no tensor map, float by float from `base`.
struct Operand {
  const float* base;
  long long ld, s, s2;           // row stride; matrix (o, i) of a batch starts o * s2 + i * s in
  int tma, chunked;              // chunked: rows contiguous, all chunks of 32 in one box
  int kbox;                      // k-blocks per box
  int heads, shift;              // tensor-map coordinates of matrix (o, i): batch i (heads) or o * inner + i, rows from o * shift
};
struct Product {
  Operand a, b;
  float* c;
  const float* bias;             // [n], added to every row; may be null
  float* relu;                   // second output max(c, 0), strides of c; may be null
  long long ldc, sc, sc2;
  int m, n, k, inner, batch;     // batch = outer * inner
  int accumulate;
  int kb_per_split;              // k-blocks of 32 that one block sums
  int tiles_m, tiles_n, vec_c;   // filled in by run()
};
constexpr int TILE_M = 64, TILE_N = 32;
constexpr int MAX_PRODUCTS = 16;
constexpr int MAX_SPLITS = 8;    // the blocks that share a tile are one cluster
constexpr int MAX_KBLOCKS = 16;  // of one block: all of its operands are in shared memory at once
constexpr int ROUND = 4;         // k-blocks that a box brings and a wait is for

// Blocks of a product, and the shared memory of one.
inline long long blocks_of(long long m, long long n, long long batch, int splits) {
  return ((m + TILE_M - 1) / TILE_M) * ((n + TILE_N - 1) / TILE_N) * batch * splits;
}
inline int smem_of(int kb_per_split) {
  const int round = kb_per_split < ROUND ? kb_per_split : ROUND;
  return (kb_per_split + round - 1) / round * round * (TILE_M + TILE_N) * 128 + 1024;
}

// Up to MAX_PRODUCTS products of one transposition as one launch; `splits` blocks share each tile (more than one: a single
// product).
cudaError_t run(Product* p, const CUtensorMap* ta, const CUtensorMap* tb, int count, int splits, bool trans_a, bool trans_b,
                int* status, cudaStream_t st);

}  // namespace tsb_small
