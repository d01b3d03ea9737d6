// Products of a few million multiply-adds, where a launch is bound by latency: the gates of a recurrent cell, the layers
// of a small perceptron or Transformer, classifier heads.
//
// Same sums, bit for bit, as the kernels of gemm_tcgen05.cu (tcgen05.mma.kind::tf32 over K in steps of 8, the same K
// ranges added in the same order), but built for the shortest path instead of throughput:
//   - 64 x 32 tiles, so 128 x 128 is on 8 SMs, and a k-block brings 12 KB into an SM, not 24 (some 64 bytes a cycle);
//   - all of a block's k-blocks are in flight at once, there is no ring; a TMA box, a wait and a fence are for four of
//     them (the issuing thread spends 80 cycles on a box, 110 on a wait that succeeds at once, and 25 on an MMA);
//   - an operand that TMA cannot read (rows of 10 or 37 floats) is fetched by cp.async, without a padding pass before;
//   - K steps past the end are left out (adding zeros changes nothing);
//   - accumulators leave by plain stores: no TMA store to wait for;
//   - the partial sums of a long K meet in distributed shared memory (a cluster per tile), not in a workspace that a
//     second kernel reads.
#include "gemm_small.h"
#include "tc_common.cuh"
#include "launch.cuh"
#include "smem_limit.h"

using namespace tsb;

namespace tsb_small {
namespace {

constexpr int TM = TILE_M, TN = TILE_N, BK = 32, UMMA_K = 8;
constexpr int A_BYTES = TM * BK * 4, B_BYTES = TN * BK * 4;
constexpr int THREADS = 6 * 32;                            // warps 0..3 store, 4 issues MMAs, 5 TMA loads
constexpr int COPY_WARPS = 16;                             // warps 0..3 and twelve more where there is something TMA cannot load
constexpr int COPY_THREADS = (COPY_WARPS + 2) * 32;
constexpr int TMEM_COLS = 32;
constexpr int PART_LD = TN + 4;                            // a partial tile for the other blocks of the cluster

template <int N>
struct Group {
  CUtensorMap ta[N], tb[N];
  Product p[N];
  int first[N + 1];                 // first tile of each product
  int count, splits;
  int* status;
};

// Rows r0 .. r0 + ROWS - 1 of `n` k-blocks from k0 on by TMA: a round, whose boxes hold `kbox` k-blocks each.  In shared
// memory K-major blocks follow one another, MN-major chunks of 32 rows are `chunk_bytes` apart with all of the round's k.
template <int ROWS, bool MN>
__device__ __forceinline__ void load_tma(uint8_t* smem, const CUtensorMap* map, uint64_t* bar, const bool chunked, int kbox,
                                         int n, int chunk_bytes, int r0, int k0, int row_shift, int z) {
  if (!MN) {
    if (kbox > 1) tma_load_4d(smem, map, bar, 0, r0 + row_shift, k0 / BK, z);
    else
      for (int i = 0; i < n; ++i) tma_load_3d(smem + i * (ROWS * BK * 4), map, bar, k0 + i * BK, r0 + row_shift, z);
  } else if (chunked) {
    tma_load_4d(smem, map, bar, 0, k0 + row_shift, r0 >> 5, z);
  } else {
#pragma unroll
    for (int c = 0; c < ROWS / 32; ++c) tma_load_3d(smem + c * chunk_bytes, map, bar, r0 + c * 32, k0 + row_shift, z);
  }
}

// The same float by float, by COPY_WARPS warps: a warp copies 32 consecutive floats at a time, to where TMA would put them
// (K contiguous: rows of 128 bytes, 128B swizzle; rows contiguous: chunks of 32 rows, 128 bytes of them per k, 128B
// swizzle with 32-byte atoms).  Rows past the end of the matrix are left as they are (what they give lands in outputs
// that nobody stores); k past the end reads as zero.
template <int ROWS, bool MN>
__device__ __forceinline__ void load_copy(uint32_t smem, const float* base, long long ld, int r0, int rows, int k0, int k,
                                          int chunk_bytes, int warp, int lane) {
  auto copy = [](uint32_t dst, const float* src, bool inside) {
    if (inside) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst), "f"(0.f) : "memory");
  };
  if (!MN) {                         // a row per warp and copy: lane is k
    const bool inside = k0 + lane < k;
    const float* src = base + (r0 + warp) * ld + k0 + lane;
    const uint32_t dst = smem + warp * 128 + (((lane >> 2) ^ (warp & 7)) << 4) + (lane & 3) * 4;
#pragma unroll
    for (int j = 0; j < ROWS / COPY_WARPS; ++j, src += COPY_WARPS * ld)
      if (r0 + warp + COPY_WARPS * j < rows) copy(dst + j * (COPY_WARPS * 128), src, inside);
  } else {                           // 32 rows of one k per warp and copy
    const float* src = base + (k0 + warp) * ld + r0 + lane;
    const uint32_t dst = smem + warp * 128 + (((lane >> 3) ^ (warp & 3)) << 5) + (lane & 7) * 4;
#pragma unroll
    for (int j = 0; j < BK / COPY_WARPS; ++j, src += COPY_WARPS * ld)
#pragma unroll
      for (int h = 0; h < ROWS / 32; ++h)
        if (r0 + h * 32 + lane < rows)
          copy(dst + h * chunk_bytes + j * (COPY_WARPS * 128), src + h * 32, k0 + warp + COPY_WARPS * j < k);
  }
}

__device__ __forceinline__ float4 load_cluster(uint32_t local, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}

// `count` > 0 of four outputs; `vec`: 16-byte accesses are aligned.  bias: of these columns; relu: where max(output, 0) goes.
__device__ __forceinline__ void store4(float* dst, int count, bool vec, bool accumulate, float4 s, const float* bias,
                                       float* relu) {
  if (bias) {                        // (16-byte aligned; past the last column it is not read)
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (count >= 4) {
      x = tsb_launch::load(reinterpret_cast<const float4*>(bias));
    } else {
      x.x = tsb_launch::load(bias);
      if (count > 1) x.y = tsb_launch::load(bias + 1);
      if (count > 2) x.z = tsb_launch::load(bias + 2);
    }
    s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
  }
  if (relu) {
    const float4 r = make_float4(fmaxf(s.x, 0.f), fmaxf(s.y, 0.f), fmaxf(s.z, 0.f), fmaxf(s.w, 0.f));
    if (vec && count >= 4) {
      *reinterpret_cast<float4*>(relu) = r;
    } else {
      relu[0] = r.x;
      if (count > 1) relu[1] = r.y;
      if (count > 2) relu[2] = r.z;
      if (count > 3) relu[3] = r.w;
    }
  }
  if (vec && count >= 4) {
    if (accumulate) {
      const float4 old = *reinterpret_cast<const float4*>(dst);
      s.x += old.x; s.y += old.y; s.z += old.z; s.w += old.w;
    }
    *reinterpret_cast<float4*>(dst) = s;
  } else {
    const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < count) dst[j] = accumulate ? dst[j] + v[j] : v[j];
  }
}

template <int N, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(COPY_THREADS) gemm_small_kernel(const __grid_constant__ Group<N> grp) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full[MAX_KBLOCKS / ROUND], done;
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(16) float part[TM * PART_LD];
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  const int splits = grp.splits, rank = splits > 1 ? (int)blockIdx.x % splits : 0;
  int item = splits > 1 ? (int)blockIdx.x / splits : (int)blockIdx.x, which = 0;
  if (N > 1)
    while (which + 1 < grp.count && grp.first[which + 1] <= item) ++which;
  const Product& p = grp.p[which];
  if (threadIdx.x == 5 * 32) {
    if (p.a.tma) tma_prefetch_desc(&grp.ta[which]);
    if (p.b.tma) tma_prefetch_desc(&grp.tb[which]);
  }
  const bool tma_a = p.a.tma != 0, tma_b = p.b.tma != 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_KBLOCKS / ROUND; ++s) mbar_init(&full[s], tma_a && tma_b ? 1 : 1 + COPY_WARPS);
    mbar_init(&done, 1);
    fence_barrier_init();
  }
  if (warp == 4) {
    tmem_alloc(&tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  item -= grp.first[which];
  const int tiles = p.tiles_m * p.tiles_n, z = p.batch > 1 ? item / tiles : 0;
  item -= z * tiles;
  const int m0 = item / p.tiles_n * TM, n0 = item % p.tiles_n * TN;
  const int o = p.batch > 1 ? z / p.inner : 0, in = z - o * p.inner;
  const int k = p.k, kblocks = (k + BK - 1) / BK, kb0 = rank * p.kb_per_split, kb1 = min(kblocks, kb0 + p.kb_per_split);
  const int blocks = kb1 - kb0, round = min(ROUND, p.kb_per_split), rounds = (blocks + round - 1) / round;
  const int chunk_bytes = round * BK * 128;                // (MN-major)
  // (parameters are read here, under the tail of the kernel before)
  const bool vec_c = p.vec_c != 0, accumulate = p.accumulate != 0;
  const int rows_left = p.m - m0, cols_left = p.n - n0;
  const long long ldc = p.ldc;
  float* c = p.c + o * p.sc2 + in * p.sc + m0 * ldc + n0;
  const float* bias = p.bias ? p.bias + n0 : nullptr;
  float* relu = p.relu ? p.relu + o * p.sc2 + in * p.sc + m0 * ldc + n0 : nullptr;
  int* status = grp.status;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t s0 = smem_u32(smem), sb0 = s0 + rounds * round * A_BYTES;

  if (warp == 5) {
    const bool chunked_a = p.a.chunked != 0, chunked_b = p.b.chunked != 0;
    const int za = p.a.heads ? in : z, zb = p.b.heads ? in : z, ra = o * p.a.shift, rb = o * p.b.shift;
    const int kbox_a = p.a.kbox, kbox_b = p.b.kbox;
    tsb_launch::enter();
    if ((tma_a || tma_b) && elect_one()) {
      for (int r = 0; r < rounds; ++r) {
        const int at = r * round, n = min(round, blocks - at), k0 = (kb0 + at) * BK;
        // (a box past the end brings zeros and counts in full)
        const int na = A_MN || kbox_a > 1 ? round : n, nb = B_MN || kbox_b > 1 ? round : n;
        mbar_expect_tx(&full[r], (tma_a ? na * A_BYTES : 0) + (tma_b ? nb * B_BYTES : 0));
        if (tma_a) load_tma<TM, A_MN>(smem + at * A_BYTES, &grp.ta[which], &full[r], chunked_a, kbox_a, n, chunk_bytes, m0, k0, ra, za);
        if (tma_b) load_tma<TN, B_MN>(smem + rounds * round * A_BYTES + at * B_BYTES, &grp.tb[which], &full[r], chunked_b, kbox_b, n,
                                      chunk_bytes, n0, k0, rb, zb);
      }
    }
  } else if (warp == 4) {
    constexpr uint32_t idesc = make_idesc_tf32(TM, TN, A_MN, B_MN);
    constexpr uint32_t A_HI = A_MN ? smem_desc_hi(512, LAYOUT_SW128_BASE32B) : smem_desc_hi(1024);
    constexpr uint32_t B_HI = B_MN ? smem_desc_hi(512, LAYOUT_SW128_BASE32B) : smem_desc_hi(1024);
    constexpr uint32_t A_KSTEP = (A_MN ? 1024 : UMMA_K * 4) >> 4, B_KSTEP = (B_MN ? 1024 : UMMA_K * 4) >> 4;
    // from one k-block to the next: K-major a block further, MN-major 32 rows of k inside the round's chunks
    constexpr uint32_t A_NEXT = (A_MN ? BK * 128 : A_BYTES) >> 4, B_NEXT = (B_MN ? BK * 128 : B_BYTES) >> 4;
    const uint32_t a_lo0 = smem_desc_lo(s0, A_MN ? chunk_bytes : 16), b_lo0 = smem_desc_lo(sb0, B_MN ? chunk_bytes : 16);
    tsb_launch::enter();
    if (elect_one()) {
      for (int r = 0; r < rounds; ++r) {
        if (!mbar_wait(&full[r], 0, status, 0x110)) {
          for (int i = 0; i < 64; ++i) __nanosleep(1000);      // let copies that are still in flight land
          break;
        }
        tc_fence_after();
        uint32_t a_lo = a_lo0 + r * round * (A_BYTES >> 4), b_lo = b_lo0 + r * round * (B_BYTES >> 4);
        const int left = min(blocks * BK, k - kb0 * BK) - r * round * BK;      // of K, in and behind this round
        int at = 0;
        for (; at < round && (at + 1) * BK <= left; ++at, a_lo += A_NEXT, b_lo += B_NEXT)
#pragma unroll
          for (int s = 0; s < BK / UMMA_K; ++s)
            umma_tf32(tmem, smem_desc_join(A_HI, a_lo + s * A_KSTEP), smem_desc_join(B_HI, b_lo + s * B_KSTEP), idesc,
                      (r > 0 || at > 0 || s > 0) ? 1u : 0u);
        if (at < round)
          for (int s = 0; at * BK + s * UMMA_K < left; ++s)
            umma_tf32(tmem, smem_desc_join(A_HI, a_lo + s * A_KSTEP), smem_desc_join(B_HI, b_lo + s * B_KSTEP), idesc,
                      (r > 0 || at > 0 || s > 0) ? 1u : 0u);
      }
      umma_commit(&done);            // (also after a wait that ran out: the storing warps go on)
    }
  } else {
    const float* a = p.a.base + o * p.a.s2 + in * p.a.s;
    const float* b = p.b.base + o * p.b.s2 + in * p.b.s;
    const long long lda = p.a.ld, ldb = p.b.ld;
    const int m = p.m, n = p.n, cw = warp < 4 ? warp : warp - 2;
    tsb_launch::enter();
    if (!(tma_a && tma_b)) {
      for (int r = 0; r <= rounds; ++r) {
        if (r < rounds)
          for (int i = r * round; i < min(blocks, r * round + round); ++i) {
            const int in_round = (i - r * round) * (BK * 128);
            if (!tma_a)
              load_copy<TM, A_MN>(A_MN ? s0 + r * round * A_BYTES + in_round : s0 + i * A_BYTES, a, lda, m0, m, (kb0 + i) * BK, k,
                                  chunk_bytes, cw, lane);
            if (!tma_b)
              load_copy<TN, B_MN>(B_MN ? sb0 + r * round * B_BYTES + in_round : sb0 + i * B_BYTES, b, ldb, n0, n, (kb0 + i) * BK, k,
                                  chunk_bytes, cw, lane);
          }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (r > 0) {                 // the round before this one is in shared memory
          asm volatile("cp.async.wait_group 1;" ::: "memory");
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&full[r - 1]);
            if (cw == 0 && !tma_a && !tma_b) mbar_arrive(&full[r - 1]);      // (in the place of the TMA thread)
          }
        }
      }
    }
    if (warp < 4) {
      // TMEM lanes 32 w .. 32 w + 15 hold rows 16 w .. 16 w + 15 of a 64-row tile
      bool ok = true;
      if (lane == 0) ok = mbar_wait(&done, 0, status, 0x111);
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      tc_fence_after();
      float v[TN];
      tmem_ld_32x32(tmem + ((uint32_t)(warp * 32) << 16), v);
      tmem_ld_wait();
      // (a thread has 32 columns of one row; through shared memory, stores of a warp are whole lines)
      if (lane < 16) {
#pragma unroll
        for (int j = 0; j < TN; j += 4)
          *reinterpret_cast<float4*>(part + (warp * 16 + lane) * PART_LD + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
      __syncwarp();
      if (splits == 1 && ok) {
        const int col = (lane & 7) * 4;
        int row = warp * 16 + (lane >> 3);
        float* dst = c + row * ldc + col;
        if (vec_c && cols_left >= TN && !accumulate && !bias && !relu) {
#pragma unroll
          for (int j = 0; j < 4; ++j, row += 4, dst += 4 * ldc)
            if (row < rows_left) *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(part + row * PART_LD + col);
        } else {
          for (int j = 0; j < 4; ++j, row += 4, dst += 4 * ldc)
            if (row < rows_left && col < cols_left)
              store4(dst, cols_left - col, vec_c, accumulate, *reinterpret_cast<const float4*>(part + row * PART_LD + col),
                     bias ? bias + col : nullptr, relu ? relu + (dst - c) : nullptr);
        }
      }
      tc_fence_before();
    }
  }
  __syncwarp();
  if (splits > 1) {
    cluster_sync_all();
    for (int e = rank * blockDim.x + threadIdx.x; e < TM * TN / 4; e += splits * blockDim.x) {
      const int row = e / (TN / 4), col = e % (TN / 4) * 4;
      if (row >= rows_left || col >= cols_left) continue;
      const uint32_t at = smem_u32(part + row * PART_LD + col);
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f), v[MAX_SPLITS];
#pragma unroll
      for (int u = 0; u < MAX_SPLITS; ++u)
        if (u < splits) v[u] = load_cluster(at, u);
#pragma unroll
      for (int u = 0; u < MAX_SPLITS; ++u)
        if (u < splits) { s.x += v[u].x; s.y += v[u].y; s.z += v[u].z; s.w += v[u].w; }
      store4(c + row * ldc + col, cols_left - col, vec_c, accumulate, s, bias ? bias + col : nullptr,
             relu ? relu + row * ldc + col : nullptr);
    }
    __syncwarp();
    cluster_sync_all();              // the partial sums stay until everybody has read them
  } else {
    __syncthreads();
  }
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

template <int N, bool A_MN, bool B_MN>
cudaError_t launch(const Group<N>& g, int tiles, int smem, bool copies, cudaStream_t st) {
  auto kern = gemm_small_kernel<N, A_MN, B_MN>;
  static tsb_launch::SmemLimit limit;
  const cudaError_t e = limit.raise(kern, smem_of(MAX_KBLOCKS));
  if (e != cudaSuccess) return e;
  return tsb_launch::launch_cluster(g.splits > 1 ? (unsigned)g.splits : 0u, kern, dim3((unsigned)(tiles * g.splits)),
                                    dim3(copies ? COPY_THREADS : THREADS), smem, st, g);
}

template <int N>
cudaError_t run_group(Product* p, const CUtensorMap* ta, const CUtensorMap* tb, int count, int splits, bool trans_a,
                      bool trans_b, int* status, cudaStream_t st) {
  Group<N> g;
  g.count = count;
  g.splits = splits;
  g.status = status;
  int tiles = 0, smem = 0;
  bool copies = false;
  for (int i = 0; i < count; ++i) {
    Product& q = p[i];
    q.tiles_m = (q.m + TM - 1) / TM;
    q.tiles_n = (q.n + TN - 1) / TN;
    q.vec_c = ((reinterpret_cast<uintptr_t>(q.c) | reinterpret_cast<uintptr_t>(q.relu)) & 15) == 0 && q.ldc % 4 == 0 &&
              (q.batch == 1 || (q.sc % 4 == 0 && q.sc2 % 4 == 0));
    g.p[i] = q;
    copies = copies || !q.a.tma || !q.b.tma;
    if (q.a.tma) g.ta[i] = ta[i];
    if (q.b.tma) g.tb[i] = tb[i];
    g.first[i] = tiles;
    tiles += q.tiles_m * q.tiles_n * q.batch;
    if (smem_of(q.kb_per_split) > smem) smem = smem_of(q.kb_per_split);
  }
  g.first[count] = tiles;
  if (!trans_a && !trans_b) return launch<N, false, true>(g, tiles, smem, copies, st);
  if (!trans_a && trans_b) return launch<N, false, false>(g, tiles, smem, copies, st);
  if (trans_a && !trans_b) return launch<N, true, true>(g, tiles, smem, copies, st);
  return launch<N, true, false>(g, tiles, smem, copies, st);
}

}  // namespace

cudaError_t run(Product* p, const CUtensorMap* ta, const CUtensorMap* tb, int count, int splits, bool trans_a, bool trans_b,
                int* status, cudaStream_t st) {
  return count == 1 ? run_group<1>(p, ta, tb, count, splits, trans_a, trans_b, status, st)
                    : run_group<MAX_PRODUCTS>(p, ta, tb, count, splits, trans_a, trans_b, status, st);
}

}  // namespace tsb_small
