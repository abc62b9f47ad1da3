// Float32 matrix product  C[M, N] = A[M, K] * W[N, K]^T  on the 5th-generation tensor cores, for weights of
// at least 1,024 x 1,024 (gemm_f32.cu has the others).
//
// A float32 number times 2^16 is exactly the sum of three bfloat16 ones (hi + mid + lo, each the rest rounded to nearest), and a
// product of two numbers is six of the nine products of their parts; the three left out come to 2^-24 of it at most, to
// 2^-27 on average (root mean square).  Products of bfloat16 are exact in float32, but what a tensor core adds up it rounds toward zero.  So
// hi * hi has a tensor-memory tile of its own, which starts from nothing every 64 columns of k: its sums of 16-bit numbers lose
// little.  The five small products of a segment (an eighth of the chunks of k) are added up in another, where what is
// cut off is 2^-8 of that.  The sums are read back and added with rounding to nearest: in ascending order within a segment, and the
// segments in ascending order.  That order depends on K alone: an element's value does not depend on M, on the tile it falls
// in or on how many blocks share the sum.  Errors against float64 are in the comment at fg_gemm_f32_split.
//
// The weights' rows are the 128 rows of the tensor core's tile, the rows of A its columns (T of them):
// 777 rows against 128,256 x 2,048: 7,870 -> 1,966 us; 5 rows: 287 -> 180 (bytes: 160).  What bounds it now is the way
// from L2: a chunk brings 32 KB of W and 384 T bytes of A's parts to a block for 12 T cycles of products.
//
//   load warp:      TMA of W (float32, 128 rows x 64) into a ring of three, and of A's parts
//   8 worker warps: W's numbers -> parts -> tensor memory (the product's left operand); the partial sums of the chunk
//                   before -> registers
//   MMA warp:       24 tcgen05.mma a chunk (6 products x 4 steps of 16)
// The left operand in tensor memory leaves shared memory to A's parts: each of them is read once a product.
// hi * hi comes last in a chunk: its sums are read during the next chunk's small products, the small ones' during the hi * hi that
// ends their segment, so that one tile of each is enough.
// Few rows (T <= 32): the workers also split A; two blocks an SM, bound by reading W.  More rows: A is split once by
// a kernel of its own, and the tensor core is what bounds the rest.
// Where the tiles are too few for the chip, a cluster of two, four or eight blocks shares a tile, its segments evenly, and
// adds the segments up over distributed shared memory.
//
// An element that is not finite (an infinity or NaN among its inputs, numbers of 2^111 and more, or an overflow) is computed
// again with float32 multiply-adds in ascending k: the parts of an infinity are an infinity and NaNs.  A block does that
// when all its tiles are stored and it waits for nothing any more.
#include "tc5_primitives.cuh"
#include "tensor_map.cuh"

namespace {
using namespace fg_tc5;

constexpr int ROWS = 128;     // rows of W a tile
constexpr int KC = 64;        // columns of k a chunk
constexpr int SEGMENTS = 8;   // stretches of chunks whose sums are added last
constexpr int W_BOX = ROWS * 128, W_STAGE = 2 * W_BOX;
constexpr int WORKERS = 256, THREADS_ALL = WORKERS + 64, LOAD_WARP_ID = 8, MMA_WARP_ID = 9;
constexpr int A_COLS = 96;    // tensor-memory columns of a chunk of W: three parts of 64 bfloat16
// What operands are multiplied by before they are split, and what that leaves on a sum.  Float32's smallest number is then
// bfloat16's smallest, and the smallest result, 2^-149, is 2^-117 in the sums, inside float32's normal range.
constexpr float SCALE = 0x1p16f, UNSCALE = 0x1p-32f;

// T rows of A a tile; SHARE blocks (a cluster) share a tile
template <int T_, int SHARE_>
struct Shape {
  static constexpr int T = T_, TC = T / 2;        // columns a worker thread keeps
  static constexpr int SHARE = SHARE_, OWN = SEGMENTS / SHARE;  // segments a block sums
  static constexpr bool SPLIT_HERE = T <= 32;     // A is split by the workers
  static constexpr bool SUM_IN_SMEM = T > 112 && SHARE == 1;  // the finished segments' sum (else in registers)
  static constexpr int W_STAGES = T == 32 || SUM_IN_SMEM ? 2 : 3;  // (two blocks an SM at T <= 32)
  static constexpr int UNIT = T * 128;            // bytes of one part of A's chunk
  static constexpr int UNITS = SPLIT_HERE ? 6 : T <= 64 ? 9 : T <= 112 ? 8 : SUM_IN_SMEM ? 4 : 6;
  static constexpr int BLOCKS = SPLIT_HERE ? 2 : 1;
  static constexpr int COL_A = 2 * T, TMEM = SPLIT_HERE ? 256 : 512;
  static constexpr int RINGS = W_STAGES * W_STAGE + UNITS * UNIT;
  static constexpr size_t SMEM = 1024 + RINGS + (SUM_IN_SMEM ? T * ROWS * 4 : 0);
  static_assert(COL_A + 2 * A_COLS <= TMEM && SMEM <= 231 * 1024, "");
  static_assert(SHARE == 1 || OWN * T * ROWS * 4 <= RINGS, "the exchange of a cluster reuses the rings");
};

__device__ __forceinline__ void tma_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];\n" ::"r"(smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}
// asks for a box in L2 only: also safe while a kernel before this one is still writing what it covers
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];\n" ::"l"(map), "r"(c0), "r"(c1) : "memory");
}
// 8 consecutive columns of this thread's lane; several may be in flight before tmem_ld_wait
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

// one arrival for the warp: arrivals on one barrier come one after the other, and three times 256 of them were half of a
// chunk's time
__device__ __forceinline__ void warp_arrive(uint64_t* bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

__device__ __forceinline__ uint32_t cvt_pair(float a, float b) {  // a in the lower half
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ uint64_t pair_of(float a, float b) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  return v;
}
// a pair of numbers and its rest, both float32, from the pair's bfloat16 (exact)
__device__ __forceinline__ uint32_t take_part(uint64_t& v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  const uint32_t part = cvt_pair(a, b);
  const uint64_t wide = pair_of(__uint_as_float(part << 16), __uint_as_float(part & 0xffff0000u));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(wide), "l"(pair_of(-1.f, -1.f)));
  return part;
}
// two numbers, times SCALE -> their three parts, packed
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  uint64_t v = pair_of(a, b);
  asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(pair_of(SCALE, SCALE)));
  hi = take_part(v);
  mid = take_part(v);
  lo = take_part(v);
}
// byte offset of the 16-byte piece `piece` of a row of 128 bytes in a swizzled tile
__device__ __forceinline__ int swizzled(int row, int piece) { return row * 128 + ((piece ^ (row & 7)) << 4); }

__device__ __forceinline__ bool finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

// The elements of C that are not finite, in the columns n0 .. n0 + ROWS - 1 of the rows m0, m0 + step, ... (`count` of them, all
// stored by this block), once more with multiply-adds in ascending k.  Called by the whole block when it waits for nothing any
// more: rows of A with a NaN give NaNs; the other rows that hold such an element go sixteen at a time, eight elements of one
// column a thread, so that a reading of W's 128 rows serves sixteen, the next 64 columns of k on their way meanwhile.  (5 rows
// against 2,048 x 2,048, all infinite: 443 us with a lane an element and W's rows side by side, here 207; 777 rows against 16,384 x
// 2,048 5,583, and 441 with a NaN in one row.)
constexpr int R_ROWS = 16, R_K = 64, R_LD = R_K + 4;
template <int T>
__device__ __noinline__ void repair(float* smem, const float* A, int lda, const float* W, int ldw, float* C, int ldc, int n0, int m0,
                                    int step, int count, int N, int K, const float* bias) {
  __shared__ int bad_rows[T], n_bad;
  float* const ws = smem;                   // [ROWS][R_LD]
  float* const as = smem + ROWS * R_LD;     // [R_ROWS][R_K]
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) n_bad = 0;
  __syncthreads();
  if (tid < WORKERS)
    for (int i = tid >> 5; i < count; i += WORKERS / 32) {
      const int m = m0 + i * step;
      float* c = C + (size_t)m * ldc + n0;
      bool bad = false, nan = false;
      for (int n = lane; n < min(ROWS, N - n0); n += 32) bad = bad || !finite(c[n]);
      if (!__any_sync(0xffffffffu, bad)) continue;
      const float* a = A + (size_t)m * lda;
#pragma unroll 4
      for (int k = lane * 4; k < K; k += 128) {
        const float4 v = *reinterpret_cast<const float4*>(a + k);
        nan = nan || v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w;
      }
      if (__any_sync(0xffffffffu, nan)) {
        for (int n = lane; n < min(ROWS, N - n0); n += 32) c[n] = __uint_as_float(0x7fffffffu);
      } else if (lane == 0) {
        bad_rows[atomicAdd(&n_bad, 1)] = m;
      }
    }
  __syncthreads();
  const int rows = n_bad, col = tid & (ROWS - 1), part = tid / ROWS, n = n0 + col;
  constexpr int PIECES = (ROWS + R_ROWS) * (R_K / 4) / WORKERS;  // of 16 bytes, a thread: the last is of A
  static_assert(PIECES * WORKERS == (ROWS + R_ROWS) * (R_K / 4) && R_ROWS * (R_K / 4) == WORKERS, "");
  const int row = tid / (R_K / 4), quad = tid % (R_K / 4);  // a thread's first piece; the others are 16 rows apart
  for (int r0 = 0; r0 < rows; r0 += R_ROWS) {
    float4 next[PIECES];
    auto fetch = [&](int k0) {
      const int k = k0 + 4 * quad;
#pragma unroll
      for (int i = 0; i < PIECES; ++i) {
        const bool ok = k < K && (i < PIECES - 1 ? n0 + row + 16 * i < N : r0 + row < rows);
        const float* src = i < PIECES - 1 ? W + (size_t)(n0 + row + 16 * i) * ldw : A + (size_t)(ok ? bad_rows[r0 + row] : 0) * lda;
        next[i] = ok ? *reinterpret_cast<const float4*>(src + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    float v[R_ROWS / 2];
#pragma unroll
    for (int i = 0; i < R_ROWS / 2; ++i) v[i] = 0.f;
    if (tid < WORKERS) fetch(0);
    for (int k0 = 0; k0 < K; k0 += R_K) {
      const int quads = min(R_K, K - k0) / 4;
      __syncthreads();  // the columns of k before are read
      if (tid < WORKERS) {
#pragma unroll
        for (int i = 0; i < PIECES - 1; ++i) *reinterpret_cast<float4*>(ws + (row + 16 * i) * R_LD + 4 * quad) = next[i];
        *reinterpret_cast<float4*>(as + row * R_K + 4 * quad) = next[PIECES - 1];
      }
      __syncthreads();
      if (tid < WORKERS) {
        if (k0 + R_K < K) fetch(k0 + R_K);
        for (int q = 0; q < quads; ++q) {
          const float4 w = *reinterpret_cast<const float4*>(ws + col * R_LD + 4 * q);
#pragma unroll
          for (int i = 0; i < R_ROWS / 2; ++i) {
            const float4 a = *reinterpret_cast<const float4*>(as + (part * (R_ROWS / 2) + i) * R_K + 4 * q);
            v[i] = fmaf(a.x, w.x, v[i]);
            v[i] = fmaf(a.y, w.y, v[i]);
            v[i] = fmaf(a.z, w.z, v[i]);
            v[i] = fmaf(a.w, w.w, v[i]);
          }
        }
      }
    }
    if (tid < WORKERS && n < N)
#pragma unroll
      for (int i = 0; i < R_ROWS / 2; ++i) {
        const int r = r0 + part * (R_ROWS / 2) + i;
        if (r >= rows) break;
        float* c = C + (size_t)bad_rows[r] * ldc + n;
        if (!finite(*c)) *c = bias != nullptr ? v[i] + bias[n] : v[i];
      }
  }
  __syncthreads();  // the list of rows is read
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_16(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(remote)
               : "memory");
  return v;
}

// With several blocks a tile, block r of them sums segments r OWN, ... one by one.  Otherwise a block walks the tiles blockIdx.x,
// blockIdx.x + gridDim.x, ...: the chunks of its tiles are one long sequence, so that the next tile's loads and
// products run while the workers store the last one's sums.
template <typename S>
__global__ void __launch_bounds__(THREADS_ALL, S::BLOCKS)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map,
                      const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                      const float* bias, int m_tiles, int tiles, int* status) {
  constexpr int T = S::T, TC = S::TC, W_STAGES = S::W_STAGES;
  constexpr bool CLUSTERED = S::SHARE > 1;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* const ws = reinterpret_cast<unsigned char*>(((uintptr_t)smem_unaligned + 1023) & ~(uintptr_t)1023);
  unsigned char* const as = ws + W_STAGES * W_STAGE;
  // w_full / w_empty: a stage of W; a_full / a_empty: a part of A (SPLIT_HERE: unused); op_full: the parts of a chunk of W
  // are in tensor memory; d_full / d_empty: a chunk's sums of hi * hi; small_full / small_empty: a segment's other sums
  __shared__ __align__(8) uint64_t w_full[W_STAGES], w_empty[W_STAGES], a_full[S::UNITS], a_empty[S::UNITS], op_full[2],
      d_full, d_empty, small_full, small_empty, drained;
  __shared__ uint32_t tmem_base;
  __shared__ int gave_up, any_bad;  // any_bad: an element that is not finite was stored
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

  pdl_trigger();
  if (warp == MMA_WARP_ID) {
    tmem_alloc(&tmem_base, S::TMEM);
    tmem_relinquish();
  }
  if (tid == 0) {
    gave_up = any_bad = 0;
    for (int i = 0; i < W_STAGES; ++i) {
      mbar_init(&w_full[i], 1);
      mbar_init(&w_empty[i], WORKERS / 32);
    }
    for (int i = 0; i < S::UNITS; ++i) {
      mbar_init(&a_full[i], 1);
      mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) mbar_init(&op_full[i], WORKERS / 32);
    mbar_init(&d_full, 1);
    mbar_init(&d_empty, WORKERS / 32);
    mbar_init(&small_full, 1);
    mbar_init(&small_empty, WORKERS / 32);
    mbar_init(&drained, 1);
    mbar_fence_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);

  // the block's chunks: `per_tile` of each of its tiles, from chunk `first` on
  const int chunks = (K + KC - 1) / KC, per_segment = (chunks + SEGMENTS - 1) / SEGMENTS;
  const int rank = CLUSTERED ? (int)cluster_rank() : 0;
  const int tile0 = blockIdx.x / S::SHARE, tile_step = CLUSTERED ? tiles : gridDim.x;
  const int first = rank * S::OWN * per_segment;
  const int per_tile = max(0, min(S::OWN * per_segment, chunks - first));
  const int total = tile0 < tiles ? ((tiles - 1 - tile0) / tile_step + 1) * per_tile : 0;

  if (warp == LOAD_WARP_ID) {
    if (elect_one()) {
      int wt = tile0, wc = 0, ws_slot = 0, w_use = 0;  // the next chunk of W: tile, chunk of it, stage, uses of the stage before
      auto load_w = [&]() {
        if (w_use > 0) mbar_wait(&w_empty[ws_slot], (w_use - 1) & 1, status, &gave_up);
        mbar_arrive_expect(&w_full[ws_slot], W_STAGE);
        const int n0 = wt / m_tiles * ROWS, k0 = (first + wc) * KC;
        tma_2d(ws + ws_slot * W_STAGE, &w_map, k0, n0, &w_full[ws_slot]);
        tma_2d(ws + ws_slot * W_STAGE + W_BOX, &w_map, k0 + 32, n0, &w_full[ws_slot]);
        if (++wc == per_tile) {
          wc = 0;
          wt += tile_step;
        }
        if (++ws_slot == W_STAGES) {
          ws_slot = 0;
          ++w_use;
        }
      };
      for (int j = 0; j < min(W_STAGES, total); ++j) {  // while the kernels before this one end
        const int n0 = (tile0 + j / per_tile * tile_step) / m_tiles * ROWS, k0 = (first + j % per_tile) * KC;
        tma_prefetch_2d(&w_map, k0, n0);
        tma_prefetch_2d(&w_map, k0 + 32, n0);
      }
      pdl_wait();
      for (int j = 0; j < min(W_STAGES, total); ++j) load_w();
      int slot = 0, use = 0, tile = tile0, c = 0;
      for (int j = 0; j < total; ++j) {
        if (!S::SPLIT_HERE) {
          const int m0 = tile % m_tiles * T, k0 = (first + c) * KC;
#pragma unroll 1
          for (int p = 0; p < 3; ++p) {  // in the order of their use: lo, mid, hi
            if (use > 0) mbar_wait(&a_empty[slot], (use - 1) & 1, status, &gave_up);
            mbar_arrive_expect(&a_full[slot], S::UNIT);
            tma_3d(as + slot * S::UNIT, &a_map, k0, m0, 2 - p, &a_full[slot]);
            if (++slot == S::UNITS) {
              slot = 0;
              ++use;
            }
          }
          if (++c == per_tile) {
            c = 0;
            tile += tile_step;
          }
        }
        if (j + W_STAGES < total) load_w();
      }
      if (*reinterpret_cast<volatile int*>(&gave_up) != 0) {
        // a wait ran out: the copies in flight land before the block leaves
        for (int i = 0; i < min(W_STAGES, total); ++i) mbar_wait(&w_full[i], (total - 1 - i) / W_STAGES & 1, status);
        if (!S::SPLIT_HERE)
          for (int i = 0; i < min(S::UNITS, 3 * total); ++i)
            mbar_wait(&a_full[i], (3 * total - 1 - i) / S::UNITS & 1, status);
      }
    }
    __syncwarp();
  } else if (warp == MMA_WARP_ID) {
    if (elect_one()) {
      constexpr uint32_t IDESC = instr_desc(T, false);
      const uint64_t a_desc = smem_desc(as, 16);
      int slot = 0, use = 0, c = 0, in_segment = 0, segments = 0;  // (segments: those begun before this one)
      for (int j = 0; j < total; ++j) {
        const int buf = j & 1;
        const uint32_t small = tmem, d = tmem + T, op = tmem + S::COL_A + buf * A_COLS;
        const bool last = in_segment + 1 == per_segment || c + 1 == per_tile;  // chunk of its segment
        mbar_wait(&op_full[buf], (j >> 1) & 1, status, &gave_up);
        if (in_segment == 0 && segments > 0) mbar_wait(&small_empty, (segments - 1) & 1, status, &gave_up);
        tc_fence_after();
#pragma unroll
        for (int p = 0; p < 3; ++p) {  // A's lo, mid, hi
          const int unit = S::SPLIT_HERE ? buf * 3 + p : slot;
          if (!S::SPLIT_HERE) {
            mbar_wait(&a_full[slot], use & 1, status, &gave_up);
            tc_fence_after();
          }
          const uint64_t bd = a_desc + (uint64_t)((unit * S::UNIT) >> 4);
#pragma unroll
          for (int q = p; q >= 0; --q) {  // W's part q (0: hi): lo * hi; mid * mid, mid * hi; hi * lo, hi * mid, hi * hi
            const bool main = p == 2 && q == 0;
            if (main) {
              if (last) umma_commit(&small_full);
              if (j > 0) {
                mbar_wait(&d_empty, (j - 1) & 1, status, &gave_up);
                tc_fence_after();
              }
            }
#pragma unroll
            for (int kk = 0; kk < KC / 16; ++kk)
              umma_f16_ts(main ? d : small, op + q * 32 + kk * 8, bd + (uint64_t)(kk * 32 >> 4), IDESC,
                          main ? (kk > 0 ? 1u : 0u) : (p > 0 || kk > 0 || in_segment > 0 ? 1u : 0u));
          }
          if (!S::SPLIT_HERE) {
            umma_commit(&a_empty[slot]);
            if (++slot == S::UNITS) {
              slot = 0;
              ++use;
            }
          }
        }
        umma_commit(&d_full);
        if (last) {
          in_segment = 0;
          ++segments;
        } else {
          ++in_segment;
        }
        if (++c == per_tile) c = 0;
      }
      if (*reinterpret_cast<volatile int*>(&gave_up) != 0) {
        umma_commit(&drained);
        mbar_wait(&drained, 0, status);
      }
    }
    __syncwarp();
  } else {
    // ================================ workers ================================
    const int half = warp >> 2, row = (warp & 3) * 32 + lane;  // half of a chunk's k, then of a tile's columns
    const uint32_t my_lane = (uint32_t)((warp & 3) * 32) << 16;
    // a segment's sum so far; the sum of the finished segments (SHARE == 1), or each of them
    float acc[TC], sum[CLUSTERED ? S::OWN : 1][S::SUM_IN_SMEM || (CLUSTERED && S::OWN == 1) ? 1 : TC];
    float* const sum_smem = reinterpret_cast<float*>(ws + S::RINGS) + half * TC * ROWS + row;
#pragma unroll
    for (int i = 0; i < TC; ++i) acc[i] = 0.f;
    pdl_wait();  // A comes from the kernels before, and C may still be read by them
    // SPLIT_HERE: this thread's numbers of A of the next chunk: rows a_row, a_row + 16, four columns
    constexpr int A_LOADS = S::SPLIT_HERE ? T / 16 : 1;
    const int a_row = tid >> 4, a_k = (tid & 15) * 4;
    float4 a_next[A_LOADS];
    int load_c = 0;
    auto fetch_a = [&]() {
      const int k = (first + load_c) * KC + a_k;
#pragma unroll
      for (int u = 0; u < A_LOADS; ++u) {
        const int m = u * 16 + a_row;  // (one tile holds all rows)
        a_next[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m < M && k < K) a_next[u] = *reinterpret_cast<const float4*>(A + (size_t)m * lda + k);
      }
      if (++load_c == per_tile) load_c = 0;
    };
    if (S::SPLIT_HERE && total > 0) fetch_a();
    int slot = 0, use = 0, tile = tile0, c = 0, in_segment = 0, segment = 0, segments = 0;  // (of the tile, of all)
    for (int j = 0; j <= total; ++j) {
      if (j < total) {
        const int buf = j & 1;
        mbar_wait(&w_full[slot], use & 1, status, &gave_up);
        const unsigned char* src = ws + slot * W_STAGE + half * W_BOX + row * 128;
        const uint32_t op = tmem + my_lane + S::COL_A + buf * A_COLS + half * 16;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t hi[8], mid[8], lo[8];
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const float4 w = *reinterpret_cast<const float4*>(src + (((h * 4 + p) ^ (row & 7)) << 4));
            split_pair(w.x, w.y, hi[2 * p], mid[2 * p], lo[2 * p]);
            split_pair(w.z, w.w, hi[2 * p + 1], mid[2 * p + 1], lo[2 * p + 1]);
          }
          tmem_st8(op + h * 8, hi);
          tmem_st8(op + 32 + h * 8, mid);
          tmem_st8(op + 64 + h * 8, lo);
        }
        warp_arrive(&w_empty[slot]);
        if (++slot == W_STAGES) {
          slot = 0;
          ++use;
        }
        if (S::SPLIT_HERE) {
#pragma unroll
          for (int u = 0; u < A_LOADS; ++u) {
            uint2 part[3];
            split_pair(a_next[u].x, a_next[u].y, part[0].x, part[1].x, part[2].x);
            split_pair(a_next[u].z, a_next[u].w, part[0].y, part[1].y, part[2].y);
            const int r = u * 16 + a_row;
#pragma unroll
            for (int p = 0; p < 3; ++p)
              *reinterpret_cast<uint2*>(as + (buf * 3 + 2 - p) * S::UNIT + swizzled(r, a_k >> 3) + (a_k & 4) * 2) = part[p];
          }
          fence_async_smem();  // written by ordinary stores, read by the tensor core
        }
        tmem_st_wait();
        tc_fence_before();
        warp_arrive(&op_full[buf]);
        if (S::SPLIT_HERE && j + 1 < total) fetch_a();
      }
      if (j == 0) continue;
      // the sums of the chunk before (and of its segment, where it is the last): tensor memory -> acc
      auto add_sums = [&](uint32_t col, uint64_t* full, uint64_t* empty, int parity) {
        mbar_wait(full, parity, status, &gave_up);
        tc_fence_after();
        const uint32_t d = tmem + my_lane + col + half * TC;
        constexpr int G = TC < 48 ? TC : 16;  // columns in flight: what the registers leave
#pragma unroll
        for (int g = 0; g < TC; g += G) {
          uint32_t v[G];
#pragma unroll
          for (int i = 0; i < G && g + i < TC; i += 8) tmem_ld8(d + g + i, v + i);
          tmem_ld_wait();
          if (g + G >= TC) {
            tc_fence_before();
            warp_arrive(empty);
          }
#pragma unroll
          for (int i = 0; i < G && g + i < TC; ++i) acc[g + i] += __uint_as_float(v[i]);
        }
      };
      if (in_segment + 1 == per_segment || c + 1 == per_tile) {
        add_sums(0, &small_full, &small_empty, segments & 1);
        ++segments;
      }
      add_sums(T, &d_full, &d_empty, (j - 1) & 1);
      ++c;
      if (++in_segment == per_segment || c == per_tile) {
        if (S::SUM_IN_SMEM) {
          if (c < per_tile) {  // (the last one meets the sum as it is stored)
#pragma unroll
            for (int i = 0; i < TC; ++i) {
              sum_smem[i * ROWS] = segment == 0 ? acc[i] : sum_smem[i * ROWS] + acc[i];
              acc[i] = 0.f;
            }
          }
        } else if (CLUSTERED && S::OWN == 1) {
          // (the block's only segment: acc is its sum)
        } else if (CLUSTERED) {
#pragma unroll
          for (int o = 0; o < S::OWN; ++o)
            if (segment == o)
#pragma unroll
              for (int i = 0; i < TC; ++i) sum[o][i] = acc[i];
#pragma unroll
          for (int i = 0; i < TC; ++i) acc[i] = 0.f;
        } else {
#pragma unroll
          for (int i = 0; i < TC; ++i) {
            sum[0][i] = segment == 0 ? acc[i] : sum[0][i] + acc[i];
            acc[i] = 0.f;
          }
        }
        in_segment = 0;
        ++segment;
      }
      if (c == per_tile && !CLUSTERED) {
        const int n0 = tile / m_tiles * ROWS + (warp & 3) * 32, m0 = tile % m_tiles * T + half * TC, n = n0 + lane;
        const float add = bias != nullptr && n < N ? bias[n] : 0.f;
        bool bad = false;
#pragma unroll
        for (int i = 0; i < TC; ++i) {
          float v;
          if (S::SUM_IN_SMEM) {
            v = segment == 1 ? acc[i] : sum_smem[i * ROWS] + acc[i];
            acc[i] = 0.f;
          } else {
            v = sum[0][i];
          }
          v *= UNSCALE;
          if (bias != nullptr) v += add;
          if (n < N && m0 + i < M) {
            C[(size_t)(m0 + i) * ldc + n] = v;
            bad = bad || !finite(v);
          }
        }
        if (bad) any_bad = 1;
        c = segment = 0;
        tile += tile_step;
      }
    }
    if (CLUSTERED) {
      // (every chunk of this block has been read out of the rings by now)
      float* part = reinterpret_cast<float*>(ws);
#pragma unroll
      for (int o = 0; o < S::OWN; ++o)
#pragma unroll
        for (int i = 0; i < TC; ++i) part[(o * T + half * TC + i) * ROWS + row] = S::OWN == 1 ? acc[i] : sum[o][S::OWN == 1 ? 0 : i];
    }
  }
  if (CLUSTERED) {
    cluster_sync();
    const int segments = (chunks + per_segment - 1) / per_segment;
    const int m0 = tile0 % m_tiles * T, rows = min(T, M - m0), n0 = tile0 / m_tiles * ROWS, n = n0 + lane * 4;
    if (tid < WORKERS) {
      // a warp a row of C, the cluster's warps in turn; a lane four numbers of it
      const bool whole = (ldc & 3) == 0 && ((uintptr_t)C & 15) == 0 && n + 4 <= N;
      for (int t = warp * S::SHARE + rank; t < rows; t += 8 * S::SHARE) {
        const uint32_t at = smem_u32(ws) + (t * ROWS + lane * 4) * 4;
        float4 p[SEGMENTS];
#pragma unroll
        for (int s = 0; s < SEGMENTS; ++s)
          if (s < segments) p[s] = ld_cluster_16(at + s % S::OWN * (T * ROWS * 4), s / S::OWN);
        float v[4] = {p[0].x, p[0].y, p[0].z, p[0].w};
#pragma unroll
        for (int s = 1; s < SEGMENTS; ++s)
          if (s < segments) {
            v[0] += p[s].x;
            v[1] += p[s].y;
            v[2] += p[s].z;
            v[3] += p[s].w;
          }
        bool bad = false;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[e] *= UNSCALE;
          if (bias != nullptr && n + e < N) v[e] += bias[n + e];
          bad = bad || (n + e < N && !finite(v[e]));
        }
        float* c = C + (size_t)(m0 + t) * ldc + n;
        if (whole) {
          *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (n + e < N) c[e] = v[e];
        }
        if (bad) any_bad = 1;
      }
    }
    __syncwarp();
    cluster_sync();  // nobody leaves while its sums are being read
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == MMA_WARP_ID) tmem_dealloc(tmem, S::TMEM);
  if (any_bad && !gave_up)
    for (int tile = tile0; tile < tiles; tile += tile_step) {
      const int m0 = tile % m_tiles * T, rows = min(T, M - m0);
      repair<T>(reinterpret_cast<float*>(ws), A, lda, W, ldw, C, ldc, tile / m_tiles * ROWS, m0 + rank, S::SHARE,
                (rows - rank + S::SHARE - 1) / S::SHARE, N, K, bias);
    }
}

// A's rows in three parts: planes [3][M][ld] (hi, mid, lo); bound by its bytes.
__global__ void split_rows_kernel(const float* A, int lda, __nv_bfloat16* planes, int ld, int M, int K) {
  pdl_trigger();
  pdl_wait();
  const int k = (blockIdx.y * blockDim.x + threadIdx.x) * 4, m = blockIdx.x;
  if (k >= K) return;
  const float4 v = *reinterpret_cast<const float4*>(A + (size_t)m * lda + k);
  uint2 part[3];
  split_pair(v.x, v.y, part[0].x, part[1].x, part[2].x);
  split_pair(v.z, v.w, part[0].y, part[1].y, part[2].y);
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(planes + ((size_t)p * M + m) * ld + k) = part[p];
}

template <typename S>
int launch(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K, const float* bias,
           const __nv_bfloat16* planes, int ld, int* status, cudaStream_t stream) {
  alignas(64) CUtensorMap w_map, a_map;
  const cuuint64_t wd[2] = {(cuuint64_t)K, (cuuint64_t)N}, wst[1] = {(cuuint64_t)ldw * 4};
  const cuuint32_t wbox[2] = {32, ROWS};
  int rc = fg_encode_tensor_map(&w_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, W, wd, wst, wbox);
  if (rc) return rc;
  a_map = w_map;
  if (!S::SPLIT_HERE) {
    const cuuint64_t ad[3] = {(cuuint64_t)K, (cuuint64_t)M, 3}, ast[2] = {(cuuint64_t)ld * 2, (cuuint64_t)ld * 2 * M};
    const cuuint32_t abox[3] = {KC, (cuuint32_t)S::T, 1};
    rc = fg_encode_tensor_map(&a_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, planes, ad, ast, abox);
    if (rc) return rc;
  }
  auto kern = gemm_f32_split_kernel<S>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  FG_CHECK_ARG(e == cudaSuccess, "fg_gemm_f32_split: shared memory: %s", cudaGetErrorString(e));
  const int m_tiles = (M + S::T - 1) / S::T;
  const long tiles = (long)m_tiles * ((N + ROWS - 1) / ROWS), resident = (long)S::BLOCKS * fg_sm_count();
  FG_CHECK_ARG(!S::SPLIT_HERE || m_tiles == 1, "fg_gemm_f32_split: %d rows in tiles of %d", M, S::T);
  FG_CHECK_ARG(tiles <= (1l << 27), "fg_gemm_f32_split: M=%d N=%d too large", M, N);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(S::SHARE > 1 ? tiles * S::SHARE : tiles < resident ? tiles : resident));
  cfg.blockDim = dim3(THREADS_ALL);
  cfg.dynamicSmemBytes = S::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = fg_pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = S::SHARE;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = S::SHARE > 1 ? 2 : 1;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, w_map, a_map, A, lda, W, ldw, C, ldc, M, N, K, bias, m_tiles,
                                            (int)tiles, status);
  FG_CHECK_ARG(le == cudaSuccess, "fg_gemm_f32_split: launch failed: %s", cudaGetErrorString(le));
  return 0;
}

// The rows of A a tile, and how many blocks share one.  Measured (us): a chunk of 64 columns takes a block that has an SM for
// itself 1.1 (T = 16) to 1.25 (T = 112) and 1.8 (T = 160), two blocks on one SM 0.65 each (T <= 32); a wave of clusters
// costs 3 more than one of single blocks.  The plan is the least of that over the busiest SM.  E.g. 2,048 x 2,048: 5 rows
// 28.6 / 18.0 / 12.0 / 8.8 with 1 / 2 / 4 / 8 blocks a tile; 16,384 x 2,048: 40.3 / 27.8 / 31.3 / 38.5; 777 rows
// against 3,072 x 2,048 79.6 in tiles of 112 and 61.4 in tiles of 160, against 2,048 x 2,048 42.4 and 60.3.
struct Plan {
  int t, share;
};
Plan choose(int M, int N, int K) {
  const int chunks = (K + KC - 1) / KC, per_segment = (chunks + SEGMENTS - 1) / SEGMENTS;
  const long n_tiles = (N + ROWS - 1) / ROWS, sms = fg_sm_count();
  const int few = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 0;
  Plan best = {0, 1};
  long best_cost = 0;
  for (int big = 0; big < (few ? 1 : 2); ++big) {
    const int t = few ? few : big ? 160 : 112;
    const long tiles = n_tiles * ((M + t - 1) / t);
    const int blocks = t <= 32 ? 2 : 1;
    for (int share = 1; share <= SEGMENTS; share *= 2) {
      if ((share == 2 && t > 16) || (share == 4 && t > 32)) continue;
      const long units = tiles * share, slots = share == 1 ? sms : sms / SEGMENTS * SEGMENTS;
      const long an_sm = (units + slots - 1) / slots;
      const long chunk = t <= 32 ? (an_sm > 1 ? 65 : 110) : t <= 112 ? 125 : 180;  // hundredths of a microsecond
      const long cost = an_sm * (SEGMENTS / share * per_segment) * chunk + (an_sm + blocks - 1) / blocks * (share == 1 ? 200 : 500);
      if (best.t == 0 || cost < best_cost) {
        best_cost = cost;
        best = {t, share};
      }
    }
  }
  return best;
}
}  // namespace

// Whether the product takes this way: by K and N and by how the rows lie, never by M (a row's sums do not
// depend on the rows beside it).
// The line lies above the sizes where a single row is slower this way than by multiply-adds.  Measured below it (us; this way, multiply-adds;
// 1, 5, 16 and 777 rows): 576 x 576 4.6 / 4.7 / 4.9 / 25 and 3.8 / 4.0 / 6.8 / 27, 3,072 x 768 6.4 / 6.6 / 7.1 / 33 and
// 5.6 / 7.2 / 10.5 / 112, 2,560 x 960 6.6 / 6.7 / 7.2 / 25 and 6.3 / 8.7 / 13 / 116, 8,192 x 512 8.1 / 8.4 / 9.0 / 52 and 6.3 / 8.8 / 19 /
// 147, 960 x 960 5.1 / 5.2 / 5.6 / 24 and 5.8 / 6.2 / 9.8 / 74.
extern "C" int fg_gemm_f32_split_takes(const float* A, int lda, const float* W, int ldw, int N, int K) {
  return K >= 1024 && N >= 1024 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
}

// bytes of scratch (16-byte aligned) of a product of M rows; 0: none is needed
extern "C" long long fg_gemm_f32_split_scratch(int M, int K) {
  return M <= 32 ? 0 : 3ll * M * ((K + 7) / 8 * 8) * 2;
}

// Against float64 (2-norm of the error over that of the result; these sums, multiply-adds in ascending k), numbers drawn from a
// normal distribution: K = 1,024 9.2e-8 and 5.8e-7, 2,048 9.8e-8 and 8.1e-7, 8,192 1.19e-7 and 1.62e-6, 14,336 1.37e-7 and
// 2.14e-6.  Rows with few numbers that are not zero (K = 2,048): one 2.6e-8 and 2.5e-8 (at most 9.7e-8 and 6.0e-8 of an element:
// the products left out), two 3.6e-8 and 3.1e-8 and four 4.5e-8 and 4.1e-8 (a segment's sum is one rounding more), eight 5.3e-8
// and 5.3e-8, sixteen 6.0e-8 and 7.4e-8, sixty-four 6.5e-8 and 14.5e-8.
extern "C" int fg_gemm_f32_split(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                                 const float* bias, void* scratch, int* status, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  FG_CHECK_ARG(K > 0 && lda >= K && ldw >= K && ldc >= N, "fg_gemm_f32_split: bad sizes M=%d N=%d K=%d", M, N, K);
  FG_CHECK_ARG(fg_gemm_f32_split_takes(A, lda, W, ldw, N, K), "fg_gemm_f32_split: rows or sizes it does not take");
  const Plan plan = choose(M, N, K);
  __nv_bfloat16* planes = static_cast<__nv_bfloat16*>(scratch);
  const int ld = (K + 7) / 8 * 8;
  if (M > 32) {
    FG_CHECK_ARG(planes != nullptr && ((uintptr_t)planes & 15) == 0, "fg_gemm_f32_split: scratch is missing or unaligned");
    const dim3 grid(M, (K / 4 + 255) / 256);
    const cudaError_t e = fg_launch_pdl(split_rows_kernel, grid, dim3(256), 0, stream, A, lda, planes, ld, M, K);
    FG_CHECK_ARG(e == cudaSuccess, "fg_gemm_f32_split: launch failed: %s", cudaGetErrorString(e));
  }
#define FG_SPLIT(rows, blocks)                      \
  if (plan.t == rows && plan.share == blocks) \
    return launch<Shape<rows, blocks>>(A, lda, W, ldw, C, ldc, M, N, K, bias, planes, ld, status, stream);
  FG_SPLIT(16, 1) FG_SPLIT(16, 2) FG_SPLIT(16, 4) FG_SPLIT(16, 8)
  FG_SPLIT(32, 1) FG_SPLIT(32, 4) FG_SPLIT(32, 8)
  FG_SPLIT(64, 1) FG_SPLIT(64, 8)
  FG_SPLIT(112, 1) FG_SPLIT(112, 8)
  FG_SPLIT(160, 1) FG_SPLIT(160, 8)
#undef FG_SPLIT
  fg_set_error("fg_gemm_f32_split: no plan");
  return -1;
}
