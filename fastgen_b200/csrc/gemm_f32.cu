// True 32-bit matrix product  C[M, N] = A[M, K] * W[N, K]^T  on the CUDA cores.
//
// This is the GEMM of the float32 path for small weights (N or K below 1,024) and for rows that do not lie on 16 bytes
// (gemm_f32_split.cu has the others): IEEE float32 fused multiply-adds, no tensor cores.  Every output element is the sum
// over k = 0 .. K-1 in ascending order in a single accumulator, so its value
// does not depend on M, on the tile it falls in, on which of the kernels below
// computes it, or on what else is in the batch.
// It stands where the reference calls F.linear (fastgen/forward.py:438-440,470,
// 491-496,513).  A bias [N], if given, is added to the finished sum.
//
// Four kernels, the same sums:
//  * gemm_f32_rows_kernel: few rows of A (decoded tokens), bound by reading W once;
//  * gemm_f32_tile_kernel: many rows (prompts), bound by the rate of multiply-adds;
//  * gemm_f32_block_kernel: in between;
//  * gemm_f32_nt_kernel: whatever the others do not take (rows that are no multiple of
//    16 bytes, a 16-bit left operand).
#include "common.cuh"

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;  // 256 threads, 4x4 outputs each

template <typename TA>
__global__ void __launch_bounds__(256)
gemm_f32_nt_kernel(const TA* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                   float* __restrict__ C, int ldc, int M, int N, int K, const float* __restrict__ bias) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;  // tx: column group, ty: row group
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  // each thread loads 4 elements of A and 4 of W per k-tile
  const int lr = tid >> 2;        // 0..63 row within tile
  const int lk = (tid & 3) * 4;   // 0,4,8,12
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int kk = k0 + lk + u;
      const int am = m0 + lr, wn = n0 + lr;
      As[lk + u][lr] = (am < M && kk < K) ? to_f32<TA>(A[(size_t)am * lda + kk]) : 0.f;
      Ws[lk + u][lr] = (wn < N && kk < K) ? W[(size_t)wn * ldw + kk] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n < N) C[(size_t)m * ldc + n] = bias != nullptr ? acc[i][j] + bias[n] : acc[i][j];
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Many rows and columns: bound by the multiply-adds (74 TFLOP/s).  A block owns 64 x 128 outputs, a thread 8 x 8
// of them.  Tiles of 16 columns of k go through registers (16-byte loads of the next tile are on their way while
// this one is multiplied) into shared memory with k as the slow index: a thread's operands of one k are
// four 16-byte reads for 64 multiply-adds, which is what the shared memory can deliver beside them (4 x 4
// outputs a thread, as in the kernel above, need twice as much).  Two multiply-adds an instruction
// (fma.rn.f32x2, each rounded as fmaf rounds).  777 x 128,256 x 2,048: 16.7 -> 8.1 ms (50 TFLOP/s).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

struct TileShape {
  static constexpr int MT = 64, NT = 128, KT = 16, THREADS = 128;
  static constexpr int LA = MT * KT / 4 / THREADS, LW = NT * KT / 4 / THREADS;  // 16-byte pieces a thread loads a tile
  static constexpr int SA = MT + 4, SW = NT + 4;                                // row strides of the transposed tiles
};

__global__ void __launch_bounds__(TileShape::THREADS, 4)
gemm_f32_tile_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                     float* __restrict__ C, int ldc, int M, int N, int K, const float* __restrict__ bias) {
  using S = TileShape;
  constexpr int KT = S::KT;
  __shared__ __align__(16) float as[2][KT][S::SA];
  __shared__ __align__(16) float ws[2][KT][S::SW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // a warp: 32 x 64 outputs; a lane's rows (columns) are two runs of four, 16 rows (32 columns) apart
  const int wm = (warp >> 1) * 32 + (lane >> 3) * 4, wn = (warp & 1) * 64 + (lane & 7) * 4;
  const int m0 = blockIdx.x * S::MT, n0 = blockIdx.y * S::NT;  // blocks that share columns of W run side by side
  unsigned long long acc[8][4];  // [row][pair of columns]
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

  // (of a tile's upper eight k, runs of eight rows change places with their neighbours: a warp's transposing stores are
  // of four k and eight rows, and fall on 32 banks that way)
  float4 ra[S::LA], rw[S::LW];
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < S::LA; ++u) {
      const int i = tid + u * S::THREADS, row = m0 + i / (KT / 4), k = k0 + i % (KT / 4) * 4;
      ra[u] = (row < M && k < K) ? *reinterpret_cast<const float4*>(A + (size_t)row * lda + k) : zero;
    }
#pragma unroll
    for (int u = 0; u < S::LW; ++u) {
      const int i = tid + u * S::THREADS, row = n0 + i / (KT / 4), k = k0 + i % (KT / 4) * 4;
      rw[u] = (row < N && k < K) ? *reinterpret_cast<const float4*>(W + (size_t)row * ldw + k) : zero;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int u = 0; u < S::LA; ++u) {
      const int i = tid + u * S::THREADS, row = i / (KT / 4), k = i % (KT / 4) * 4;
      as[buf][k][row ^ (k & 8)] = ra[u].x;
      as[buf][k + 1][row ^ (k & 8)] = ra[u].y;
      as[buf][k + 2][row ^ (k & 8)] = ra[u].z;
      as[buf][k + 3][row ^ (k & 8)] = ra[u].w;
    }
#pragma unroll
    for (int u = 0; u < S::LW; ++u) {
      const int i = tid + u * S::THREADS, row = i / (KT / 4), k = i % (KT / 4) * 4;
      ws[buf][k][row ^ (k & 8)] = rw[u].x;
      ws[buf][k + 1][row ^ (k & 8)] = rw[u].y;
      ws[buf][k + 2][row ^ (k & 8)] = rw[u].z;
      ws[buf][k + 3][row ^ (k & 8)] = rw[u].w;
    }
  };

  load(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += KT) {
    const bool more = k0 + KT < K;
    if (more) load(k0 + KT);
    float4 a[2][2];
    ulonglong2 b[2][2];
    auto fetch = [&](int kk, int f) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[f][i] = *reinterpret_cast<const float4*>(&as[buf][kk][(wm + 16 * i) ^ (kk & 8)]);
        b[f][i] = *reinterpret_cast<const ulonglong2*>(&ws[buf][kk][(wn + 32 * i) ^ (kk & 8)]);
      }
    };
    fetch(0, 0);
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) {
      const int f = kk & 1;
      // the next tile goes to the other buffer (free since the last barrier) while this one is multiplied
      if (kk == KT * 3 / 4 && more) store(buf ^ 1);
      if (kk + 1 < KT) fetch(kk + 1, f ^ 1);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 av = a[f][i >> 2];
        const float x = (i & 3) == 0 ? av.x : (i & 3) == 1 ? av.y : (i & 3) == 2 ? av.z : av.w;
        const unsigned long long xx = pack2(x, x);
        fma2(acc[i][0], xx, b[f][0].x);
        fma2(acc[i][1], xx, b[f][0].y);
        fma2(acc[i][2], xx, b[f][1].x);
        fma2(acc[i][3], xx, b[f][1].y);
      }
    }
    __syncthreads();
    buf ^= 1;
  }
  const bool whole = (ldc & 3) == 0 && ((uintptr_t)C & 15) == 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + wm + (i >> 2) * 16 + (i & 3);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int n = n0 + wn + 32 * j;
      float v[4];
      unpack2(acc[i][2 * j], v[0], v[1]);
      unpack2(acc[i][2 * j + 1], v[2], v[3]);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (bias != nullptr && n + e < N) v[e] += bias[n + e];
      float* c = C + (size_t)m * ldc + n;
      if (whole && n + 4 <= N) {
        *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < N) c[e] = v[e];
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Few rows: bound by reading W once, or by the chain of K dependent multiply-adds (4 cycles each).  A block owns 16 rows of W; a half of a warp's lanes hold one each, against TOK rows of A
// (four warps: 8 TOK rows of A a block).  Chunks of COLS columns of W and A come through a ring of
// 16-byte asynchronous copies (the pieces of W's rows swizzled so that eight lanes read eight bank
// groups); a lane walks its row of W with 16-byte reads, A is the same address for sixteen lanes.
// (5 rows, launches back to back: 2,048 x 2,048 150 -> 13 us; 16,384 x 2,048 221 -> 49; 2,048 x 8,192 583 -> 38;
// 128,256 x 2,048 1,186 -> 291, its bytes 160.)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void copy_16(uint32_t dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

template <int TOK_, int COLS_, int STAGES_>
struct RowsShape {
  static constexpr int ROWS = 16, TOK = TOK_, COLS = COLS_, STAGES = STAGES_, THREADS = 128;
  static constexpr int A_ROWS = 8 * TOK, PIECES = COLS / 4;
  static constexpr int STAGE = (ROWS + A_ROWS) * COLS;  // floats
  static constexpr size_t SMEM = sizeof(float) * STAGE * STAGES;
  static constexpr int STEP = THREADS / PIECES;  // rows a pass of the block's copies covers
  static_assert(THREADS % PIECES == 0 && ROWS % STEP == 0 && A_ROWS % STEP == 0, "");
};

template <typename S>
__global__ void __launch_bounds__(S::THREADS)
gemm_f32_rows_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                     float* __restrict__ C, int ldc, int M, int N, int K, const float* __restrict__ bias) {
  extern __shared__ __align__(16) float ring[];  // [STAGES][ROWS + A_ROWS][COLS]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n0 = blockIdx.x * S::ROWS, m0 = blockIdx.y * S::A_ROWS;
  const int chunks = (K + S::COLS - 1) / S::COLS;
  const int rows = min(S::ROWS, N - n0), toks = min(S::A_ROWS, M - m0);

  // a thread copies piece `cp` of every STEP-th row
  const int cp = tid % S::PIECES, cr = tid / S::PIECES;
  const float* const src_w = W + (size_t)n0 * ldw + cp * 4;
  const float* const src_a = A + (size_t)m0 * lda + cp * 4;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(ring);
  auto issue = [&](int c, int slot) {
    const int k0 = c * S::COLS;
    const bool in_k = k0 + cp * 4 < K;
    const uint32_t dst = base + slot * (S::STAGE * 4);
#pragma unroll
    for (int r = 0; r < S::ROWS; r += S::STEP) {
      const int row = r + cr;
      const bool ok = in_k && row < rows;
      copy_16(dst + (row * S::COLS + (cp ^ (row & 7)) * 4) * 4, ok ? src_w + (size_t)row * ldw + k0 : W, ok);
    }
#pragma unroll
    for (int r = 0; r < S::A_ROWS; r += S::STEP) {
      const int row = r + cr;
      if (row < toks) copy_16(dst + ((S::ROWS + row) * S::COLS + cp * 4) * 4, in_k ? src_a + (size_t)row * lda + k0 : A, in_k);
    }
  };

#pragma unroll
  for (int c = 0; c < S::STAGES - 1; ++c) {
    if (c < chunks) issue(c, c);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  float acc[S::TOK];
#pragma unroll
  for (int t = 0; t < S::TOK; ++t) acc[t] = 0.f;
  const int row = lane & 15, tok0 = (warp * 2 + (lane >> 4)) * S::TOK;
  const bool busy = warp * 2 * S::TOK < toks;  // a warp without rows of A only copies
  int slot = 0, fill = S::STAGES - 1;
  for (int c = 0; c < chunks; ++c) {
    // all groups but the newest STAGES - 2 are complete: chunk c has landed for this thread; the
    // barrier makes it so for all, and lets nobody overwrite a stage that is still being read
    asm volatile("cp.async.wait_group %0;\n" ::"n"(S::STAGES - 2) : "memory");
    __syncthreads();
    if (c + S::STAGES - 1 < chunks) issue(c + S::STAGES - 1, fill);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* pw = ring + slot * S::STAGE + row * S::COLS;
    const float* pa = ring + slot * S::STAGE + (S::ROWS + tok0) * S::COLS;
    auto step = [&](int p) {
      const float4 w = *reinterpret_cast<const float4*>(pw + ((p ^ (row & 7)) * 4));
      float4 a[S::TOK];
#pragma unroll
      for (int t = 0; t < S::TOK; ++t) a[t] = *reinterpret_cast<const float4*>(pa + t * S::COLS + p * 4);
#pragma unroll
      for (int t = 0; t < S::TOK; ++t) acc[t] = fmaf(a[t].x, w.x, acc[t]);
#pragma unroll
      for (int t = 0; t < S::TOK; ++t) acc[t] = fmaf(a[t].y, w.y, acc[t]);
#pragma unroll
      for (int t = 0; t < S::TOK; ++t) acc[t] = fmaf(a[t].z, w.z, acc[t]);
#pragma unroll
      for (int t = 0; t < S::TOK; ++t) acc[t] = fmaf(a[t].w, w.w, acc[t]);
    };
    const int pieces = min(S::COLS, K - c * S::COLS) / 4;
    if (busy) {
      if (pieces == S::PIECES) {
#pragma unroll
        for (int p = 0; p < S::PIECES; ++p) step(p);
      } else {
        for (int p = 0; p < pieces; ++p) step(p);
      }
    }
    slot = slot + 1 == S::STAGES ? 0 : slot + 1;
    fill = fill + 1 == S::STAGES ? 0 : fill + 1;
  }
  if (row < rows) {
#pragma unroll
    for (int t = 0; t < S::TOK; ++t)
      if (tok0 + t < toks)
        C[(size_t)(m0 + tok0 + t) * ldc + n0 + row] = bias != nullptr ? acc[t] + bias[n0 + row] : acc[t];
  }
}

// ---------------------------------------------------------------------------------------------
// In between: too many rows for the kernel above, too few tiles for the one before it.  A lane holds TOK rows of A against NC columns of C (rows of W, 32 apart); the block's warps
// (any number of them) share out the rows of A.  Both operands come through the same kind of ring, 32
// columns of k a stage, rows as they lie in memory: four k of a row of W are one 16-byte read (eight lanes
// on eight bank groups), four k of a row of A one read of the same address for the whole warp.
// (2,048 x 2,048: 100 rows 153 -> 63 us, 300 rows 220 -> 124, 777 rows 309 -> 205.)
// ---------------------------------------------------------------------------------------------
template <int TOK_, int NC_, int STAGES_, int BLOCKS_, int MAX_WARPS_>
struct BlockShape {
  static constexpr int TOK = TOK_, NC = NC_, STAGES = STAGES_, BLOCKS = BLOCKS_, MAX_WARPS = MAX_WARPS_;
  static constexpr int COLS = 32, PIECES = COLS / 4, NT = 32 * NC;
};

template <typename S>
__global__ void __launch_bounds__(S::MAX_WARPS * 32, S::BLOCKS)
gemm_f32_block_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                      float* __restrict__ C, int ldc, int M, int N, int K, const float* __restrict__ bias) {
  extern __shared__ __align__(16) float ring[];  // [STAGES][NT + warps * TOK][COLS]
  constexpr int COLS = S::COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x;
  const int mt = (threads >> 5) * S::TOK;
  const int m0 = blockIdx.x * mt, n0 = blockIdx.y * S::NT;  // blocks that share columns of W run side by side
  const int chunks = (K + COLS - 1) / COLS;
  const int cols = min(S::NT, N - n0), toks = min(mt, M - m0);
  const int stage = (S::NT + mt) * COLS;
  const int cp = tid % S::PIECES, cr = tid / S::PIECES, step_rows = threads / S::PIECES;
  const float* const src_w = W + (size_t)n0 * ldw + cp * 4;
  const float* const src_a = A + (size_t)m0 * lda + cp * 4;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(ring);
  auto issue = [&](int c, int slot) {
    const int k0 = c * COLS;
    const bool in_k = k0 + cp * 4 < K;
    const uint32_t dst = base + slot * stage * 4;
    for (int row = cr; row < S::NT; row += step_rows) {
      const bool ok = in_k && row < cols;
      copy_16(dst + (row * COLS + (cp ^ (row & 7)) * 4) * 4, ok ? src_w + (size_t)row * ldw + k0 : W, ok);
    }
    for (int row = cr; row < toks; row += step_rows)
      copy_16(dst + ((S::NT + row) * COLS + cp * 4) * 4, in_k ? src_a + (size_t)row * lda + k0 : A, in_k);
  };
#pragma unroll
  for (int c = 0; c < S::STAGES - 1; ++c) {
    if (c < chunks) issue(c, c);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  float acc[S::TOK][S::NC];
#pragma unroll
  for (int t = 0; t < S::TOK; ++t)
#pragma unroll
    for (int j = 0; j < S::NC; ++j) acc[t][j] = 0.f;
  const int tok0 = warp * S::TOK;
  int slot = 0, fill = S::STAGES - 1;
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(S::STAGES - 2) : "memory");  // as in the kernel above
    __syncthreads();
    if (c + S::STAGES - 1 < chunks) issue(c + S::STAGES - 1, fill);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* pw = ring + slot * stage + lane * COLS;
    const float* pa = ring + slot * stage + (S::NT + tok0) * COLS;
    auto step = [&](int p) {
      float4 w[S::NC];
#pragma unroll
      for (int j = 0; j < S::NC; ++j) w[j] = *reinterpret_cast<const float4*>(pw + j * 32 * COLS + ((p ^ (lane & 7)) * 4));
#pragma unroll
      for (int t = 0; t < S::TOK; t += 2) {
        const float4 a0 = *reinterpret_cast<const float4*>(pa + t * COLS + p * 4);
        const float4 a1 = *reinterpret_cast<const float4*>(pa + (t + 1) * COLS + p * 4);
#define FG_ONE_K(e)                                                                     \
  _Pragma("unroll") for (int j = 0; j < S::NC; ++j) {                                   \
    acc[t][j] = fmaf(a0.e, w[j].e, acc[t][j]);                                          \
    acc[t + 1][j] = fmaf(a1.e, w[j].e, acc[t + 1][j]);                                  \
  }
        FG_ONE_K(x) FG_ONE_K(y) FG_ONE_K(z) FG_ONE_K(w)
#undef FG_ONE_K
      }
    };
    const int pieces = min(COLS, K - c * COLS) / 4;
    if (pieces == S::PIECES) {
#pragma unroll
      for (int p = 0; p < S::PIECES; ++p) step(p);
    } else {
      for (int p = 0; p < pieces; ++p) step(p);
    }
    slot = slot + 1 == S::STAGES ? 0 : slot + 1;
    fill = fill + 1 == S::STAGES ? 0 : fill + 1;
  }
#pragma unroll
  for (int j = 0; j < S::NC; ++j) {
    const int n = n0 + lane + 32 * j;
    if (n >= N) continue;
    const float add = bias != nullptr ? bias[n] : 0.f;
#pragma unroll
    for (int t = 0; t < S::TOK; ++t)
      if (tok0 + t < toks) C[(size_t)(m0 + tok0 + t) * ldc + n] = bias != nullptr ? acc[t][j] + add : acc[t][j];
  }
}

template <int TOK, int NC, int STAGES, int BLOCKS, int MAX_WARPS>
int launch_block(int warps, const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                 const float* bias, cudaStream_t stream) {
  using S = BlockShape<TOK, NC, STAGES, BLOCKS, MAX_WARPS>;
  auto kern = gemm_f32_block_kernel<S>;
  auto bytes = [](int w) { return (int)(sizeof(float) * S::STAGES * (S::NT + w * TOK) * S::COLS); };
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes(MAX_WARPS));
  FG_CHECK_ARG(e == cudaSuccess, "fg_gemm_f32_nt: shared memory: %s", cudaGetErrorString(e));
  const dim3 grid((M + warps * TOK - 1) / (warps * TOK), (N + S::NT - 1) / S::NT);
  FG_CHECK_ARG(grid.y <= 65535, "fg_gemm_f32_nt: N=%d too large", N);
  kern<<<grid, warps * 32, bytes(warps), stream>>>(A, lda, W, ldw, C, ldc, M, N, K, bias);
  return 0;
}

template <int TOK, int COLS, int STAGES>
int launch_rows(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K, const float* bias,
                cudaStream_t stream) {
  using S = RowsShape<TOK, COLS, STAGES>;
  auto kern = gemm_f32_rows_kernel<S>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  FG_CHECK_ARG(e == cudaSuccess, "fg_gemm_f32_nt: shared memory: %s", cudaGetErrorString(e));
  const dim3 grid((N + S::ROWS - 1) / S::ROWS, (M + S::A_ROWS - 1) / S::A_ROWS);
  kern<<<grid, S::THREADS, S::SMEM, stream>>>(A, lda, W, ldw, C, ldc, M, N, K, bias);
  return 0;
}
}  // namespace

extern "C" int fg_gemm_f32_nt(const float* A, int lda, const float* W, int ldw, float* C, int ldc,
                              int M, int N, int K, const float* bias, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  FG_CHECK_ARG(K > 0 && lda >= K && ldw >= K && ldc >= N, "fg_gemm_f32_nt: bad sizes M=%d N=%d K=%d", M, N, K);
  if (K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0 && N <= 64 * 65535) {
    // Which kernel, by what was measured over 1 to 777 rows and the products of the 1B and 3B layers (2,048 to
    // 16,384 columns, 2,048 to 8,192 of k) and their 128,256 logits (us):
    //  * up to 8 rows the kernel of few rows with a row of A a lane; up to 64 rows with four rows a lane while its
    //    blocks of 16 columns are not more than about two an SM (48 rows: 2,048 x 2,048 30 against 62 of the next
    //    one, 5,120 x 3,072 101 against 133; but 16,384 x 2,048 181 against 134);
    //  * two 64 x 128 tiles an SM or more (296 on 148 SMs): the tile kernel (160 rows, 16,384 x 2,048: 358 against 369);
    //  * between them the small block while it is about two an SM (300 rows, 2,048 x 2,048: 124 against 136), else
    //    128 columns by as many rows as divide the launch best.
    auto up = [](long a, long b) { return (a + b - 1) / b; };
    const long two_an_sm = 2 * fg_sm_count(), about_two = two_an_sm + two_an_sm / 12;  // (296 and 320)
    int rc = 0;
    if (M <= 8) rc = launch_rows<1, 128, 4>(A, lda, W, ldw, C, ldc, M, N, K, bias, stream);
    else if (M <= 64 && up(N, 16) <= about_two) rc = launch_rows<4, 128, 4>(A, lda, W, ldw, C, ldc, M, N, K, bias, stream);
    else if (M > 32 && up(M, 64) * up(N, 128) >= two_an_sm) {
      const dim3 grid((unsigned)up(M, TileShape::MT), (unsigned)up(N, TileShape::NT));
      FG_CHECK_ARG(grid.y <= 65535, "fg_gemm_f32_nt: N=%d too large", N);
      gemm_f32_tile_kernel<<<grid, TileShape::THREADS, 0, stream>>>(A, lda, W, ldw, C, ldc, M, N, K, bias);
    } else if (M <= 32 || up(M, 32) * up(N, 64) <= about_two) {
      rc = launch_block<8, 2, 4, 4, 4>(M <= 16 ? 2 : M <= 24 ? 3 : 4, A, lda, W, ldw, C, ldc, M, N, K, bias, stream);
    } else {
      // warps of 8 rows: the fewest rounds of two blocks an SM, and of those the fewest rows
      int warps = 8;
      long best = 1l << 40;
      for (int w = 8; w >= 3; --w) {
        const long cost = up(up(M, 8 * w) * up(N, 128), two_an_sm) * (w + 1);
        if (cost < best) {
          best = cost;
          warps = w;
        }
      }
      rc = launch_block<8, 4, 4, 2, 8>(warps, A, lda, W, ldw, C, ldc, M, N, K, bias, stream);
    }
    if (rc) return rc;
    FG_CHECK_LAUNCH("fg_gemm_f32_nt");
    return 0;
  }
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  FG_CHECK_ARG(grid.y <= 65535, "fg_gemm_f32_nt: M=%d too large", M);
  gemm_f32_nt_kernel<float><<<grid, 256, 0, stream>>>(A, lda, W, ldw, C, ldc, M, N, K, bias);
  FG_CHECK_LAUNCH("fg_gemm_f32_nt");
  return 0;
}

// The same product with a left operand of either type (a_dtype): 16-bit activations are widened
// as they are loaded and everything after that is float32.  For the small products that a design
// wants in 32-bit whatever the serving type is (a router's logits).
extern "C" int fg_gemm_f32_nt_from(const void* A, int a_dtype, int lda, const float* W, int ldw, float* C, int ldc,
                                   int M, int N, int K, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  FG_CHECK_ARG(K > 0 && lda >= K && ldw >= K && ldc >= N, "fg_gemm_f32_nt_from: bad sizes M=%d N=%d K=%d", M, N, K);
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  FG_CHECK_ARG(grid.y <= 65535, "fg_gemm_f32_nt_from: M=%d too large", M);
  if (a_dtype == FG_F32)
    gemm_f32_nt_kernel<float><<<grid, 256, 0, stream>>>((const float*)A, lda, W, ldw, C, ldc, M, N, K, nullptr);
  else
    gemm_f32_nt_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)A, lda, W, ldw, C, ldc, M, N, K,
                                                                nullptr);
  FG_CHECK_LAUNCH("fg_gemm_f32_nt_from");
  return 0;
}
