// The gated delta rule: a matrix state per head that forgets per key channel and is corrected
// towards each new value.  Per head, with q, k unit vectors (q also times d^-1/2), a decay
// g in (0, 1)^d, a step size beta and the value v, in float32 and in this order:
//
//     S <- diag(g) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q          (S is [d, dv])
//
// The read-out sees the token's own write.  With R = diag(g) S_old, o = R^T q + u (k . q): both
// sums over the rows of the old state are formed side by side and k . q comes with the token.
//
// Two kernels.  The first prepares every token by itself (a warp a (token, head)): unit norms,
// k . q, the decay exp(-exp(A) softplus(a + bias)) per key channel, sigmoid of the step size, all
// float32, written as padded float32 rows that the second can copy in 16-byte words:
//   qn, kn [T, kv heads, DP]; rec [T, heads, DP + 4] = the decay's DP numbers, beta, k . q, 0, 0;
//   vp [T, heads, DVP]        (DP: d rounded up to the kernel's row count, DVP: dv up to a multiple of 4)
// The second runs the recurrence, which is a chain from token to token whose length, not the
// arithmetic, sets the time, so nothing else is left in it (with one decay per head instead of one per
// channel, `rec` holds g, beta, k . q, 0 and the decay is one number a token).  A block of eight warps works on
// (sequence, head, a run of the state's columns).  A column's rows are spread over LPC lanes, RPL
// rows a lane in registers (in runs of four: a lane reads its part of k, g and q as 16-byte words);
// a warp holds 32 / LPC columns and the sums over a column's rows end in log2(LPC) exchanges.
// (Measured at key size 64, 2,048 tokens: 16 lanes x 4 rows 536 us, 32 x 4 591 us, 8 x 8 601 us, 2 x 32 669 us.)
// Tokens arrive eight at a time through a ring of cp.async buffers, several stages ahead; whole
// stages run unrolled, so that a token's operands are read while the one before it is reduced.
// The recurrence runs token by token, so prompt portions, single tokens and mixed batches take these kernels and give the
// same numbers however a prompt is cut; the exception is 16-bit serving with one decay a head, where sequences that bring
// many tokens (chunk_min() and more, which looks at the step's tokens too) go chunk by chunk, with sums of another
// order.  The state of a slot is
// [heads][dv][d] float32 (a column's rows side by side), zero at admission.
#include <type_traits>

#include "common.cuh"
#include "long_sequences.cuh"

constexpr int DELTA_WARPS = 8;
constexpr int DELTA_TOKENS = 8;  // tokens a stage
constexpr int DELTA_STAGES = 4;  // buffers of the ring
constexpr int DELTA_THREADS = DELTA_WARPS * 32;
constexpr int DELTA_MAX_NRP = 8;  // key sizes up to 256

__device__ __forceinline__ float softplus_f32(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// HEAD: a is [T, heads] and dt_bias [heads], one decay per head
template <typename TA, bool HEAD>
__global__ void __launch_bounds__(128)
delta_prepare_kernel(const float* qkv, long qkv_stride, const TA* a, long a_stride, const TA* b, long b_stride,
                     const float* __restrict__ dt_bias, const float* __restrict__ a_log, const int* __restrict__ req,
                     float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ rec, float* __restrict__ vp,
                     int n_tokens, int n_heads, int n_kv_heads, int d, int dv, int DP, int DVP) {
  const int item = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= n_tokens * n_heads) return;
  const int t = item / n_heads, h = item - t * n_heads;
  if (req[t] < 0) return;
  const int group = n_heads / n_kv_heads, hk = h / group;
  const float* row = qkv + (size_t)t * qkv_stride;
  const int q_off = hk * d, k_off = (n_kv_heads + hk) * d, v_off = 2 * n_kv_heads * d + h * dv;
  const int nrp = DP / 32;
  float fq[DELTA_MAX_NRP], fk[DELTA_MAX_NRP];
  float ssq = 0.f, ssk = 0.f;
#pragma unroll
  for (int i = 0; i < DELTA_MAX_NRP; ++i) {
    const int r = lane + 32 * i;
    const bool ok = i < nrp && r < d;
    fq[i] = ok ? row[q_off + r] : 0.f;
    fk[i] = ok ? row[k_off + r] : 0.f;
    ssq = fmaf(fq[i], fq[i], ssq);
    ssk = fmaf(fk[i], fk[i], ssk);
  }
  ssq = warp_sum(ssq);
  ssk = warp_sum(ssk);
  const float rq = (1.f / sqrtf((float)d)) / sqrtf(ssq + 1e-6f), rk = 1.f / sqrtf(ssk + 1e-6f);
  const float rate = expf(a_log[h]);
  const int REC = HEAD ? 4 : DP + 4;
  float* rec_row = rec + ((size_t)t * n_heads + h) * REC;
  const bool first = h == hk * group;  // the group's first head writes the group's q and k
  float* qn_row = qn + ((size_t)t * n_kv_heads + hk) * DP;
  float* kn_row = kn + ((size_t)t * n_kv_heads + hk) * DP;
  float kq = 0.f;
#pragma unroll
  for (int i = 0; i < DELTA_MAX_NRP; ++i) {
    const int r = lane + 32 * i;
    if (i < nrp) {
      const float qv = fq[i] * rq, kv = fk[i] * rk;
      kq = fmaf(qv, kv, kq);
      if (first) {
        qn_row[r] = qv;
        kn_row[r] = kv;
      }
      // rows beyond d: k and q are zero there, and so is the state
      if (!HEAD)
        rec_row[r] = r < d ? expf(-rate * softplus_f32(to_f32<TA>(a[(size_t)t * a_stride + h * d + r]) + dt_bias[h * d + r])) : 0.f;
    }
  }
  kq = warp_sum(kq);
  if (lane < 4) {
    const float beta = 1.f / (1.f + expf(-to_f32<TA>(b[(size_t)t * b_stride + h])));
    if (HEAD) {
      const float g = expf(-rate * softplus_f32(to_f32<TA>(a[(size_t)t * a_stride + h]) + dt_bias[h]));
      rec_row[lane] = lane == 0 ? g : (lane == 1 ? beta : (lane == 2 ? kq : 0.f));
    } else {
      rec_row[DP + lane] = lane == 0 ? beta : (lane == 1 ? kq : 0.f);
    }
  }
  float* vp_row = vp + ((size_t)t * n_heads + h) * DVP;
  for (int c = lane; c < DVP; c += 32) vp_row[c] = c < dv ? row[v_off + c] : 0.f;
}

__device__ __forceinline__ void delta_copy16(float* dst, const float* src, bool pred) {
  const int bytes = pred ? 16 : 0;  // 0: the 16 bytes are zero-filled, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes) : "memory");
}

template <int LPC, int RPL, bool HEAD>
__global__ void __launch_bounds__(DELTA_THREADS)
delta_scan_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ rec,
                  const float* __restrict__ vp, float* __restrict__ out, long out_stride, float* __restrict__ state,
                  long state_stride, const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int n_heads,
                  int n_kv_heads, int d, int dv, int DVP, int most) {
  constexpr int DP = LPC * RPL;            // rows, padded
  constexpr int CPW = 32 / LPC;            // columns a warp
  constexpr int COLS = DELTA_WARPS * CPW;  // columns a block
  constexpr int REC = HEAD ? 4 : DP + 4;
  static_assert(DP % 32 == 0 && RPL % 4 == 0 && COLS % 4 == 0, "rows in runs of four, a multiple of 32 in all");
  extern __shared__ __align__(16) float smem[];
  // per token of a buffer: q[DP], k[DP], rec (g, beta, k . q), v[COLS]
  constexpr int TOKF = 2 * DP + REC + COLS;
  constexpr int BUF = DELTA_TOKENS * TOKF;
  constexpr int CHUNKS = TOKF / 4;  // 16-byte words a token
  const int slot = seq_slot[blockIdx.z];
  if (slot < 0) return;
  const int start = seq_start[blockIdx.z], n = seq_start[blockIdx.z + 1] - start;
  if (n <= 0 || n > most) return;  // (more than `most`: delta_chunk_kernel's)
  const int h = blockIdx.y, hk = h / (n_heads / n_kv_heads);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane % LPC, cw = warp * CPW + lane / LPC;  // the lane's part of a column; its column in the block
  const int col0 = blockIdx.x * COLS, j = col0 + cw;
  const bool live_col = j < dv;

  // the lane's rows: 4 (sub + LPC jj) + e for jj < RPL / 4, e < 4
  float S[RPL];
  float* st = state + (size_t)slot * state_stride + ((size_t)h * dv + (live_col ? j : 0)) * d;
#pragma unroll
  for (int i = 0; i < RPL; ++i) {
    const int r = 4 * (sub + LPC * (i >> 2)) + (i & 3);
    S[i] = (live_col && r < d) ? st[r] : 0.f;
  }

  // the copies of one stage: every thread takes 16-byte words of the stage's tokens in turn
  auto issue = [&](int stage) {
    float* buf = smem + (stage % DELTA_STAGES) * BUF;
    for (int c = threadIdx.x; c < DELTA_TOKENS * CHUNKS; c += DELTA_THREADS) {
      const int tt = c / CHUNKS, w = c - tt * CHUNKS, t = stage * DELTA_TOKENS + tt;
      const bool live = t < n;
      const size_t tok = (size_t)(start + (live ? t : 0));
      const float* src;
      bool ok = live;
      if (w < DP / 4) {
        src = qn + (tok * n_kv_heads + hk) * DP + 4 * w;
      } else if (w < 2 * (DP / 4)) {
        src = kn + (tok * n_kv_heads + hk) * DP + 4 * (w - DP / 4);
      } else if (w < 2 * (DP / 4) + REC / 4) {
        src = rec + (tok * n_heads + h) * REC + 4 * (w - 2 * (DP / 4));
      } else {
        const int c4 = 4 * (w - 2 * (DP / 4) - REC / 4);
        ok = live && col0 + c4 < DVP;
        src = vp + (tok * n_heads + h) * DVP + (ok ? col0 + c4 : 0);
      }
      delta_copy16(buf + tt * TOKF + 4 * w, src, ok);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  // one token of the recurrence, its operands at `tokp`
  auto step = [&](const float* tokp, size_t out_row) {
    const float4* sq = reinterpret_cast<const float4*>(tokp);
    const float4* sk = reinterpret_cast<const float4*>(tokp + DP);
    const float4* sg = reinterpret_cast<const float4*>(tokp + 2 * DP);
    constexpr int AT = HEAD ? 2 * DP + 1 : 3 * DP;  // beta's place
    const float beta = tokp[AT], kq = tokp[AT + 1], v = tokp[2 * DP + REC + cw];
    const float g_head = HEAD ? tokp[2 * DP] : 0.f;
    float kr[RPL];
    float rk2[4] = {0.f, 0.f, 0.f, 0.f}, rq2[4] = {0.f, 0.f, 0.f, 0.f};  // four chains a sum: a lane's rows are many
#pragma unroll
    for (int jj = 0; jj < RPL / 4; ++jj) {
      const float4 kv = sk[sub + LPC * jj], gv = HEAD ? make_float4(g_head, g_head, g_head, g_head) : sg[sub + LPC * jj], qv = sq[sub + LPC * jj];
      const float ke[4] = {kv.x, kv.y, kv.z, kv.w}, ge[4] = {gv.x, gv.y, gv.z, gv.w}, qe[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 4 * jj + e;
        kr[i] = ke[e];
        S[i] *= ge[e];
        rk2[e] = fmaf(S[i], ke[e], rk2[e]);
        rq2[e] = fmaf(S[i], qe[e], rq2[e]);
      }
    }
    float rk_sum = (rk2[0] + rk2[1]) + (rk2[2] + rk2[3]), rq_sum = (rq2[0] + rq2[1]) + (rq2[2] + rq2[3]);
#pragma unroll
    for (int o = LPC / 2; o > 0; o >>= 1) {
      rk_sum += __shfl_xor_sync(0xffffffffu, rk_sum, o);
      rq_sum += __shfl_xor_sync(0xffffffffu, rq_sum, o);
    }
    const float u = beta * (v - rk_sum);
#pragma unroll
    for (int i = 0; i < RPL; ++i) S[i] = fmaf(kr[i], u, S[i]);
    if (sub == 0 && live_col) out[out_row * out_stride + h * dv + j] = fmaf(u, kq, rq_sum);
  };

  const int n_stages = (n + DELTA_TOKENS - 1) / DELTA_TOKENS;
#pragma unroll
  for (int s = 0; s < DELTA_STAGES - 1; ++s) {
    if (s < n_stages) issue(s);
    else asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  for (int stage = 0; stage < n_stages; ++stage) {
    // this stage's copies have landed (the groups after it may be in flight), for every thread
    asm volatile("cp.async.wait_group %0;\n" ::"n"(DELTA_STAGES - 2) : "memory");
    __syncthreads();
    // the buffer of the stage before this one is free now: fill it with the stage three ahead
    if (stage + DELTA_STAGES - 1 < n_stages) issue(stage + DELTA_STAGES - 1);
    else asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* buf = smem + (stage % DELTA_STAGES) * BUF;
    const int n_tok = min(DELTA_TOKENS, n - stage * DELTA_TOKENS);
    const size_t row0 = (size_t)start + (size_t)stage * DELTA_TOKENS;
    if (n_tok == DELTA_TOKENS) {
#pragma unroll
      for (int tt = 0; tt < DELTA_TOKENS; ++tt) step(buf + tt * TOKF, row0 + tt);
    } else {
      for (int tt = 0; tt < n_tok; ++tt) step(buf + tt * TOKF, row0 + tt);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if (live_col) {
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      const int r = 4 * (sub + LPC * (i >> 2)) + (i & 3);
      if (r < d) st[r] = S[i];
    }
  }
}

// ---- sequences of many tokens with one decay a head: chunks ------------------------------------------
// The recurrence above is a chain of about 450 cycles a token.  Over a chunk of C = 32 tokens from state S0 it
// is also, with D[i][j] = g_{j+1} .. g_i (a product, never a quotient) and c_i = g_1 .. g_i,
//
//     (I + A) U = beta (V - c K S0),   A[i][j] = beta_i D[i][j] k_i . k_j  (j < i)
//     O = c Q S0 + (D o Q K^T) U       S <- c_C S0 + (D[C] o K)^T U
//
// and all that does not hold S0 is each chunk's own.  delta_wy_kernel forms it for all chunks side by side
// (a block a (chunk, head); the triangular system by forward substitution, a thread a column):
//     W = (I + A)^-1 beta c K,  V' = (I + A)^-1 beta V,  c Q,  (D[C] o K)^T,  D o Q K^T
// and delta_chunk_kernel walks the chunks: U = V' - W S0, then O and the next state, two small products
// and two barriers for 32 tokens.  1,501 tokens, 16 heads of 64: 347 -> 63 us and 28 of forming the chunks.
// float32, but for the products of decays, K K^T and Q K^T, which are added up in 64 bits.  (As single float32 chains these,
// the substitution and the sums over the state's rows made the outputs 2.6e-7 off at key size 64 and 3.2e-7 at
// 128, against 2.0e-7 and 2.3e-7 of the token kernel; with short chains 1.9e-7 and 2.1e-7.)  The order of the
// sums is not the token kernel's, so the float32 mode, whose results do not depend on how a prompt is cut, keeps that.
// (The chunked form is published, for instance in Yang et al., "Parallelizing Linear Transformers with the Delta
// Rule over Sequence Length", 2024.)
constexpr int CHUNK = 32;
constexpr int CHUNK_RUN = 8;     // rows of the state that are summed by themselves
constexpr int CHUNK_THREADS = 128;
constexpr int CHUNK_COLS = 8;    // columns of the state a block of the walk
constexpr int CHUNK_STAGES = 3;  // chunks in its ring
// Fewest tokens of a sequence that takes this way: where the two meet, which depends on how many such sequences the
// step's tokens leave room for (16 heads of 64).  Chunks, formed and walked, against tokens, us: one sequence of 80 / 96 / 128
// 19.5 / 19.7 / 21.0 against 20.7 / 24.4 / 31.8 (of 64: 18.0 against 17.0), two of 96 / 128 23.2 / 26.6 against 24.6 / 32.2,
// four 33.1 / 39.4 against 30.1 / 39.2, eight 49.5 / 66.7 against 46.7 / 66.9.
inline int chunk_min(int n_tokens) { return n_tokens < 2 * 80 ? 80 : n_tokens < 3 * 96 ? 96 : 128; }

// Chunks formed and walked at a time: a step of more goes in stretches, through the same room (at 32 heads of 128 a chunk
// takes 2.2 MB, and 16,384 tokens of 256 requests would take 1.7 GB).  One sequence of 8,192
// tokens, 16 heads of 64: walked in 328 us either way; 16 of 512: 251 instead of 227.
constexpr int CHUNK_ROOM = 128;

// floats of a (chunk, head): W [32][D], c Q [32][D], (D[C] o K)^T [D][32], D o Q K^T [32][32], V' [32][DVP], c_C
__host__ __device__ constexpr long chunk_floats(int D, int DVP) { return 96L * D + CHUNK * CHUNK + CHUNK * DVP + 4; }

template <int D>
__global__ void __launch_bounds__(CHUNK_THREADS)
delta_wy_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ rec,
                const float* __restrict__ vp, long_seq::Head* list, float* __restrict__ chunks,
                const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int n_seqs, int n_heads, int n_kv_heads,
                int DVP, int min_tokens, int base) {
  constexpr int SK = D + 4, SA = CHUNK + 4;
  __shared__ __align__(16) float ks[CHUNK][SK];
  __shared__ __align__(16) float qs[CHUNK][SK];
  __shared__ __align__(16) float at[CHUNK][SA];  // A transposed: [m][i]
  __shared__ double dm[CHUNK][CHUNK + 1];        // D[i][j], j <= i
  __shared__ float gs[CHUNK], betas[CHUNK], cs[CHUNK];
  const int h = blockIdx.y, hk = h / (n_heads / n_kv_heads), tid = threadIdx.x;
  const auto found = long_seq::find_chunk<CHUNK, CHUNK_THREADS>(seq_slot, seq_start, n_seqs, min_tokens, base + blockIdx.x,
                                                                blockIdx.x + h == 0 ? list : nullptr);
  if (found.seq < 0) return;
  const int c = base + blockIdx.x - found.first_chunk;
  const int t0 = seq_start[found.seq] + c * CHUNK, nt = min(CHUNK, found.tokens - c * CHUNK);
  float* const dst = chunks + ((size_t)blockIdx.x * n_heads + h) * chunk_floats(D, DVP);
  for (int i = tid; i < CHUNK * (D / 4); i += CHUNK_THREADS) {
    const int t = i / (D / 4), w = i % (D / 4) * 4;
    float4 k = make_float4(0.f, 0.f, 0.f, 0.f), q = k;
    if (t < nt) {
      k = *reinterpret_cast<const float4*>(kn + ((size_t)(t0 + t) * n_kv_heads + hk) * D + w);
      q = *reinterpret_cast<const float4*>(qn + ((size_t)(t0 + t) * n_kv_heads + hk) * D + w);
    }
    *reinterpret_cast<float4*>(&ks[t][w]) = k;
    *reinterpret_cast<float4*>(&qs[t][w]) = q;
  }
  if (tid < CHUNK) {  // tokens beyond the sequence change nothing: no decay, no step
    const float* r = rec + ((size_t)(t0 + tid) * n_heads + h) * 4;
    gs[tid] = tid < nt ? r[0] : 1.f;
    betas[tid] = tid < nt ? r[1] : 0.f;
  }
  __syncthreads();
  if (tid <= CHUNK) {  // column tid of D; thread 32: the decays from the chunk's start
    const int j = tid < CHUNK ? tid : -1;
    double x = 1.0;
    for (int i = j < 0 ? 0 : j; i < CHUNK; ++i) {
      if (i > j) x *= gs[i];
      if (j < 0) cs[i] = (float)x;
      else dm[i][j] = x;
    }
  }
  __syncthreads();
  {  // K K^T (the first half of the threads) and Q K^T: 4 x 4 places a thread, 8 apart
    const bool of_q = tid >= 64;
    const int ib = (tid & 63) >> 3, jb = tid & 7;
    const float (*left)[SK] = of_q ? qs : ks;
    // short chains: stretches of 16 products that are four chains each, added up in 64 bits
    double acc[4][4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int f = 0; f < 4; ++f) acc[e][f] = 0.0;
#pragma unroll 1
    for (int w0 = 0; w0 < D; w0 += 16) {
      float4 run[4][4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int f = 0; f < 4; ++f) run[e][f] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = w0; w < w0 + 16; w += 4) {
        float4 a[4], k[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          a[e] = *reinterpret_cast<const float4*>(&left[ib + 8 * e][w]);
          k[e] = *reinterpret_cast<const float4*>(&ks[jb + 8 * e][w]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            run[e][f].x = fmaf(a[e].x, k[f].x, run[e][f].x);
            run[e][f].y = fmaf(a[e].y, k[f].y, run[e][f].y);
            run[e][f].z = fmaf(a[e].z, k[f].z, run[e][f].z);
            run[e][f].w = fmaf(a[e].w, k[f].w, run[e][f].w);
          }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int f = 0; f < 4; ++f) acc[e][f] += (run[e][f].x + run[e][f].y) + (run[e][f].z + run[e][f].w);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const int i = ib + 8 * e, j = jb + 8 * f;
        if (of_q) dst[96 * D + i * CHUNK + j] = j <= i ? (float)(dm[i][j] * acc[e][f]) : 0.f;
        else at[j][i] = j < i ? (float)(betas[i] * dm[i][j] * acc[e][f]) : 0.f;
      }
  }
  __syncthreads();
  for (int col = tid; col < D + DVP; col += CHUNK_THREADS) {
    float x[CHUNK];
    if (col < D) {
#pragma unroll
      for (int i = 0; i < CHUNK; i += 4) {
        float kd[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float k = ks[i + e][col];
          kd[e] = (float)dm[CHUNK - 1][i + e] * k;
          x[i + e] = betas[i + e] * cs[i + e] * k;
          dst[32 * D + (i + e) * D + col] = cs[i + e] * qs[i + e][col];
        }
        *reinterpret_cast<float4*>(dst + 64 * D + col * CHUNK + i) = make_float4(kd[0], kd[1], kd[2], kd[3]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < CHUNK; ++i)
        x[i] = i < nt ? betas[i] * vp[((size_t)(t0 + i) * n_heads + h) * DVP + col - D] : 0.f;
    }
    // what the tokens before it take off a token is summed by itself: it is small beside the token's own number
    float off[CHUNK];
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) off[i] = 0.f;
#pragma unroll
    for (int m = 0; m < CHUNK; ++m) {
      x[m] -= off[m];
#pragma unroll
      for (int i = (m + 1) / 4 * 4; i < CHUNK; i += 4) {
        const float4 a = *reinterpret_cast<const float4*>(&at[m][i]);  // zero up to i = m
        if (i > m) off[i] = fmaf(a.x, x[m], off[i]);
        if (i + 1 > m) off[i + 1] = fmaf(a.y, x[m], off[i + 1]);
        if (i + 2 > m) off[i + 2] = fmaf(a.z, x[m], off[i + 2]);
        off[i + 3] = fmaf(a.w, x[m], off[i + 3]);
      }
    }
#pragma unroll
    for (int i = 0; i < CHUNK; ++i) {
      if (col < D) dst[i * D + col] = x[i];
      else dst[96 * D + CHUNK * CHUNK + i * DVP + col - D] = x[i];
    }
  }
  if (tid == 0) dst[96 * D + CHUNK * CHUNK + CHUNK * DVP] = cs[CHUNK - 1];
}

template <int D>
struct ChunkWalk {
  static constexpr int SW = D + 4, SK = CHUNK + 4;  // padded rows: eight lanes read eight bank groups
  static constexpr int W = 0, Q = W + CHUNK * SW, K = Q + CHUNK * SW, A = K + D * SK, V = A + CHUNK * SK;
  static constexpr int END = V + CHUNK * CHUNK_COLS, BUF = END + 4;
  static constexpr size_t SMEM = sizeof(float) * (CHUNK_STAGES * BUF + CHUNK_COLS * (SW + SK));
};

__device__ __forceinline__ float dot4(float4 a, float4 b, float acc) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}

// v's numbers up to place n, zeros behind it
__device__ __forceinline__ float4 up_to(float4 v, int n) {
  return make_float4(n >= 0 ? v.x : 0.f, n >= 1 ? v.y : 0.f, n >= 2 ? v.z : 0.f, n >= 3 ? v.w : 0.f);
}

// (Two blocks an SM said outright, which is what the ring leaves room for at key size 64: the registers of a chunk's operands
// stay in flight; left to itself the compiler keeps to 72 and the walk takes 82 us instead of 63.)
template <int D>
__global__ void __launch_bounds__(CHUNK_THREADS, 2)
delta_chunk_kernel(long_seq::Head* list, const float* __restrict__ chunks, float* __restrict__ out, long out_stride, float* __restrict__ state,
                   long state_stride, const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int n_heads,
                   int d, int dv, int DVP, int base) {
  using L = ChunkWalk<D>;
  constexpr int ND = D / 32;
  extern __shared__ __align__(16) float smem[];
  float* const s_t = smem + CHUNK_STAGES * L::BUF;   // the state, a column a row: [COLS][SW]
  float* const u_t = s_t + CHUNK_COLS * L::SW;       // U, a column a row: [COLS][SK]
  const int tid = threadIdx.x;
  const int r = tid >> 2, c0 = (tid & 3) * 2;
  const int columns = (dv + CHUNK_COLS - 1) / CHUNK_COLS;
  const long REC = chunk_floats(D, DVP);
  for (long_seq::Items items(list, n_heads * columns); items.more(); items.draw()) {
    const auto sequence = items.sequence();
    const int h = items.part() / columns, col0 = items.part() % columns * CHUNK_COLS;
    const int n = sequence.tokens, first = sequence.first_chunk - base, start = seq_start[sequence.seq];
    // the sequence's chunks of this stretch
    const int c_lo = max(0, -first), c_hi = min((n + CHUNK - 1) / CHUNK, CHUNK_ROOM - first);
    if (c_lo >= c_hi) continue;

    auto issue = [&](int c) {
      const float* src = chunks + ((size_t)(first + c) * n_heads + h) * REC;
      float* buf = smem + c % CHUNK_STAGES * L::BUF;
      for (int i = tid; i < 2 * CHUNK * (D / 4); i += CHUNK_THREADS)  // W and c Q
        delta_copy16(buf + i / (D / 4) * L::SW + i % (D / 4) * 4, src + i * 4, true);
      for (int i = tid; i < (D + CHUNK) * (CHUNK / 4); i += CHUNK_THREADS)  // (D[C] o K)^T and D o Q K^T
        delta_copy16(buf + L::K + i / (CHUNK / 4) * L::SK + i % (CHUNK / 4) * 4, src + 64 * D + i * 4, true);
      if (tid < CHUNK * CHUNK_COLS / 4) {
        const int r = tid / (CHUNK_COLS / 4), w = tid % (CHUNK_COLS / 4) * 4;
        const bool ok = col0 + w < DVP;
        delta_copy16(buf + L::V + r * CHUNK_COLS + w, src + 96 * D + CHUNK * CHUNK + r * DVP + (ok ? col0 + w : 0), ok);
      }
      if (tid == 64) delta_copy16(buf + L::END, src + 96 * D + CHUNK * CHUNK + CHUNK * DVP, true);
    };
    // a thread: row r of the chunk (or rows r + 32 i of the state) against two columns
    float* const st = state + (size_t)seq_slot[sequence.seq] * state_stride + ((size_t)h * dv + col0) * d;
    // An infinity or NaN in U reaches the tokens before its own through the zeros of D o Q K^T (0 * inf): where an output is
    // not finite, the block walks once more with U cut off behind each token (CAUSAL; in the first walk the cuts,
    // or a test in every chunk, cost 5 to 12 % of the time).  The state is stored at the walk's end, so that both start alike.
    auto walk = [&](auto causal) {
      constexpr bool CAUSAL = decltype(causal)::value;
#pragma unroll
      for (int c = c_lo; c < c_lo + CHUNK_STAGES - 1; ++c) {
        if (c < c_hi) issue(c);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
      }
      float s[ND][2];
#pragma unroll
      for (int i = 0; i < ND; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int row = r + 32 * i, col = c0 + e;
          s[i][e] = (row < d && col0 + col < dv) ? st[(size_t)col * d + row] : 0.f;
          s_t[col * L::SW + row] = s[i][e];
        }
      float finite = 0.f;
      for (int c = c_lo; c < c_hi; ++c) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(CHUNK_STAGES - 2) : "memory");
        __syncthreads();  // the chunk has landed, and the state of the chunk before stands in shared memory
        if (c + CHUNK_STAGES - 1 < c_hi) issue(c + CHUNK_STAGES - 1);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const float* buf = smem + c % CHUNK_STAGES * L::BUF;
        float w0 = 0.f, w1 = 0.f, q0 = 0.f, q1 = 0.f;
#pragma unroll
        for (int k0 = 0; k0 < D; k0 += CHUNK_RUN) {
          float rw0 = 0.f, rw1 = 0.f, rq0 = 0.f, rq1 = 0.f;
#pragma unroll
          for (int k = k0; k < k0 + CHUNK_RUN; k += 4) {
            const float4 w = *reinterpret_cast<const float4*>(buf + L::W + r * L::SW + k);
            const float4 q = *reinterpret_cast<const float4*>(buf + L::Q + r * L::SW + k);
            const float4 a = *reinterpret_cast<const float4*>(s_t + c0 * L::SW + k);
            const float4 e = *reinterpret_cast<const float4*>(s_t + (c0 + 1) * L::SW + k);
            rw0 = dot4(w, a, rw0);
            rw1 = dot4(w, e, rw1);
            rq0 = dot4(q, a, rq0);
            rq1 = dot4(q, e, rq1);
          }
          w0 += rw0;
          w1 += rw1;
          q0 += rq0;
          q1 += rq1;
        }
        const float2 v = *reinterpret_cast<const float2*>(buf + L::V + r * CHUNK_COLS + c0);
        u_t[c0 * L::SK + r] = v.x - w0;
        u_t[(c0 + 1) * L::SK + r] = v.y - w1;
        __syncthreads();
        const float gc = buf[L::END];
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          s[i][0] *= gc;
          s[i][1] *= gc;
        }
        float m0 = 0.f, m1 = 0.f;
#pragma unroll
        for (int k = 0; k < CHUNK; k += 4) {
          const float4 a = *reinterpret_cast<const float4*>(u_t + c0 * L::SK + k);
          const float4 e = *reinterpret_cast<const float4*>(u_t + (c0 + 1) * L::SK + k);
          const float4 m = *reinterpret_cast<const float4*>(buf + L::A + r * L::SK + k);
          m0 = dot4(m, CAUSAL ? up_to(a, r - k) : a, m0);
          m1 = dot4(m, CAUSAL ? up_to(e, r - k) : e, m1);
#pragma unroll
          for (int i = 0; i < ND; ++i) {
            const float4 kd = *reinterpret_cast<const float4*>(buf + L::K + (r + 32 * i) * L::SK + k);
            s[i][0] = dot4(kd, a, s[i][0]);
            s[i][1] = dot4(kd, e, s[i][1]);
          }
        }
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          s_t[c0 * L::SW + r + 32 * i] = s[i][0];
          s_t[(c0 + 1) * L::SW + r + 32 * i] = s[i][1];
        }
        q0 += m0;
        q1 += m1;
        if (!CAUSAL) finite = fmaf(0.f, q0, fmaf(0.f, q1, finite));
        if (c * CHUNK + r < n) {
          float* o = out + (size_t)(start + c * CHUNK + r) * out_stride + h * dv + col0 + c0;
          if (col0 + c0 < dv) o[0] = q0;
          if (col0 + c0 + 1 < dv) o[1] = q1;
        }
      }
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      if (!CAUSAL && __syncthreads_or(finite != 0.f)) return false;
#pragma unroll
      for (int i = 0; i < ND; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int row = r + 32 * i, col = c0 + e;
          if (row < d && col0 + col < dv) st[(size_t)col * d + row] = s[i][e];
        }
      return true;
    };
    if (!walk(std::false_type())) walk(std::true_type());
  }
}

// rows of the prepared arrays for key size d (the row count of the kernel that takes it)
static int delta_rows(int d) { return d <= 32 ? 32 : d <= 64 ? 64 : d <= 128 ? 128 : 256; }

template <bool HEAD>
static int launch_scan(cudaStream_t stream, const float* qn, const float* kn, const float* rec, const float* vp,
                       float* out, long out_stride, float* state, long state_stride, const int* seq_slot,
                       const int* seq_start, int n_seqs, int n_heads, int n_kv_heads, int d, int dv, int DVP, int most) {
#define CASE(LPC, RPL)                                                                                         \
  {                                                                                                            \
    constexpr int COLS = DELTA_WARPS * (32 / LPC);                                                             \
    const size_t smem = (size_t)DELTA_STAGES * DELTA_TOKENS * ((HEAD ? 2 : 3) * LPC * RPL + 4 + COLS) * sizeof(float); \
    auto kern = delta_scan_kernel<LPC, RPL, HEAD>;                                                              \
    if (smem > 48 * 1024) {                                                                                     \
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);       \
      FG_CHECK_ARG(e == cudaSuccess, "fg_delta_scan: shared memory: %s", cudaGetErrorString(e));                \
    }                                                                                                           \
    dim3 grid((dv + COLS - 1) / COLS, n_heads, n_seqs);                                                         \
    kern<<<grid, DELTA_THREADS, smem, stream>>>(qn, kn, rec, vp, out, out_stride, state, state_stride, seq_slot, \
                                                seq_start, n_heads, n_kv_heads, d, dv, DVP, most);              \
  }
  if (d <= 32) CASE(8, 4)
  else if (d <= 64) CASE(16, 4)
  else if (d <= 128) CASE(16, 8)
  else CASE(16, 16)
#undef CASE
  return 0;
}

// Whether a step may hold sequences for delta_chunk_kernel: 16-bit serving, one decay a head, key sizes whose
// rows are 64 or 128, and enough tokens (`longest`: the most that one of its sequences can bring).
static bool chunks_apply(int n_tokens, int longest, int d, int dtype, int head_decay) {
  return dtype == FG_BF16 && head_decay && d > 32 && d <= 128 && longest >= chunk_min(n_tokens);
}
static long most_chunks(int n_tokens, int n_seqs) { return long_seq::most_chunks(n_tokens, n_seqs, chunk_min(n_tokens), CHUNK); }

// kernels that fg_delta_scan launches
extern "C" int fg_delta_scan_launches(int n_tokens, int longest, int n_seqs, int d, int dtype, int head_decay) {
  return 2 + (chunks_apply(n_tokens, longest, d, dtype, head_decay) ? 2 * (int)((most_chunks(n_tokens, n_seqs) + CHUNK_ROOM - 1) / CHUNK_ROOM) : 0);
}

// floats of the scratch that fg_delta_scan needs for `n_tokens` tokens
extern "C" long fg_delta_scan_scratch_floats(int n_tokens, int longest, int n_seqs, int n_heads, int n_kv_heads, int d, int dv,
                                             int dtype, int head_decay) {
  const long DP = delta_rows(d), DVP = (dv + 3) / 4 * 4;
  const long rows = (long)n_tokens * (2 * n_kv_heads * DP + n_heads * (DP + 4) + n_heads * DVP);
  if (!chunks_apply(n_tokens, longest, d, dtype, head_decay)) return rows;
  const long most = most_chunks(n_tokens, n_seqs);
  return rows + long_seq::list_floats(n_tokens, n_seqs, chunk_min(n_tokens)) +
         (most < CHUNK_ROOM ? most : CHUNK_ROOM) * n_heads * chunk_floats((int)DP, (int)DVP);
}

// qkv: float32 [T, q (kv heads x d) | k (kv heads x d) | v (heads x dv)], the convolutions' outputs.
// a: [T, heads x d] decay logits ([T, heads] with head_decay: one decay per head) and b: [T, .] step-size logits (column h of row t at b[t * b_stride + h]),
// both of `dtype`.  dt_bias: float32 [heads x d] or [heads]; a_log: float32 [heads].  out: float32 [T, heads x dv].
// state: float32 [slots, state_stride], a slot's first heads * dv * d numbers.
extern "C" int fg_delta_scan(const float* qkv, long qkv_stride, const void* a, long a_stride, const void* b,
                             long b_stride, int dtype, const float* dt_bias, const float* a_log, float* out,
                             long out_stride, float* state, long state_stride, const int* seq_slot,
                             const int* seq_start, int n_seqs, const int* req, int n_tokens, int longest, float* scratch,
                             int n_heads, int n_kv_heads, int d, int dv, int head_decay, cudaStream_t stream) {
  if (n_seqs == 0 || n_tokens == 0) return 0;
  FG_CHECK_ARG(n_heads > 0 && n_kv_heads > 0 && n_heads % n_kv_heads == 0, "fg_delta_scan: %d heads over %d key heads",
               n_heads, n_kv_heads);
  FG_CHECK_ARG(d >= 1 && d <= 256 && dv >= 1, "fg_delta_scan: key size %d (1 to 256), value size %d", d, dv);
  FG_CHECK_ARG(n_heads <= 65535 && n_seqs <= 65535, "fg_delta_scan: too many heads or sequences");
  FG_CHECK_ARG(scratch != nullptr && ((uintptr_t)scratch & 15) == 0, "fg_delta_scan: scratch missing or unaligned");
  const int DP = delta_rows(d), DVP = (dv + 3) / 4 * 4;
  float* qn = scratch;
  float* kn = qn + (size_t)n_tokens * n_kv_heads * DP;
  float* rec = kn + (size_t)n_tokens * n_kv_heads * DP;
  float* vp = rec + (size_t)n_tokens * n_heads * (head_decay ? 4 : DP + 4);
  const int blocks = (int)(((long)n_tokens * n_heads + 3) / 4);
  FG_CHECK_ARG(dtype == FG_F32 || dtype == FG_BF16, "fg_delta_scan: bad dtype %d", dtype);
#define PREPARE(T, HEAD)                                                                                        \
  delta_prepare_kernel<T, HEAD><<<blocks, 128, 0, stream>>>(qkv, qkv_stride, (const T*)a, a_stride, (const T*)b,  \
                                                            b_stride, dt_bias, a_log, req, qn, kn, rec, vp,       \
                                                            n_tokens, n_heads, n_kv_heads, d, dv, DP, DVP)
  if (dtype == FG_F32) {
    if (head_decay) PREPARE(float, true); else PREPARE(float, false);
  } else {
    if (head_decay) PREPARE(__nv_bfloat16, true); else PREPARE(__nv_bfloat16, false);
  }
#undef PREPARE
  FG_CHECK_LAUNCH("fg_delta_scan (prepare)");
  int most = 0x7fffffff;  // tokens of the longest sequence that the token kernel takes
  if (chunks_apply(n_tokens, longest, d, dtype, head_decay)) {
    most = chunk_min(n_tokens) - 1;
    float* const behind = scratch + (size_t)n_tokens * (2 * n_kv_heads * DP + n_heads * (DP + 4) + n_heads * DVP);
    long_seq::Head* const list = reinterpret_cast<long_seq::Head*>(behind);
    float* const chunks = behind + long_seq::list_floats(n_tokens, n_seqs, chunk_min(n_tokens));
    const int all = (int)most_chunks(n_tokens, n_seqs);
    const long items = long_seq::most_sequences(n_tokens, n_seqs, chunk_min(n_tokens)) * n_heads * ((dv + CHUNK_COLS - 1) / CHUNK_COLS);
#define CHUNKS(D)                                                                                                       \
  for (int base = 0; base < all; base += CHUNK_ROOM) {                                                                  \
    const dim3 wy_grid(all - base < CHUNK_ROOM ? all - base : CHUNK_ROOM, n_heads);                                     \
    delta_wy_kernel<D><<<wy_grid, CHUNK_THREADS, 0, stream>>>(qn, kn, rec, vp, list, chunks, seq_slot, seq_start, n_seqs, \
                                                              n_heads, n_kv_heads, DVP, most + 1, base);                \
    FG_CHECK_LAUNCH("fg_delta_scan (chunks)");                                                                          \
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,            \
                                         (int)ChunkWalk<D>::SMEM);                                                      \
    FG_CHECK_ARG(e == cudaSuccess, "fg_delta_scan: shared memory: %s", cudaGetErrorString(e));                          \
    const long resident = (long)fg_sm_count() * fg_blocks_per_sm(CHUNK_THREADS, ChunkWalk<D>::SMEM);                    \
    delta_chunk_kernel<D><<<(unsigned)(items < resident ? items : resident), CHUNK_THREADS, ChunkWalk<D>::SMEM, stream>>>( \
        list, chunks, out, out_stride, state, state_stride, seq_slot, seq_start, n_heads, d, dv, DVP, base);            \
    FG_CHECK_LAUNCH("fg_delta_scan (walk)");                                                                            \
  }
    if (DP == 64) {
      CHUNKS(64)
    } else {
      CHUNKS(128)
    }
#undef CHUNKS
  }
  const auto scan = head_decay ? launch_scan<true> : launch_scan<false>;
  const int rc = scan(stream, qn, kn, rec, vp, out, out_stride, state, state_stride, seq_slot, seq_start, n_seqs,
                      n_heads, n_kv_heads, d, dv, DVP, most);
  if (rc != 0) return rc;
  FG_CHECK_LAUNCH("fg_delta_scan");
  return 0;
}

// ---- the read-out's norm and gate -------------------------------------------------------------
// out[t, h, :] = o[t, h, :] * rsqrt(mean(o[t, h, :]^2) + eps) * w[:] * sigmoid(z[t, h, :]), or silu(z) with
// `silu`; a warp a
// (token, head), float32 arithmetic, one rounding.
template <typename TZ>
__global__ void __launch_bounds__(128)
head_norm_gate_kernel(const float* o, long o_stride, const TZ* z, long z_stride, const float* __restrict__ w,
                      TZ* __restrict__ out, long out_stride, const int* __restrict__ req, int n_tokens, int n_heads,
                      int dv, float eps, int silu) {
  const int item = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= n_tokens * n_heads) return;
  const int t = item / n_heads, h = item - t * n_heads;
  if (req[t] < 0) return;
  const float* src = o + (size_t)t * o_stride + h * dv;
  float ss = 0.f;
  for (int c = lane; c < dv; c += 32) ss = fmaf(src[c], src[c], ss);
  ss = warp_sum(ss);
  const float rstd = rsqrtf(ss / (float)dv + eps);
  for (int c = lane; c < dv; c += 32) {
    const float zc = to_f32<TZ>(z[(size_t)t * z_stride + h * dv + c]);
    const float gate = (silu ? zc : 1.f) / (1.f + expf(-zc));
    out[(size_t)t * out_stride + h * dv + c] = from_f32<TZ>(src[c] * rstd * w[c] * gate);
  }
}

extern "C" int fg_head_norm_gate(const float* o, long o_stride, const void* z, long z_stride, int dtype,
                                 const float* w, void* out, long out_stride, const int* req, int n_tokens,
                                 int n_heads, int dv, float eps, int silu, cudaStream_t stream) {
  if (n_tokens == 0) return 0;
  const int blocks = (n_tokens * n_heads + 3) / 4;
  if (dtype == FG_F32)
    head_norm_gate_kernel<float><<<blocks, 128, 0, stream>>>(o, o_stride, (const float*)z, z_stride, w, (float*)out,
                                                             out_stride, req, n_tokens, n_heads, dv, eps, silu);
  else if (dtype == FG_BF16)
    head_norm_gate_kernel<__nv_bfloat16><<<blocks, 128, 0, stream>>>(o, o_stride, (const __nv_bfloat16*)z, z_stride, w,
                                                                     (__nv_bfloat16*)out, out_stride, req, n_tokens,
                                                                     n_heads, dv, eps, silu);
  else
    FG_CHECK_ARG(false, "fg_head_norm_gate: bad dtype %d", dtype);
  FG_CHECK_LAUNCH("fg_head_norm_gate");
  return 0;
}
