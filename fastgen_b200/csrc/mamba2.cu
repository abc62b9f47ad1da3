// The state-space mixer (Mamba-2 form): short causal convolution with SiLU, the recurrence
// over a per-head matrix state, and the gated norm of its output.
//
// The mixer's input projection gives, per token, a row [z | x | B | C | dt] (inner, inner,
// groups*N, groups*N, heads columns).  x, B and C ("xBC", `channels` columns) pass the
// convolution; then, per head h with group g = h / (heads / groups), in float32:
//
//   dt = softplus(dt_raw + dt_bias[h]);   a = exp(-exp(A_log[h]) * dt)
//   S <- a * S + dt * B x^T      (S is N x P, P the head's value size)
//   y = S^T C + D[h] * x
//
// A request's state lives in one float32 row per slot: [heads, P, N] for S (a column's rows side
// by side, as the recurrence's threads hold them), then
// [taps-1, channels] for the convolution's last inputs (oldest first).  It is zero at
// admission, which is also "zeros before the start" for the convolution.  A step may bring a
// sequence any number of tokens; sequences are consecutive runs of tokens with one slot, and
// tokens of slot < 0 are padding that touches nothing.
//
// No sum depends on what else is in the batch.  The recurrence runs token by token, so that its sums do not depend on how
// a prompt was cut either, except in 16-bit serving for sequences that bring many tokens (SC_MIN and more): those go
// chunk by chunk, with float32 sums of another order that are as close to 64 bits.
#include "common.cuh"
#include "long_sequences.cuh"

// ---- convolution + SiLU ---------------------------------------------------------------------
// out[t, c] = silu(bias[c] + sum_k w[c, k] * in[t - (taps-1-k), c]); inputs before the step's
// first token of the sequence come from the state.
constexpr int CONV_THREADS = 128;
constexpr int CONV_MAX_TAPS = 8;

// A thread computes one channel of four consecutive tokens.  Nothing here waits for anything
// else: the slots of the tokens around them are read first, then all the taps' inputs (from the
// step's tokens, or from the state where a sequence's part of the step began less than taps-1
// tokens ago), and neighbouring threads' re-reads hit the cache.
constexpr int CONV_TOKENS = 4;

// TO: the output's type; SILU: whether the sum passes SiLU (else it is stored as it is).
template <typename T, typename TO, bool SILU>
__global__ void __launch_bounds__(CONV_THREADS)
conv_silu_kernel(const T* __restrict__ in, long in_stride, TO* __restrict__ out, long out_stride,
                 const float* __restrict__ w, const float* __restrict__ bias, const float* __restrict__ state,
                 long state_stride, long conv_offset, const int* __restrict__ req, int n_tokens, int channels,
                 int taps) {
  const int c = blockIdx.y * CONV_THREADS + threadIdx.x;
  if (c >= channels) return;
  const int t0 = blockIdx.x * CONV_TOKENS;
  constexpr int BACK = CONV_MAX_TAPS - 1;
  int rq[CONV_TOKENS + BACK];  // rq[j]: the slot of token t0 - BACK + j
#pragma unroll
  for (int j = 0; j < CONV_TOKENS + BACK; ++j) {
    const int t = t0 - BACK + j;
    rq[j] = (t >= 0 && t < n_tokens) ? req[t] : -1;
  }
  float wk[CONV_MAX_TAPS];
#pragma unroll
  for (int k = 0; k < CONV_MAX_TAPS; ++k) wk[k] = k < taps ? w[(size_t)c * taps + k] : 0.f;
  const float bc = bias ? bias[c] : 0.f;
  float v[CONV_TOKENS][CONV_MAX_TAPS];
#pragma unroll
  for (int u = 0; u < CONV_TOKENS; ++u) {
    const int t = t0 + u, slot = rq[u + BACK];
    // how many of the taps-1 tokens before t the step itself brings
    int have = 0;
#pragma unroll
    for (int b = 1; b <= BACK; ++b)
      if (have == b - 1 && b <= taps - 1 && rq[u + BACK - b] == slot) have = b;
#pragma unroll
    for (int k = 0; k < CONV_MAX_TAPS; ++k) {
      v[u][k] = 0.f;
      if (slot >= 0 && k < taps) {
        const int back = taps - 1 - k;  // this tap meets the input `back` tokens ago
        v[u][k] = back <= have ? to_f32<T>(in[(size_t)(t - back) * in_stride + c])
                               : state[(size_t)slot * state_stride + conv_offset +
                                       (size_t)(taps - 1 + have - back) * channels + c];
      }
    }
  }
#pragma unroll
  for (int u = 0; u < CONV_TOKENS; ++u) {
    if (rq[u + BACK] < 0) continue;
    float acc = bc;
#pragma unroll
    for (int k = 0; k < CONV_MAX_TAPS; ++k)
      if (k < taps) acc = fmaf(wk[k], v[u][k], acc);
    out[(size_t)(t0 + u) * out_stride + c] = from_f32<TO>(SILU ? acc / (1.f + expf(-acc)) : acc);
  }
}

// The same for four taps, four channels a thread and CONV_RUN consecutive tokens: where those tokens and the
// three before them are one sequence's, every input is read once, 8 or 16 bytes at a time, and all reads are
// in flight together (the kernel above reads every input four times, a channel at a time).  Other runs (a
// sequence's start, padding) look up each tap's place as above.  The sums are the kernel's above, bit for bit.
// 2,048 tokens of 6,144 channels, bfloat16 -> float32: 105 -> 23 us (its 75 MB take 11.5).
constexpr int CONV_RUN = 8;

template <typename T>
__device__ __forceinline__ float4 conv_load4(const T* p);
template <>
__device__ __forceinline__ float4 conv_load4<float>(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}
template <>
__device__ __forceinline__ float4 conv_load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 r = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void conv_store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void conv_store4(__nv_bfloat16* p, float4 v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 r;
  r.x = *reinterpret_cast<const uint32_t*>(&a);
  r.y = *reinterpret_cast<const uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = r;
}

template <typename T, typename TO, bool SILU>
__global__ void __launch_bounds__(CONV_THREADS)
conv4_silu_kernel(const T* in, long in_stride, TO* out, long out_stride, const float* __restrict__ w,
                  const float* __restrict__ bias, const float* state,
                  long state_stride, long conv_offset, const int* __restrict__ req, int n_tokens, int channels) {
  constexpr int TAPS = 4, BACK = TAPS - 1;
  const int c = (blockIdx.y * CONV_THREADS + threadIdx.x) * 4;
  pdl_trigger();
  if (c >= channels) return;
  const int t0 = blockIdx.x * CONV_RUN;
  int rq[CONV_RUN + BACK];  // rq[j]: the slot of token t0 - BACK + j
  bool one = t0 >= BACK && t0 + CONV_RUN <= n_tokens;
#pragma unroll
  for (int j = 0; j < CONV_RUN + BACK; ++j) {
    const int t = t0 - BACK + j;
    rq[j] = (t >= 0 && t < n_tokens) ? req[t] : -1;
    one = one && rq[j] == rq[0];
  }
  one = one && rq[0] >= 0;
  float wk[4][TAPS];
#pragma unroll
  for (int e = 0; e < 4; ++e)
    *reinterpret_cast<float4*>(wk[e]) = *reinterpret_cast<const float4*>(w + (size_t)(c + e) * TAPS);
  const float4 bc = bias ? *reinterpret_cast<const float4*>(bias + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  pdl_wait();  // (the weights and the slots are the step's from its start)
  auto emit = [&](int t, const float4& v0, const float4& v1, const float4& v2, const float4& v3) {
    float r[4] = {bc.x, bc.y, bc.z, bc.w};
    const float x[TAPS][4] = {{v0.x, v0.y, v0.z, v0.w}, {v1.x, v1.y, v1.z, v1.w}, {v2.x, v2.y, v2.z, v2.w}, {v3.x, v3.y, v3.z, v3.w}};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
#pragma unroll
      for (int k = 0; k < TAPS; ++k) r[e] = fmaf(wk[e][k], x[k][e], r[e]);
      if (SILU) r[e] = r[e] / (1.f + expf(-r[e]));
    }
    conv_store4(out + (size_t)t * out_stride + c, make_float4(r[0], r[1], r[2], r[3]));
  };
  if (one) {
    float4 v[CONV_RUN + BACK];
#pragma unroll
    for (int j = 0; j < CONV_RUN + BACK; ++j) v[j] = conv_load4<T>(in + (size_t)(t0 - BACK + j) * in_stride + c);
#pragma unroll
    for (int u = 0; u < CONV_RUN; ++u) emit(t0 + u, v[u], v[u + 1], v[u + 2], v[u + 3]);
    return;
  }
#pragma unroll
  for (int u = 0; u < CONV_RUN; ++u) {
    const int t = t0 + u, slot = rq[u + BACK];
    if (slot < 0) continue;
    int have = 0;  // how many of the three tokens before t the step itself brings
#pragma unroll
    for (int b = 1; b <= BACK; ++b)
      if (have == b - 1 && rq[u + BACK - b] == slot) have = b;
    float4 v[TAPS];
#pragma unroll
    for (int k = 0; k < TAPS; ++k) {
      const int back = BACK - k;
      v[k] = back <= have ? conv_load4<T>(in + (size_t)(t - back) * in_stride + c)
                          : *reinterpret_cast<const float4*>(state + (size_t)slot * state_stride + conv_offset +
                                                             (size_t)(BACK + have - back) * channels + c);
    }
    emit(t, v[0], v[1], v[2], v[3]);
  }
}

// The state's convolution inputs after the step: the last taps-1 of (old inputs, new inputs).
template <typename T>
__global__ void __launch_bounds__(CONV_THREADS)
conv_state_kernel(const T* in, long in_stride, float* state, long state_stride,
                  long conv_offset, const int* __restrict__ seq_slot, const int* __restrict__ seq_start,
                  int channels, int taps) {
  const int c = blockIdx.y * CONV_THREADS + threadIdx.x;
  pdl_trigger();
  const int slot = seq_slot[blockIdx.x];
  pdl_wait();  // (every block)
  if (c >= channels || slot < 0) return;
  const int start = seq_start[blockIdx.x], n = seq_start[blockIdx.x + 1] - start;
  float* st = state + (size_t)slot * state_stride + conv_offset;
  // ascending k: entry k + n is read before any write reaches it
  for (int k = 0; k < taps - 1; ++k) {
    const int j = n - (taps - 1) + k;
    const float v = j >= 0 ? to_f32<T>(in[(size_t)(start + j) * in_stride + c]) : st[(size_t)(k + n) * channels + c];
    st[(size_t)k * channels + c] = v;
  }
}

// ---- the recurrence ---------------------------------------------------------------------------
// A block works on (sequence, head, 16 columns of P); LANES threads share a column p, each with
// every LANES-th row n of the state in registers (8 threads a column for small states, a warp a
// column from 64 rows on: the recurrence has heads * P * N independent chains and nothing else
// to fill the GPU with).  Tokens are staged through shared
// memory sixteen at a time in two buffers: while a stage is computed, the next one's B, C and x
// arrive by asynchronous copies and its raw step sizes wait in a register.
constexpr int SCAN_PB = 16;      // columns of P a block
constexpr int SCAN_TOKENS = 16;  // tokens a stage
constexpr int SCAN_GROUP = 8;    // tokens whose sums are reduced together

__device__ __forceinline__ void cp_async_4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

template <typename T, int NPT, int SCAN_LANES>
__global__ void __launch_bounds__(SCAN_PB * SCAN_LANES)
ssm_scan_kernel(const float* __restrict__ xbc, long xbc_stride, const T* __restrict__ dt_raw, long dt_stride,
                const float* __restrict__ dt_bias, const float* __restrict__ a_log, const float* __restrict__ d_skip,
                float* __restrict__ y, long y_stride, float* __restrict__ state, long state_stride,
                const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int heads, int groups,
                int N, int P) {
  constexpr int SCAN_THREADS = SCAN_PB * SCAN_LANES;
  extern __shared__ float smem[];
  const int stage_floats = 2 * SCAN_TOKENS * N + SCAN_TOKENS * SCAN_PB + 2 * SCAN_TOKENS;
  auto Bs = [&](int buf) { return smem + buf * stage_floats; };               // [SCAN_TOKENS][N]
  auto Cs = [&](int buf) { return Bs(buf) + SCAN_TOKENS * N; };               // [SCAN_TOKENS][N]
  auto xs = [&](int buf) { return Cs(buf) + SCAN_TOKENS * N; };               // [SCAN_TOKENS][SCAN_PB]
  auto dts = [&](int buf) { return xs(buf) + SCAN_TOKENS * SCAN_PB; };        // [SCAN_TOKENS]
  auto decs = [&](int buf) { return dts(buf) + SCAN_TOKENS; };                // [SCAN_TOKENS]

  const int slot = seq_slot[blockIdx.x];
  if (slot < 0) return;
  const int start = seq_start[blockIdx.x], n_tok = seq_start[blockIdx.x + 1] - start;
  if (n_tok <= 0) return;
  const int h = blockIdx.y, g = h / (heads / groups);
  const int p0 = blockIdx.z * SCAN_PB;
  const int tid = threadIdx.x;
  const int pl = tid / SCAN_LANES, lane = tid % SCAN_LANES;
  const int p = p0 + pl;
  const bool p_ok = p < P;
  const int inner = heads * P;
  const float bias = dt_bias[h];
  const float a = -expf(a_log[h]);
  const float dsk = d_skip[h];

  float* S = state + (size_t)slot * state_stride + (size_t)h * N * P;
  float s[NPT];
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const int n = lane + SCAN_LANES * i;
    s[i] = (p_ok && n < N) ? S[(size_t)p * N + n] : 0.f;
  }

  const int n_stages = (n_tok + SCAN_TOKENS - 1) / SCAN_TOKENS;
  auto issue = [&](int k) {
    const int buf = k & 1, t0 = k * SCAN_TOKENS, nt = min(SCAN_TOKENS, n_tok - t0);
    float *bs = Bs(buf), *cs = Cs(buf), *xx = xs(buf);
    for (int i = tid; i < nt * N; i += SCAN_THREADS) {
      const int tt = i / N, n = i - tt * N;
      const float* row = xbc + (size_t)(start + t0 + tt) * xbc_stride + inner + g * N + n;
      cp_async_4(bs + i, row);
      cp_async_4(cs + i, row + groups * N);
    }
    for (int i = tid; i < nt * SCAN_PB; i += SCAN_THREADS) {
      const int tt = i / SCAN_PB, pp = i - tt * SCAN_PB;
      if (p0 + pp < P) cp_async_4(xx + i, xbc + (size_t)(start + t0 + tt) * xbc_stride + h * P + p0 + pp);
      else xx[i] = 0.f;
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto raw_dt = [&](int k) {
    const int t = k * SCAN_TOKENS + tid;
    return (tid < SCAN_TOKENS && t < n_tok) ? to_f32<T>(dt_raw[(size_t)(start + t) * dt_stride + h]) : 0.f;
  };
  issue(0);
  float dtr = raw_dt(0);

  for (int k = 0; k < n_stages; ++k) {
    const int buf = k & 1, t0 = k * SCAN_TOKENS, nt = min(SCAN_TOKENS, n_tok - t0);
    if (tid < nt) {
      const float v = dtr + bias;
      const float dt = v > 20.f ? v : log1pf(expf(v));
      dts(buf)[tid] = dt;
      decs(buf)[tid] = expf(a * dt);
    }
    if (k + 1 < n_stages) {
      issue(k + 1);
      dtr = raw_dt(k + 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const float *bs = Bs(buf), *cs = Cs(buf), *xx = xs(buf), *dd = dts(buf), *de = decs(buf);
    // eight tokens at a time: their sums over the state's rows are reduced across the column's
    // threads together, and thread j of the column stores token j's output
    for (int tt0 = 0; tt0 < nt; tt0 += SCAN_GROUP) {
      float acc[SCAN_GROUP];
#pragma unroll
      for (int u = 0; u < SCAN_GROUP; ++u) {
        const int tt = tt0 + u;
        float a0 = 0.f, a1 = 0.f;
        if (tt < nt) {
          const float dec = de[tt];
          const float dx = dd[tt] * xx[tt * SCAN_PB + pl];
#pragma unroll
          for (int i = 0; i < NPT; ++i) {
            const int n = lane + SCAN_LANES * i;
            if (n < N) {
              s[i] = fmaf(dec, s[i], bs[tt * N + n] * dx);
              if (i & 1) a1 = fmaf(s[i], cs[tt * N + n], a1);
              else a0 = fmaf(s[i], cs[tt * N + n], a0);
            }
          }
        }
        acc[u] = a0 + a1;
      }
#pragma unroll
      for (int o = SCAN_LANES / 2; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < SCAN_GROUP; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
      float mine = 0.f;
#pragma unroll
      for (int u = 0; u < SCAN_GROUP; ++u)
        if (lane == u) mine = acc[u];
      const int tt = tt0 + lane;
      if (lane < SCAN_GROUP && tt < nt && p_ok) y[(size_t)(start + t0 + tt) * y_stride + h * P + p] = fmaf(dsk, xx[tt * SCAN_PB + pl], mine);
    }
    __syncthreads();  // the stage is read to its end before the copies after next overwrite it
  }
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const int n = lane + SCAN_LANES * i;
    if (p_ok && n < N) S[(size_t)p * N + n] = s[i];
  }
}

// ---- the recurrence, states of 64, 128 or 256 rows ------------------------------------------------
// The same recurrence with fewer instructions a state element: N = 32 * NPT is a compile-time
// number (no bounds to test, every address an immediate), B and C of a token sit side by side in
// shared memory (one 8-byte load brings both), a warp owns two columns of P (a loaded pair serves
// both), and the sums of 8 tokens x 2 columns over the state's rows are reduced by halving
// exchanges (16 shuffles for the 16 sums) that leave sum k in lanes 2k and 2k + 1.
constexpr int TS_COLS = 2;                       // columns of P a warp
constexpr int TS_WARPS = SCAN_PB / TS_COLS;      // warps a block
constexpr int TS_THREADS = 32 * TS_WARPS;

template <typename T, int NPT>
__global__ void __launch_bounds__(TS_THREADS)
ssm_scan_tiled_kernel(const float* xbc, long xbc_stride, const T* dt_raw, long dt_stride,
                      const float* __restrict__ dt_bias, const float* __restrict__ a_log,
                      const float* __restrict__ d_skip, float* y, long y_stride,
                      float* state, long state_stride, const int* __restrict__ seq_slot,
                      const int* __restrict__ seq_start, int heads, int groups, int P, int most) {
  pdl_trigger();
  constexpr int N = 32 * NPT;
  constexpr int STAGE = 2 * SCAN_TOKENS * N + SCAN_TOKENS * SCAN_PB + 2 * SCAN_TOKENS;  // floats
  extern __shared__ __align__(16) float smem[];
  auto BC = [&](int buf) { return reinterpret_cast<float2*>(smem + buf * STAGE); };      // [TOKENS][N] (B, C)
  auto xs = [&](int buf) { return smem + buf * STAGE + 2 * SCAN_TOKENS * N; };           // [TOKENS][SCAN_PB]
  auto dts = [&](int buf) { return xs(buf) + SCAN_TOKENS * SCAN_PB; };
  auto decs = [&](int buf) { return dts(buf) + SCAN_TOKENS; };

  const int slot = seq_slot[blockIdx.x];
  pdl_wait();  // (every block: one that left before would let the next kernel pass the one before this)
  if (slot < 0) return;
  const int start = seq_start[blockIdx.x], n_tok = seq_start[blockIdx.x + 1] - start;
  if (n_tok <= 0 || n_tok > most) return;  // (more than `most`: ssm_chunk_kernel's)
  const int h = blockIdx.y, g = h / (heads / groups);
  const int p0 = blockIdx.z * SCAN_PB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int pc = p0 + TS_COLS * warp;  // this warp's first column
  const int inner = heads * P;
  const float bias = dt_bias[h];
  const float a = -expf(a_log[h]);
  const float dsk = d_skip[h];

  float* S = state + (size_t)slot * state_stride + (size_t)h * N * P;
  float s[TS_COLS][NPT];
#pragma unroll
  for (int c = 0; c < TS_COLS; ++c)
#pragma unroll
    for (int i = 0; i < NPT; ++i) s[c][i] = pc + c < P ? S[(size_t)(pc + c) * N + lane + 32 * i] : 0.f;

  const int n_stages = (n_tok + SCAN_TOKENS - 1) / SCAN_TOKENS;
  auto issue = [&](int k) {
    const int buf = k & 1, t0 = k * SCAN_TOKENS, nt = min(SCAN_TOKENS, n_tok - t0);
    float* bc = smem + buf * STAGE;
    float* xx = xs(buf);
    for (int i = tid; i < nt * N; i += TS_THREADS) {
      const int tt = i / N, n = i - tt * N;
      const float* row = xbc + (size_t)(start + t0 + tt) * xbc_stride + inner + g * N + n;
      cp_async_4(bc + 2 * i, row);
      cp_async_4(bc + 2 * i + 1, row + groups * N);
    }
    for (int i = tid; i < nt * SCAN_PB; i += TS_THREADS) {
      const int tt = i / SCAN_PB, pp = i - tt * SCAN_PB;
      if (p0 + pp < P) cp_async_4(xx + i, xbc + (size_t)(start + t0 + tt) * xbc_stride + h * P + p0 + pp);
      else xx[i] = 0.f;
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto raw_dt = [&](int k) {
    const int t = k * SCAN_TOKENS + tid;
    return (tid < SCAN_TOKENS && t < n_tok) ? to_f32<T>(dt_raw[(size_t)(start + t) * dt_stride + h]) : 0.f;
  };
  issue(0);
  float dtr = raw_dt(0);

  for (int k = 0; k < n_stages; ++k) {
    const int buf = k & 1, t0 = k * SCAN_TOKENS, nt = min(SCAN_TOKENS, n_tok - t0);
    if (tid < nt) {
      const float v = dtr + bias;
      const float dt = v > 20.f ? v : log1pf(expf(v));
      dts(buf)[tid] = dt;
      decs(buf)[tid] = expf(a * dt);
    }
    if (k + 1 < n_stages) {
      issue(k + 1);
      dtr = raw_dt(k + 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const float2* bc = BC(buf);
    const float *xx = xs(buf), *dd = dts(buf), *de = decs(buf);
    for (int tt0 = 0; tt0 < nt; tt0 += SCAN_GROUP) {
      float acc[TS_COLS * SCAN_GROUP];  // [column][token of the group]
#pragma unroll
      for (int u = 0; u < SCAN_GROUP; ++u) {
        const int tt = tt0 + u;
        float a0 = 0.f, a1 = 0.f;
        if (tt < nt) {
          const float dec = de[tt], dtv = dd[tt];
          const float2 xv = *reinterpret_cast<const float2*>(xx + tt * SCAN_PB + TS_COLS * warp);
          const float dx0 = dtv * xv.x, dx1 = dtv * xv.y;
#pragma unroll
          for (int i = 0; i < NPT; ++i) {
            const float2 v = bc[tt * N + lane + 32 * i];
            s[0][i] = fmaf(dec, s[0][i], v.x * dx0);
            a0 = fmaf(s[0][i], v.y, a0);
            s[1][i] = fmaf(dec, s[1][i], v.x * dx1);
            a1 = fmaf(s[1][i], v.y, a1);
          }
        }
        acc[u] = a0;
        acc[SCAN_GROUP + u] = a1;
      }
      // halving exchanges: after the step with mask m a lane keeps the half of its sums that its
      // bit m chooses, with the partner's share added
#pragma unroll
      for (int half = TS_COLS * SCAN_GROUP / 2, mask = 16; half >= 1; half >>= 1, mask >>= 1) {
        const bool upper = (lane & mask) != 0;
#pragma unroll
        for (int j = 0; j < half; ++j) {
          const float send = upper ? acc[j] : acc[j + half];
          const float keep = upper ? acc[j + half] : acc[j];
          acc[j] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
        }
      }
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);  // (16 sums use the masks 16, 8, 4, 2)
      const int kidx = (lane >> 1) & 15, c = kidx >> 3, tt = tt0 + (kidx & 7);
      if (!(lane & 1) && tt < nt && pc + c < P)
        y[(size_t)(start + t0 + tt) * y_stride + h * P + pc + c] =
            fmaf(dsk, xx[tt * SCAN_PB + TS_COLS * warp + c], acc[0]);
    }
    __syncthreads();  // the stage is read to its end before the copies after next overwrite it
  }
#pragma unroll
  for (int c = 0; c < TS_COLS; ++c)
#pragma unroll
    for (int i = 0; i < NPT; ++i)
      if (pc + c < P) S[(size_t)(pc + c) * N + lane + 32 * i] = s[c][i];
}

// ---- sequences of many tokens, 16-bit serving: chunks ---------------------------------------------------
// Token by token the recurrence takes about 390 cycles a token and reads its operands from shared memory once per
// token.  Over a chunk of 32 tokens from state S0 it is also, with D[i][j] = a_{j+1} .. a_i (a product of the
// tokens' decays), e_i = a_1 .. a_i and w_j = D[32][j] dt_j,
//
//     Y = e (C S0) + M X + D_skip X,  M[i][j] = (C_i . B_j) D[i][j] dt_j  (j <= i)
//     S <- e_32 S0 + B^T (w X)
//
// 2,048 tokens of 64 heads, 128 x 64 states: 420 -> 202 us and 17 of preparing (the multiply-adds alone take 75; what
// bounds the walk is shared memory: a 16-byte read a lane takes its 4 cycles whoever shares the address, and 4 x 4
// numbers a thread want two such reads for 16 multiply-adds).
//
// ssm_chunk_prepare_kernel forms M, e and w for all chunks side by side (a block a (chunk, group): C B^T once for the
// group's heads); ssm_chunk_kernel walks the chunks of one (sequence, head, 32 columns), a state of 4 x 4 numbers a
// thread.  float32 multiply-adds (the decays and C B^T in 64 bits); the sums have another order than the token kernel's,
// so the float32 mode, whose results do not depend on how a prompt is cut, keeps that one.  (The chunked form is
// published, for instance in Dao and Gu, "Transformers are SSMs", 2024.)
constexpr int SC_TOKENS = 32;   // tokens a chunk
constexpr int SC_COLS = 32;     // columns of P a block of the walk
constexpr int SC_THREADS = 256;
constexpr int SC_STAGES = 2;
// Fewest tokens of a sequence that takes this way (prepared and walked): where the two meet.  Chunks against tokens, us at
// 96 / 112 / 128 tokens: one sequence 22.8 / 25.8 / 25.8 against 22.0 / 25.3 / 28.6, four 60 / 75 / 75 against
// 64 / 74 / 84, eight 101 / 125 / 125 against 121 / 143 / 165.  (At 64: 19.3 against 15.5, 47 against 44, 79 against 83.)
constexpr int SC_MIN = 112;
// Products of the state that are summed by themselves before they join a token's sum: the token kernel's sums over N are
// trees (a few products a lane, then exchanges), and one chain over N is twice as far from 64 bits as those
// (1.9e-7 against 1.05e-7 at N = 128; with runs of 16 and C B^T summed in 64 bits 1.0e-7, for 5 % of the walk's time).
constexpr int SC_RUN = 16;
template <int V>
struct Whole {
  static constexpr int value = V;
};
constexpr int SC_REC = SC_TOKENS * SC_TOKENS + 2 * SC_TOKENS;  // floats of a (chunk, head): M, e, w

__device__ __forceinline__ void cp_async_16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(ok ? 16 : 0)
               : "memory");
}

template <typename T, int N>
__global__ void __launch_bounds__(SC_THREADS)
ssm_chunk_prepare_kernel(const float* __restrict__ xbc, long xbc_stride, const T* __restrict__ dt_raw, long dt_stride,
                         const float* __restrict__ dt_bias, const float* __restrict__ a_log, long_seq::Head* list,
                         float* __restrict__ chunks, const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int n_seqs, int heads,
                         int groups, int P) {
  __shared__ __align__(16) float bs[SC_TOKENS][N + 4];
  __shared__ __align__(16) float cs[SC_TOKENS][N + 4];
  __shared__ double gram[SC_TOKENS][SC_TOKENS + 1];
  __shared__ float decs[SC_THREADS / 32][SC_TOKENS];
  const int g = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const auto found = long_seq::find_chunk<SC_TOKENS, SC_THREADS>(seq_slot, seq_start, n_seqs, SC_MIN, blockIdx.x,
                                                                 blockIdx.x + g == 0 ? list : nullptr);
  if (found.seq < 0) return;
  const int c = blockIdx.x - found.first_chunk;
  const int t0 = seq_start[found.seq] + c * SC_TOKENS, nt = min(SC_TOKENS, found.tokens - c * SC_TOKENS), inner = heads * P;
  for (int i = tid; i < SC_TOKENS * (N / 4); i += SC_THREADS) {
    const int t = i / (N / 4), w = i % (N / 4) * 4;
    float4 bv = make_float4(0.f, 0.f, 0.f, 0.f), cv = bv;
    if (t < nt) {
      const float* row = xbc + (size_t)(t0 + t) * xbc_stride + inner + g * N + w;
      bv = *reinterpret_cast<const float4*>(row);
      cv = *reinterpret_cast<const float4*>(row + groups * N);
    }
    *reinterpret_cast<float4*>(&bs[t][w]) = bv;
    *reinterpret_cast<float4*>(&cs[t][w]) = cv;
  }
  __syncthreads();
  {
    const int ib = tid >> 4, jb = tid & 15;
    // short chains: a sum over N in stretches of 16 that are four chains each, added up in 64 bits (see SC_RUN)
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 2
    for (int w0 = 0; w0 < N; w0 += 16) {
      float4 run[2][2];
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int f = 0; f < 2; ++f) run[e][f] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = w0; w < w0 + 16; w += 4) {
        float4 cv[2], bv[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          cv[e] = *reinterpret_cast<const float4*>(&cs[ib + 16 * e][w]);
          bv[e] = *reinterpret_cast<const float4*>(&bs[jb + 16 * e][w]);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int f = 0; f < 2; ++f) {
            run[e][f].x = fmaf(cv[e].x, bv[f].x, run[e][f].x);
            run[e][f].y = fmaf(cv[e].y, bv[f].y, run[e][f].y);
            run[e][f].z = fmaf(cv[e].z, bv[f].z, run[e][f].z);
            run[e][f].w = fmaf(cv[e].w, bv[f].w, run[e][f].w);
          }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int f = 0; f < 2; ++f) acc[e][f] += (run[e][f].x + run[e][f].y) + (run[e][f].z + run[e][f].w);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int f = 0; f < 2; ++f) gram[ib + 16 * e][jb + 16 * f] = acc[e][f];
  }
  __syncthreads();
  const int per = heads / groups;
  for (int hh = warp; hh < per; hh += SC_THREADS / 32) {  // a warp a head, a lane a column j
    const int h = g * per + hh;
    float dt = 0.f, dec = 1.f;  // tokens beyond the sequence change nothing
    if (lane < nt) {
      const float v = to_f32<T>(dt_raw[(size_t)(t0 + lane) * dt_stride + h]) + dt_bias[h];
      dt = v > 20.f ? v : log1pf(expf(v));
      dec = expf(-expf(a_log[h]) * dt);
    }
    decs[warp][lane] = dec;
    __syncwarp();
    float* rec = chunks + ((size_t)blockIdx.x * heads + h) * SC_REC;
    // M is rounded once, from 64 bits: its error, unlike that of a state's numbers, is the same for all of P
    double d = 1.0, e = 1.0;
    for (int i = 0; i < SC_TOKENS; ++i) {
      const double ai = decs[warp][i];
      e *= ai;
      if (i > lane) d *= ai;
      rec[i * SC_TOKENS + lane] = i >= lane ? (float)(gram[i][lane] * (d * dt)) : 0.f;
      if (lane == 0) rec[SC_TOKENS * SC_TOKENS + i] = (float)e;
    }
    rec[SC_TOKENS * SC_TOKENS + SC_TOKENS + lane] = (float)(d * dt);
    __syncwarp();
  }
}

template <int N>
struct ScanWalk {
  static constexpr int SCN = N + 4, SM = SC_TOKENS + 4, SP = SC_COLS;
  static constexpr int C = 0, B = C + SC_TOKENS * SCN, M = B + SC_TOKENS * N, X = M + SC_TOKENS * SM, E = X + SC_TOKENS * SP,
                       W = E + SC_TOKENS, BUF = W + SC_TOKENS;
  static constexpr int GROUPS = 4;  // groups of threads that share out the sums of C S0 and M X
  static constexpr int S = SC_STAGES * BUF, XW = S + N * SP, PART = XW + SC_TOKENS * SP, SPART = SP + 4;
  static constexpr size_t SMEM = sizeof(float) * (PART + GROUPS * SC_TOKENS * SPART);
};

template <int N>
__global__ void __launch_bounds__(SC_THREADS, 1)
ssm_chunk_kernel(const float* __restrict__ xbc, long xbc_stride, long_seq::Head* list, const float* __restrict__ chunks,
                 const float* __restrict__ d_skip, float* __restrict__ y, long y_stride, float* __restrict__ state,
                 long state_stride, const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int heads,
                 int groups, int P) {
  using L = ScanWalk<N>;
  constexpr int NROWS = N / 32;  // rows of the state a thread, side by side
  extern __shared__ __align__(16) float smem[];
  float *const s_s = smem + L::S, *const xw_s = smem + L::XW, *const part = smem + L::PART;
  const int tid = threadIdx.x, pb = tid & 7, nb = tid >> 3;
  const int columns = (P + SC_COLS - 1) / SC_COLS, inner = heads * P;
  for (long_seq::Items items(list, heads * columns); items.more(); items.draw()) {
    const auto sequence = items.sequence();
    const int h = items.part() / columns, p0 = items.part() % columns * SC_COLS, g = h / (heads / groups);
    const int n = sequence.tokens, first = sequence.first_chunk, start = seq_start[sequence.seq];
    const int n_chunks = (n + SC_TOKENS - 1) / SC_TOKENS;
    const float dsk = d_skip[h];

    auto issue = [&](int c) {
      float* buf = smem + c % SC_STAGES * L::BUF;
      const int t0 = start + c * SC_TOKENS, nt = min(SC_TOKENS, n - c * SC_TOKENS);
      for (int i = tid; i < SC_TOKENS * (N / 4); i += SC_THREADS) {
        const int t = i / (N / 4), w = i % (N / 4) * 4;
        const float* row = xbc + (size_t)(t < nt ? t0 + t : t0) * xbc_stride + inner + g * N + w;
        cp_async_16(buf + L::B + t * N + w, row, t < nt);
        cp_async_16(buf + L::C + t * L::SCN + w, row + groups * N, t < nt);
      }
      const float* rec = chunks + ((size_t)(first + c) * heads + h) * SC_REC;
      {
        const int t = tid / 8, w = tid % 8 * 4;  // 32 rows of 32 numbers: M and x
        cp_async_16(buf + L::M + t * L::SM + w, rec + t * SC_TOKENS + w, true);
        const bool ok = t < nt && p0 + w < P;
        cp_async_16(buf + L::X + t * L::SP + w, ok ? xbc + (size_t)(t0 + t) * xbc_stride + h * P + p0 + w : xbc, ok);
      }
      if (tid < 2 * SC_TOKENS / 4) cp_async_16(buf + L::E + tid * 4, rec + SC_TOKENS * SC_TOKENS + tid * 4, true);
    };
    issue(0);
    asm volatile("cp.async.commit_group;\n" ::: "memory");

    // the state: rows NROWS nb + r, columns 4 pb .. + 3
    float* const st = state + (size_t)seq_slot[sequence.seq] * state_stride + (size_t)h * N * P;
    float s[NROWS][4];
#pragma unroll
    for (int r = 0; r < NROWS; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int p = p0 + 4 * pb + e;
        s[r][e] = p < P ? st[(size_t)p * N + NROWS * nb + r] : 0.f;
      }
    // the sums of C S0 and M X: group q takes a quarter of the state's rows and of the tokens, a thread 4 x 4 places
    const int q = tid >> 6, ib = (tid & 63) >> 3;
    for (int c = 0; c < n_chunks; ++c) {
      const float* buf = smem + c % SC_STAGES * L::BUF;
#pragma unroll
      for (int r = 0; r < NROWS; ++r)
        *reinterpret_cast<float4*>(s_s + (NROWS * nb + r) * L::SP + 4 * pb) = make_float4(s[r][0], s[r][1], s[r][2], s[r][3]);
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      __syncthreads();  // the chunk has landed, the state stands in shared memory, the buffer of the chunk before is free
      if (c + 1 < n_chunks) issue(c + 1);
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      bool finite;
      {  // w X for the state's update
        const int t = tid / 8, w = tid % 8 * 4;
        const float4 x = *reinterpret_cast<const float4*>(buf + L::X + t * L::SP + w);
        finite = isfinite(x.x) && isfinite(x.y) && isfinite(x.z) && isfinite(x.w);
        const float wt = buf[L::W + t];
        *reinterpret_cast<float4*>(xw_s + t * L::SP + w) = make_float4(x.x * wt, x.y * wt, x.z * wt, x.w * wt);
      }
      float acc[4][4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int f = 0; f < 4; ++f) acc[e][f] = 0.f;
      auto products = [&](const float* left, int left_stride, const float* right, int from, auto count, auto run_length) {
        constexpr int COUNT = decltype(count)::value, RUN = decltype(run_length)::value;
#pragma unroll 1
        for (int k0 = from; k0 < from + COUNT; k0 += RUN) {
          float run[4][4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int f = 0; f < 4; ++f) run[e][f] = 0.f;
#pragma unroll 2
          for (int k = k0; k < k0 + RUN; k += 4) {
            float4 a[4], v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              a[e] = *reinterpret_cast<const float4*>(left + (ib + 8 * e) * left_stride + k);
              v[e] = *reinterpret_cast<const float4*>(right + (k + e) * L::SP + 4 * pb);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float ae[4] = {a[e].x, a[e].y, a[e].z, a[e].w};
#pragma unroll
              for (int f = 0; f < 4; ++f) {
                run[e][0] = fmaf(ae[f], v[f].x, run[e][0]);
                run[e][1] = fmaf(ae[f], v[f].y, run[e][1]);
                run[e][2] = fmaf(ae[f], v[f].z, run[e][2]);
                run[e][3] = fmaf(ae[f], v[f].w, run[e][3]);
              }
            }
          }
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int f = 0; f < 4; ++f) acc[e][f] += run[e][f];
        }
      };
      products(buf + L::C, L::SCN, s_s, q * (N / 4), Whole<N / 4>(), Whole<SC_RUN>());
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float ei = buf[L::E + ib + 8 * e];
#pragma unroll
        for (int f = 0; f < 4; ++f) acc[e][f] *= ei;
      }
      products(buf + L::M, L::SM, buf + L::X, q * (SC_TOKENS / 4), Whole<SC_TOKENS / 4>(), Whole<SC_TOKENS / 4>());
#pragma unroll
      for (int e = 0; e < 4; ++e)
        *reinterpret_cast<float4*>(part + (q * SC_TOKENS + ib + 8 * e) * L::SPART + 4 * pb) =
            make_float4(acc[e][0], acc[e][1], acc[e][2], acc[e][3]);
      // (an infinity or NaN in X would reach the tokens before its own through M's zeros)
      const bool causal = __syncthreads_or(!finite) != 0;
      {  // a token's four columns a thread: the groups' sums in order
        const int t = tid / 8, w = tid % 8 * 4;
        const float4 x = *reinterpret_cast<const float4*>(buf + L::X + t * L::SP + w);
        float4 v = *reinterpret_cast<const float4*>(part + t * L::SPART + w);
#pragma unroll
        for (int i = 1; i < L::GROUPS; ++i) {
          const float4 u = *reinterpret_cast<const float4*>(part + (i * SC_TOKENS + t) * L::SPART + w);
          v.x += u.x;
          v.y += u.y;
          v.z += u.z;
          v.w += u.w;
        }
        if (causal) {  // the token's sums once more, over the tokens up to it alone
          v = make_float4(0.f, 0.f, 0.f, 0.f);
          auto add = [&](float a, const float* row) {
            const float4 u = *reinterpret_cast<const float4*>(row + w);
            v = make_float4(fmaf(a, u.x, v.x), fmaf(a, u.y, v.y), fmaf(a, u.z, v.z), fmaf(a, u.w, v.w));
          };
          for (int k = 0; k < N; ++k) add(buf[L::C + t * L::SCN + k], s_s + k * L::SP);
          const float et = buf[L::E + t];
          v = make_float4(v.x * et, v.y * et, v.z * et, v.w * et);
          for (int k = 0; k <= t; ++k) add(buf[L::M + t * L::SM + k], buf + L::X + k * L::SP);
          __syncthreads();  // the state in shared memory has been read
        }
        if (c * SC_TOKENS + t < n && p0 + w < P)
          *reinterpret_cast<float4*>(y + (size_t)(start + c * SC_TOKENS + t) * y_stride + h * P + p0 + w) =
              make_float4(fmaf(dsk, x.x, v.x), fmaf(dsk, x.y, v.y), fmaf(dsk, x.z, v.z), fmaf(dsk, x.w, v.w));
      }
      const float whole = buf[L::E + SC_TOKENS - 1];
#pragma unroll
      for (int r = 0; r < NROWS; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[r][e] *= whole;
#pragma unroll 8
      for (int t = 0; t < SC_TOKENS; ++t) {
        const float4 x = *reinterpret_cast<const float4*>(xw_s + t * L::SP + 4 * pb);
        __align__(16) float bt[NROWS];
        if (NROWS == 4) *reinterpret_cast<float4*>(bt) = *reinterpret_cast<const float4*>(buf + L::B + t * N + 4 * nb);
        else *reinterpret_cast<float2*>(bt) = *reinterpret_cast<const float2*>(buf + L::B + t * N + 2 * nb);
#pragma unroll
        for (int r = 0; r < NROWS; ++r) {
          const float bv = bt[r];
          s[r][0] = fmaf(bv, x.x, s[r][0]);
          s[r][1] = fmaf(bv, x.y, s[r][1]);
          s[r][2] = fmaf(bv, x.z, s[r][2]);
          s[r][3] = fmaf(bv, x.w, s[r][3]);
        }
      }
      // (the next chunk's state goes to shared memory at once: its readers are through since the barrier above;
      // w X is written behind the next barrier)
    }
#pragma unroll
    for (int r = 0; r < NROWS; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int p = p0 + 4 * pb + e;
        if (p < P) st[(size_t)p * N + NROWS * nb + r] = s[r][e];
      }
  }
}

// ---- gate, then RMS norm in equal parts ---------------------------------------------------------
// out[t, part] = v * rsqrt(mean(v^2) + eps) * w with v = y * silu(z) over the part's columns.
constexpr int GN_THREADS = 256;

template <typename T>
__global__ void __launch_bounds__(GN_THREADS)
gated_part_norm_kernel(const float* __restrict__ y, long y_stride, const T* __restrict__ z, long z_stride,
                       const float* __restrict__ w, T* __restrict__ out, long out_stride, const int* __restrict__ req,
                       int part, float eps) {
  __shared__ float scratch[32];
  const int t = blockIdx.x, c0 = blockIdx.y * part;
  if (req[t] < 0) return;
  const float* yr = y + (size_t)t * y_stride + c0;
  const T* zr = z + (size_t)t * z_stride + c0;
  float ss = 0.f;
  for (int d = threadIdx.x; d < part; d += GN_THREADS) {
    const float zv = to_f32<T>(zr[d]);
    const float v = yr[d] * (zv / (1.f + expf(-zv)));
    ss += v * v;
  }
  ss = block_sum(ss, scratch);
  const float rstd = 1.f / sqrtf(ss / (float)part + eps);
  for (int d = threadIdx.x; d < part; d += GN_THREADS) {
    const float zv = to_f32<T>(zr[d]);
    const float v = yr[d] * (zv / (1.f + expf(-zv)));
    out[(size_t)t * out_stride + c0 + d] = from_f32<T>(v * rstd * w[c0 + d]);
  }
}

// Parts of up to 1,024 columns: a warp a (token, part), the part's values in registers between the
// sum of squares and the scaling, so y and z are read once.
constexpr int GW_WARPS = 8;
constexpr int GW_ITEMS = 32;

template <typename T>
__global__ void __launch_bounds__(GW_WARPS * 32)
gated_part_norm_warp_kernel(const float* __restrict__ y, long y_stride, const T* __restrict__ z, long z_stride,
                            const float* __restrict__ w, T* __restrict__ out, long out_stride,
                            const int* __restrict__ req, int n_tokens, int parts, int part, float eps) {
  const int lane = threadIdx.x & 31;
  const long item = (long)blockIdx.x * GW_WARPS + (threadIdx.x >> 5);
  if (item >= (long)n_tokens * parts) return;
  const int t = item / parts, c0 = (item - (long)t * parts) * part;
  if (req[t] < 0) return;
  const float* yr = y + (size_t)t * y_stride + c0;
  const T* zr = z + (size_t)t * z_stride + c0;
  float v[GW_ITEMS];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < GW_ITEMS; ++i) {
    const int d = lane + 32 * i;
    v[i] = 0.f;
    if (d < part) {
      const float zv = to_f32<T>(zr[d]);
      v[i] = yr[d] * (zv / (1.f + expf(-zv)));
    }
    ss += v[i] * v[i];
  }
  ss = warp_sum(ss);
  const float rstd = 1.f / sqrtf(ss / (float)part + eps);
#pragma unroll
  for (int i = 0; i < GW_ITEMS; ++i) {
    const int d = lane + 32 * i;
    if (d < part) out[(size_t)t * out_stride + c0 + d] = from_f32<T>(v[i] * rstd * w[c0 + d]);
  }
}

// Parts of 128, 256, 512 or 1,024 columns: the same sums with a compile-time number of columns a lane, so that
// all of a part's loads are in flight together and nothing is tested (2,048 tokens of 8 parts of 512: 43 -> 19 us;
// its 67 MB take 10).
template <typename T, int ITEMS>
__global__ void __launch_bounds__(GW_WARPS * 32)
gated_part_norm_whole_kernel(const float* y, long y_stride, const T* z, long z_stride,
                             const float* __restrict__ w, T* out, long out_stride,
                             const int* __restrict__ req, int n_tokens, int parts, float eps) {
  constexpr int PART = ITEMS * 32;
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const long item = (long)blockIdx.x * GW_WARPS + (threadIdx.x >> 5);
  pdl_wait();
  if (item >= (long)n_tokens * parts) return;
  const int t = item / parts, c0 = (int)(item - (long)t * parts) * PART;
  if (req[t] < 0) return;
  const float* yr = y + (size_t)t * y_stride + c0 + lane;
  const T* zr = z + (size_t)t * z_stride + c0 + lane;
  float v[ITEMS], zv[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    v[i] = yr[32 * i];
    zv[i] = to_f32<T>(zr[32 * i]);
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    v[i] *= zv[i] / (1.f + expf(-zv[i]));
    ss += v[i] * v[i];
  }
  ss = warp_sum(ss);
  const float rstd = 1.f / sqrtf(ss / (float)PART + eps);
#pragma unroll
  for (int i = 0; i < ITEMS; ++i)
    out[(size_t)t * out_stride + c0 + lane + 32 * i] = from_f32<T>(v[i] * rstd * w[c0 + lane + 32 * i]);
}

// ---- C interface -----------------------------------------------------------------------------------

// A causal convolution over time per channel, from and into the state's last inputs, with a choice
// of activation (act 1: SiLU, 0: none) and of the output's type (out_dtype).
template <typename T, typename TO>
static int launch_time_conv(const T* in, long proj_stride, TO* out, long out_stride, const float* w, const float* bias,
                            float* state, long state_stride, long conv_offset, const int* req, const int* seq_slot,
                            const int* seq_start, int n_tokens, int n_seqs, int channels, int taps, int act,
                            cudaStream_t stream) {
  const dim3 grid((n_tokens + CONV_TOKENS - 1) / CONV_TOKENS, (channels + CONV_THREADS - 1) / CONV_THREADS);
  const dim3 sgrid(n_seqs, grid.y);
  // four taps, and every row of inputs, weights, state and results in whole aligned groups of four channels
  const bool fours = taps == 4 && channels % 4 == 0 && proj_stride % 4 == 0 && out_stride % 4 == 0 && state_stride % 4 == 0 &&
                     conv_offset % 4 == 0 && (uintptr_t)in % (4 * sizeof(T)) == 0 && (uintptr_t)out % (4 * sizeof(TO)) == 0 &&
                     (((uintptr_t)w | (uintptr_t)bias | (uintptr_t)state) & 15) == 0;
  const dim3 fgrid((n_tokens + CONV_RUN - 1) / CONV_RUN, (channels / 4 + CONV_THREADS - 1) / CONV_THREADS);
  if (fours && act)
    fg_launch_pdl(conv4_silu_kernel<T, TO, true>, fgrid, dim3(CONV_THREADS), 0, stream, in, proj_stride, out, out_stride, w,
                  bias, state, state_stride, conv_offset, req, n_tokens, channels);
  else if (fours)
    fg_launch_pdl(conv4_silu_kernel<T, TO, false>, fgrid, dim3(CONV_THREADS), 0, stream, in, proj_stride, out, out_stride, w,
                  bias, state, state_stride, conv_offset, req, n_tokens, channels);
  else if (act)
    conv_silu_kernel<T, TO, true><<<grid, CONV_THREADS, 0, stream>>>(in, proj_stride, out, out_stride, w, bias, state,
                                                                     state_stride, conv_offset, req, n_tokens, channels,
                                                                     taps);
  else
    conv_silu_kernel<T, TO, false><<<grid, CONV_THREADS, 0, stream>>>(in, proj_stride, out, out_stride, w, bias, state,
                                                                      state_stride, conv_offset, req, n_tokens,
                                                                      channels, taps);
  FG_CHECK_LAUNCH("fg_time_conv");
  if (taps > 1)
    fg_launch_pdl(conv_state_kernel<T>, sgrid, dim3(CONV_THREADS), 0, stream, in, proj_stride, state, state_stride, conv_offset,
                  seq_slot, seq_start, channels, taps);
  FG_CHECK_LAUNCH("fg_time_conv (state)");
  return 0;
}

extern "C" int fg_time_conv(const void* proj, long proj_stride, long offset, int dtype, void* out, long out_stride,
                            int out_dtype, const float* w, const float* bias, float* state, long state_stride,
                            long conv_offset, const int* req, const int* seq_slot, const int* seq_start, int n_tokens,
                            int n_seqs, int channels, int taps, int act, cudaStream_t stream) {
  if (n_tokens == 0) return 0;
  FG_CHECK_ARG(taps >= 1 && taps <= CONV_MAX_TAPS, "fg_time_conv: %d taps (1 to %d)", taps, CONV_MAX_TAPS);
  FG_CHECK_ARG((dtype == FG_F32 || dtype == FG_BF16) && (out_dtype == FG_F32 || out_dtype == dtype),
               "fg_time_conv: types %d -> %d", dtype, out_dtype);
#define FG_CONV_ARGS w, bias, state, state_stride, conv_offset, req, seq_slot, seq_start, n_tokens, n_seqs, channels, taps, act, stream
  if (dtype == FG_F32)
    return launch_time_conv((const float*)proj + offset, proj_stride, (float*)out, out_stride, FG_CONV_ARGS);
  if (out_dtype == FG_F32)
    return launch_time_conv((const __nv_bfloat16*)proj + offset, proj_stride, (float*)out, out_stride, FG_CONV_ARGS);
  return launch_time_conv((const __nv_bfloat16*)proj + offset, proj_stride, (__nv_bfloat16*)out, out_stride, FG_CONV_ARGS);
#undef FG_CONV_ARGS
}

extern "C" int fg_mamba2_conv(const void* proj, long proj_stride, long xbc_offset, int dtype, float* out,
                              long out_stride, const float* w, const float* bias, float* state, long state_stride,
                              long conv_offset, const int* req, const int* seq_slot, const int* seq_start,
                              int n_tokens, int n_seqs, int channels, int taps, cudaStream_t stream) {
  return fg_time_conv(proj, proj_stride, xbc_offset, dtype, out, out_stride, FG_F32, w, bias, state, state_stride,
                      conv_offset, req, seq_slot, seq_start, n_tokens, n_seqs, channels, taps, 1, stream);
}

// Whether a step may hold sequences for ssm_chunk_kernel: 16-bit serving, states of 64 or 128 rows, rows in
// whole groups of four, and enough tokens for one such sequence.
static bool sc_apply(int n_tokens, int n_state, int head_dim, int dtype) {
  return dtype == FG_BF16 && (n_state == 64 || n_state == 128) && head_dim % 4 == 0 && n_tokens >= SC_MIN;
}
// floats of the scratch that fg_mamba2_scan takes (0: none; without it every token goes through the token kernels, as
// it does where no sequence of the step brings more than `longest` tokens and those are too few)
extern "C" long fg_mamba2_scan_scratch_floats(int n_tokens, int longest, int n_seqs, int heads, int n_state, int head_dim,
                                              int dtype) {
  return sc_apply(longest, n_state, head_dim, dtype)
             ? long_seq::list_floats(n_tokens, n_seqs, SC_MIN) + long_seq::most_chunks(n_tokens, n_seqs, SC_MIN, SC_TOKENS) * heads * SC_REC
             : 0;
}

template <typename T>
static int launch_scan(const float* xbc, long xbc_stride, const T* dt_raw, long dt_stride, const float* dt_bias,
                       const float* a_log, const float* d_skip, float* y, long y_stride, float* state, long state_stride,
                       const int* seq_slot, const int* seq_start, int n_seqs, int heads, int groups, int N, int P,
                       int n_tokens, float* scratch, cudaStream_t stream) {
  const dim3 grid(n_seqs, heads, (P + SCAN_PB - 1) / SCAN_PB);
  const size_t smem = 2 * sizeof(float) * (size_t)(2 * SCAN_TOKENS * N + SCAN_TOKENS * SCAN_PB + 2 * SCAN_TOKENS);
  if (N == 64 || N == 128 || N == 256) {
    const size_t tsmem = 2 * sizeof(float) * (size_t)(2 * SCAN_TOKENS * N + SCAN_TOKENS * SCAN_PB + 2 * SCAN_TOKENS);
    int most = 0x7fffffff;  // tokens of the longest sequence that the token kernel takes
    if (scratch != nullptr) {
      most = SC_MIN - 1;
      long_seq::Head* const list = reinterpret_cast<long_seq::Head*>(scratch);
      float* const chunks = scratch + long_seq::list_floats(n_tokens, n_seqs, SC_MIN);
      const dim3 prepare((unsigned)long_seq::most_chunks(n_tokens, n_seqs, SC_MIN, SC_TOKENS), groups);
      const long items = long_seq::most_sequences(n_tokens, n_seqs, SC_MIN) * heads * ((P + SC_COLS - 1) / SC_COLS);
#define CHUNKS(NN)                                                                                                     \
  do {                                                                                                                 \
    ssm_chunk_prepare_kernel<T, NN><<<prepare, SC_THREADS, 0, stream>>>(xbc, xbc_stride, dt_raw, dt_stride, dt_bias,    \
                                                                        a_log, list, chunks, seq_slot, seq_start,      \
                                                                        n_seqs, heads, groups, P);                     \
    cudaFuncSetAttribute(ssm_chunk_kernel<NN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ScanWalk<NN>::SMEM);   \
    const long resident = (long)fg_sm_count() * fg_blocks_per_sm(SC_THREADS, ScanWalk<NN>::SMEM);                      \
    ssm_chunk_kernel<NN><<<(unsigned)(items < resident ? items : resident), SC_THREADS, ScanWalk<NN>::SMEM, stream>>>(  \
        xbc, xbc_stride, list, chunks, d_skip, y, y_stride, state, state_stride, seq_slot, seq_start, heads, groups, P); \
  } while (0)
      if (N == 64) CHUNKS(64);
      else CHUNKS(128);
#undef CHUNKS
      FG_CHECK_LAUNCH("fg_mamba2_scan (chunks)");
    }
#define TILED(NPT)                                                                                              \
  do {                                                                                                          \
    auto kern = ssm_scan_tiled_kernel<T, NPT>;                                                                  \
    if (tsmem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsmem); \
    fg_launch_pdl(kern, grid, dim3(TS_THREADS), tsmem, stream, xbc, xbc_stride, dt_raw, dt_stride, dt_bias,     \
                  a_log, d_skip, y, y_stride, state, state_stride, seq_slot, seq_start, heads, groups, P, most); \
  } while (0)
    if (N == 64) TILED(2);
    else if (N == 128) TILED(4);
    else TILED(8);
#undef TILED
    return 0;
  }
  const int lanes = N >= 64 ? 32 : 8;
  const int npt = (N + lanes - 1) / lanes;
#define SCAN(NPT, LANES)                                                                                        \
  do {                                                                                                          \
    auto kern = ssm_scan_kernel<T, NPT, LANES>;                                                                 \
    if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
    kern<<<grid, SCAN_PB * LANES, smem, stream>>>(xbc, xbc_stride, dt_raw, dt_stride, dt_bias, a_log, d_skip, y, \
                                                  y_stride, state, state_stride, seq_slot, seq_start, heads,    \
                                                  groups, N, P);                                                \
  } while (0)
  if (lanes == 32) {
    if (npt <= 2) SCAN(2, 32);
    else if (npt <= 4) SCAN(4, 32);
    else SCAN(8, 32);
  } else {
    if (npt <= 1) SCAN(1, 8);
    else if (npt <= 2) SCAN(2, 8);
    else if (npt <= 4) SCAN(4, 8);
    else SCAN(8, 8);
  }
#undef SCAN
  return 0;
}

extern "C" int fg_mamba2_scan(const float* xbc, long xbc_stride, const void* proj, long proj_stride, long dt_offset,
                              int dtype, const float* dt_bias, const float* a_log, const float* d_skip, float* y,
                              long y_stride, float* state, long state_stride, const int* seq_slot,
                              const int* seq_start, int n_seqs, int heads, int groups, int N, int P,
                              int n_tokens, float* scratch, cudaStream_t stream) {
  if (n_seqs == 0) return 0;
  FG_CHECK_ARG(heads > 0 && groups > 0 && heads % groups == 0 && N > 0 && P > 0,
               "fg_mamba2_scan: bad sizes heads=%d groups=%d N=%d P=%d", heads, groups, N, P);
  // the chunks' copies are of 16 bytes
  if (!sc_apply(n_tokens, N, P, dtype) || xbc_stride % 4 != 0 || y_stride % 4 != 0 ||
      (((uintptr_t)xbc | (uintptr_t)y | (uintptr_t)scratch) & 15) != 0)
    scratch = nullptr;
  int rc;
  if (dtype == FG_F32)
    rc = launch_scan<float>(xbc, xbc_stride, (const float*)proj + dt_offset, proj_stride, dt_bias,
                            a_log, d_skip, y, y_stride, state, state_stride, seq_slot,
                            seq_start, n_seqs, heads, groups, N, P, n_tokens, scratch, stream);
  else if (dtype == FG_BF16)
    rc = launch_scan<__nv_bfloat16>(xbc, xbc_stride, (const __nv_bfloat16*)proj + dt_offset, proj_stride,
                                    dt_bias, a_log, d_skip, y, y_stride, state, state_stride, seq_slot,
                                    seq_start, n_seqs, heads, groups, N, P, n_tokens, scratch, stream);
  else
    FG_CHECK_ARG(false, "fg_mamba2_scan: bad dtype %d", dtype);
  if (rc) return rc;
  FG_CHECK_LAUNCH("fg_mamba2_scan");
  return 0;
}

extern "C" int fg_gated_part_norm(const float* y, long y_stride, const void* z, long z_stride, int dtype,
                                  const float* w, void* out, long out_stride, const int* req, int n_tokens, int width,
                                  int parts, float eps, cudaStream_t stream) {
  if (n_tokens == 0) return 0;
  FG_CHECK_ARG(parts > 0 && width % parts == 0, "fg_gated_part_norm: %d columns in %d parts", width, parts);
  const dim3 grid(n_tokens, parts);
  const int part = width / parts;
  if ((dtype == FG_F32 || dtype == FG_BF16) && (part == 128 || part == 256 || part == 512 || part == 1024)) {
    const int blocks = (int)(((long)n_tokens * parts + GW_WARPS - 1) / GW_WARPS);
#define GATED(T, I)                                                                                                       \
  fg_launch_pdl(gated_part_norm_whole_kernel<T, I>, dim3(blocks), dim3(GW_WARPS * 32), 0, stream, y, y_stride, (const T*)z, \
                z_stride, w, (T*)out, out_stride, req, n_tokens, parts, eps)
#define GATED_I(T)                      \
  do {                                  \
    if (part == 128) GATED(T, 4);       \
    else if (part == 256) GATED(T, 8);  \
    else if (part == 512) GATED(T, 16); \
    else GATED(T, 32);                  \
  } while (0)
    if (dtype == FG_F32) GATED_I(float);
    else GATED_I(__nv_bfloat16);
#undef GATED_I
#undef GATED
    FG_CHECK_LAUNCH("fg_gated_part_norm");
    return 0;
  }
  if (part <= 32 * GW_ITEMS) {
    const long items = (long)n_tokens * parts;
    const int blocks = (int)((items + GW_WARPS - 1) / GW_WARPS);
    if (dtype == FG_F32)
      gated_part_norm_warp_kernel<float><<<blocks, GW_WARPS * 32, 0, stream>>>(
          y, y_stride, (const float*)z, z_stride, w, (float*)out, out_stride, req, n_tokens, parts, part, eps);
    else if (dtype == FG_BF16)
      gated_part_norm_warp_kernel<__nv_bfloat16><<<blocks, GW_WARPS * 32, 0, stream>>>(
          y, y_stride, (const __nv_bfloat16*)z, z_stride, w, (__nv_bfloat16*)out, out_stride, req, n_tokens, parts,
          part, eps);
    else
      FG_CHECK_ARG(false, "fg_gated_part_norm: bad dtype %d", dtype);
    FG_CHECK_LAUNCH("fg_gated_part_norm");
    return 0;
  }
  if (dtype == FG_F32)
    gated_part_norm_kernel<float><<<grid, GN_THREADS, 0, stream>>>(y, y_stride, (const float*)z, z_stride,
                                                                    w, (float*)out, out_stride, req,
                                                                    width / parts, eps);
  else if (dtype == FG_BF16)
    gated_part_norm_kernel<__nv_bfloat16><<<grid, GN_THREADS, 0, stream>>>(
        y, y_stride, (const __nv_bfloat16*)z, z_stride, w, (__nv_bfloat16*)out, out_stride, req,
        width / parts, eps);
  else
    FG_CHECK_ARG(false, "fg_gated_part_norm: bad dtype %d", dtype);
  FG_CHECK_LAUNCH("fg_gated_part_norm");
  return 0;
}
