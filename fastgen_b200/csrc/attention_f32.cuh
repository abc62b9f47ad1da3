// Paged causal attention in float32 for prompts in tiles of 64 rows, and for single tokens.  Every score, weight and output
// is the sum of attention_simt.cuh in the same order (tiles of 32 keys from position 0, running maximum and sum a tile,
// keys in ascending order), bit for bit: a token's result does not depend on which of the kernels computes it.
// A key that a row does not see contributes nothing to it here, whatever its value holds.
//
// Pools start on 16 bytes (head sizes are multiples of 16 numbers, so that all rows do).
#pragma once

#include "attention_simt.cuh"

namespace fg_attn {

__device__ __forceinline__ void cp_async_row16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(ok ? 16 : 0)
               : "memory");
}

// ---------------------------------------------------------------------------------------------------------------
// Prompts: a block holds 64 rows (tokens x heads of a group), a thread the scores of 4 rows x 4 keys and the outputs of the
// same 4 rows x HD / 8 columns, so that only keys and values meet at a barrier (one a tile; the next tile's arrive by
// asynchronous copies meanwhile).  What bounds it is shared memory: 8 reads of 16 bytes for 64 multiply-adds.
// 777 tokens, 32 / 8 heads of 64: 16 rows a block (attention_simt.cuh) 248 us, here 146; 300 tokens 61 and 42.  Which prompts come
// here: fg_attention_f32_prompt_rows.
// ---------------------------------------------------------------------------------------------------------------
constexpr int P_ROWS = 64;

template <int HD>
struct PromptShape {
  static constexpr int HP = HD + 4, PP = KEYS + 4;
  static constexpr size_t SMEM = sizeof(float) * ((P_ROWS + 4 * KEYS) * HP + P_ROWS * PP);
};

template <int HD>
__global__ void __launch_bounds__(128, 3)
attention_prompt_f32_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, int out_stride,
                            const float* __restrict__ k_pages, const float* __restrict__ v_pages,
                            const int* __restrict__ block_table, int table_width, int page_size, int n_pages,
                            const int* __restrict__ pos, const int* __restrict__ tile_req,
                            const int* __restrict__ tile_tok0, const int* __restrict__ tile_ntok, int n_kv_heads,
                            int group, int heads_per_block, int window, int keep_first, float scale, int* status,
                            float softcap, const float* __restrict__ sinks, int n_tiles, int slices, int wave) {
  constexpr int HP = PromptShape<HD>::HP, PP = PromptShape<HD>::PP;
  extern __shared__ __align__(16) float smem_f[];
  float* const Qs = smem_f;                 // [P_ROWS][HP]
  float* const Ks = Qs + P_ROWS * HP;       // [2][KEYS][HP]
  float* const Vs = Ks + 2 * KEYS * HP;     // [2][KEYS][HP]
  float* const Ps = Vs + 2 * KEYS * HP;     // [P_ROWS][PP]; -1: a key that the row does not see
  __shared__ int key_ok[2][KEYS];

  // The list is in ascending order of keys: the longest tiles first.  The launch's blocks are mostly on the chip at once,
  // `wave` of them side by side: every second such run goes backwards, or the SM with the longest block of one had the
  // longest of all (777 tokens: 183 us instead of 165 when this was measured).
  const int run = blockIdx.x / wave, in_run = blockIdx.x % wave;
  const int item = (run & 1) && (run + 1) * wave <= gridDim.x ? run * wave + wave - 1 - in_run : blockIdx.x;
  const int tile = n_tiles - 1 - item / (n_kv_heads * slices), g = item % n_kv_heads, sub = item / n_kv_heads % slices;
  const int b = tile_req[tile], tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
  if (b < 0 || ntok <= 0) return;  // padding of a captured list
  const int tid = threadIdx.x;
  auto row_token = [&](int r) { return r / heads_per_block; };
  auto row_head = [&](int r) { return sub * heads_per_block + (r % heads_per_block); };
  auto row_valid = [&](int r) { return row_token(r) < ntok && row_head(r) < group; };
  // two threads a row: copies of 16 bytes where the queries lie on them (waited for with the first tile), else one by one
  {
    const int r = tid >> 1;
    const bool ok = row_valid(r);
    const float* src = ok ? q + (size_t)(tok0 + row_token(r)) * q_stride + (size_t)(g * group + row_head(r)) * HD : q;
    if (q_stride % 4 == 0 && ((uintptr_t)q & 15) == 0) {
#pragma unroll
      for (int d = (tid & 1) * 4; d < HD; d += 8) cp_async_row16(Qs + r * HP + d, ok ? src + d : q, ok);
    } else {
#pragma unroll 8
      for (int d = tid & 1; d < HD; d += 2) Qs[r * HP + d] = ok ? src[d] : 0.f;
    }
  }
  // the tokens of a tile are consecutive positions of one request
  const int min_pos = pos[tok0], max_pos = min_pos + ntok - 1;
  const int lo_min = first_visible(min_pos, window);
  int k_win = 0, k_keep_end = 0;  // tiles between the kept positions and the window are skipped
  if (window != 0) {
    k_win = lo_min / KEYS * KEYS;
    k_keep_end = min(k_win, (max(keep_first, 0) + KEYS - 1) / KEYS * KEYS);
  }
  auto settle = [&](int k0) { return k0 >= k_keep_end && k0 < k_win ? k_win : k0; };

  // a thread copies a quarter of one key's row (and of its value's); where that row lies is looked up a tile ahead
  constexpr unsigned NONE = 0xffffffffu;
  const int ck = tid >> 2, cp = tid & 3;
  auto row_of = [&](int k0) {
    const int j = k0 + ck;
    if (j > max_pos) return NONE;
    const int logical = j / page_size;
    const int page = logical < table_width ? block_table[(size_t)b * table_width + logical] : -1;
    if (page < 0 || page >= n_pages) {
      // a key some row must see has no page
      if ((j >= lo_min || j < keep_first) && cp == 0 && status) atomicOr(status, FG_STATUS_BAD_PAGE);
      return NONE;
    }
    return ((unsigned)page * n_kv_heads + g) * page_size + (j - logical * page_size);
  };
  float* const k_dst = Ks + ck * HP + cp * 4;
  float* const v_dst = Vs + ck * HP + cp * 4;
  auto issue = [&](unsigned row, int buf) {
    const size_t base = row != NONE ? (size_t)row * HD + cp * 4 : 0;
#pragma unroll
    for (int i = 0; i < HD / 16; ++i) {
      cp_async_row16(k_dst + buf * KEYS * HP + i * 16, k_pages + base + i * 16, row != NONE);
      cp_async_row16(v_dst + buf * KEYS * HP + i * 16, v_pages + base + i * 16, row != NONE);
    }
    if (cp == 0) key_ok[buf][ck] = row != NONE;
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  // this thread's rows rg + 16 i, keys kg + 8 j of a tile, columns 32 c + 4 kg (and two of the last 16 of an odd HD / 16)
  const int rg = tid >> 3, kg = tid & 7;
  constexpr int QUADS = HD / 32, REST = HD % 32 != 0 ? 2 : 0;
  float m_run[4], l_run[4];
  int p_row[4], lo_row[4];
  float4 o4[4][QUADS > 0 ? QUADS : 1];
  float2 o2[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = rg + 16 * i;
    p_row[i] = row_valid(r) ? min_pos + row_token(r) : -1;
    lo_row[i] = first_visible(p_row[i], window);
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
    if (sinks != nullptr && row_head(r) < group) {
      m_run[i] = sinks[g * group + row_head(r)];
      l_run[i] = 1.f;
    }
#pragma unroll
    for (int c = 0; c < QUADS; ++c) o4[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
    o2[i] = make_float2(0.f, 0.f);
  }

  int k0 = settle(0), buf = 0;
  issue(row_of(k0), 0);
  int next = settle(k0 + KEYS);
  unsigned next_row = row_of(next);
  while (k0 <= max_pos) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // the tile has landed for all, and the other buffer is read by nobody
    if (next <= max_pos) issue(next_row, buf ^ 1);
    const int after = settle(next + KEYS);
    next_row = row_of(after);
    // whether some row does not see some key of the tile (rows without a query are computed and not stored)
    const bool masked = k0 + KEYS - 1 > min_pos || (window != 0 && k0 < first_visible(max_pos, window));
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
    const float* kt = Ks + buf * KEYS * HP;
#pragma unroll 2
    for (int d = 0; d < HD; d += 4) {
      float4 kv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(kt + (kg + 8 * j) * HP + d);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 qv = *reinterpret_cast<const float4*>(Qs + (rg + 16 * i) * HP + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = fmaf(qv.x, kv[j].x, s[i][j]);
          s[i][j] = fmaf(qv.y, kv[j].y, s[i][j]);
          s[i][j] = fmaf(qv.z, kv[j].z, s[i][j]);
          s[i][j] = fmaf(qv.w, kv[j].w, s[i][j]);
        }
      }
    }
    // (no branches but the cap's, the same for all: the four rows' exponentials and exchanges run side by side)
    unsigned visible = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool ok = key_ok[buf][kg + 8 * j] != 0;
      const int key = k0 + kg + 8 * j;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        s[i][j] *= scale;
        if (ok && key <= p_row[i] && (key >= lo_row[i] || key < keep_first)) visible |= 1u << (4 * i + j);
      }
    }
    if (softcap > 0.f)
#pragma unroll
      for (int i = 0; i < 16; ++i) s[i / 4][i % 4] = softcap * tanhf(s[i / 4][i % 4] / softcap);
    float mx[4], al[4], sum[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (!(visible >> (4 * i + j) & 1)) s[i][j] = -INFINITY;
      mx[i] = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < 4; ++i) mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], o));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float m_new = fmaxf(m_run[i], mx[i]), base = m_new == -INFINITY ? 0.f : m_new;  // (-inf: no key so far)
      al[i] = m_run[i] == -INFINITY ? (m_new == -INFINITY ? 1.f : 0.f) : expf(m_run[i] - base);
      m_run[i] = m_new;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool seen = visible >> (4 * i + j) & 1;
        s[i][j] = seen ? expf(s[i][j] - base) : 0.f;
        Ps[(rg + 16 * i) * PP + kg + 8 * j] = seen || !masked ? s[i][j] : -1.f;
      }
      // the tree of a warp's sum over 32 keys: distances 16, 8, 4, 2, 1
      sum[i] = (s[i][0] + s[i][2]) + (s[i][1] + s[i][3]);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < 4; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
#pragma unroll
    for (int i = 0; i < 4; ++i) l_run[i] = l_run[i] * al[i] + sum[i];
    __syncwarp();  // a row's weights are written and read by the same eight lanes
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int c = 0; c < QUADS; ++c)
        o4[i][c] = make_float4(o4[i][c].x * al[i], o4[i][c].y * al[i], o4[i][c].z * al[i], o4[i][c].w * al[i]);
      o2[i] = make_float2(o2[i].x * al[i], o2[i].y * al[i]);
    }
    const float* vt = Vs + buf * KEYS * HP;
    auto add = [&](bool guarded) {
#pragma unroll 1
      for (int c = 0; c < KEYS; c += 4) {
        float4 p4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) p4[i] = *reinterpret_cast<const float4*>(Ps + (rg + 16 * i) * PP + c);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float4 v[QUADS > 0 ? QUADS : 1];
          float2 vr = make_float2(0.f, 0.f);
#pragma unroll
          for (int n = 0; n < QUADS; ++n) v[n] = *reinterpret_cast<const float4*>(vt + (c + e) * HP + 32 * n + 4 * kg);
          if (REST) vr = *reinterpret_cast<const float2*>(vt + (c + e) * HP + 32 * QUADS + 2 * kg);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float pr = e == 0 ? p4[i].x : e == 1 ? p4[i].y : e == 2 ? p4[i].z : p4[i].w;
            auto sum_up = [&](float value, float& o) { o = guarded && pr < 0.f ? o : fmaf(pr, value, o); };
#pragma unroll
            for (int n = 0; n < QUADS; ++n) {
              sum_up(v[n].x, o4[i][n].x);
              sum_up(v[n].y, o4[i][n].y);
              sum_up(v[n].z, o4[i][n].z);
              sum_up(v[n].w, o4[i][n].w);
            }
            if (REST) {
              sum_up(vr.x, o2[i].x);
              sum_up(vr.y, o2[i].y);
            }
          }
        }
      }
    };
    if (masked)
      add(true);
    else
      add(false);
    k0 = next;
    next = after;
    buf ^= 1;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = rg + 16 * i;
    if (!row_valid(r)) continue;
    const float inv = l_run[i] > 0.f ? 1.f / l_run[i] : 0.f;
    float* o = out + (size_t)(tok0 + row_token(r)) * out_stride + (g * group + row_head(r)) * HD;
#pragma unroll
    for (int c = 0; c < QUADS; ++c) {
      float* at = o + 32 * c + 4 * kg;
      at[0] = o4[i][c].x * inv;
      at[1] = o4[i][c].y * inv;
      at[2] = o4[i][c].z * inv;
      at[3] = o4[i][c].w * inv;
    }
    if (REST) {
      o[32 * QUADS + 2 * kg] = o2[i].x * inv;
      o[32 * QUADS + 2 * kg + 1] = o2[i].y * inv;
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Single tokens: a block holds one token and R heads of a group (as many as there are, rounded up to 4 or 8).  The walk over the
// keys is a chain only in the outputs' sums: a run of several tiles of 32 keys is scored at once, a warp one or two of
// them, their maxima meet in shared memory, every warp finds the running maximum that its tile starts from, and only then
// the outputs walk the run's keys, four rows a thread side by side.  The next run's keys come by asynchronous copies
// during that walk, their values behind it.
//
// One block's time falls with the run's length, its shared memory grows with it (head size 64: 139 KB at 8 tiles, 71 at 4, 37 at 2),
// and a launch of more blocks than fit at once takes another turn for the rest.  So the longest run whose blocks fit at
// once, else the shortest that is there: form 0 (256 threads; 8 tiles up to head size 80, 4 up to 160, 2 beyond), form 1 (128
// threads, 4 tiles, up to head size 80), form 2 (2 tiles, 48 to 160).  Measured (us; 32 / 8 heads of 64; tile after tile in blocks of 16
// rows as in attention_simt.cuh, then forms 0, 1, 2): one token on 4,000 keys 320 / 112 / 149 / 203, 32 tokens 365 / 231 / 208 / 272,
// 64 tokens 501 / 458 / 410 / 300, and on 20 keys 8 / 21 / 10 / 6; 128 tokens on 250 77 / 71 / 47 / 41.  Head size 128, 64 tokens on 1,000
// 289 / 213 / - / 159.  5 tokens on 100 to 500 keys of 64 38 / 16.  Blocks of 16 rows stay ahead on a few tens of keys at groups of
// 8 (7 us to 8) and at head sizes 16 and 32 (4 to 5), and with 768 blocks at head size 16 (240 to 276 on 4,000 keys).
// ---------------------------------------------------------------------------------------------------------------
template <int HD, int R, int FORM>
struct SingleShape {
  static constexpr bool THERE = FORM == 0 || (FORM == 1 ? HD <= 80 : HD > 32 && HD <= 160);
  static constexpr int TILES = FORM == 1 ? 4 : FORM == 2 ? 2 : HD <= 80 ? 8 : HD <= 160 ? 4 : 2;  // what shared memory holds
  static constexpr int THREADS = FORM == 0 ? 256 : 128, A_WARP = FORM == 0 ? 2 : 1;  // tiles that a warp scores
  static constexpr int CHUNK = TILES * KEYS, KP = HD + 4;  // padded rows of keys: eight lanes read eight bank groups
  static constexpr size_t SMEM = sizeof(float) * (CHUNK * (HD + KP) + R * HD + CHUNK * R);
  // blocks an SM: by shared memory (4 KB beside the above) and by 128 registers a thread (4 rows, 128 threads: 96)
  static constexpr int FIT = (int)(228 * 1024 / (SMEM + 4096)), MOST = FORM == 0 ? 2 : R == 4 ? 5 : 4;
  static constexpr int BLOCKS = FIT < 1 ? 1 : FIT < MOST ? FIT : MOST;
};

template <int HD, int R, int FORM>
__global__ void __launch_bounds__(SingleShape<HD, R, FORM>::THREADS, SingleShape<HD, R, FORM>::BLOCKS)
attention_single_f32_kernel(const float* q, int q_stride, float* out, int out_stride, const float* k_pages,
                            const float* v_pages, const int* __restrict__ block_table, int table_width, int page_size,
                            int n_pages, const int* __restrict__ pos, const int* __restrict__ req_of,
                            const int* __restrict__ single_req, const int* __restrict__ single_tok, int n_kv_heads,
                            int group, int window, int keep_first, float scale, int* status, float softcap,
                            const float* __restrict__ sinks) {
  using S = SingleShape<HD, R, FORM>;
  constexpr int TILES = S::TILES, CHUNK = S::CHUNK, KP = S::KP, THREADS = S::THREADS, H = S::A_WARP;
  extern __shared__ __align__(16) float smem_f[];
  float* const Vs = smem_f;                 // [CHUNK][HD]
  float* const Ks = Vs + CHUNK * HD;        // [CHUNK][KP]
  float* const Qs = Ks + CHUNK * KP;        // [R][HD]
  float* const Ps = Qs + R * HD;       // [CHUNK][R]; -1: a key that is not seen
  __shared__ __align__(16) float max_s[TILES][R], sum_s[TILES][R], al_s[TILES][R], l_s[R];
  __shared__ unsigned row_s[2][CHUNK];  // the keys' rows in the pools, of this run of tiles and of the next

  const int g = blockIdx.y, head0 = blockIdx.z * R, rows = min(R, group - head0);
  const int b = single_req[blockIdx.x], tok = single_tok[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* const o = out + (size_t)tok * out_stride + (size_t)(g * group + head0) * HD;
  pdl_trigger();
  pdl_wait();
  if (b < 0) {
    // padding of a fixed-size batch: no request; the rows of a token that belongs to none are zeroed
    if (req_of[tok] < 0)
      for (int i = tid; i < rows * HD; i += THREADS) o[i] = 0.f;
    return;
  }
  const int p = pos[tok], lo = first_visible(p, window);
  int k_win = 0, kept = 0;  // tiles: those of the kept positions, then the window's
  if (window != 0) {
    k_win = lo / KEYS;
    kept = min(k_win, (max(keep_first, 0) + KEYS - 1) / KEYS);
  }
  const int n_tiles = kept + p / KEYS - k_win + 1;
  auto tile_pos = [&](int t) { return (t < kept ? t : t - kept + k_win) * KEYS; };
  // the walk's last tile and the window's edges hold keys that are not seen: the same ones for all rows
  auto masked = [&](int t) {
    const int first = tile_pos(t);
    return first + KEYS - 1 > p || (first < lo && first + KEYS > keep_first);
  };
  // the row of a key in the pools
  constexpr unsigned NONE = 0xffffffffu;
  auto key_row = [&](int t, int key) -> unsigned {
    const int j = tile_pos(t) + key;
    if (t >= n_tiles || j > p) return NONE;
    const int logical = j / page_size;
    const int page = logical < table_width ? block_table[(size_t)b * table_width + logical] : -1;
    if (page < 0 || page >= n_pages) {
      if ((j >= lo || j < keep_first) && status) atomicOr(status, FG_STATUS_BAD_PAGE);
      return NONE;
    }
    return ((unsigned)page * n_kv_heads + g) * page_size + j % page_size;
  };
  for (int i = tid; i < R * HD; i += THREADS)
    Qs[i] = i < rows * HD ? q[(size_t)tok * q_stride + (size_t)(g * group + head0) * HD + i] : 0.f;

  // every thread keeps the running maxima; the sums' and outputs' state: thread -> column, four rows
  float m_run[R];
#pragma unroll
  for (int r = 0; r < R; ++r) m_run[r] = sinks != nullptr && r < rows ? sinks[g * group + head0 + r] : -INFINITY;
  float l_run = sinks != nullptr ? 1.f : 0.f;  // of row `tid` (tid < R)
  constexpr int SLOTS = (R / 4 * (HD / 2) + THREADS - 1) / THREADS;  // (two columns, four rows) a thread
  float2 acc[SLOTS][4];
#pragma unroll
  for (int u = 0; u < SLOTS; ++u)
#pragma unroll
    for (int r = 0; r < 4; ++r) acc[u][r] = make_float2(0.f, 0.f);

  auto look_up = [&](int t0, int buf) {
    for (int i = tid; i < CHUNK; i += THREADS) row_s[buf][i] = key_row(t0 + i / KEYS, i % KEYS);
  };
  auto copy = [&](float* dst, int stride, const float* pool, int buf, int tiles) {
#pragma unroll 4
    for (int u = 0; u < CHUNK * (HD / 4) / THREADS; ++u) {
      const int i = tid + u * THREADS, key = i / (HD / 4), c = i % (HD / 4) * 4;
      if (key >= tiles * KEYS) break;
      const unsigned row = row_s[buf][key];
      cp_async_row16(dst + key * stride + c, pool + (row != NONE ? (size_t)row * HD + c : 0), row != NONE);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  int buf = 0;
  look_up(0, 0);
  __syncthreads();  // (and the queries)
  copy(Ks, KP, k_pages, 0, min(TILES, n_tiles));
  for (int t0 = 0; t0 < n_tiles; t0 += TILES, buf ^= 1) {
    const int tiles = min(TILES, n_tiles - t0);
    copy(Vs, HD, v_pages, buf, tiles);
    if (t0 + TILES < n_tiles) look_up(t0 + TILES, buf ^ 1);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();  // the keys have landed for all
    // a warp H tiles, a lane a key of each: a read of the queries serves all
    const int w0 = warp * H;
    float s[H][R];
    bool visible[H];
    if (w0 < tiles) {
#pragma unroll
      for (int r = 0; r < H * R; ++r) s[r / R][r % R] = 0.f;
      const float* kr = Ks + (w0 * KEYS + lane) * KP;
#pragma unroll 4
      for (int d = 0; d < HD; d += 4) {
        float4 kv[H];
#pragma unroll
        for (int h = 0; h < H; ++h) kv[h] = *reinterpret_cast<const float4*>(kr + h * KEYS * KP + d);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float4 qv = *reinterpret_cast<const float4*>(Qs + r * HD + d);
#pragma unroll
          for (int h = 0; h < H; ++h) s[h][r] = fmaf(qv.x, kv[h].x, s[h][r]);
#pragma unroll
          for (int h = 0; h < H; ++h) s[h][r] = fmaf(qv.y, kv[h].y, s[h][r]);
#pragma unroll
          for (int h = 0; h < H; ++h) s[h][r] = fmaf(qv.z, kv[h].z, s[h][r]);
#pragma unroll
          for (int h = 0; h < H; ++h) s[h][r] = fmaf(qv.w, kv[h].w, s[h][r]);
        }
      }
      float mx[H][R];
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const int j = tile_pos(t0 + w0 + h) + lane;
        visible[h] = w0 + h < tiles && row_s[buf][(w0 + h) * KEYS + lane] != NONE && j <= p && (j >= lo || j < keep_first);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          s[h][r] *= scale;
          if (softcap > 0.f) s[h][r] = softcap * tanhf(s[h][r] / softcap);
          mx[h][r] = s[h][r] = visible[h] ? s[h][r] : -INFINITY;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < H * R; ++r) mx[r / R][r % R] = fmaxf(mx[r / R][r % R], __shfl_xor_sync(0xffffffffu, mx[r / R][r % R], o));
      if (lane == 0)
#pragma unroll
        for (int r = 0; r < H * R; ++r) max_s[w0 + r / R][r % R] = mx[r / R][r % R];
    }
    __syncthreads();
    // the keys are read: the next ones are on their way during the rest (an empty group keeps the count where there are none)
    if (t0 + TILES < n_tiles)
      copy(Ks, KP, k_pages, buf ^ 1, min(TILES, n_tiles - t0 - TILES));
    else
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (w0 < tiles) {
      float before[H][R], sum[H][R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float m = m_run[r];
#pragma unroll
        for (int u = 0; u < TILES - H; ++u) m = fmaxf(m, u < w0 ? max_s[u][r] : -INFINITY);
#pragma unroll
        for (int h = 0; h < H; ++h) before[h][r] = m = h == 0 ? m : fmaxf(m, max_s[w0 + h - 1][r]);
      }
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const bool hide = w0 + h < tiles && masked(t0 + w0 + h);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float here = fmaxf(before[h][r], max_s[w0 + h][r]), base = here == -INFINITY ? 0.f : here;
          const float pr = visible[h] ? expf(s[h][r] - base) : 0.f;
          sum[h][r] = pr;
          Ps[((w0 + h) * KEYS + lane) * R + r] = visible[h] || !hide ? pr : -1.f;
          if (lane == 0)
            al_s[w0 + h][r] = before[h][r] == -INFINITY ? (here == -INFINITY ? 1.f : 0.f) : expf(before[h][r] - base);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < H * R; ++r) sum[r / R][r % R] += __shfl_xor_sync(0xffffffffu, sum[r / R][r % R], o);
      if (lane == 0)
#pragma unroll
        for (int r = 0; r < H * R; ++r) sum_s[w0 + r / R][r % R] = sum[r / R][r % R];
    }
#pragma unroll
    for (int u = 0; u < TILES; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r) m_run[r] = fmaxf(m_run[r], u < tiles ? max_s[u][r] : -INFINITY);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();  // the values have landed, the weights are written
    if (tid < R)
      for (int u = 0; u < tiles; ++u) l_run = l_run * al_s[u][tid] + sum_s[u][tid];
#pragma unroll
    for (int u = 0; u < SLOTS; ++u) {
      const int at = tid + u * THREADS, col = at % (HD / 2) * 2, r0 = at / (HD / 2) * 4;
      if (r0 >= R) continue;
      auto one_tile = [&](int n, bool guarded) {
        const float* vt = Vs + n * KEYS * HD + col;
        const float* pt = Ps + n * KEYS * R + r0;
#pragma unroll 16
        for (int k = 0; k < KEYS; ++k) {
          const float4 pr = *reinterpret_cast<const float4*>(pt + k * R);
          const float2 v = *reinterpret_cast<const float2*>(vt + k * HD);
          if (guarded && pr.x < 0.f) continue;  // (the same for the whole block)
          acc[u][0].x = fmaf(pr.x, v.x, acc[u][0].x);
          acc[u][0].y = fmaf(pr.x, v.y, acc[u][0].y);
          acc[u][1].x = fmaf(pr.y, v.x, acc[u][1].x);
          acc[u][1].y = fmaf(pr.y, v.y, acc[u][1].y);
          acc[u][2].x = fmaf(pr.z, v.x, acc[u][2].x);
          acc[u][2].y = fmaf(pr.z, v.y, acc[u][2].y);
          acc[u][3].x = fmaf(pr.w, v.x, acc[u][3].x);
          acc[u][3].y = fmaf(pr.w, v.y, acc[u][3].y);
        }
      };
      for (int n = 0; n < tiles; ++n) {
        const float4 al = *reinterpret_cast<const float4*>(&al_s[n][r0]);
        acc[u][0] = make_float2(acc[u][0].x * al.x, acc[u][0].y * al.x);
        acc[u][1] = make_float2(acc[u][1].x * al.y, acc[u][1].y * al.y);
        acc[u][2] = make_float2(acc[u][2].x * al.z, acc[u][2].y * al.z);
        acc[u][3] = make_float2(acc[u][3].x * al.w, acc[u][3].y * al.w);
        if (masked(t0 + n))
          one_tile(n, true);
        else
          one_tile(n, false);
      }
    }
    __syncthreads();  // values, weights and maxima are free
  }
  if (tid < R) l_s[tid] = l_run;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < SLOTS; ++u) {
    const int at = tid + u * THREADS, col = at % (HD / 2) * 2, r0 = at / (HD / 2) * 4;
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (r0 + r < rows) {
        const float l = l_s[r0 + r], inv = l > 0.f ? 1.f / l : 0.f;
        o[(r0 + r) * HD + col] = acc[u][r].x * inv;
        o[(r0 + r) * HD + col + 1] = acc[u][r].y * inv;
      }
  }
}

}  // namespace fg_attn
