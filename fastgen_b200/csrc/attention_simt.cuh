// Paged causal attention on the CUDA cores, float32 arithmetic throughout.
//
// Prompt portions of few tokens, and all tokens where pages do not start on 16 bytes (attention_f32.cuh has
// single tokens and the prompts of many): the host cuts the step's query tokens into tiles (request, first token, token count)
// and each thread block handles one tile for one group of query heads that
// share a key/value head.  Keys and values come only from the cache pages
// (the step's own keys were written before), in tiles of 32 positions that
// always start at multiples of 32 from position 0, so that the order of every
// sum depends only on the query's own position -- not on how the prompt was
// cut, what else is in the batch, or which pages hold the keys.
//
// Semantics of fastgen/forward.py:176-258: softmax(q.k * scale) v over the
// positions j <= pos(query) of the query's own request (and, when a window is given,
// j > pos - window or j < keep_first: the first positions stay visible; with a negative window only the
// positions of the query's own chunk, see first_visible), grouped-query heads h -> h / (Hq/Hkv).
// Running maximum, sum and output accumulator are float32; exp is expf.  With `sinks` (float32 per
// query head) the denominator also holds exp(sink_h): a score without a key, unscaled, counted once.
//
// Storage type T (float or bf16) only affects loads and the final store.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace fg_attn {

constexpr int ROWS = 16;      // query rows (token x head-of-group) per block
constexpr int KEYS = 32;      // key positions per tile
constexpr int THREADS = 128;

template <typename T, int HD>
__global__ void __launch_bounds__(THREADS)
attention_simt_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, int out_stride,
                      const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                      const int* __restrict__ block_table, int table_width, int page_size,
                      int n_pages, const int* __restrict__ pos, const int* __restrict__ tile_req,
                      const int* __restrict__ tile_tok0, const int* __restrict__ tile_ntok,
                      int n_kv_heads, int group, int heads_per_block, int window, int keep_first,
                      float scale, int* status, float softcap, const float* __restrict__ sinks) {
  constexpr int HP = HD + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float(*Qs)[HP] = reinterpret_cast<float(*)[HP]>(smem_raw);
  float(*Ks)[HP] = reinterpret_cast<float(*)[HP]>(Qs + ROWS);
  float(*Vs)[HP] = reinterpret_cast<float(*)[HP]>(Ks + KEYS);
  float(*Ps)[KEYS + 1] = reinterpret_cast<float(*)[KEYS + 1]>(Vs + KEYS);
  __shared__ float alpha_s[ROWS];
  __shared__ float l_s[ROWS];
  __shared__ long long key_base[KEYS];
  __shared__ int row_pos[ROWS];

  const int tile = blockIdx.x;
  const int g = blockIdx.y;        // key/value head
  const int sub = blockIdx.z;      // which slice of the group's heads
  const int b = tile_req[tile];
  const int tok0 = tile_tok0[tile];
  const int ntok = tile_ntok[tile];
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;

  // row r -> (token r / heads_per_block, head-of-group sub*hpb + r % hpb)
  auto row_token = [&](int r) { return r / heads_per_block; };
  auto row_head = [&](int r) { return sub * heads_per_block + (r % heads_per_block); };
  auto row_valid = [&](int r) { return row_token(r) < ntok && row_head(r) < group; };

  if (b < 0) {
    // padding of a fixed-size batch: no request, the output rows are zeroed
    for (int i = tid; i < ROWS * HD; i += THREADS) {
      const int r = i / HD, d = i - r * HD;
      if (row_valid(r))
        out[(size_t)(tok0 + row_token(r)) * out_stride + (g * group + row_head(r)) * HD + d] = from_f32<T>(0.f);
    }
    return;
  }
  if (tid < ROWS) row_pos[tid] = row_valid(tid) ? pos[tok0 + row_token(tid)] : -1;
  for (int i = tid; i < ROWS * HD; i += THREADS) {
    const int r = i / HD, d = i - r * HD;
    float v = 0.f;
    if (row_valid(r))
      v = to_f32<T>(q[(size_t)(tok0 + row_token(r)) * q_stride + (g * group + row_head(r)) * HD + d]);
    Qs[r][d] = v;
  }
  __syncthreads();

  int max_pos = -1, min_pos = 0x7fffffff;
  for (int r = 0; r < ROWS; ++r) {
    const int p = row_pos[r];
    if (p >= 0) {
      max_pos = max(max_pos, p);
      min_pos = min(min_pos, p);
    }
  }
  if (max_pos < 0) return;
  // with a window, tiles that lie wholly before the earliest row's window are skipped, apart
  // from those that hold some of the first `keep_first` positions, which stay visible for good
  const int lo_min = first_visible(min_pos, window);
  int k_win = 0, k_keep_end = 0;
  if (window != 0) {
    k_win = lo_min / KEYS * KEYS;
    k_keep_end = min(k_win, (max(keep_first, 0) + KEYS - 1) / KEYS * KEYS);
  }

  // this thread's 4 score rows: warp, warp+4, warp+8, warp+12; column = lane
  float m_run[4], l_run[4];
  int row_lo[4];  // the first position each of them sees
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
    row_lo[i] = first_visible(row_pos[warp + 4 * i], window);
    // a sink: a learned score per query head that has no key and no value and counts once in the
    // denominator; the running maximum and sum start from it
    if (sinks != nullptr && row_head(warp + 4 * i) < group) {
      m_run[i] = sinks[g * group + row_head(warp + 4 * i)];
      l_run[i] = 1.f;
    }
  }
  // this thread's output elements: row tid/8, columns tid%8 + 8*i
  constexpr int OD = HD / 8;
  float o_acc[OD];
#pragma unroll
  for (int i = 0; i < OD; ++i) o_acc[i] = 0.f;
  const int o_row = tid >> 3, o_col = tid & 7;

  for (int k0 = 0; k0 <= max_pos; k0 += KEYS) {
    if (k0 >= k_keep_end && k0 < k_win) k0 = k_win;
    if (tid < KEYS) {
      const int j = k0 + tid;
      long long base = -1;
      if (j <= max_pos) {
        const int logical = j / page_size;
        const int page = logical < table_width ? block_table[(size_t)b * table_width + logical] : -1;
        if (page >= 0 && page < n_pages) {
          base = (((long long)page * n_kv_heads + g) * page_size + (j - logical * page_size)) * HD;
        } else if (j >= lo_min || j < keep_first) {
          // a key some row must see has no page
          if (status) atomicOr(status, FG_STATUS_BAD_PAGE);
        }
      }
      key_base[tid] = base;
    }
    __syncthreads();
    for (int i = tid; i < KEYS * HD; i += THREADS) {
      const int c = i / HD, d = i - c * HD;
      const long long base = key_base[c];
      float kv = 0.f, vv = 0.f;
      if (base >= 0) {
        kv = to_f32<T>(k_pages[base + d]);
        vv = to_f32<T>(v_pages[base + d]);
      }
      Ks[c][d] = kv;
      Vs[c][d] = vv;
    }
    __syncthreads();

    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int d = 0; d < HD; ++d) {
      const float kv = Ks[lane][d];
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] = fmaf(Qs[warp + 4 * i][d], kv, s[i]);
    }
    const int j = k0 + lane;
    const bool has_key = key_base[lane] >= 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = warp + 4 * i;
      const int p = row_pos[r];
      const bool visible = has_key && p >= 0 && j <= p && (j >= row_lo[i] || j < keep_first);
      // with a cap, the scaled score is squashed to cap * tanh(score / cap)
      float sc = s[i] * scale;
      if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
      const float sv = visible ? sc : -INFINITY;
      const float m_tile = warp_max(sv);
      const float m_new = fmaxf(m_run[i], m_tile);
      float pr = 0.f, al = 1.f;
      if (m_new != -INFINITY) {
        pr = visible ? expf(sv - m_new) : 0.f;
        al = (m_run[i] == -INFINITY) ? 0.f : expf(m_run[i] - m_new);
      }
      const float psum = warp_sum(pr);
      l_run[i] = l_run[i] * al + psum;
      m_run[i] = m_new;
      Ps[r][lane] = pr;
      if (lane == 0) alpha_s[r] = al;
    }
    __syncthreads();

    {
      const float al = alpha_s[o_row];
#pragma unroll
      for (int i = 0; i < OD; ++i) o_acc[i] *= al;
#pragma unroll 4
      for (int c = 0; c < KEYS; ++c) {
        const float pr = Ps[o_row][c];
#pragma unroll
        for (int i = 0; i < OD; ++i) o_acc[i] = fmaf(pr, Vs[c][o_col + 8 * i], o_acc[i]);
      }
    }
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (lane == 0) l_s[warp + 4 * i] = l_run[i];
  __syncthreads();
  if (row_valid(o_row)) {
    const float l = l_s[o_row];
    const float inv = l > 0.f ? 1.f / l : 0.f;
    T* o = out + (size_t)(tok0 + row_token(o_row)) * out_stride + (g * group + row_head(o_row)) * HD;
#pragma unroll
    for (int i = 0; i < OD; ++i) o[o_col + 8 * i] = from_f32<T>(o_acc[i] * inv);
  }
}

// The same for float32 pages, bit for bit (every score, weight and output is the same sum in the same order).  A
// query's keys stay one sequential walk, so what a launch waits for is the walk's length times a tile's latency: the
// next tile's keys and values arrive by 16-byte asynchronous copies while this one is worked on, its page numbers a
// tile earlier still, operands are read four numbers at a time, and rows without a query are skipped.  A key that a row does
// not see contributes nothing to it here, whatever its value holds.
// A tile's work is there twice, for tiles that all rows see whole and for the others: with the guard in one body for both, 8
// tokens on 4,000 keys took 439 us instead of 387 (32 / 8 heads of 64); with as many registers as its blocks leave
// 387 instead of 392, at head size 128 543 instead of 618.  Which prompts come here: fg_attention_f32_prompt_rows.
template <int HD>
struct SimtShape {
  static constexpr int HP = HD + 4, PP = KEYS + 4;  // padded rows: eight lanes read eight bank groups
  static constexpr size_t SMEM = sizeof(float) * ((ROWS + 4 * KEYS) * HP + ROWS * PP);
  // Blocks an SM: by shared memory (2 KB beside the above), 6 at most.  Up to head size 32 the compiler's own choice (70
  // registers): 64 portions of 4 tokens on 500 keys 49 us, with room for 7 blocks asked for 54.
  static constexpr int FIT = (int)(228 * 1024 / (SMEM + 2048)), BLOCKS = HD <= 32 ? 0 : FIT < 1 ? 1 : FIT < 6 ? FIT : 6;
};

template <int HD>
__global__ void __launch_bounds__(THREADS, SimtShape<HD>::BLOCKS)
attention_simt_f32_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, int out_stride,
                          const float* __restrict__ k_pages, const float* __restrict__ v_pages,
                          const int* __restrict__ block_table, int table_width, int page_size, int n_pages,
                          const int* __restrict__ pos, const int* __restrict__ tile_req,
                          const int* __restrict__ tile_tok0, const int* __restrict__ tile_ntok, int n_kv_heads,
                          int group, int heads_per_block, int window, int keep_first, float scale, int* status,
                          float softcap, const float* __restrict__ sinks) {
  constexpr int HP = SimtShape<HD>::HP, PP = SimtShape<HD>::PP;
  extern __shared__ __align__(16) float smem_f[];
  float* const Qs = smem_f;                 // [ROWS][HP]
  float* const Ks = Qs + ROWS * HP;         // [2][KEYS][HP]
  float* const Vs = Ks + 2 * KEYS * HP;     // [2][KEYS][HP]
  float* const Ps = Vs + 2 * KEYS * HP;     // [ROWS][PP]; -1: a key that the row does not see
  __shared__ float alpha_s[ROWS], l_s[ROWS];
  __shared__ int key_ok[2][KEYS], row_pos[ROWS];

  const int tile = blockIdx.x, g = blockIdx.y, sub = blockIdx.z;
  const int b = tile_req[tile], tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto row_token = [&](int r) { return r / heads_per_block; };
  auto row_head = [&](int r) { return sub * heads_per_block + (r % heads_per_block); };
  auto row_valid = [&](int r) { return row_token(r) < ntok && row_head(r) < group; };

  if (b < 0) {
    // padding of a fixed-size batch: no request, the output rows are zeroed
    for (int i = tid; i < ROWS * HD; i += THREADS) {
      const int r = i / HD, d = i - r * HD;
      if (row_valid(r)) out[(size_t)(tok0 + row_token(r)) * out_stride + (g * group + row_head(r)) * HD + d] = 0.f;
    }
    return;
  }
  if (tid < ROWS) row_pos[tid] = row_valid(tid) ? pos[tok0 + row_token(tid)] : -1;
  for (int i = tid; i < ROWS * HD; i += THREADS) {
    const int r = i / HD, d = i - r * HD;
    Qs[r * HP + d] = row_valid(r) ? q[(size_t)(tok0 + row_token(r)) * q_stride + (g * group + row_head(r)) * HD + d] : 0.f;
  }
  __syncthreads();

  int max_pos = -1, min_pos = 0x7fffffff;
  for (int r = 0; r < ROWS; ++r) {
    const int p = row_pos[r];
    if (p >= 0) {
      max_pos = max(max_pos, p);
      min_pos = min(min_pos, p);
    }
  }
  if (max_pos < 0) return;
  const int lo_min = first_visible(min_pos, window);
  int k_win = 0, k_keep_end = 0;  // tiles between the kept positions and the window are skipped
  if (window != 0) {
    k_win = lo_min / KEYS * KEYS;
    k_keep_end = min(k_win, (max(keep_first, 0) + KEYS - 1) / KEYS * KEYS);
  }
  auto settle = [&](int k0) { return k0 >= k_keep_end && k0 < k_win ? k_win : k0; };

  // a thread copies a quarter of one key's row (and of its value's)
  const int ck = tid >> 2, cp = tid & 3;
  auto page_of = [&](int k0) {
    const int j = k0 + ck;
    if (j > max_pos) return -1;
    const int logical = j / page_size;
    return logical < table_width ? block_table[(size_t)b * table_width + logical] : -1;
  };
  auto issue = [&](int k0, int page, int buf) {
    const int j = k0 + ck;
    const bool ok = j <= max_pos && page >= 0 && page < n_pages;
    // a key some row must see has no page
    if (!ok && j <= max_pos && (j >= lo_min || j < keep_first) && cp == 0 && status) atomicOr(status, FG_STATUS_BAD_PAGE);
    const size_t base = ok ? (((size_t)page * n_kv_heads + g) * page_size + j % page_size) * HD : 0;
    const uint32_t kd = (uint32_t)__cvta_generic_to_shared(Ks + (buf * KEYS + ck) * HP);
    const uint32_t vd = (uint32_t)__cvta_generic_to_shared(Vs + (buf * KEYS + ck) * HP);
#pragma unroll
    for (int i = cp; i < HD / 4; i += 4) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(kd + i * 16), "l"(k_pages + base + i * 4), "r"(ok ? 16 : 0) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(vd + i * 16), "l"(v_pages + base + i * 4), "r"(ok ? 16 : 0) : "memory");
    }
    if (cp == 0) key_ok[buf][ck] = ok;
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  float m_run[4], l_run[4];
  int row_lo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
    row_lo[i] = first_visible(row_pos[warp + 4 * i], window);
    if (sinks != nullptr && row_head(warp + 4 * i) < group) {
      m_run[i] = sinks[g * group + row_head(warp + 4 * i)];
      l_run[i] = 1.f;
    }
  }
  // this thread's output elements: row tid / 8; runs of four columns 32 apart, and two of the last 16 of an odd HD / 16
  constexpr int QUADS = HD / 32, REST = HD % 32 != 0 ? 2 : 0;
  float4 o4[QUADS > 0 ? QUADS : 1];
  float2 o2 = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < QUADS; ++i) o4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int o_row = tid >> 3, o_col = tid & 7;
  const bool o_live = row_pos[o_row] >= 0;

  int k0 = settle(0), buf = 0;
  issue(k0, page_of(k0), 0);
  int next = settle(k0 + KEYS);
  int next_page = page_of(next);
  while (k0 <= max_pos) {
    const bool more = next <= max_pos;
    if (more) {
      issue(next, next_page, buf ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    const int after = settle(next + KEYS);
    next_page = page_of(after);
    __syncthreads();
    auto work = [&](auto guard) {
      constexpr bool guarded = decltype(guard)::value;  // some row does not see some key of the tile
      const float* kt = Ks + (buf * KEYS + lane) * HP;
      float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
      for (int d = 0; d < HD; d += 4) {
        const float4 kv = *reinterpret_cast<const float4*>(kt + d);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 qv = *reinterpret_cast<const float4*>(Qs + (warp + 4 * i) * HP + d);
          s[i] = fmaf(qv.x, kv.x, s[i]);
          s[i] = fmaf(qv.y, kv.y, s[i]);
          s[i] = fmaf(qv.z, kv.z, s[i]);
          s[i] = fmaf(qv.w, kv.w, s[i]);
        }
      }
      const int j = k0 + lane;
      const bool has_key = key_ok[buf][lane] != 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = warp + 4 * i;
        const int p = row_pos[r];
        if (p < 0) continue;  // (the same for the whole warp)
        const bool visible = has_key && j <= p && (j >= row_lo[i] || j < keep_first);
        float sc = s[i] * scale;
        if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
        const float sv = visible ? sc : -INFINITY;
        const float m_tile = warp_max(sv);
        const float m_new = fmaxf(m_run[i], m_tile);
        float pr = 0.f, al = 1.f;
        if (m_new != -INFINITY) {
          pr = visible ? expf(sv - m_new) : 0.f;
          al = (m_run[i] == -INFINITY) ? 0.f : expf(m_run[i] - m_new);
        }
        const float psum = warp_sum(pr);
        l_run[i] = l_run[i] * al + psum;
        m_run[i] = m_new;
        Ps[r * PP + lane] = visible || !guarded ? pr : -1.f;
        if (lane == 0) alpha_s[r] = al;
      }
      __syncthreads();
      if (o_live) {
        const float al = alpha_s[o_row];
#pragma unroll
        for (int i = 0; i < QUADS; ++i) o4[i] = make_float4(o4[i].x * al, o4[i].y * al, o4[i].z * al, o4[i].w * al);
        o2 = make_float2(o2.x * al, o2.y * al);
        const float* vt = Vs + buf * KEYS * HP;
#pragma unroll 2
        for (int c = 0; c < KEYS; c += 4) {
          const float4 p4 = *reinterpret_cast<const float4*>(Ps + o_row * PP + c);
          const float pr[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            auto sum_up = [&](float value, float& o) { o = guarded && pr[e] < 0.f ? o : fmaf(pr[e], value, o); };
#pragma unroll
            for (int i = 0; i < QUADS; ++i) {
              const float4 v = *reinterpret_cast<const float4*>(vt + (c + e) * HP + 32 * i + 4 * o_col);
              sum_up(v.x, o4[i].x);
              sum_up(v.y, o4[i].y);
              sum_up(v.z, o4[i].z);
              sum_up(v.w, o4[i].w);
            }
            if (REST) {
              const float2 v = *reinterpret_cast<const float2*>(vt + (c + e) * HP + 32 * QUADS + 2 * o_col);
              sum_up(v.x, o2.x);
              sum_up(v.y, o2.y);
            }
          }
        }
      }
    };
    if (k0 + KEYS - 1 > min_pos || (window != 0 && k0 < first_visible(max_pos, window)))
      work(std::true_type());
    else
      work(std::false_type());
    __syncthreads();  // the tile's buffer, the weights and the factors are free
    k0 = next;
    next = after;
    buf ^= 1;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (lane == 0) l_s[warp + 4 * i] = l_run[i];
  __syncthreads();
  if (o_live) {
    const float l = l_s[o_row];
    const float inv = l > 0.f ? 1.f / l : 0.f;
    float* o = out + (size_t)(tok0 + row_token(o_row)) * out_stride + (g * group + row_head(o_row)) * HD;
#pragma unroll
    for (int i = 0; i < QUADS; ++i) {
      float* at = o + 32 * i + 4 * o_col;
      at[0] = o4[i].x * inv;
      at[1] = o4[i].y * inv;
      at[2] = o4[i].z * inv;
      at[3] = o4[i].w * inv;
    }
    if (REST) {
      o[32 * QUADS + 2 * o_col] = o2.x * inv;
      o[32 * QUADS + 2 * o_col + 1] = o2.y * inv;
    }
  }
}

template <int HD>
constexpr size_t simt_smem_bytes() {
  return sizeof(float) * ((ROWS + 2 * KEYS) * (HD + 1) + ROWS * (KEYS + 1));
}

}  // namespace fg_attn
