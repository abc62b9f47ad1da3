// The sequences of a step that the recurrences walk chunk by chunk: those of `min_tokens` tokens and more.
//
// A captured step holds a place for every request the engine admits (256 by default), most of them empty, so nothing
// may be launched by places.  The blocks that prepare the chunks are launched for the most chunks the step's tokens
// can make, and find their sequence here; the first of them also writes the list of the long sequences, and
// the blocks that walk draw their work from it: (sequence, part) items, the parts of a sequence side by side.
// With a block a (place, part), one prompt of 2,048 tokens among 256 places took the state-space walk (64 heads) 373 us
// and its preparation 36, alone 198 and 16; this way 202 and 19, alone 201 and 17.  The delta rule's (16
// heads of 64): 145 and 80 us, alone 110 and 42; this way 85 and 39 both times.
#pragma once

#include "common.cuh"

namespace long_seq {

struct Found {
  int seq, tokens, first_chunk;  // seq < 0: no such sequence
};

// In front of the chunks' scratch: the number of long sequences, that of the items drawn so far and those of the blocks
// that have come up on each SM, then the sequences.
constexpr int SMS = 252;
struct Head {
  int n_seqs, drawn, pad[2], on_sm[SMS];
};
struct Entry {
  int seq, tokens, first_chunk, pad;
};
// most sequences of `min_tokens` tokens in a step, most chunks of them, and the floats of head and list
inline long most_sequences(int n_tokens, int n_seqs, int min_tokens) {
  return n_seqs < n_tokens / min_tokens ? n_seqs : n_tokens / min_tokens;
}
inline long most_chunks(int n_tokens, int n_seqs, int min_tokens, int chunk) {
  return n_tokens / chunk + most_sequences(n_tokens, n_seqs, min_tokens);
}
inline long list_floats(int n_tokens, int n_seqs, int min_tokens) {
  return sizeof(Head) / 4 + sizeof(Entry) / 4 * most_sequences(n_tokens, n_seqs, min_tokens);
}

// The sequence that holds chunk `target` (the long sequences' chunks are numbered one after another).  With `list`,
// the whole list is written too.  For all threads of a block, THREADS of them; places are read THREADS at a time.
template <int CHUNK, int THREADS>
__device__ __forceinline__ Found find_chunk(const int* __restrict__ seq_slot, const int* __restrict__ seq_start, int n_seqs,
                                            int min_tokens, int target, Head* list) {
  constexpr int WARPS = THREADS / 32;
  __shared__ int seqs_s[WARPS], chunks_s[WARPS];
  __shared__ Found found_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int seqs = 0, chunks = 0;  // before this stretch of places
  if (tid == 0) found_s.seq = -1;
  for (int base = 0; base < n_seqs; base += THREADS) {
    const int i = base + tid;
    int n = 0;
    if (i < n_seqs && seq_slot[i] >= 0) n = seq_start[i + 1] - seq_start[i];
    const bool is_long = n >= min_tokens;
    const int own = is_long ? (n + CHUNK - 1) / CHUNK : 0;
    const unsigned longs = __ballot_sync(0xffffffffu, is_long);
    int upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    if (lane == 31) {
      seqs_s[warp] = __popc(longs);
      chunks_s[warp] = upto;
    }
    __syncthreads();
    int rank = seqs + __popc(longs & ((1u << lane) - 1)), first = chunks + upto - own;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      if (w < warp) {
        rank += seqs_s[w];
        first += chunks_s[w];
      }
      seqs += seqs_s[w];
      chunks += chunks_s[w];
    }
    if (is_long) {
      if (target >= first && target < first + own) found_s = {i, n, first};
      if (list) reinterpret_cast<Entry*>(list + 1)[rank] = {i, n, first, 0};
    }
    __syncthreads();
    if (list == nullptr && chunks > target) break;
  }
  __syncthreads();
  if (list) {
    if (tid == 0) {
      list->n_seqs = seqs;
      list->drawn = 0;
    }
    for (int i = tid; i < SMS; i += THREADS) list->on_sm[i] = 0;
  }
  return found_s;
}

// The blocks of a walk take the items (list.n_seqs sequences of `parts` parts) in order, each the next one when it is
// through; draw() is called by all threads, between two items.  A launch may have more blocks than there are
// items, and two neighbours may come up on one SM while others have none: a block that finds as many on its SM as each
// would have items waits a microsecond or two before it draws.
struct Items {
  Head* list;
  int parts, total, item;
  __device__ __forceinline__ Items(Head* l, int parts_) : list(l), parts(parts_) {
    total = l->n_seqs * parts;
    item = blockIdx.x;
    if (total > 0 && total < (int)gridDim.x) {
      unsigned sm, sms;
      asm volatile("mov.u32 %0, %%smid;\n" : "=r"(sm));
      asm volatile("mov.u32 %0, %%nsmid;\n" : "=r"(sms));
      take([&] {
        if (sm < SMS && atomicAdd(&list->on_sm[sm], 1) * (int)sms >= total) {
          __nanosleep(1500);
        }
        return atomicAdd(&list->drawn, 1);
      });
    }
  }
  __device__ __forceinline__ bool more() const { return item < total; }
  __device__ __forceinline__ Entry sequence() const { return reinterpret_cast<const Entry*>(list + 1)[item / parts]; }
  __device__ __forceinline__ int part() const { return item % parts; }
  __device__ __forceinline__ void draw() {
    if (total == (int)gridDim.x) item = total;  // a block an item
    else take([&] { return (total < (int)gridDim.x ? 0 : gridDim.x) + atomicAdd(&list->drawn, 1); });
  }
  template <typename F>
  __device__ __forceinline__ void take(F next) {
    __shared__ int next_s;
    __syncthreads();  // everybody is through with the item and with the last draw
    if (threadIdx.x == 0) next_s = next();
    __syncthreads();
    item = next_s;
  }
};

}  // namespace long_seq
