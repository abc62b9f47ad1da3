// Changes of a block table, carried to the device in the launch's own arguments.
//
// A step's new pages are a few entries (a 2,048-token prompt takes 32 pages of 64), known on the host.  A copy from
// pageable memory makes the host wait until everything before it on the stream has run, so that the step's
// own host work (some 0.3 to 0.6 ms for a prompt of 2,048 tokens) starts only when the device is idle; a
// copy from pinned memory needs buffers whose allocation costs milliseconds an engine.  Launch arguments are read
// when the launch is made: nothing waits, and nothing has to outlive the call.
#include "common.cuh"

namespace {
constexpr int ENTRIES = 480;  // a launch's arguments hold 4 KB

struct Entries {
  int at[ENTRIES], value[ENTRIES];
};

__global__ void table_entries_kernel(int* __restrict__ table, const __grid_constant__ Entries e, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) table[e.at[i]] = e.value[i];
}
}  // namespace

// table[at[i]] = value[i] for n entries with different places; `at` and `value` are host memory, read before the call
// returns.  The caller has checked the places.
extern "C" int fg_set_table_entries(int* table, const int* at, const int* value, int n, cudaStream_t stream) {
  for (int done = 0; done < n; done += ENTRIES) {
    Entries e;
    const int m = n - done < ENTRIES ? n - done : ENTRIES;
    for (int i = 0; i < m; ++i) {
      e.at[i] = at[done + i];
      e.value[i] = value[done + i];
    }
    table_entries_kernel<<<(m + 127) / 128, 128, 0, stream>>>(table, e, m);
    FG_CHECK_LAUNCH("fg_set_table_entries");
  }
  return 0;
}
