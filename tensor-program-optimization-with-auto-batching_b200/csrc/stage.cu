// Small tables of a pass on their way to the device: the values travel in the launch's own parameters.
//
// A pinned buffer and a copy per table cost the host 25 to 60 us in front of a prompt pass's first kernel and the GPU a copy
// engine's start for each; a launch costs 4 us and needs no buffer that has to outlive it.  Rows of a prompt pass go as one
// record per sequence, not as three numbers per row.  With the engine's status words read at once and the stream's handle taken
// without its object: two Llama layers, 2 prompts of 17 tokens 858 -> 711 us a pass, 5 of 17 to 301 1268 -> 1161; the
// peft-style layer, 8 rows 68 -> 52 (570 -> 555 on the first pass over new inputs).
#include "common.cuh"

namespace mlora {
namespace {

constexpr int kPutInts = 896;   // values of one launch (kernel parameters hold 4 KB)
constexpr int kPutSeqs = 128;   // sequences of one launch

struct PutArgs {
  int32_t* dst;
  int n, repeat;
  int32_t v[kPutInts];
};
__global__ void __launch_bounds__(256) put_i32_kernel(const __grid_constant__ PutArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i < (long long)a.n * a.repeat) a.dst[i] = a.v[i / a.repeat];
}

struct RowsArgs {
  int32_t *slots, *row_slot, *row_pos;
  int n, row0, rows;  // sequences; the first one's first row, rows of all
  int4 seq[kPutSeqs];  // first row, cache slot, adapter slot, position of the first row
};
__global__ void __launch_bounds__(256) put_rows_kernel(const __grid_constant__ RowsArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= a.rows) return;
  const int r = a.row0 + i;
  int lo = 0, hi = a.n - 1;  // the last sequence that starts at or before r (those without rows end where the next begins)
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (a.seq[mid].x <= r)
      lo = mid;
    else
      hi = mid - 1;
  }
  const int4 s = a.seq[lo];
  a.slots[r] = s.z;
  a.row_slot[r] = s.y;
  a.row_pos[r] = s.w + (r - s.x);
}

}  // namespace
}  // namespace mlora

using namespace mlora;

extern "C" int mlora_put_i32(int32_t* d_dst, const int32_t* h_values, int32_t n, int32_t repeat, void* stream) {
  MLORA_REQUIRE(n >= 0 && repeat > 0 && d_dst && h_values, "put_i32: bad arguments (n=%d repeat=%d)", n, repeat);
  MLORA_REQUIRE((long long)n * repeat <= 2147483647ll, "put_i32: %d values %d times", n, repeat);
  for (int first = 0; first < n; first += kPutInts) {
    PutArgs a;
    a.n = n - first < kPutInts ? n - first : kPutInts;
    a.repeat = repeat;
    a.dst = d_dst + (size_t)first * repeat;
    for (int i = 0; i < a.n; ++i) a.v[i] = h_values[first + i];
    launch_pdl(put_i32_kernel, (unsigned)(((long long)a.n * repeat + 255) / 256), 256, 0, (cudaStream_t)stream, a);
    count_launch();
    MLORA_CHECK_LAUNCH("put_i32_kernel");
  }
  return MLORA_OK;
}

extern "C" int mlora_put_rows(const int32_t* h_seqs, int32_t n, int32_t* d_slots, int32_t* d_row_slot, int32_t* d_row_pos, void* stream) {
  MLORA_REQUIRE(n >= 0 && h_seqs && d_slots && d_row_slot && d_row_pos, "put_rows: bad arguments (n=%d)", n);
  long long row = 0;
  for (int i = 0; i < n; ++i) {
    MLORA_REQUIRE(h_seqs[4 * i + 2] >= 0, "put_rows: sequence %d has %d rows", i, h_seqs[4 * i + 2]);
    row += h_seqs[4 * i + 2];
  }
  MLORA_REQUIRE(row <= 2147483647ll, "put_rows: too many rows");
  int at = 0;
  for (int first = 0; first < n; first += kPutSeqs) {
    RowsArgs a;
    a.slots = d_slots;
    a.row_slot = d_row_slot;
    a.row_pos = d_row_pos;
    a.n = n - first < kPutSeqs ? n - first : kPutSeqs;
    a.row0 = at;
    for (int i = 0; i < a.n; ++i) {
      const int32_t* s = h_seqs + 4 * (size_t)(first + i);  // cache slot, adapter slot, rows, position of the first row
      a.seq[i] = make_int4(at, s[0], s[1], s[3]);
      at += s[2];
    }
    a.rows = at - a.row0;
    if (a.rows == 0) continue;
    launch_pdl(put_rows_kernel, (unsigned)((a.rows + 255) / 256), 256, 0, (cudaStream_t)stream, a);
    count_launch();
    MLORA_CHECK_LAUNCH("put_rows_kernel");
  }
  return MLORA_OK;
}
