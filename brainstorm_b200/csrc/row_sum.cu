// Sum of rows by destination index: out[o] = sum of in[r] over the rows r with index[r] == o,
// added in ascending r.  This is the tag-index branch of combine (the reference's binding
// does it with torch: scatter_reduce("sum") over the inverse indices of unique(tags),
// src/backend/torch/router.cc:449-459; its launcher refuses tag indices,
// src/router/route.cu:519-521).
//
// Destination-major and deterministic: the rows are first grouped by destination, then one
// thread per 16-byte piece of a destination row walks that row's list of row addresses,
// accumulates in fp32 in ascending source order and writes the piece once.  Every input row is
// read once, every output row is written once (rows nobody points at as zeros); no atomics on
// data, no pre-zeroed output.  The input may lie in several pieces (one tensor per path): the
// list holds addresses, so nothing has to be concatenated first (64 samples of 3 MiB over 8
// paths: the concatenation alone took 253 us, the sum takes 158).
//
// Grouping by a given index: count, scan, fill, per-destination sort of the usually very short
// lists.  Grouping by tag (the destination of a row is the rank of its tag among the distinct
// tags): up to kTagRows rows are sorted by one CTA in shared memory, which also yields the
// distinct tags and their number.
#include "common.cuh"

namespace brt_b200 {
namespace {

constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads)
index_count_kernel(const int* __restrict__ index, int64_t rows_in, int64_t rows_out,
                   int* __restrict__ seg /* [rows_out + 1], zeroed */) {
  for (int64_t r = (int64_t)blockIdx.x * kThreads + threadIdx.x; r < rows_in;
       r += (int64_t)gridDim.x * kThreads) {
    const int o = index[r];
    if (o >= 0 && o < rows_out) atomicAdd(&seg[o + 1], 1);
  }
}

// In-place inclusive scan of seg[0 .. n] (seg[0] == 0) by one CTA, so that seg[o] becomes the
// first list slot of destination o; cursor[o] starts at the same value.
__global__ void __launch_bounds__(1024)
index_scan_kernel(int* __restrict__ seg, int* __restrict__ cursor, int64_t n) {
  __shared__ int s_warp[32];
  __shared__ int s_carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int64_t base = 0; base <= n; base += 1024) {
    const int64_t i = base + threadIdx.x;
    const int v = i <= n ? seg[i] : 0;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += up;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int before = s_carry;
    for (int w = 0; w < warp; w++) before += s_warp[w];
    const int mine = before + incl;
    if (i <= n) {
      seg[i] = mine;
      if (i < n) cursor[i] = mine;
    }
    __syncthreads();
    if (threadIdx.x == 1023) s_carry = mine;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kThreads)
index_fill_kernel(const int* __restrict__ index, int64_t rows_in, int64_t rows_out,
                  int* __restrict__ cursor, int* __restrict__ list) {
  for (int64_t r = (int64_t)blockIdx.x * kThreads + threadIdx.x; r < rows_in;
       r += (int64_t)gridDim.x * kThreads) {
    const int o = index[r];
    if (o >= 0 && o < rows_out) list[atomicAdd(&cursor[o], 1)] = (int)r;
  }
}

// Input rows in up to kMaxPieces tensors, numbered through.
constexpr int kMaxPieces = 128;
struct Pieces {
  const char* ptr[kMaxPieces];
  int start[kMaxPieces + 1];  // first row of each piece
  int n;
  long long row_bytes;
};
// The address of row r; `start` is a copy of the table in shared memory.
__device__ __forceinline__ const void* row_address(const Pieces& p, const int* start, int r) {
  int lo = 0, hi = p.n - 1;  // last piece that starts at or before r (empty ones skipped)
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (start[mid] <= r) lo = mid; else hi = mid - 1;
  }
  return p.ptr[lo] + (long long)(r - start[lo]) * p.row_bytes;
}

// The fill order inside a destination's list depends on scheduling; sort every list so the
// sums are taken in ascending source order (lists hold one entry per path at most in the
// router's use, so an insertion sort by one thread is the cheapest).
__global__ void __launch_bounds__(kThreads)
index_sort_kernel(const int* __restrict__ seg, int* __restrict__ list,
                  const void** __restrict__ rows, const __grid_constant__ Pieces pieces,
                  int64_t rows_out) {
  __shared__ int s_start[kMaxPieces];
  for (int i = threadIdx.x; i < pieces.n; i += kThreads) s_start[i] = pieces.start[i];
  __syncthreads();
  for (int64_t o = (int64_t)blockIdx.x * kThreads + threadIdx.x; o < rows_out;
       o += (int64_t)gridDim.x * kThreads) {
    const int lo = seg[o], hi = seg[o + 1];
    for (int i = lo + 1; i < hi; i++) {
      const int v = list[i];
      int j = i - 1;
      while (j >= lo && list[j] > v) {
        list[j + 1] = list[j];
        j--;
      }
      list[j + 1] = v;
    }
    for (int i = lo; i < hi; i++) rows[i] = row_address(pieces, s_start, list[i]);
  }
}

// Tags of up to kTagRows rows -> distinct tags in ascending order, the segment of every tag in
// the list of its rows' addresses (ascending rows), and the number of tags.  One CTA: the keys
// (tag, row) are sorted in shared memory by a bitonic network.  drop_zero: a tag 0 (rows that
// only pad) is left out.  270 rows: 11 us; torch.unique, a bincount-like grouping and the copies
// around them took 45 us of GPU time in 18 launches, with two synchronisations.
constexpr int kTagRows = 4096;
constexpr int kTagThreads = 1024;
__global__ void __launch_bounds__(kTagThreads)
tag_group_kernel(const __grid_constant__ Pieces tags, const __grid_constant__ Pieces pieces,
                 int drop_zero, int* __restrict__ tags_out, int* __restrict__ seg,
                 const void** __restrict__ rows, int* __restrict__ count) {
  __shared__ unsigned long long s_key[kTagRows];
  __shared__ int s_start[kMaxPieces];
  __shared__ int s_warp[kTagThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < tags.n; i += kTagThreads) s_start[i] = tags.start[i];
  __syncthreads();
  const int n = tags.start[tags.n];
  int size = 2;
  while (size < n) size <<= 1;
  for (int i = tid; i < size; i += kTagThreads) {
    unsigned long long key = ~0ull;
    if (i < n) {
      const int tag = *static_cast<const int*>(row_address(tags, s_start, i));
      key = ((unsigned long long)((unsigned)tag ^ 0x80000000u) << 32) | (unsigned)i;
    }
    s_key[i] = key;
  }
  for (int k = 2; k <= size; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      for (int p = tid; p < size >> 1; p += kTagThreads) {
        const int i = ((p & ~(j - 1)) << 1) | (p & (j - 1));  // bit j clear
        const unsigned long long a = s_key[i], b = s_key[i + j];
        if ((a > b) == ((i & k) == 0)) {
          s_key[i] = b;
          s_key[i + j] = a;
        }
      }
    }
  }
  __syncthreads();
  auto tag_at = [&](int i) { return (unsigned)(s_key[i] >> 32); };
  const int skip = drop_zero && tag_at(0) == 0x80000000u ? 1 : 0;
  // heads of segments, numbered through: a thread owns kPer neighbours
  constexpr int kPer = kTagRows / kTagThreads;
  int heads = 0;
  for (int u = 0; u < kPer; u++) {
    const int i = tid * kPer + u;
    if (i < n && (i == 0 || tag_at(i) != tag_at(i - 1))) heads++;
  }
  int incl = heads;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += up;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  int at = incl - heads, total = 0;
  for (int w = 0; w < kTagThreads / 32; w++) {
    if (w < warp) at += s_warp[w];
    total += s_warp[w];
  }
  for (int u = 0; u < kPer; u++) {
    const int i = tid * kPer + u;
    if (i >= n) break;
    rows[i] = row_address(pieces, s_start, (int)(unsigned)s_key[i]);
    if (i == 0 || tag_at(i) != tag_at(i - 1)) {
      if (at >= skip) {
        tags_out[at - skip] = (int)(tag_at(i) ^ 0x80000000u);
        seg[at - skip] = i;
      }
      at++;
    }
  }
  if (tid == 0) {
    seg[total - skip] = n;
    count[0] = total - skip;
  }
}

// VB-byte pieces: one thread per (destination row, piece).
template <int DT, int VB>
__global__ void __launch_bounds__(kThreads)
row_sum_kernel(const void* const* __restrict__ rows, void* __restrict__ out,
               const int* __restrict__ seg, int64_t rows_out,
               int64_t row_vecs) {
  using T = typename Elem<DT>::type;
  using V = typename Chunk<VB>::type;
  constexpr int N = VB / (int)sizeof(T);
  V* __restrict__ dst = static_cast<V*>(out);
  const int64_t items = rows_out * row_vecs;
  for (int64_t it = (int64_t)blockIdx.x * kThreads + threadIdx.x; it < items;
       it += (int64_t)gridDim.x * kThreads) {
    const int64_t o = it / row_vecs;
    const int64_t v = it - o * row_vecs;
    float acc[N];
#pragma unroll
    for (int i = 0; i < N; i++) acc[i] = 0.f;
    const int lo = seg[o], hi = seg[o + 1];
    for (int k = lo; k < hi; k++) {
      const V piece = load_stream(static_cast<const V*>(rows[k]) + v);
      const T* e = reinterpret_cast<const T*>(&piece);
#pragma unroll
      for (int i = 0; i < N; i++) acc[i] = __fadd_rn(acc[i], Elem<DT>::to_f32(e[i]));
    }
    V res;
    T* e = reinterpret_cast<T*>(&res);
#pragma unroll
    for (int i = 0; i < N; i++) e[i] = Elem<DT>::from_f32(acc[i]);
    store_stream(dst + it, res);
  }
}

size_t group_scratch_bytes(int64_t rows_in, int64_t rows_out) {
  return round_up((size_t)(rows_out + 1) * 4, 256) + round_up((size_t)rows_out * 4 + 4, 256) +
         round_up((size_t)rows_in * 4 + 4, 256) + round_up((size_t)rows_in * 8 + 8, 256);
}

template <int DT>
void launch_row_sum(int vb, const void* const* rows, void* out, const int* seg,
                    int64_t rows_out, int64_t row_bytes, cudaStream_t st) {
  const int64_t row_vecs = row_bytes / vb;
  int64_t blocks = (rows_out * row_vecs + kThreads - 1) / kThreads;
  // one piece per thread, CTAs in launch order: 64 x 3 MiB from 270 rows 158 us, 167 with resident
  // CTAs that stride (DRAM likes the narrow window of CTAs launched in order)
  const int64_t cap = 0x7fffffff;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  const KernelTimer timer("row_sum_kernel", st);
  constexpr int kElem = DT == BRT_F32 ? 4 : 2;
  if (vb == 16)
    row_sum_kernel<DT, 16><<<(unsigned)blocks, kThreads, 0, st>>>(rows, out, seg, rows_out,
                                                                   row_vecs), note_launch();
  else
    row_sum_kernel<DT, kElem><<<(unsigned)blocks, kThreads, 0, st>>>(rows, out, seg, rows_out,
                                                                      row_vecs), note_launch();
}

int sum_grouped(const Pieces& pieces, const void* const* rows, const int* seg, void* out,
                int64_t rows_out, int dtype, cudaStream_t st) {
  const int es = dtype_size(dtype);
  bool wide = pieces.row_bytes % 16 == 0 && aligned_to(out, 16);
  bool fits = aligned_to(out, es);
  for (int i = 0; i < pieces.n; i++) {
    if (pieces.start[i + 1] == pieces.start[i]) continue;
    wide = wide && aligned_to(pieces.ptr[i], 16);
    fits = fits && aligned_to(pieces.ptr[i], es);
  }
  BRT_REQUIRE(fits, "misaligned rows");
  const int vb = wide ? 16 : es;
  switch (dtype) {
    case BRT_F32: launch_row_sum<BRT_F32>(vb, rows, out, seg, rows_out, pieces.row_bytes, st); break;
    case BRT_F16: launch_row_sum<BRT_F16>(vb, rows, out, seg, rows_out, pieces.row_bytes, st); break;
    default: launch_row_sum<BRT_BF16>(vb, rows, out, seg, rows_out, pieces.row_bytes, st); break;
  }
  BRT_LAUNCH_CHECK("row_sum_kernel");
  return BRT_OK;
}

// The table of the caller's pieces; more than 2^31 - 1 rows or kMaxPieces pieces are refused.
int pieces_of(Pieces* out, const void* const* ptrs, const int64_t* rows, int n, int64_t row_bytes) {
  BRT_REQUIRE(n >= 1 && n <= kMaxPieces && ptrs != nullptr && rows != nullptr,
              "between 1 and %d pieces", kMaxPieces);
  int64_t at = 0;
  for (int i = 0; i < n; i++) {
    BRT_REQUIRE(rows[i] >= 0 && (rows[i] == 0 || ptrs[i] != nullptr), "bad piece %d", i);
    out->ptr[i] = static_cast<const char*>(ptrs[i]);
    out->start[i] = (int)at;
    at += rows[i];
    BRT_REQUIRE(at <= 0x7fffffffLL, "too many rows");
  }
  out->start[n] = (int)at;
  out->n = n;
  out->row_bytes = row_bytes;
  return BRT_OK;
}

}  // namespace
}  // namespace brt_b200

using namespace brt_b200;

extern "C" {

BRT_API size_t brt_sum_rows_scratch_bytes(int64_t rows_in, int64_t rows_out) {
  if (rows_in < 0 || rows_out < 0) return 0;
  return group_scratch_bytes(rows_in, rows_out);
}

BRT_API int brt_sum_rows_by_index(const void* in_rows, const int32_t* row_index, void* out_rows,
                                  int64_t rows_in, int64_t rows_out, int64_t cell_size,
                                  int dtype, void* scratch, size_t scratch_bytes, void* stream) {
  return brt_sum_pieces_by_index(&in_rows, &rows_in, 1, row_index, out_rows, rows_out, cell_size,
                                 dtype, scratch, scratch_bytes, stream);
}

BRT_API int brt_sum_pieces_by_index(const void* const* in_pieces, const int64_t* piece_rows,
                                    int pieces, const int32_t* row_index, void* out_rows,
                                    int64_t rows_out, int64_t cell_size, int dtype,
                                    void* scratch, size_t scratch_bytes, void* stream) {
  clear_error();
  BRT_REQUIRE(dtype == BRT_F32 || dtype == BRT_F16 || dtype == BRT_BF16, "bad dtype %d", dtype);
  BRT_REQUIRE(rows_out >= 0 && cell_size >= 0, "negative size");
  BRT_REQUIRE(rows_out <= 0x7ffffffeLL, "too many rows");
  if (rows_out == 0 || cell_size == 0) return BRT_OK;
  Pieces table;
  if (int rc = pieces_of(&table, in_pieces, piece_rows, pieces, cell_size * dtype_size(dtype)))
    return rc;
  const int64_t rows_in = table.start[table.n];
  BRT_REQUIRE(out_rows != nullptr && (rows_in == 0 || row_index != nullptr),
              "null pointer argument");
  BRT_REQUIRE(scratch != nullptr && aligned_to(scratch, 256),
              "scratch must be a 256-byte aligned device buffer");
  const size_t need = group_scratch_bytes(rows_in, rows_out);
  if (scratch_bytes < need)
    return set_error(BRT_ERR_SCRATCH_TOO_SMALL, "scratch holds %zu bytes, %zu needed",
                     scratch_bytes, need);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  char* p = static_cast<char*>(scratch);
  int* seg = reinterpret_cast<int*>(p);
  p += round_up((size_t)(rows_out + 1) * 4, 256);
  int* cursor = reinterpret_cast<int*>(p);
  p += round_up((size_t)rows_out * 4 + 4, 256);
  int* list = reinterpret_cast<int*>(p);
  p += round_up((size_t)rows_in * 4 + 4, 256);
  const void** rows = reinterpret_cast<const void**>(p);
  BRT_CUDA_TRY(cudaMemsetAsync(seg, 0, (size_t)(rows_out + 1) * 4, st));
  int64_t blocks = (rows_in + kThreads - 1) / kThreads;
  const int64_t cap = (int64_t)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  index_count_kernel<<<(unsigned)blocks, kThreads, 0, st>>>(row_index, rows_in, rows_out, seg),
      note_launch();
  index_scan_kernel<<<1, 1024, 0, st>>>(seg, cursor, rows_out), note_launch();
  index_fill_kernel<<<(unsigned)blocks, kThreads, 0, st>>>(row_index, rows_in, rows_out, cursor,
                                                           list),
      note_launch();
  int64_t sort_blocks = (rows_out + kThreads - 1) / kThreads;
  if (sort_blocks > cap) sort_blocks = cap;
  index_sort_kernel<<<(unsigned)sort_blocks, kThreads, 0, st>>>(seg, list, rows, table, rows_out),
      note_launch();
  BRT_LAUNCH_CHECK("row grouping kernels");
  return sum_grouped(table, rows, seg, out_rows, rows_out, dtype, st);
}

BRT_API size_t brt_tag_group_bytes(int64_t rows_in) {
  if (rows_in < 2 || rows_in > kTagRows) return 0;
  return round_up((size_t)(rows_in + 1) * 4, 256) + (size_t)rows_in * 8;
}

BRT_API int brt_group_pieces_by_tag(const void* const* in_pieces, const void* const* tag_pieces,
                                    const int64_t* piece_rows, int pieces, int64_t cell_size,
                                    int dtype, int drop_zero, int32_t* tags_out, int32_t* count,
                                    void* groups, size_t group_bytes, void* stream) {
  clear_error();
  BRT_REQUIRE(dtype == BRT_F32 || dtype == BRT_F16 || dtype == BRT_BF16, "bad dtype %d", dtype);
  BRT_REQUIRE(cell_size > 0, "empty cells");
  Pieces table, tags;
  if (int rc = pieces_of(&table, in_pieces, piece_rows, pieces, cell_size * dtype_size(dtype)))
    return rc;
  if (int rc = pieces_of(&tags, tag_pieces, piece_rows, pieces, 4)) return rc;
  const int64_t rows_in = table.start[table.n];
  const size_t need = brt_tag_group_bytes(rows_in);
  if (need == 0)
    return set_error(BRT_ERR_UNSUPPORTED, "%lld rows: between 2 and %d are grouped by tag",
                     (long long)rows_in, kTagRows);
  BRT_REQUIRE(tags_out != nullptr && count != nullptr && groups != nullptr &&
                  aligned_to(groups, 256),
              "null or misaligned pointer argument");
  for (int i = 0; i < pieces; i++)
    BRT_REQUIRE(piece_rows[i] == 0 || aligned_to(tag_pieces[i], 4), "misaligned tags");
  if (group_bytes < need)
    return set_error(BRT_ERR_SCRATCH_TOO_SMALL, "groups holds %zu bytes, %zu needed", group_bytes,
                     need);
  char* p = static_cast<char*>(groups);
  tag_group_kernel<<<1, kTagThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      tags, table, drop_zero, tags_out, reinterpret_cast<int*>(p),
      reinterpret_cast<const void**>(p + round_up((size_t)(rows_in + 1) * 4, 256)), count),
      note_launch();
  BRT_LAUNCH_CHECK("tag_group_kernel");
  return BRT_OK;
}

BRT_API int brt_sum_grouped_pieces(const void* const* in_pieces, const int64_t* piece_rows,
                                   int pieces, const void* groups, void* out_rows,
                                   int64_t rows_out, int64_t cell_size, int dtype,
                                   void* stream) {
  clear_error();
  BRT_REQUIRE(dtype == BRT_F32 || dtype == BRT_F16 || dtype == BRT_BF16, "bad dtype %d", dtype);
  BRT_REQUIRE(rows_out >= 0 && cell_size >= 0, "negative size");
  if (rows_out == 0 || cell_size == 0) return BRT_OK;
  Pieces table;
  if (int rc = pieces_of(&table, in_pieces, piece_rows, pieces, cell_size * dtype_size(dtype)))
    return rc;
  const int64_t rows_in = table.start[table.n];
  BRT_REQUIRE(rows_out <= rows_in, "more groups than rows");
  BRT_REQUIRE(groups != nullptr && out_rows != nullptr, "null pointer argument");
  const char* p = static_cast<const char*>(groups);
  return sum_grouped(table,
                     reinterpret_cast<const void* const*>(
                         p + round_up((size_t)(rows_in + 1) * 4, 256)),
                     reinterpret_cast<const int*>(p), out_rows, rows_out, dtype,
                     static_cast<cudaStream_t>(stream));
}

}  // extern "C"
