// pmp_store.cu -- the droplet store: hand-over (pmp_spray_set_particles),
// packing into the cell-sorted structure of arrays the update kernels read,
// and write-back (pmp_spray_get_particles).
//
// A box's droplets are handed over into staging rows (one 128- or 160-byte
// row per droplet: the reals, the id and the caller's index) and a sort key
// each (box, then cell), whatever the caller's layout.  The first operation
// that needs the droplets packs all boxes at once: one sort over every box (by
// counting into cells, cell_sort.cuh, or a radix sort), one gather of whole
// rows into the store's component arrays.  A row is whole 32-byte sectors, so
// the gather in sorted (random) order moves no byte it does not use, where
// gathering 8 bytes from each of 14-17 component arrays read four times the
// data; write-back to records goes the same way round.  Staging rows, store,
// sort arrays and maps stay with the handle between calls (KeptBuffer), so
// that a caller who hands its droplets over for every call, in device memory
// that the kernels read directly, allocates nothing in the steady state
// (droplets that come another way pass through a buffer, given back when it is
// above 64 MB).  A buffer above 256 MB of which a packing leaves three quarters
// idle is given back.  Measured, hand-over, update and write-back: 2M
// two-fuel droplets in 8 boxes, FP64, 56.0 -> 2.82 ms (2.15 ms of it the
// update; with a cudaMalloc and cudaFree per array and box the allocator took
// 46 ms and moving droplets 1.8 ms), 0.78M droplets in 64 uneven boxes
// 72.9 -> 2.24 ms, 8M droplets in the mixed form 79.9 -> 4.31 ms.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

#include "cell_sort.cuh"
#include "pmp_handle.h"

namespace pmp {

namespace {

int check(pmp_spray* h, cudaError_t e, const char* what)
{
  if (e != cudaSuccess) {
    char b[160];
    snprintf(b, sizeof(b), "%s: %s", what, cudaGetErrorString(e));
    cudaGetLastError();  // reported here, not by the next call
    return set_err(h, PMP_ERR_CUDA, b);
  }
  return PMP_OK;
}

#define PMP_TRY(h, call)                        \
  do {                                          \
    const int rc_ = check((h), (call), #call);  \
    if (rc_ != PMP_OK) {                        \
      return rc_;                               \
    }                                           \
  } while (0)

constexpr int kTile = 128;  // droplets per CTA of the kernels below
constexpr int kMaxWords = 4 + PMP_PSTATE_NUM(PMP_MAX_FUEL);

// A droplet's staging row: 3 + NR reals, then {id, caller's index} in one
// word, padded to whole sectors.
template <int NF>
struct Row {
  static constexpr int kReals = 3 + PMP_PSTATE_NUM(NF);
  static constexpr int kWords = kReals + 1;
  static constexpr int kStride = (kWords + 3) / 4 * 4;  // doubles
  static constexpr int kPieces = (kWords + 1) / 2;      // 16-byte pieces that hold words
  static constexpr int kPitch = kWords | 1;             // shared-memory tile: odd, so that a column is conflict-free
};
int row_stride(int nf) { return (PMP_PSTATE_NUM(nf) + 4 + 3) / 4 * 4; }

struct Columns {
  double* c[kMaxWords - 1];
  int* id;
};

// The sort key of a droplet of one box: the box above `shift` bits of its
// cell's place in the box's sort order (brick_key over the box and kSortPad
// cells around it; a droplet further out counts to the edge).
struct KeyOf {
  double plo[3], dxi[3];
  int lo[3], ext[3];
  unsigned long long base;  // box << shift
  int kept;                 // the rows are in the store's order: keep it
};
__device__ __forceinline__ unsigned long long sort_key(const KeyOf& k, double x, double y, double z)
{
  if (k.kept) {
    return k.base;
  }
  const double p[3] = {x, y, z};
  int c[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int v = static_cast<int>(floor(__dmul_rn(__dsub_rn(p[d], k.plo[d]), k.dxi[d]))) - k.lo[d] + kSortPad;
    c[d] = v < 0 ? 0 : (v >= k.ext[d] ? k.ext[d] - 1 : v);
  }
  return k.base | brick_key(c[0], c[1], c[2], k.ext[0], k.ext[1]);
}

// Where a staging kernel leaves each row's key and index (narrow keys; null:
// formed from the rows when they are packed); with counts, the row is counted
// into its cell and its rank takes the index's place
struct KeyOut {
  unsigned* keys;
  int* idx;
  long long row0;  // index of the kernel's first row
  unsigned* counts;
  int* crowded;
};

// A thread's row in the keys, before and after the CTA writes its rows (all
// lanes call both); valid: the thread has a row, i its number among the kernel's
struct RowKey {
  unsigned key;
  Counted count;
};
__device__ __forceinline__ RowKey begin_key(const KeyOut& out, const KeyOf& key, bool valid, const double* pos)
{
  RowKey k{};
  if (out.keys) {
    k.key = valid ? (unsigned)sort_key(key, pos[0], pos[1], pos[2]) : kNoCell;
    if (out.counts) {
      k.count = count_cell(out.counts, k.key);
    }
  }
  return k;
}
__device__ __forceinline__ void end_key(const KeyOut& out, const RowKey& k, bool valid, long long i)
{
  if (out.keys) {
    const int v = out.counts ? rank_of(k.count, k.key, out.crowded) : (int)(out.row0 + i);
    if (valid) {
      out.keys[i] = k.key;
      out.idx[i] = v;
    }
  }
}

__device__ __forceinline__ double pack_ints(int lo, int hi) { return __hiloint2double(hi, lo); }

// tile[r][w] of the CTA's rows -> staging rows, 16 bytes a lane
template <int NF>
__device__ __forceinline__ void tile_to_rows(const double (*tile)[Row<NF>::kPitch], double* rows, int m)
{
  using R = Row<NF>;
  for (int i = threadIdx.x; i < m * R::kPieces; i += kTile) {
    const int r = i / R::kPieces, w = 2 * (i % R::kPieces);
    double2 v;
    v.x = tile[r][w];
    v.y = w + 1 < R::kWords ? tile[r][w + 1] : 0.;
    *reinterpret_cast<double2*>(rows + (long long)r * R::kStride + w) = v;
  }
}

// AMReX records {pos[3], rdata[10 + F], id, cpu} -> rows.  Records are read as
// one stream of words (the caller's buffer is 8-byte aligned, a record with
// one fuel is 120 bytes), and turned in shared memory.
template <int NF>
__global__ void __launch_bounds__(kTile) k_aos_to_rows(const double* aos, long long n, double* rows,
                                                       const __grid_constant__ KeyOf key, const KeyOut out)
{
  using R = Row<NF>;
  __shared__ double tile[kTile][R::kPitch];
  const long long s0 = (long long)blockIdx.x * kTile;
  const int m = (int)min((long long)kTile, n - s0);
  const double* src = aos + s0 * R::kWords;
  for (int i = threadIdx.x; i < m * R::kWords; i += kTile) {
    tile[i / R::kWords][i % R::kWords] = __ldcs(src + i);
  }
  __syncthreads();
  double* t = tile[threadIdx.x];
  const bool valid = (int)threadIdx.x < m;
  if (valid) {
    const int id = __double2loint(t[R::kReals]);
    t[R::kReals] = pack_ints(id, (int)(s0 + threadIdx.x));
  }
  const RowKey k = begin_key(out, key, valid, t);
  __syncthreads();
  tile_to_rows<NF>(tile, rows + s0 * R::kStride, m);
  end_key(out, k, valid, s0 + threadIdx.x);
}

// component arrays -> rows; a null component is zero.  caller: the droplets'
// caller indices, or null for 0, 1, ...
template <int NF>
__global__ void __launch_bounds__(kTile) k_columns_to_rows(const __grid_constant__ Columns C, const long long* caller,
                                                           long long n, double* rows,
                                                           const __grid_constant__ KeyOf key, const KeyOut out)
{
  using R = Row<NF>;
  __shared__ double tile[kTile][R::kPitch];
  const long long s0 = (long long)blockIdx.x * kTile;
  const int m = (int)min((long long)kTile, n - s0);
  const long long s = s0 + threadIdx.x;
  const bool valid = (int)threadIdx.x < m;
  double* t = tile[threadIdx.x];
  if (valid) {
#pragma unroll
    for (int c = 0; c < R::kReals; ++c) {
      t[c] = C.c[c] ? __ldcs(C.c[c] + s) : 0.;
    }
    t[R::kReals] = pack_ints(C.id[s], caller ? (int)caller[s] : (int)s);
  }
  const RowKey k = begin_key(out, key, valid, t);
  __syncthreads();
  tile_to_rows<NF>(tile, rows + s0 * R::kStride, m);
  end_key(out, k, valid, s);
}

// One box's staging rows, in the order of the packed store (box by box).
struct Region {
  long long row;    // first staging row
  long long begin;  // first slot of the box
  KeyOf key;
};

__device__ __forceinline__ int region_of(const Region* reg, int nb, long long s)
{
  int lo = 0, hi = nb;
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (reg[mid].begin <= s) {
      lo = mid;
    } else {
      hi = mid;
    }
  }
  return lo;
}

// Wide keys (the boxes' bits do not fit 32, or 2^31 rows and more), from the
// rows, and the rows' indices.
__global__ void __launch_bounds__(256) k_row_keys(const double* rows, int stride, const Region* reg, int nb, long long n,
                                                  unsigned long long* keys, long long* idx)
{
  const long long s = blockIdx.x * 256LL + threadIdx.x;
  if (s >= n) {
    return;
  }
  const Region& g = reg[region_of(reg, nb, s)];
  const long long r = g.row + (s - g.begin);
  const double* q = rows + r * stride;
  keys[s] = sort_key(g.key, q[0], q[1], q[2]);
  idx[s] = r;
}

// rows [0, n): key (keys null: unchanged) and their own index
__global__ void __launch_bounds__(256) k_fill_keys(unsigned* keys, int* idx, long long row0, long long n, unsigned key)
{
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  if (i < n) {
    if (keys) {
      keys[row0 + i] = key;
    }
    idx[row0 + i] = (int)(row0 + i);
  }
}

// rows in sorted order -> the store.  Eight or nine lanes read one row.
template <int NF, typename V>
__global__ void __launch_bounds__(kTile) k_rows_to_store(const double* rows, const V* order, long long n, double* soa,
                                                         int* ids, long long* perm)
{
  using R = Row<NF>;
  __shared__ double tile[kTile][R::kPitch];
  const long long s0 = (long long)blockIdx.x * kTile;
  const int m = (int)min((long long)kTile, n - s0);
#pragma unroll
  for (int it = 0; it < R::kPieces; ++it) {
    const int i = it * kTile + threadIdx.x;
    const int r = i / R::kPieces, w = 2 * (i % R::kPieces);
    if (r < m) {
      const double2 v = __ldcs(reinterpret_cast<const double2*>(rows + (long long)order[s0 + r] * R::kStride + w));
      tile[r][w] = v.x;
      if (w + 1 < R::kWords) {
        tile[r][w + 1] = v.y;
      }
    }
  }
  __syncthreads();
  if ((int)threadIdx.x < m) {
    const long long s = s0 + threadIdx.x;
#pragma unroll
    for (int c = 0; c < R::kReals; ++c) {
      soa[c * n + s] = tile[threadIdx.x][c];
    }
    const double t = tile[threadIdx.x][R::kReals];
    ids[s] = __double2loint(t);
    perm[s] = (long long)__double2hiint(t);
  }
}

// the store's slots of one box -> records in the caller's order: whole
// records per droplet, turned in shared memory
template <int NF>
__global__ void __launch_bounds__(kTile) k_store_to_aos(const double* soa, long long total, const int* ids,
                                                        const long long* perm, long long n, double* aos)
{
  using R = Row<NF>;
  __shared__ double tile[kTile][R::kPitch];
  __shared__ long long at[kTile];
  const long long s0 = (long long)blockIdx.x * kTile;
  const int m = (int)min((long long)kTile, n - s0);
  if ((int)threadIdx.x < m) {
    const long long s = s0 + threadIdx.x;
#pragma unroll
    for (int c = 0; c < R::kReals; ++c) {
      tile[threadIdx.x][c] = __ldcs(soa + c * total + s);
    }
    tile[threadIdx.x][R::kReals] = pack_ints(ids[s], 0);
    at[threadIdx.x] = perm[s] * R::kWords;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < m * R::kWords; i += kTile) {
    const int r = i / R::kWords, w = i % R::kWords;
    aos[at[r] + w] = tile[r][w];
  }
}

// the store's slots of one box -> component arrays in the caller's order, a
// component per blockIdx.y: the CTAs in flight then write one or two
// components of the box, which stay in L2 until their sectors are full (with
// every component in flight, k_unsort's 8-byte stores left L2 as partial
// sectors: 2929 us of GPU time for 8M droplets of 17 words)
__global__ void __launch_bounds__(256) k_store_to_columns(const double* soa, long long total, const int* ids,
                                                          const long long* perm, long long n, int nreal, const Columns C)
{
  const long long s = blockIdx.x * 256LL + threadIdx.x;
  if (s >= n) {
    return;
  }
  const int c = blockIdx.y;
  if (c < nreal) {
    if (C.c[c]) {
      C.c[c][perm[s]] = __ldcs(soa + c * total + s);
    }
  } else if (C.id) {
    C.id[perm[s]] = ids[s];
  }
}

// staging rows of one box (not packed yet) -> the caller's order
__global__ void __launch_bounds__(256) k_rows_out(const double* rows, int stride, int nreal, long long n, const Columns C,
                                                  double* aos)
{
  const long long s = blockIdx.x * 256LL + threadIdx.x;
  if (s >= n) {
    return;
  }
  const double* q = rows + s * stride;
  const int id = __double2loint(q[nreal]);
  const long long j = (long long)__double2hiint(q[nreal]);
  if (aos) {
    double* o = aos + j * (nreal + 1);
    for (int c = 0; c < nreal; ++c) {
      o[c] = q[c];
    }
    o[nreal] = pack_ints(id, 0);
    return;
  }
  for (int c = 0; c < nreal; ++c) {
    if (C.c[c]) {
      C.c[c][j] = q[c];
    }
  }
  if (C.id) {
    C.id[j] = id;
  }
}

// (box, first slot) of each CTA of the update's map: kBlock slots of one box
__global__ void __launch_bounds__(256) k_cta_map(const long long* box_begin, const int* first, int nb, int ncta,
                                                 int* cta_box, long long* cta_start)
{
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= ncta) {
    return;
  }
  int lo = 0, hi = nb;  // the box b with first[b] <= i < first[b + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (first[mid] <= i) {
      lo = mid;
    } else {
      hi = mid;
    }
  }
  cta_box[i] = lo;
  cta_start[i] = box_begin[lo] + (long long)(i - first[lo]) * kBlock;
}

#define PMP_BY_FUELS(h, CALL) \
  switch ((h)->nfuel) {       \
    case 1: {                 \
      constexpr int F = 1;    \
      CALL;                   \
    } break;                  \
    case 2: {                 \
      constexpr int F = 2;    \
      CALL;                   \
    } break;                  \
    case 3: {                 \
      constexpr int F = 3;    \
      CALL;                   \
    } break;                  \
    default: {                \
      constexpr int F = 4;    \
      CALL;                   \
    } break;                  \
  }

unsigned nblk(long long n, int b) { return (unsigned)((n + b - 1) / b); }

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

size_t row_bytes(const pmp_spray* h) { return sizeof(double) * row_stride(h->nfuel); }

double* staged_row(const pmp_spray* h, long long r)
{
  return reinterpret_cast<double*>(static_cast<char*>(h->spare.p) + (size_t)r * row_bytes(h));
}

// sort-key extent of a box: its cells and kSortPad around them
void sort_extent(const pmp_box& bx, int* ext)
{
  for (int d = 0; d < 3; ++d) {
    ext[d] = bx.hi[d] - bx.lo[d] + 1 + 2 * kSortPad;
  }
}

KeyOf key_of(const pmp_spray* h, int box, bool kept)
{
  KeyOf k;
  memset(&k, 0, sizeof(k));
  const pmp_box& bx = h->boxes[box];
  sort_extent(bx, k.ext);
  for (int d = 0; d < 3; ++d) {
    k.plo[d] = h->geom.plo[d];
    k.dxi[d] = 1. / h->geom.dx[d];
    k.lo[d] = bx.lo[d];
  }
  k.base = (unsigned long long)box << h->sort_shift;
  k.kept = kept ? 1 : 0;
  return k;
}

// 32-bit keys: every box's fit below 2^31, the key of rows given up lies above
bool narrow_keys(const pmp_spray* h) { return h->sort_bits <= 31; }

// the narrow keys and indices of the staging rows, from row `row` on
KeyOut key_out(const pmp_spray* h, long long row)
{
  const long long cap = (long long)(h->row_keys.bytes / (2 * sizeof(unsigned)));
  unsigned* keys = static_cast<unsigned*>(h->row_keys.p);
  return {keys + row, reinterpret_cast<int*>(keys + cap) + row, row, nullptr, nullptr};
}

long long sort_cells(const pmp_spray* h) { return padded_cells((long long)h->boxes.size(), h->sort_shift); }

// Whether the rows of a hand-over are counted into their cells while they are
// staged: decided at its first box, of n droplets, as if there were as many in
// all as in the last hand-over; cell_sorted() looks at the whole.  In a handle's
// first one the other boxes count as full as this one, which says little: the
// counts are then at most kGuessedCells (64 MB).  512 boxes of 64^3 cells with
// 300k droplets in the first and 50 in each of the others: without these bounds
// 1 GB of counts, cleared and left for the radix sort in every pass.
constexpr long long kGuessedCells = 1LL << 24;
bool count_first(const pmp_spray* h, long long n)
{
  const long long cells = sort_cells(h);
  const bool known = h->last_total >= 0;
  const long long total = known ? std::max(n, h->last_total) : n * (long long)h->boxes.size();
  return narrow_keys(h) && counting_pays(cells, total, h->grid_cells, kDenseStaged) && (known || cells <= kGuessedCells);
}
bool cell_sorted(const pmp_spray* h, long long m)
{
  return h->counted && *h->crowded() == 0 && counting_pays(sort_cells(h), m, h->grid_cells, kDenseStaged);
}

// Room for n more staging rows in the spare buffer (and their keys); the live
// boxes' rows move to its front when it is exchanged for a larger one.
int stage_room(pmp_spray* h, long long n)
{
  const size_t rb = row_bytes(h);
  const size_t kb = 2 * sizeof(unsigned);
  if ((size_t)(h->staged_rows + n) * rb <= h->spare.bytes && (size_t)(h->staged_rows + n) * kb <= h->row_keys.bytes) {
    return PMP_OK;
  }
  long long live = 0;
  bool whole = true;  // every box is handed over: no rows were unpacked or given up
  for (const StagedBox& s : h->staged) {
    live += s.n;
    whole = whole && !s.kept;
  }
  whole = whole && live == h->staged_rows;
  // the first boxes of a hand-over say little about the rest of it: doubling,
  // so that many boxes exchange the buffer a few times only, up to what the last
  // hand-over came to, or to what the boxes so far let expect and a quarter more
  // than they need (boxes handed over again also need the rows that they give
  // up: 64 boxes one by one, without the doubling, exchange the buffer 64 times)
  size_t rows = (size_t)(live > 0 ? 2 * (live + n) : n);
  if (whole && live > 0) {
    const long long nb = (long long)h->boxes.size();
    const long long so_far = 1 + std::count(h->box_set.begin(), h->box_set.end(), true);
    const long long all = h->last_total >= live + n ? h->last_total
                          : so_far >= nb            ? live + n
                                                    : std::max((live + n) * 5 / 4, (live + n) / so_far * nb + nb);
    rows = std::min(rows, (size_t)all);
  }
  if (live == 0 && h->last_total < 0) {
    // a handle's first: as if every box held as many, within 64 MB
    rows = std::max(rows, std::min(rows * h->boxes.size(), ((size_t)64 << 20) / rb));
  }
  KeptBuffer nw, nk;
  if (store_alloc(h, &nw.p, rows * rb) != cudaSuccess) {
    cudaGetLastError();
    rows = (size_t)(live + n);
    PMP_TRY(h, store_alloc(h, &nw.p, rows * rb));
  }
  nw.bytes = rows * rb;
  nk.bytes = rows * kb;
  cudaError_t e = store_alloc(h, &nk.p, nk.bytes);
  const KeptBuffer old_rows = h->spare, old_keys = h->row_keys;
  const KeyOut from = key_out(h, 0);
  h->row_keys = nk;
  const KeyOut to = key_out(h, 0);
  long long at = 0;
  for (const StagedBox& s : h->staged) {
    if (s.n > 0 && e == cudaSuccess) {
      e = cudaMemcpy(static_cast<char*>(nw.p) + (size_t)at * rb, staged_row(h, s.row), (size_t)s.n * rb,
                     cudaMemcpyDeviceToDevice);
      if (e == cudaSuccess) {
        e = cudaMemcpy(to.keys + at, from.keys + s.row, sizeof(unsigned) * s.n, cudaMemcpyDeviceToDevice);
      }
      if (e == cudaSuccess && h->ranked) {
        e = cudaMemcpy(to.idx + at, from.idx + s.row, sizeof(int) * s.n, cudaMemcpyDeviceToDevice);
      }
      at += s.n;
    }
  }
  if (e == cudaSuccess && at > 0 && !h->ranked) {
    k_fill_keys<<<nblk(at, 256), 256>>>(nullptr, to.idx, 0, at, 0);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    h->row_keys = old_keys;
    cudaFree(nw.p);
    cudaFree(nk.p);
    return check(h, e, "staging rows");
  }
  at = 0;
  for (StagedBox& s : h->staged) {
    if (s.n > 0) {
      s.row = at;
      at += s.n;
    }
  }
  h->staged_rows = at;
  h->spare = nw;
  cudaFree(old_rows.p);  // waits for the copies
  cudaFree(old_keys.p);
  return PMP_OK;
}

// The packed droplets back into staging rows, in the store's order (which a
// later pack keeps), except box `skip`, whose droplets are being replaced.
int unpack(pmp_spray* h, int skip)
{
  const int nb = (int)h->boxes.size();
  const int nc = h->ncomp();
  const long long T = h->total;
  h->staged_rows = 0;
  h->counted = h->ranked = false;
  for (int b = 0; b < nb; ++b) {
    h->staged[b] = StagedBox{};
  }
  long long n = T - (h->box_begin[skip + 1] - h->box_begin[skip]);
  int rc = stage_room(h, n);
  if (rc != PMP_OK) {
    return rc;
  }
  for (int b = 0; b < nb; ++b) {
    const long long o = h->box_begin[b], m = h->box_begin[b + 1] - o;
    if (b == skip || m == 0) {
      continue;
    }
    StagedBox& s = h->staged[b];
    s.n = m;
    s.row = h->staged_rows;
    s.kept = true;
    h->staged_rows += m;
    const KeyOf key = key_of(h, b, true);
    const KeyOut out = narrow_keys(h) ? key_out(h, s.row) : KeyOut{};
    Columns C;
    memset(&C, 0, sizeof(C));
    for (int c = 0; c < nc; ++c) {
      C.c[c] = h->soa + (long long)c * T + o;
    }
    C.id = h->ids + o;
    PMP_BY_FUELS(h, (k_columns_to_rows<F><<<nblk(m, kTile), kTile>>>(C, h->perm() + o, m, staged_row(h, s.row), key,
                                                                   out)));
  }
  PMP_TRY(h, cudaGetLastError());
  store_reset(h);
  return PMP_OK;
}

// Ranges of device allocations of the handle's GPU that a call has seen: a
// caller's array inside one, and suitably aligned, is read or written by the
// kernels directly.  Everything else (host, managed or another GPU's memory,
// a range that leaves its allocation) goes through cudaMemcpy, which accepts
// or refuses it.
class DeviceRanges {
 public:
  explicit DeviceRanges(int device) : device_(device) {}
  bool holds(const void* p, size_t bytes, size_t align)
  {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    if (!p || a % align != 0) {
      return false;
    }
    if (a >= lo_ && a + bytes <= hi_) {
      return true;
    }
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    if (at.type != cudaMemoryTypeDevice || at.device != device_) {
      return false;
    }
    CUdeviceptr base = 0;
    size_t size = 0;
    if (!range_of() || range_of()(&base, &size, (CUdeviceptr)a) != CUDA_SUCCESS) {
      return false;
    }
    lo_ = (uintptr_t)base;
    hi_ = lo_ + size;
    return a + bytes <= hi_;
  }

 private:
  using RangeFn = CUresult (*)(CUdeviceptr*, size_t*, CUdeviceptr);
  static RangeFn range_of()
  {
    static const RangeFn fn = [] {
      void* p = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &p, cudaEnableDefault, &q) != cudaSuccess ||
          q != cudaDriverEntryPointSuccess) {
        cudaGetLastError();
        p = nullptr;
      }
      return reinterpret_cast<RangeFn>(p);
    }();
    return fn;
  }
  int device_;
  uintptr_t lo_ = 1, hi_ = 0;
};

// A device buffer for droplets on their way from or to memory the kernels do
// not touch directly; given back when it grew large.
struct Transit {
  pmp_spray* h;
  explicit Transit(pmp_spray* handle) : h(handle) {}
  ~Transit()
  {
    if (h->transit.bytes > ((size_t)64 << 20)) {
      cudaFree(h->transit.p);
      h->transit = KeptBuffer{};
    }
  }
};

// Kernels that a hand-over has launched on the legacy stream and not waited
// for.  Whatever way the call returns, they have run by then: the next
// operation packs on its own stream, which may be one that the legacy stream
// does not order.
struct InFlight {
  bool launched = false;
  cudaError_t wait()
  {
    const cudaError_t e = launched ? cudaStreamSynchronize(nullptr) : cudaSuccess;
    launched = false;
    return e;
  }
  ~InFlight() { wait(); }
};

// columns of nreal components of n doubles, then n ids, in one buffer
Columns columns_in(void* base, int nreal, long long n)
{
  Columns C;
  memset(&C, 0, sizeof(C));
  double* d = static_cast<double*>(base);
  for (int c = 0; c < nreal; ++c) {
    C.c[c] = d + (long long)c * n;
  }
  C.id = reinterpret_cast<int*>(d + (long long)nreal * n);
  return C;
}

// the sort of m keyed rows: the sorted row indices at *order
template <typename K, typename V>
int sort_rows(pmp_spray* h, const K* keys, const V* idx, long long m, int end_bit, size_t used, cudaStream_t st,
              const V** order)
{
  using N = V;  // the count type decides CUB's offsets
  const size_t kb = align256(sizeof(K) * m), vb = align256(sizeof(V) * m);
  char* base = static_cast<char*>(h->sort_scratch.p) + used;
  size_t tbytes = h->sort_scratch.bytes - used - kb - vb;
  PMP_TRY(h, (cub::DeviceRadixSort::SortPairs(base + kb + vb, tbytes, keys, reinterpret_cast<K*>(base), idx,
                                              reinterpret_cast<V*>(base + kb), (N)m, 0, end_bit, st)));
  *order = reinterpret_cast<V*>(base + kb);
  return PMP_OK;
}

template <typename K, typename V>
size_t sort_bytes(long long m, int end_bit)
{
  size_t tbytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, tbytes, (const K*)nullptr, (K*)nullptr, (const V*)nullptr, (V*)nullptr, (V)m, 0,
                                  end_bit, nullptr);
  return align256(sizeof(K) * m) + align256(sizeof(V) * m) + align256(std::max(tbytes, (size_t)1));
}

}  // namespace

// Every allocation of the store; the fail_alloc-th from now fails as cudaMalloc
// does without memory.
cudaError_t store_alloc(pmp_spray* h, void** p, size_t bytes)
{
  if (h->fail_alloc > 0 && --h->fail_alloc == 0) {
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  h->allocs += 1;
  return cudaMalloc(p, bytes);
}

// a buffer of which `bytes` are used is large and mostly unused
static bool idle(const KeptBuffer& b, size_t bytes) { return b.bytes > ((size_t)256 << 20) && b.bytes / 4 > bytes; }

// A kept buffer of at least `bytes`: exchanged when too small, and when it is
// idle (its content is not kept).
cudaError_t try_keep(pmp_spray* h, KeptBuffer& b, size_t bytes)
{
  if (b.p && b.bytes >= bytes && !idle(b, bytes)) {
    return cudaSuccess;
  }
  cudaFree(b.p);
  b = KeptBuffer{};
  const size_t want = std::max(bytes, (size_t)256);
  const cudaError_t e = store_alloc(h, &b.p, want);
  if (e != cudaSuccess) {
    cudaGetLastError();  // reported here, not by the next call
    return e;
  }
  b.bytes = want;
  return cudaSuccess;
}
int keep(pmp_spray* h, KeptBuffer& b, size_t bytes)
{
  PMP_TRY(h, try_keep(h, b, bytes));
  return PMP_OK;
}

size_t store_bytes(const pmp_spray* h, long long n) { return (size_t)n * (sizeof(double) * h->ncomp() + sizeof(int)); }

void store_attach(pmp_spray* h, long long n)
{
  h->total = n;
  h->soa = static_cast<double*>(h->store.p);
  h->ids = reinterpret_cast<int*>(h->soa + (long long)h->ncomp() * n);
}

// Zeroed counts of `cells` cells, for a sort on st, which leaves them zero
// again: `zero_cells` says how many are (0 while they are in use).  *have:
// false when there is no memory for them (the radix sort needs none).
int count_cells(pmp_spray* h, long long cells, cudaStream_t st, bool* have)
{
  const KeptBuffer before = h->counts;
  *have = try_keep(h, h->counts, sizeof(unsigned) * (size_t)cells) == cudaSuccess;
  if (!*have) {
    h->zero_cells = 0;
    return PMP_OK;
  }
  // another buffer may lie at the old one's address: its size differs
  if (h->counts.p != before.p || h->counts.bytes != before.bytes || h->zero_cells < cells) {
    h->zero_cells = 0;
    PMP_TRY(h, cudaMemsetAsync(h->counts.p, 0, sizeof(unsigned) * (size_t)cells, st));
  }
  h->zero_cells = 0;
  *h->crowded() = 0;
  return PMP_OK;
}

// Sort-key layout of new grids: bits of a cell's place in its box, and of the
// box above them.
void store_layout(pmp_spray* h)
{
  int sh = 0;
  h->grid_cells = 0;
  for (const pmp_box& bx : h->boxes) {
    int ext[3];
    sort_extent(bx, ext);
    h->grid_cells += (long long)(bx.hi[0] - bx.lo[0] + 1) * (bx.hi[1] - bx.lo[1] + 1) * (bx.hi[2] - bx.lo[2] + 1);
    const unsigned long long cells = brick_key_count(ext[0], ext[1], ext[2]);
    while (sh < 40 && (1ULL << sh) < cells) {
      ++sh;
    }
  }
  h->sort_shift = sh;
  h->sort_bits = std::max(sh, 1);
  while (h->sort_bits < 63 && (1ULL << (h->sort_bits - sh)) < h->boxes.size()) {
    ++h->sort_bits;
  }
}

void store_reset(pmp_spray* h)
{
  h->soa = nullptr;
  h->ids = nullptr;
  h->packed = false;
  h->ncta = 0;
  batch_reset(h);
}

void store_free(pmp_spray* h)
{
  store_reset(h);
  for (KeptBuffer* b : {&h->store, &h->spare, &h->row_keys, &h->perm_b, &h->fb_b, &h->map_b, &h->sort_scratch,
                        &h->transit, &h->counts}) {
    cudaFree(b->p);
    *b = KeptBuffer{};
  }
  h->zero_cells = 0;
}

// Box offsets and the CTA -> (box, first slot) map of the packed droplets,
// and the fallback list, enqueued on st.  When it fails, the map counts as not
// built (ncta < 0), and the next ensure_packed builds it.
int build_cta_map(pmp_spray* h, cudaStream_t st)
{
  const int nb = (int)h->boxes.size();
  std::vector<int> first(nb + 1, 0);
  for (int b = 0; b < nb; ++b) {
    const long long n = h->box_begin[b + 1] - h->box_begin[b];
    first[b + 1] = first[b] + (int)((n + kBlock - 1) / kBlock);
  }
  const int ncta = first[nb];
  h->ncta = -1;
  // {box_begin[nb + 1], first[nb + 1]} uploaded, then cta_start, cta_box
  const size_t bb = sizeof(long long) * (nb + 1), fb = align256(sizeof(int) * (nb + 1));
  const size_t cs = align256(bb + fb), cb = align256(sizeof(long long) * ncta);
  int rc = keep(h, h->map_b, cs + cb + sizeof(int) * (size_t)ncta);
  if (rc == PMP_OK) {
    rc = keep(h, h->fb_b, sizeof(long long) * (size_t)std::max(h->total, 1LL));
  }
  if (rc != PMP_OK) {
    return rc;
  }
  char* base = static_cast<char*>(h->map_b.p);
  std::vector<char> up(bb + fb);
  memcpy(up.data(), h->box_begin.data(), bb);
  memcpy(up.data() + bb, first.data(), sizeof(int) * (nb + 1));
  PMP_TRY(h, cudaMemcpyAsync(base, up.data(), bb + sizeof(int) * (nb + 1), cudaMemcpyHostToDevice, st));
  h->d_box_begin = reinterpret_cast<long long*>(base);
  h->d_cta_start = reinterpret_cast<long long*>(base + cs);
  h->d_cta_box = reinterpret_cast<int*>(base + cs + cb);
  if (ncta > 0) {
    k_cta_map<<<nblk(ncta, 256), 256, 0, st>>>(h->d_box_begin, reinterpret_cast<const int*>(base + bb), nb, ncta,
                                               h->d_cta_box, h->d_cta_start);
    PMP_TRY(h, cudaGetLastError());
  }
  h->ncta = ncta;
  h->packed = true;
  return PMP_OK;
}

namespace {

// The staged boxes packed into the store, enqueued on st.  No work of the
// handle is pending (whoever staged droplets waited for it).
int pack(pmp_spray* h, cudaStream_t st)
{
  const int nb = (int)h->boxes.size();
  h->box_begin.assign(nb + 1, 0);
  for (int b = 0; b < nb; ++b) {
    h->box_begin[b + 1] = h->box_begin[b] + h->staged[b].n;
  }
  const long long n = h->box_begin[nb];
  int rc = keep(h, h->store, store_bytes(h, std::max(n, 1LL)));
  if (rc == PMP_OK) {
    rc = keep(h, h->perm_b, sizeof(long long) * (size_t)std::max(n, 1LL));
  }
  if (rc != PMP_OK) {
    return rc;
  }
  store_attach(h, n);
  if (n > 0) {
    const int end_bit = h->sort_bits;
    if (narrow_keys(h) && h->staged_rows < (1LL << 31)) {
      // rows given up carry the key of no box, above every other
      const long long m = h->staged_rows;
      const int bits = m == n ? end_bit : 32;
      const long long cells = sort_cells(h);
      if (h->counted && *h->crowded() != 0) {
        found_crowded(h);
      }
      const bool by_cell = m == n && cell_sorted(h, m) &&
                           try_keep(h, h->sort_scratch, cell_sort_layout(cells, m).total) == cudaSuccess;
      rc = by_cell ? PMP_OK : keep(h, h->sort_scratch, sort_bytes<unsigned, int>(m, bits));
      const KeyOut k = key_out(h, 0);
      const int* order = nullptr;
      if (rc == PMP_OK && by_cell) {
        char* buf = static_cast<char*>(h->sort_scratch.p);
        h->counted = false;
        cell_sort(static_cast<unsigned*>(h->counts.p), cells, k.keys, k.idx, m, buf, st);
        h->cell_sorts += 1;
        PMP_TRY(h, cudaGetLastError());
        h->zero_cells = cells;
        order = reinterpret_cast<const int*>(buf + cell_sort_layout(cells, m).order);
      } else if (rc == PMP_OK) {
        if (h->ranked) {  // counted, and not sorted by it
          k_fill_keys<<<nblk(m, 256), 256, 0, st>>>(nullptr, k.idx, 0, m, 0);
          h->counted = h->ranked = false;
        }
        rc = sort_rows<unsigned, int>(h, k.keys, k.idx, m, bits, 0, st, &order);
      }
      if (rc == PMP_OK) {
        PMP_BY_FUELS(h, (k_rows_to_store<F, int><<<nblk(n, kTile), kTile, 0, st>>>(staged_row(h, 0), order, n, h->soa,
                                                                                  h->ids, h->perm())));
      }
    } else {
      std::vector<Region> reg(nb);
      for (int b = 0; b < nb; ++b) {
        reg[b] = Region{h->staged[b].row, h->box_begin[b], key_of(h, b, h->staged[b].kept)};
      }
      const size_t kb = align256(sizeof(unsigned long long) * n), used = 2 * kb + align256(sizeof(Region) * nb);
      rc = keep(h, h->sort_scratch, used + sort_bytes<unsigned long long, long long>(n, end_bit));
      const long long* order = nullptr;
      if (rc == PMP_OK) {
        char* base = static_cast<char*>(h->sort_scratch.p);
        unsigned long long* keys = reinterpret_cast<unsigned long long*>(base);
        long long* idx = reinterpret_cast<long long*>(base + kb);
        Region* d_reg = reinterpret_cast<Region*>(base + 2 * kb);
        PMP_TRY(h, cudaMemcpyAsync(d_reg, reg.data(), sizeof(Region) * nb, cudaMemcpyHostToDevice, st));
        k_row_keys<<<nblk(n, 256), 256, 0, st>>>(staged_row(h, 0), row_stride(h->nfuel), d_reg, nb, n, keys, idx);
        rc = sort_rows<unsigned long long, long long>(h, keys, idx, n, end_bit, used, st, &order);
      }
      if (rc == PMP_OK) {
        PMP_BY_FUELS(h, (k_rows_to_store<F, long long><<<nblk(n, kTile), kTile, 0, st>>>(staged_row(h, 0), order, n,
                                                                                        h->soa, h->ids, h->perm())));
      }
    }
    if (rc != PMP_OK) {
      return rc;
    }
    PMP_TRY(h, cudaGetLastError());
  }
  rc = build_cta_map(h, st);
  if (rc != PMP_OK) {
    return rc;
  }
  for (StagedBox& s : h->staged) {
    s = StagedBox{};
  }
  h->staged_rows = 0;
  h->counted = h->ranked = false;
  h->last_total = n;
  return PMP_OK;
}

// What n packed droplets leave idle of the buffers that a hand-over fills,
// which grow with it and go through keep() only in a re-binning, or not at all:
// given back.  The packing on st still reads them.
void give_back(pmp_spray* h, long long n, cudaStream_t st)
{
  const size_t m = (size_t)n;
  const bool rows = idle(h->spare, m * row_bytes(h)), counts = idle(h->counts, m * 2 * sizeof(unsigned));
  if (!rows && !counts) {
    return;
  }
  cudaStreamSynchronize(st);
  if (rows) {
    cudaFree(h->spare.p);
    cudaFree(h->row_keys.p);
    h->spare = h->row_keys = KeptBuffer{};
  }
  if (counts) {
    cudaFree(h->counts.p);
    h->counts = KeptBuffer{};
    h->zero_cells = 0;
  }
}

}  // namespace

// The droplets packed, and their map built, in the order of st.
int ensure_packed(pmp_spray* h, cudaStream_t st)
{
  for (int b = 0; !h->packed && b < (int)h->boxes.size(); ++b) {
    if (!h->box_set[b]) {
      return set_err(h, PMP_ERR_INVALID, "set_particles was not called for every box", b);
    }
  }
  const bool built = h->packed && h->ncta >= 0;
  if (built && !(h->packing && st != h->pack_stream)) {
    return PMP_OK;
  }
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  PMP_TRY(h, cudaStreamIsCapturing(st, &cap));
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  if (built) {
    // packed by a call on another stream, which may have been refused after that
    if (capturing) {
      // a capture takes no event from outside, and a wait for one is allowed
      // beside it in the relaxed mode alone
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      PMP_TRY(h, cudaThreadExchangeStreamCaptureMode(&mode));
      const cudaError_t e = cudaEventSynchronize(h->ev_pack);
      cudaThreadExchangeStreamCaptureMode(&mode);
      PMP_TRY(h, e);
      h->packing = false;
      return PMP_OK;
    }
    PMP_TRY(h, cudaStreamWaitEvent(st, h->ev_pack, 0));
    return PMP_OK;
  }
  if (capturing) {
    // packing is not part of the caller's graph: it runs at once, beside the
    // capture, where the capture's mode lets a call allocate
    void* p = nullptr;
    PMP_TRY(h, cudaMalloc(&p, 256));
    cudaFree(p);
    st = nullptr;
  }
  const bool packing = !h->packed;
  const int rc = packing ? pack(h, st) : build_cta_map(h, st);
  if (rc == PMP_OK && packing) {
    give_back(h, h->total, st);
  }
  if (rc != PMP_OK) {
    // no kernel of it may still read rows that the caller replaces next
    cudaStreamSynchronize(st);
    cudaGetLastError();
    return rc;
  }
  if (capturing) {
    PMP_TRY(h, cudaStreamSynchronize(st));
    return PMP_OK;
  }
  // entry points on other streams wait for the store
  PMP_TRY(h, cudaEventRecord(h->ev_pack, st));
  h->pack_stream = st;
  h->packing = true;
  return PMP_OK;
}

}  // namespace pmp

using namespace pmp;

extern "C" {

int pmp_spray_set_particles(pmp_spray* h, int box, const pmp_particles* p)
{
  if (!h || !p || box < 0 || box >= (int)h->boxes.size() || p->n < 0) {
    return PMP_ERR_INVALID;
  }
  if (!h->have_geom) {
    return set_err(h, PMP_ERR_INVALID, "set_geometry must precede set_particles");
  }
  cudaSetDevice(h->device);
  pmp::quiesce(h);
  int rc = PMP_OK;
  InFlight flight;
  if (h->packed) {
    flight.launched = true;
    rc = unpack(h, box);
    if (rc != PMP_OK) {
      return rc;
    }
  }
  const long long n = p->n;
  StagedBox& s = h->staged[box];
  if (s.n > 0) {
    h->counted = false;  // with the rows that are given up
  }
  if (s.n > 0 && s.row + s.n == h->staged_rows) {
    h->staged_rows = s.row;  // its rows are the last ones
  } else if (s.n > 0 && narrow_keys(h)) {
    // given up: the key above every box's
    const KeyOut k = key_out(h, 0);
    flight.launched = true;
    k_fill_keys<<<nblk(s.n, 256), 256>>>(k.keys, k.idx, s.row, s.n, 0xffffffffu);
    PMP_TRY(h, cudaGetLastError());
  }
  s = StagedBox{};
  h->box_set[box] = false;  // until its droplets are in
  int ext[3];
  sort_extent(h->boxes[box], ext);
  if (n > 0 && brick_key_count(ext[0], ext[1], ext[2]) >= (1ULL << 32)) {
    return set_err(h, PMP_ERR_INVALID, "box too large for the droplet sort key", box);
  }
  if (n >= (1LL << 31)) {
    return set_err(h, PMP_ERR_INVALID, "2^31 droplets or more in one box", box);
  }
  if (n == 0) {
    PMP_TRY(h, flight.wait());
    h->box_set[box] = true;
    return PMP_OK;
  }
  if (p->layout != PMP_LAYOUT_SOA && p->layout != PMP_LAYOUT_AOS) {
    return set_err(h, PMP_ERR_INVALID, "unknown particle layout");
  }
  flight.launched = true;
  rc = stage_room(h, n);
  if (rc != PMP_OK) {
    return rc;
  }
  const int nc = h->ncomp();
  const int nr = h->nr();
  double* rows = staged_row(h, h->staged_rows);
  const KeyOf key = key_of(h, box, false);
  KeyOut out = narrow_keys(h) ? key_out(h, h->staged_rows) : KeyOut{};
  if (h->staged_rows == 0) {
    h->ranked = false;
    h->counted = count_first(h, n) && try_counting(h);
    if (h->counted) {
      rc = count_cells(h, sort_cells(h), nullptr, &h->counted);
      if (rc != PMP_OK) {
        h->counted = false;
        return rc;
      }
    }
  }
  const bool counting = h->counted;
  h->counted = false;  // until the box is in
  if (counting) {
    out.counts = static_cast<unsigned*>(h->counts.p);
    out.crowded = h->crowded();
    h->ranked = true;
  }
  const cudaMemcpyKind kind = p->where == PMP_WHERE_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  DeviceRanges ranges(h->device);
  Transit transit(h);
  if (p->layout == PMP_LAYOUT_SOA) {
    Columns C;
    memset(&C, 0, sizeof(C));
    for (int d = 0; d < 3; ++d) {
      if (!p->pos[d]) {
        return set_err(h, PMP_ERR_INVALID, "missing position array");
      }
      C.c[d] = const_cast<double*>(p->pos[d]);
    }
    for (int r = 0; r < nr; ++r) {
      C.c[3 + r] = const_cast<double*>(p->rdata[r]);
    }
    if (!p->id) {
      return set_err(h, PMP_ERR_INVALID, "missing id array");
    }
    C.id = const_cast<int*>(p->id);
    bool direct = p->where == PMP_WHERE_DEVICE && ranges.holds(C.id, sizeof(int) * n, sizeof(int));
    for (int c = 0; c < nc && direct; ++c) {
      direct = !C.c[c] || ranges.holds(C.c[c], sizeof(double) * n, sizeof(double));
    }
    if (!direct) {
      rc = keep(h, h->transit, store_bytes(h, n));
      if (rc != PMP_OK) {
        return rc;
      }
      Columns D = columns_in(h->transit.p, nc, n);
      for (int c = 0; c < nc; ++c) {
        if (C.c[c]) {
          PMP_TRY(h, cudaMemcpy(D.c[c], C.c[c], sizeof(double) * n, kind));
        } else {
          D.c[c] = nullptr;
        }
      }
      PMP_TRY(h, cudaMemcpy(D.id, C.id, sizeof(int) * n, kind));
      C = D;
    }
    PMP_BY_FUELS(h, (k_columns_to_rows<F><<<nblk(n, kTile), kTile>>>(C, nullptr, n, rows, key, out)));
  } else {
    const size_t bytes = sizeof(double) * (nc + 1) * (size_t)n;
    const double* src = static_cast<const double*>(p->aos);
    if (p->where != PMP_WHERE_DEVICE || !ranges.holds(p->aos, bytes, sizeof(double))) {
      rc = keep(h, h->transit, bytes);
      if (rc != PMP_OK) {
        return rc;
      }
      PMP_TRY(h, cudaMemcpy(h->transit.p, p->aos, bytes, kind));
      src = static_cast<const double*>(h->transit.p);
    }
    PMP_BY_FUELS(h, (k_aos_to_rows<F><<<nblk(n, kTile), kTile>>>(src, n, rows, key, out)));
  }
  PMP_TRY(h, cudaGetLastError());
  // the caller's arrays are read when the call returns
  PMP_TRY(h, flight.wait());
  s.n = n;
  s.row = h->staged_rows;
  h->staged_rows += n;
  h->counted = counting;
  h->box_set[box] = true;
  return PMP_OK;
}

int pmp_spray_num_particles(const pmp_spray* h, int box, long long* n)
{
  if (!h || !n || box < 0 || box >= (int)h->boxes.size()) {
    return PMP_ERR_INVALID;
  }
  *n = h->packed ? h->box_begin[box + 1] - h->box_begin[box] : h->staged[box].n;
  return PMP_OK;
}

int pmp_spray_get_particles(pmp_spray* h, int box, pmp_particles* out)
{
  if (!h || !out || box < 0 || box >= (int)h->boxes.size()) {
    return PMP_ERR_INVALID;
  }
  cudaSetDevice(h->device);
  pmp::quiesce(h);
  long long n = 0;
  pmp_spray_num_particles(h, box, &n);
  if (out->n != n) {
    return set_err(h, PMP_ERR_INVALID, "output count differs from the box's droplet count", box);
  }
  if (n == 0) {
    return PMP_OK;
  }
  const int nc = h->ncomp();
  const int nr = h->nr();
  const bool soa = out->layout == PMP_LAYOUT_SOA;
  const size_t rec_bytes = sizeof(double) * (nc + 1) * (size_t)n;
  const cudaMemcpyKind kind = out->where == PMP_WHERE_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  DeviceRanges ranges(h->device);
  Transit transit(h);
  Columns user;
  memset(&user, 0, sizeof(user));
  bool direct = out->where == PMP_WHERE_DEVICE;
  if (soa) {
    for (int d = 0; d < 3; ++d) {
      user.c[d] = out->pos[d];
    }
    for (int r = 0; r < nr; ++r) {
      user.c[3 + r] = out->rdata[r];
    }
    user.id = out->id;
    direct = direct && (!user.id || ranges.holds(user.id, sizeof(int) * n, sizeof(int)));
    for (int c = 0; c < nc && direct; ++c) {
      direct = !user.c[c] || ranges.holds(user.c[c], sizeof(double) * n, sizeof(double));
    }
  } else {
    direct = direct && ranges.holds(out->aos, rec_bytes, sizeof(double));
  }
  Columns C = user;
  double* aos = static_cast<double*>(out->aos);
  if (!direct) {
    const int rc = keep(h, h->transit, soa ? store_bytes(h, n) : rec_bytes);
    if (rc != PMP_OK) {
      return rc;
    }
    aos = static_cast<double*>(h->transit.p);
    C = columns_in(h->transit.p, nc, n);
  }
  if (!h->packed) {
    k_rows_out<<<nblk(n, 256), 256>>>(staged_row(h, h->staged[box].row), row_stride(h->nfuel), nc, n, C,
                                      soa ? nullptr : aos);
  } else {
    const long long o = h->box_begin[box];
    const long long T = h->total;
    if (soa) {
      const dim3 grid(nblk(n, 256), (unsigned)(nc + 1));
      k_store_to_columns<<<grid, 256>>>(h->soa + o, T, h->ids + o, h->perm() + o, n, nc, C);
    } else {
      PMP_BY_FUELS(h, (k_store_to_aos<F><<<nblk(n, kTile), kTile>>>(h->soa + o, T, h->ids + o, h->perm() + o, n, aos)));
    }
  }
  PMP_TRY(h, cudaGetLastError());
  if (!direct) {
    if (soa) {
      for (int c = 0; c < nc; ++c) {
        if (user.c[c]) {
          PMP_TRY(h, cudaMemcpy(user.c[c], C.c[c], sizeof(double) * n, kind));
        }
      }
      if (user.id) {
        PMP_TRY(h, cudaMemcpy(user.id, C.id, sizeof(int) * n, kind));
      }
    } else {
      PMP_TRY(h, cudaMemcpy(out->aos, aos, rec_bytes, kind));
    }
  }
  // the droplets are there when the call returns
  PMP_TRY(h, cudaStreamSynchronize(nullptr));
  return PMP_OK;
}

int pmp_spray_debug_fail_alloc(pmp_spray* h, int k)
{
  if (!h || k < 0) {
    return PMP_ERR_INVALID;
  }
  h->fail_alloc = k;
  return PMP_OK;
}

int pmp_spray_debug_store(const pmp_spray* h, long long* allocs, long long* cell_sorts)
{
  if (!h || !allocs || !cell_sorts) {
    return PMP_ERR_INVALID;
  }
  *allocs = h->allocs;
  *cell_sorts = h->cell_sorts;
  return PMP_OK;
}

}  // extern "C"
