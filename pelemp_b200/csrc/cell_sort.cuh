// cell_sort.cuh -- stable sort of droplets by cell, by counting.
//
// The kernel that forms a droplet's key also counts it into its cell, and
// keeps the count it found there (its rank, in an order that depends on the
// run).  Four passes over the cells or the droplets then give the order a
// stable sort of the keys gives: sums of 4096 cells, each cell's first slot
// (which also leaves the counts zero for the next sort), the droplets to
// first slot + rank, and each cell's few droplets into their original order.
// A radix sort moves every key and index in two or three passes, of which each
// costs 10-14 us for any number up to a million.  From the staged keys to the
// order, radix sort and counting: 100k droplets of a 32^3 box 52 -> 21 us
// (8 operations, 4), 1M in 4 boxes 92 -> 36, 8M in 8 boxes 290 -> 130; the
// counting adds 0-2 us to the staging of 100k, 10 us (of 48, the atomics) to
// that of 1M records.  With the re-binning of 4M droplets: 232 -> 94 us from
// the keys' kernel to the box bounds.
//
// The last pass is quadratic in a cell's droplets, so a cell with more than
// kCrowd of them raises `crowded`, and the caller takes the radix sort: the
// counting was for nothing, so the next kCrowdSkip sorts of the handle do not
// try it.  1M droplets, 30 % of them in 50 cells of a 32^3 box: re-binning 178 us,
// 265 when each tries; hand-over and packing 243 and 265; 4M with the same in 25
// cells of each of 8 boxes, re-binning 436 and 551.  The radix sort remains the
// better one also for a few thousand droplets (one CTA sorts them in one launch)
// and for sparse meshes (the passes over the cells).
#pragma once

#include <cuda_runtime.h>

#include "pmp_handle.h"

namespace pmp {
namespace {

constexpr unsigned kCrowd = 64;        // droplets of a cell
constexpr int kCrowdSkip = 15;         // sorts without an attempt after a crowded one
constexpr int kSumCells = 4096;        // cells of a CTA of the first two passes
constexpr int kOrderCells = 256;       // of the last
constexpr int kOrderTile = 4096;       // droplets it holds in shared memory
constexpr long long kOneTile = 4096;   // droplets that the radix sort takes in one launch
constexpr long long kFewCells = 1LL << 22;   // cells (16 MB of counts)
constexpr long long kMostCells = 1LL << 27;  // (512 MB)
constexpr unsigned kNoCell = ~0u;      // key of a droplet that is not sorted

// Count a droplet (key kNoCell: none); all 32 lanes call.  A run of lanes of
// one cell counts with one atomic, so that a cell that holds most of a box
// costs few atomics of one address.  The rank is asked for later (rank_of),
// when other work has covered the atomic's way to L2.
struct Counted {
  unsigned head, base;  // lane of the run's first droplet; its count
};
__device__ __forceinline__ Counted count_cell(unsigned* counts, unsigned key)
{
  const unsigned lane = threadIdx.x & 31u;
  const unsigned prev = __shfl_up_sync(0xffffffffu, key, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || key != prev);
  Counted c;
  c.head = 31u - (unsigned)__clz((int)(heads & (0xffffffffu >> (31u - lane))));
  c.base = 0;
  if (c.head == lane && key != kNoCell) {
    const unsigned next = lane == 31u ? 0u : heads >> (lane + 1u);  // heads after this one
    c.base = atomicAdd(counts + key, next ? (unsigned)__ffs((int)next) : 32u - lane);
  }
  return c;
}
__device__ __forceinline__ int rank_of(const Counted& c, unsigned key, int* crowded)
{
  const unsigned rank = __shfl_sync(0xffffffffu, c.base, (int)c.head) + (threadIdx.x & 31u) - c.head;
  if (rank == kCrowd && key != kNoCell) {  // one droplet of a crowded cell has this rank
    *(volatile int*)crowded = 1;  // page-locked host memory: one write a cell
  }
  return (int)rank;
}

__device__ __forceinline__ unsigned warp_sum(unsigned v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v += __shfl_xor_sync(0xffffffffu, v, o);
  }
  return v;
}

// sum over the CTA's 256 threads, for all of them
__device__ __forceinline__ unsigned block_sum(unsigned v, unsigned* part)
{
  v = warp_sum(v);
  __syncthreads();
  if (threadIdx.x % 32 == 0) {
    part[threadIdx.x / 32] = v;
  }
  __syncthreads();
  unsigned t = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    t += part[i];
  }
  return t;
}

__global__ void __launch_bounds__(256) k_cell_sums(const uint4* counts, unsigned* sums)
{
  __shared__ unsigned part[8];
  const uint4* c = counts + (long long)blockIdx.x * (kSumCells / 4);
  unsigned v = 0;
#pragma unroll
  for (int i = 0; i < kSumCells / 1024; ++i) {
    const uint4 q = c[i * 256 + threadIdx.x];
    v += q.x + q.y + q.z + q.w;
  }
  v = block_sum(v, part);
  if (threadIdx.x == 0) {
    sums[blockIdx.x] = v;
  }
}

// starts[c]: droplets of the cells before c (one more entry: of all cells).
// Each CTA adds the sums before its own by itself, from L2: at most 32768
// (kMostCells; 2 GB of reads, in a re-binning of 5.3 ms).
__global__ void __launch_bounds__(256) k_cell_starts(uint4* counts, const unsigned* sums, unsigned* starts)
{
  __shared__ unsigned part[8], wsum[8];
  const int b = blockIdx.x;
  unsigned before = 0;
  for (int i = threadIdx.x; i < b; i += 256) {
    before += sums[i];
  }
  before = block_sum(before, part);
  uint4* c = counts + (long long)b * (kSumCells / 4);
  unsigned* s = starts + (long long)b * kSumCells;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4 q[kSumCells / 1024];
#pragma unroll
  for (int i = 0; i < kSumCells / 1024; ++i) {
    q[i] = c[i * 256 + threadIdx.x];
  }
#pragma unroll
  for (int i = 0; i < kSumCells / 1024; ++i) {
    const unsigned mine = q[i].x + q[i].y + q[i].z + q[i].w;
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
      incl += lane >= o ? u : 0u;
    }
    if (lane == 31) {
      wsum[warp] = incl;
    }
    __syncthreads();
    unsigned at = before + incl - mine, all = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      at += w < warp ? wsum[w] : 0u;
      all += wsum[w];
    }
    before += all;
    __syncthreads();
    uint4 r;
    r.x = at;
    r.y = r.x + q[i].x;
    r.z = r.y + q[i].y;
    r.w = r.z + q[i].z;
    reinterpret_cast<uint4*>(s)[i * 256 + threadIdx.x] = r;
    c[i * 256 + threadIdx.x] = make_uint4(0, 0, 0, 0);
  }
  if (b == (int)gridDim.x - 1 && threadIdx.x == 0) {
    s[kSumCells] = before;
  }
}

// droplets to their cell's slots, in the order of their ranks: four a thread,
// loads first
__global__ void __launch_bounds__(256) k_cell_scatter(const unsigned* keys, const int* ranks, long long n,
                                                      const unsigned* starts, int* slots)
{
  const long long s0 = blockIdx.x * 1024LL + threadIdx.x;
  unsigned key[4], at[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const long long s = s0 + i * 256;
    key[i] = s < n ? keys[s] : kNoCell;
    at[i] = s < n ? (unsigned)ranks[s] : 0u;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    at[i] += key[i] != kNoCell ? starts[key[i]] : 0u;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (key[i] != kNoCell) {
      slots[at[i]] = (int)(s0 + i * 256);
    }
  }
}

// each cell's droplets into ascending order, a droplet's place by counting
// the smaller ones: a thread per droplet, so that the lanes of a warp store
// into few sectors (8M droplets, 16 a cell: 78 us with a thread per cell)
__global__ void __launch_bounds__(kOrderCells) k_cell_order(const unsigned* starts, const int* slots, int* order)
{
  __shared__ int tile[kOrderTile];
  __shared__ unsigned char cell[kOrderTile];
  __shared__ unsigned begin[kOrderCells + 1];
  const unsigned* s = starts + (long long)blockIdx.x * kOrderCells;
  const unsigned first = s[0], m = s[kOrderCells] - first;
  if (m == 0) {
    return;
  }
  const unsigned a = s[threadIdx.x] - first, k = s[threadIdx.x + 1] - first - a;
  if (m > kOrderTile) {  // from L2, a thread per cell
    for (unsigned e = 0; e < (k > kCrowd ? 0u : k); ++e) {
      const int v = slots[first + a + e];
      unsigned r = 0;
      for (unsigned j = 0; j < k; ++j) {
        r += slots[first + a + j] < v ? 1u : 0u;
      }
      order[first + a + r] = v;
    }
    return;
  }
  begin[threadIdx.x] = a;
  if (threadIdx.x == kOrderCells - 1) {
    begin[kOrderCells] = m;
  }
  for (unsigned i = threadIdx.x; i < m; i += kOrderCells) {
    tile[i] = slots[first + i];
  }
  for (unsigned e = 0; e < k; ++e) {
    cell[a + e] = (unsigned char)threadIdx.x;
  }
  __syncthreads();
  for (unsigned i = threadIdx.x; i < m; i += kOrderCells) {
    const unsigned c = cell[i], b = begin[c], e = begin[c + 1];
    if (e - b > kCrowd) {
      continue;  // `crowded` is set: the order is not used
    }
    const int v = tile[i];
    unsigned r = b;
    for (unsigned j = b; j < e; ++j) {
      r += tile[j] < v ? 1u : 0u;
    }
    order[first + r] = v;
  }
}

// cells of the counts: those that a shifted box number reaches, rounded up
inline long long padded_cells(long long boxes, int shift)
{
  if (shift > 40) {
    return 1LL << 62;  // more than are counted
  }
  return ((boxes << shift) + kSumCells - 1) / kSumCells * kSumCells;
}

// Whether n droplets over `cells` are sorted by counting: there are more of
// them than the radix sort takes in one launch, and the cells are not many
// more than the droplets, or few.  Measured on both sides: 4096 droplets 9 us
// in one launch, 4097 in 19 by counting (45 by a radix sort of several
// launches); 64k droplets over 4.2M cells, whose passes take 20 us, 211 us of
// GPU time in 73 (radix) and 215 in 38 from the last staging on (counting),
// fewer droplets the other way round.  Beyond kMostCells it was not measured
// (k_cell_starts reads a number of sums that grows with their square): a whole
// re-binning by counting and by radix sort, half a droplet a cell, 1.05M droplets
// 159 and 200 us, 8.5M 748 and 865, 16.9M 1396 and 1619, 67M 5293 and 6003.
// At the other end the last pass decides, which is quadratic in a cell's droplets
// and holds 16 a cell in shared memory.  One box of 32^3 and of 64^3, droplets a
// cell of the grids (`held`), radix sort and counting: hand-over and packing 16 a
// cell 181 and 163 us, 20: 196 and 216, 31: 245 and 317 (8M: 1183 and 1536);
// re-binning, whose key kernel costs as much as the sort, 20: 156 and 147, 24: 162
// and 161, 31: 175 and 208 (8M: 738 and 996).
constexpr int kDenseStaged = 16, kDenseRebin = 24;
inline bool counting_pays(long long cells, long long n, long long held, int dense)
{
  return n > kOneTile && cells <= 64 * n && (cells <= kFewCells || cells <= 2 * n) && cells <= kMostCells &&
         n <= dense * held;
}

// Whether a sort that counting_pays for tries it: not for a while after one
// that found a crowded cell (found_crowded)
inline bool try_counting(pmp_spray* h)
{
  if (h->crowd_skip > 0) {
    --h->crowd_skip;
    return false;
  }
  return true;
}
inline void found_crowded(pmp_spray* h) { h->crowd_skip = kCrowdSkip; }

// The passes' arrays within a buffer: starts, sums, slots, order.
struct CellSortLayout {
  size_t sums, slots, order, total;
};
inline CellSortLayout cell_sort_layout(long long cells, long long n)
{
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  CellSortLayout L;
  L.sums = up(sizeof(unsigned) * (size_t)(cells + 1));
  L.slots = L.sums + up(sizeof(unsigned) * (size_t)(cells / kSumCells));
  L.order = L.slots + up(sizeof(int) * (size_t)n);
  L.total = L.order + up(sizeof(int) * (size_t)n);
  return L;
}

// The order of n counted droplets, on st.  cells: a multiple of kSumCells.
inline void cell_sort(unsigned* counts, long long cells, const unsigned* keys, const int* ranks, long long n, char* buf,
                      cudaStream_t st)
{
  const CellSortLayout L = cell_sort_layout(cells, n);
  unsigned* starts = reinterpret_cast<unsigned*>(buf);
  unsigned* sums = reinterpret_cast<unsigned*>(buf + L.sums);
  int* slots = reinterpret_cast<int*>(buf + L.slots);
  const unsigned blocks = (unsigned)(cells / kSumCells);
  k_cell_sums<<<blocks, 256, 0, st>>>(reinterpret_cast<const uint4*>(counts), sums);
  k_cell_starts<<<blocks, 256, 0, st>>>(reinterpret_cast<uint4*>(counts), sums, starts);
  k_cell_scatter<<<(unsigned)((n + 1023) / 1024), 256, 0, st>>>(keys, ranks, n, starts, slots);
  k_cell_order<<<(unsigned)(cells / kOrderCells), kOrderCells, 0, st>>>(starts, slots,
                                                                       reinterpret_cast<int*>(buf + L.order));
}

}  // namespace
}  // namespace pmp
