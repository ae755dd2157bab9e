// pmp_mesh.cu -- the operations on either side of the update that a time step
// of the host code needs every step, on the device:
//  * estTimestep (SprayParticles.cpp:89-140): particle CFL time step, a min
//    reduction over the droplets;
//  * computeDerivedVars (SprayDerive.cpp:9-155): droplet mass, number,
//    volume, surface, d10, d32, temperature and velocity fields by atomic
//    deposition into the cell holding each droplet, then the protected
//    divisions;
//  * transferSource (SprayParticles.H:250-319), level 0: the source ghost
//    fold (SumBoundary with periodicity), the add into the caller's state
//    source (MultiFab::Add or addSpraySrc), and the reset of the temporary;
//  * redistribute: after a move, droplets are re-binned to the box whose
//    valid region holds their cell, positions wrapped across periodic faces,
//    and dead droplets (id <= 0) dropped -- what AMReX's Redistribute does for
//    this container.  AMReX is not in the reference tree, so its periodic
//    shift is restated here as: while x >= phi, x -= L; while x < plo, x += L
//    (periodic directions only); a droplet whose cell lies in no box is dropped.
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "cell_sort.cuh"
#include "pmp_handle.h"
#include "spray_fp64.cuh"

namespace pmp {

namespace {

struct View32 {
  double* p;
  int lo[3], hi[3];
  int js, ks, ns;
  int ncomp;
};

int check(pmp_spray* h, cudaError_t e, const char* what)
{
  if (e != cudaSuccess) {
    char b[160];
    snprintf(b, sizeof(b), "%s: %s", what, cudaGetErrorString(e));
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

inline unsigned nblk(long long n, int b = 256) { return (unsigned)std::max(1LL, (n + b - 1) / b); }

long long view_elems(const pmp_box_view& v)
{
  return (long long)(v.hi[0] - v.lo[0]) + (long long)(v.hi[1] - v.lo[1]) * v.jstride +
         (long long)(v.hi[2] - v.lo[2]) * v.kstride + (long long)(v.ncomp - 1) * v.nstride + 1;
}

int to_view32(pmp_spray* h, const pmp_box_view& v, View32& o)
{
  if (!v.p || v.ncomp < 1 || view_elems(v) >= (1LL << 31)) {
    return set_err(h, PMP_ERR_INVALID, "view is empty or spans 2^31 elements or more");
  }
  o.p = v.p;
  for (int d = 0; d < 3; ++d) {
    o.lo[d] = v.lo[d];
    o.hi[d] = v.hi[d];
  }
  o.js = (int)v.jstride;
  o.ks = (int)v.kstride;
  o.ns = (int)v.nstride;
  o.ncomp = v.ncomp;
  return PMP_OK;
}

__device__ __forceinline__ bool inside(const View32& v, int i, int j, int k)
{
  return i >= v.lo[0] && i <= v.hi[0] && j >= v.lo[1] && j <= v.hi[1] && k >= v.lo[2] && k <= v.hi[2];
}

__device__ __forceinline__ double* at(const View32& v, int i, int j, int k, int n)
{
  return v.p + ((i - v.lo[0]) + (j - v.lo[1]) * v.js + (k - v.lo[2]) * v.ks + n * v.ns);
}

// item -> (box, local index) over a prefix of per-box counts
__device__ __forceinline__ int find_box(const long long* prefix, int nb, long long i)
{
  int lo = 0, hi = nb;
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (prefix[mid] <= i) {
      lo = mid;
    } else {
      hi = mid;
    }
  }
  return lo;
}

// the handle's scratch for the small per-call tables of this file
int scratch(pmp_spray* h, size_t bytes, void** out)
{
  if (h->mesh_scratch_bytes < bytes) {
    cudaFree(h->mesh_scratch);
    h->mesh_scratch = nullptr;
    h->mesh_scratch_bytes = 0;
    PMP_TRY(h, cudaMalloc(&h->mesh_scratch, bytes));
    h->mesh_scratch_bytes = bytes;
  }
  *out = h->mesh_scratch;
  return PMP_OK;
}

// --------------------------------------------------------------------------
// cell -> box map over the domain

__global__ void k_fill_box_map(int* map, int b, int lo0, int lo1, int lo2, int nx, int ny, int nz, int dlo0, int dlo1,
                               int dlo2, int dnx, int dny)
{
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)nx * ny * nz) {
    return;
  }
  const int i = lo0 + (int)(t % nx);
  const int j = lo1 + (int)((t / nx) % ny);
  const int k = lo2 + (int)(t / ((long long)nx * ny));
  map[(long long)(k - dlo2) * dny * dnx + (long long)(j - dlo1) * dnx + (i - dlo0)] = b;
}

int ensure_box_map(pmp_spray* h, cudaStream_t st)
{
  if (h->box_map_version == h->grids_version && h->d_box_map) {
    return PMP_OK;
  }
  const pmp_geometry& g = h->geom;
  const long long dnx = g.domain_hi[0] - g.domain_lo[0] + 1;
  const long long dny = g.domain_hi[1] - g.domain_lo[1] + 1;
  const long long dnz = g.domain_hi[2] - g.domain_lo[2] + 1;
  const long long ncell = dnx * dny * dnz;
  cudaFree(h->d_box_map);
  h->d_box_map = nullptr;
  PMP_TRY(h, cudaMalloc(&h->d_box_map, sizeof(int) * ncell));
  PMP_TRY(h, cudaMemsetAsync(h->d_box_map, 0xff, sizeof(int) * ncell, st));  // -1: no box
  for (int b = 0; b < (int)h->boxes.size(); ++b) {
    const pmp_box& bx = h->boxes[b];
    for (int d = 0; d < 3; ++d) {
      if (bx.lo[d] < g.domain_lo[d] || bx.hi[d] > g.domain_hi[d]) {
        return set_err(h, PMP_ERR_INVALID, "box outside the domain", b);
      }
    }
    const int nx = bx.hi[0] - bx.lo[0] + 1, ny = bx.hi[1] - bx.lo[1] + 1, nz = bx.hi[2] - bx.lo[2] + 1;
    k_fill_box_map<<<nblk((long long)nx * ny * nz), 256, 0, st>>>(h->d_box_map, b, bx.lo[0], bx.lo[1], bx.lo[2], nx,
                                                                    ny, nz, g.domain_lo[0], g.domain_lo[1],
                                                                    g.domain_lo[2], (int)dnx, (int)dny);
  }
  PMP_TRY(h, cudaGetLastError());
  h->box_map_version = h->grids_version;
  return PMP_OK;
}

struct Domain {
  int lo[3], n[3];
  int periodic[3];
};

Domain domain_of(const pmp_spray* h)
{
  Domain D;
  for (int d = 0; d < 3; ++d) {
    D.lo[d] = h->geom.domain_lo[d];
    D.n[d] = h->geom.domain_hi[d] - h->geom.domain_lo[d] + 1;
    D.periodic[d] = h->geom.bndry_lo[d] == 0;
  }
  return D;
}

// box whose valid region holds cell (i,j,k) after periodic wrap; -1 if none
__device__ __forceinline__ int owner(const int* map, const Domain& D, int* c)
{
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    int r = c[d] - D.lo[d];
    if (D.periodic[d]) {
      r %= D.n[d];
      r += r < 0 ? D.n[d] : 0;
    } else if (r < 0 || r >= D.n[d]) {
      return -1;
    }
    c[d] = D.lo[d] + r;
  }
  return map[((long long)(c[2] - D.lo[2]) * D.n[1] + (c[1] - D.lo[1])) * D.n[0] + (c[0] - D.lo[0])];
}

// --------------------------------------------------------------------------
// estTimestep

// A double as an unsigned integer of the same order (no NaN), and back
__host__ __device__ inline unsigned long long ordered(double v)
{
  unsigned long long u;
#ifdef __CUDA_ARCH__
  u = (unsigned long long)__double_as_longlong(v);
#else
  memcpy(&u, &v, sizeof(u));
#endif
  return u >> 63 ? ~u : u | (1ULL << 63);
}
inline double from_ordered(unsigned long long k)
{
  const unsigned long long u = k >> 63 ? k & ~(1ULL << 63) : ~k;
  double v;
  memcpy(&v, &u, sizeof(v));
  return v;
}

// The minimum over the droplets into *out (an ordered double): four droplets a
// thread, all their fields asked for first (one at a time, the loads of a
// thread waited for one another: 43 us for 4M droplets, 2.6 TB/s).
constexpr int kEstPer = 4;
__global__ void __launch_bounds__(256) k_est_dt(const double* vx, const double* vy, const double* vz, const int* id,
                                                long long n, double dxi0, double dxi1, double dxi2, double cfl,
                                                unsigned long long* out)
{
  const long long base = blockIdx.x * (256LL * kEstPer) + threadIdx.x;
  int live[kEstPer];
  double u[kEstPer][3];
#pragma unroll
  for (int q = 0; q < kEstPer; ++q) {
    const long long i = base + 256 * q;
    live[q] = i < n ? __ldg(id + i) : 1;
    u[q][0] = i < n ? __ldg(vx + i) : 0.;
    u[q][1] = i < n ? __ldg(vy + i) : 0.;
    u[q][2] = i < n ? __ldg(vz + i) : 0.;
  }
  double m = DBL_MAX;
#pragma unroll
  for (int q = 0; q < kEstPer; ++q) {
    double v = -1.;
    if (live[q] > 0) {
      const double mv = fmax(fmax(fabs(u[q][0]) * dxi0, fabs(u[q][1]) * dxi1), fabs(u[q][2]) * dxi2);
      v = mv > 0. ? cfl / mv : 1.E50;
    }
    m = base + 256 * q < n ? fmin(m, v) : m;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m = fmin(m, __shfl_down_sync(0xffffffffu, m, o));
  }
  __shared__ double red[8];
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5] = m;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      m = fmin(m, red[w]);
    }
    atomicMin(out, ordered(m));
  }
}

// --------------------------------------------------------------------------
// computeDerivedVars

struct DeriveArgs {
  const double* pos[3];
  const double* vel[3];
  const double* T;
  const double* dia;
  const double* Y[PMP_MAX_FUEL];
  const double* numdens;
  const double* film;
  const int* id;
  long long n;
  const long long* box_begin;
  int nboxes;
  const View32* views;
  int start;
  int species;  // deposit the per-fuel liquid masses
  int nf;
  double rho_coef[4 * PMP_MAX_FUEL];
  double plo[3], dx[3], dxi[3];
  double cell_vol;
  int* error;  // first slot whose cell the view does not hold (+1), 0 if none
};

// component offsets (relative to start) in the reference's order
enum { kMass = 0, kDens, kNum, kVol, kSurf, kVolf, kD10, kD32, kWfh, kWfm, kTemp, kNump, kVel, kSpec = kVel + 3 };

// The droplets are sorted by cell, so a warp's neighbouring lanes deposit into
// the same cell: each run of lanes with one cell is summed by shuffles into its
// first lane, which alone adds to the cell.  One FP64 atomic per droplet and
// field (34M for 2M two-fuel droplets) held k_derive at L2's atomic rate,
// 180 us; a run is 4-8 droplets at the usual densities.
template <int NF>
__global__ void __launch_bounds__(128) k_derive(const __grid_constant__ DeriveArgs A)
{
  constexpr int NV = 13 + (NF > 1 ? NF : 0);  // deposited fields, in the order of `comp`
  const long long s = blockIdx.x * 128LL + threadIdx.x;
  const int lane = threadIdx.x & 31;
  double v[NV];
  double* cell = nullptr;  // field A.start of the droplet's cell; null: nothing to deposit
  int stride = 0;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    v[i] = 0.;
  }
  // every field of the droplet is asked for before the first one is used
  const bool held = s < A.n;
  const int id = held ? __ldcs(A.id + s) : 0;
  double pos[3], vel[3], Y[NF];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    pos[d] = held ? __ldcs(A.pos[d] + s) : 0.;
    vel[d] = held ? __ldcs(A.vel[d] + s) : 0.;
  }
  const double T_part = held ? __ldcs(A.T + s) : 1.;
  const double dia_part = held ? __ldcs(A.dia + s) : 0.;
#pragma unroll
  for (int spf = 0; spf < NF; ++spf) {
    Y[spf] = held ? __ldcs(A.Y[spf] + s) : 0.;
  }
  const double num_ppp = held ? __ldcs(A.numdens + s) : 0.;
  const double film = held ? __ldcs(A.film + s) : 0.;
  if (id > 0) {
    const int b = find_box(A.box_begin, A.nboxes, s);
    const View32& V = A.views[b];
    int c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      c[d] = static_cast<int>(floor(__dmul_rn(__dsub_rn(pos[d], A.plo[d]), A.dxi[d])));
    }
    if (!inside(V, c[0], c[1], c[2])) {
      atomicCAS(A.error, 0, (int)min(s + 1, 0x7fffffffLL));
    } else {
      double rho_part = 0.;
#pragma unroll
      for (int spf = 0; spf < NF; ++spf) {
        const double* rc = A.rho_coef + 4 * spf;
        rho_part += Y[spf] / (rc[0] + T_part * (rc[1] + T_part * (rc[2] + T_part * rc[3])));
      }
      rho_part = 1. / rho_part;
      const double surf = PMP_PI * dia_part * dia_part;
      const double vol = PMP_PI / 6. * (dia_part * dia_part * dia_part);
      const double pmass = vol * rho_part;
      double* at0 = at(V, c[0], c[1], c[2], A.start);
      if (film == 0.) {
        cell = at0;
        stride = V.ns;
        v[0] = num_ppp * pmass;
        v[1] = num_ppp * pmass / A.cell_vol;
        v[2] = num_ppp;
        v[3] = num_ppp * vol;
        v[4] = num_ppp * surf;
        v[5] = num_ppp * vol / A.cell_vol;
        v[6] = num_ppp * dia_part;
        v[7] = num_ppp * vol * 6.;
        v[8] = num_ppp * pmass * T_part;
        v[9] = 1.;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          v[10 + d] = num_ppp * pmass * vel[d];
        }
        if (NF > 1) {
#pragma unroll
          for (int spf = 0; spf < NF; ++spf) {
            v[NF > 1 ? 13 + spf : 0] = Y[spf] * pmass;  // no parcel count, as the reference
          }
        }
      } else {
        const double face_area = A.dx[0] * A.dx[0];
        const double rad2 = (0.5 * dia_part) * (0.5 * dia_part);
        const double cur_vol = PMP_PI / 6. * film * (3. * rad2 + film * film);
        atomicAdd(at0 + kWfh * V.ns, cur_vol / face_area);
        atomicAdd(at0 + kWfm * V.ns, rho_part * cur_vol);
      }
    }
  }
  // runs of neighbouring lanes with the same cell
  const unsigned all = 0xffffffffu;
  const unsigned long long key = reinterpret_cast<unsigned long long>(cell);
  const unsigned long long before = __shfl_up_sync(all, key, 1);
  const unsigned heads = __ballot_sync(all, lane == 0 || key != before);
  const unsigned after = lane == 31 ? 0u : heads >> (lane + 1);
  const int end = after ? lane + __ffs(after) - 1 : 31;  // last lane of this lane's run
  const int longest = (int)__reduce_max_sync(all, cell ? (unsigned)(end - lane) : 0u);
  for (int o = 1; o <= longest; o <<= 1) {
    const bool take = lane + o <= end;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const double t = __shfl_down_sync(all, v[i], o);
      v[i] = take ? v[i] + t : v[i];
    }
  }
  if (cell && (heads >> lane & 1u)) {
    constexpr int comp[13] = {kMass, kDens, kNum, kVol, kSurf, kVolf, kD10, kD32, kTemp, kNump, kVel, kVel + 1, kVel + 2};
#pragma unroll
    for (int i = 0; i < 13; ++i) {
      red_add(cell + comp[i] * stride, v[i]);
    }
    if (NF > 1 && A.species) {
#pragma unroll
      for (int spf = 0; spf < NF; ++spf) {
        red_add(cell + (kSpec + spf) * stride, v[NF > 1 ? 13 + spf : 0]);
      }
    }
  }
}

// FArrayBox::protected_divide over every cell of each view (ghost cells too)
__global__ void k_protected_divide(const View32* views, const long long* prefix, int nb, long long total, int start)
{
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= total) {
    return;
  }
  const int b = find_box(prefix, nb, t);
  const View32& V = views[b];
  const long long l = t - prefix[b];
  const int nx = V.hi[0] - V.lo[0] + 1, ny = V.hi[1] - V.lo[1] + 1;
  const int i = V.lo[0] + (int)(l % nx);
  const int j = V.lo[1] + (int)((l / nx) % ny);
  const int k = V.lo[2] + (int)(l / ((long long)nx * ny));
  const int pairs[6][2] = {{kNum, kD10}, {kSurf, kD32}, {kMass, kTemp}, {kMass, kVel}, {kMass, kVel + 1}, {kMass, kVel + 2}};
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const double den = *at(V, i, j, k, start + pairs[q][0]);
    if (den != 0.) {
      double* num = at(V, i, j, k, start + pairs[q][1]);
      *num = *num / den;
    }
  }
}

// --------------------------------------------------------------------------
// transferSource

// SumBoundary: every ghost cell of every box adds into the valid cell that
// owns its (periodically wrapped) location
__global__ void k_sum_boundary(const View32* tmp, const pmp_box* boxes, const long long* prefix, int nb,
                               long long total, int g, const int* map, Domain D, int ncomp)
{
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= total) {
    return;
  }
  const int b = find_box(prefix, nb, t);
  const pmp_box& bx = boxes[b];
  const long long l = t - prefix[b];
  const int nx = bx.hi[0] - bx.lo[0] + 1 + 2 * g, ny = bx.hi[1] - bx.lo[1] + 1 + 2 * g;
  const int i = bx.lo[0] - g + (int)(l % nx);
  const int j = bx.lo[1] - g + (int)((l / nx) % ny);
  const int k = bx.lo[2] - g + (int)(l / ((long long)nx * ny));
  if (i >= bx.lo[0] && i <= bx.hi[0] && j >= bx.lo[1] && j <= bx.hi[1] && k >= bx.lo[2] && k <= bx.hi[2]) {
    return;  // valid cell: a destination, not a source
  }
  int c[3] = {i, j, k};
  const int o = owner(map, D, c);
  if (o < 0) {
    return;
  }
  const View32& S = tmp[b];
  const View32& T = tmp[o];
  for (int n = 0; n < ncomp; ++n) {
    const double v = *at(S, i, j, k, n);
    if (v != 0.) {
      atomicAdd(at(T, c[0], c[1], c[2], n), v);
    }
  }
}

struct AddMap {
  int same;  // add every component
  int mom_src, rho_src, eng_src, spec_src;
  int mom, rho, eng, spec;
  int nf;
  int dep[PMP_MAX_FUEL];
};

// MultiFab::Add or addSpraySrc over each box grown by nghost, and the reset of
// the temporary over its whole view, in one pass: a thread per cell of the view
// (consecutive threads, consecutive cells of a component).  As two kernels, the
// reset one thread per value with a 64-bit division each, 60 us for 8 boxes of
// 64 x 32 x 32 and 7 components.
__global__ void __launch_bounds__(256) k_add_reset(const View32* tmp, const View32* act, const pmp_box* boxes,
                                                   const long long* prefix, int nb, long long total, int ng,
                                                   const __grid_constant__ AddMap M)
{
  const long long t = blockIdx.x * 256LL + threadIdx.x;
  if (t >= total) {
    return;
  }
  const int b = find_box(prefix, nb, t);
  const View32& S = tmp[b];
  const pmp_box& bx = boxes[b];
  const unsigned l = (unsigned)(t - prefix[b]);  // a view spans fewer than 2^31 elements
  const unsigned nx = (unsigned)(S.hi[0] - S.lo[0] + 1), ny = (unsigned)(S.hi[1] - S.lo[1] + 1);
  const unsigned row = l / nx;
  const int i = S.lo[0] + (int)(l - row * nx);
  const int k = S.lo[2] + (int)(row / ny);
  const int j = S.lo[1] + (int)(row - row / ny * ny);
  double* s = at(S, i, j, k, 0);
  const bool in = i >= bx.lo[0] - ng && i <= bx.hi[0] + ng && j >= bx.lo[1] - ng && j <= bx.hi[1] + ng &&
                  k >= bx.lo[2] - ng && k <= bx.hi[2] + ng;
  if (in) {
    const View32& A = act[b];
    double* a = at(A, i, j, k, 0);
    if (M.same) {
      for (int n = 0; n < A.ncomp; ++n) {
        a[n * A.ns] += s[n * S.ns];
      }
    } else {
      for (int d = 0; d < 3; ++d) {
        a[(M.mom + d) * A.ns] += s[(M.mom_src + d) * S.ns];
      }
      a[M.rho * A.ns] += s[M.rho_src * S.ns];
      a[M.eng * A.ns] += s[M.eng_src * S.ns];
      for (int sp = 0; sp < M.nf; ++sp) {
        a[(M.spec + M.dep[sp]) * A.ns] += s[(M.spec_src + sp) * S.ns];
      }
    }
  }
  for (int n = 0; n < S.ncomp; ++n) {
    s[n * S.ns] = 0.;
  }
}

// --------------------------------------------------------------------------
// redistribute

struct Wrap {
  double lo[3], hi[3], dxi[3];
};

// Sort key of a droplet: its new box o above `shift` bits of its cell's
// place in the box's sort order (pmp::brick_key); dead droplets and droplets
// in no box get box nb, so that they sort last.  K / V: 32-bit keys and slot
// indices when the key fits 32 bits and the count 2^31, else 64-bit.
// COUNT: the live droplets are counted into their cells, the others get key
// kNoCell, and the ranks take the indices' place.  Two droplets a thread, each
// of the dependent loads (id and position, owner, box, count) for both at
// once; the position of a dead droplet is loaded for nothing.
constexpr int kRebinPer = 2;
template <typename K, typename V, bool COUNT>
__global__ void __launch_bounds__(256) k_rebin_keys(double* px, double* py, double* pz, const int* id, long long n,
                                                    const int* map, const Domain D, const Wrap w, const pmp_box* boxes,
                                                    int nb, int shift, K* keys, V* idx, unsigned* counts, int* crowded)
{
  const long long s0 = blockIdx.x * (256LL * kRebinPer) + threadIdx.x;
  double* p[3] = {px, py, pz};
  int alive[kRebinPer], o[kRebinPer], c[kRebinPer][3];
  double x[kRebinPer][3];
#pragma unroll
  for (int u = 0; u < kRebinPer; ++u) {
    const long long s = s0 + 256 * u;
    alive[u] = s < n ? id[s] : 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      x[u][d] = s < n ? p[d][s] : 0.;
    }
  }
#pragma unroll
  for (int u = 0; u < kRebinPer; ++u) {
    o[u] = -1;
    if (alive[u] > 0) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        double y = x[u][d];
        if (D.periodic[d]) {
          const double L = w.hi[d] - w.lo[d];
          for (int it = 0; it < 64 && y >= w.hi[d]; ++it) {
            y -= L;
          }
          for (int it = 0; it < 64 && y < w.lo[d]; ++it) {
            y += L;
          }
          if (y != x[u][d]) {
            p[d][s0 + 256 * u] = y;
          }
        }
        c[u][d] = static_cast<int>(floor(__dmul_rn(__dsub_rn(y, w.lo[d]), w.dxi[d])));
      }
      o[u] = owner(map, D, c[u]);
    }
  }
  K key[kRebinPer];
  Counted q[kRebinPer];
#pragma unroll
  for (int u = 0; u < kRebinPer; ++u) {
    key[u] = COUNT ? (K)kNoCell : (K)nb << shift;
    if (o[u] >= 0) {
      const pmp_box& bx = boxes[o[u]];
      const int ex = bx.hi[0] - bx.lo[0] + 1, ey = bx.hi[1] - bx.lo[1] + 1;
      const unsigned long long local =
        pmp::brick_key(c[u][0] - bx.lo[0], c[u][1] - bx.lo[1], c[u][2] - bx.lo[2], ex, ey);
      key[u] = ((K)o[u] << shift) | (K)local;
    }
    if (COUNT) {
      q[u] = count_cell(counts, (unsigned)key[u]);
    }
  }
#pragma unroll
  for (int u = 0; u < kRebinPer; ++u) {
    const long long s = s0 + 256 * u;
    const V v = COUNT ? (V)rank_of(q[u], (unsigned)key[u], crowded) : (V)s;
    if (s < n) {
      keys[s] = key[u];
      idx[s] = v;
    }
  }
}

// begin[b] of counted droplets: the first slot of box b's first cell (b = nb:
// their number)
__global__ void k_box_starts(const unsigned* starts, int nb, int shift, long long* begin)
{
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b <= nb) {
    begin[b] = starts[(long long)b << shift];
  }
}

// begin[b]: the first sorted position of box b (b = nb: the dead)
template <typename K>
__global__ void k_box_bounds(const K* keys, long long n, int nb, int shift, long long* begin)
{
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b > nb) {
    return;
  }
  const K key = (K)b << shift;
  long long lo = 0, hi = n;  // first index with keys[i] >= key
  while (lo < hi) {
    const long long mid = (lo + hi) / 2;
    if (keys[mid] < key) {
      lo = mid + 1;
    } else {
      hi = mid;
    }
  }
  begin[b] = lo;
}

template <typename V>
__global__ void k_gather_soa(const double* src, long long stride_src, const int* sid, const V* perm, long long n,
                             int ncomp, double* dst, int* did)
{
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (s >= n) {
    return;
  }
  const long long j = (long long)perm[s];
  for (int c = 0; c < ncomp; ++c) {
    dst[c * n + s] = src[c * stride_src + j];
  }
  did[s] = sid[j];
}

// perm[s] = s - begin[b] for the slots s of box b (the re-binned order is
// each box's caller order)
__global__ void k_rebin_perm(long long* perm, const long long* begin, int nb, long long n)
{
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (s >= n) {
    return;
  }
  int lo = 0, hi = nb;  // the box b with begin[b] <= s < begin[b + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (begin[mid] <= s) {
      lo = mid;
    } else {
      hi = mid;
    }
  }
  perm[s] = s - begin[lo];
}

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Offsets of the re-binning's working arrays in the handle's sort_scratch:
// keys, sorted keys, slot indices, sorted indices (the gather order), box
// bounds, the box list, CUB's temporary storage.
struct RebinLayout {
  size_t keys2, idx, perm, begin, boxes, tmp, total;
};
RebinLayout rebin_layout(long long n, int nb, size_t kbytes, size_t vbytes, size_t tbytes)
{
  const size_t cap = (size_t)std::max(n, 1LL);
  RebinLayout L;
  L.keys2 = align256(kbytes * cap);
  L.idx = L.keys2 + align256(kbytes * cap);
  L.perm = L.idx + align256(vbytes * cap);
  L.begin = L.perm + align256(vbytes * cap);
  L.boxes = L.begin + align256(sizeof(long long) * (nb + 1));
  L.tmp = L.boxes + align256(sizeof(pmp_box) * std::max(nb, 1));
  L.total = L.tmp + align256(std::max(tbytes, (size_t)1));
  return L;
}

}  // namespace

void mesh_free(pmp_spray* h)
{
  cudaFree(h->d_box_map);
  h->d_box_map = nullptr;
  h->box_map_version = -1;
  cudaFree(h->mesh_scratch);
  h->mesh_scratch = nullptr;
  h->mesh_scratch_bytes = 0;
}

}  // namespace pmp

using namespace pmp;

extern "C" int pmp_spray_est_timestep(pmp_spray* h, double cfl, double max_jet_vel, double* dt, void* stream)
{
  if (!h || !dt) {
    return PMP_ERR_INVALID;
  }
  if (!h->have_data || !h->have_geom) {
    return set_err(h, PMP_ERR_INVALID, "setup and geometry must be set first");
  }
  cudaSetDevice(h->device);
  pmp::quiesce(h);
  cudaStream_t st = (cudaStream_t)stream;
  if (h->data.fixed_parts) {
    *dt = -1.;
    return PMP_OK;
  }
  int rc = ensure_packed(h, st);
  if (rc != PMP_OK) {
    return rc;
  }
  const pmp_geometry& g = h->geom;
  double r = DBL_MAX;
  const long long n = h->total;
  if (n > 0) {
    void* sp = nullptr;
    rc = scratch(h, sizeof(unsigned long long), &sp);
    if (rc != PMP_OK) {
      return rc;
    }
    unsigned long long* least = static_cast<unsigned long long*>(sp);
    unsigned long long* hl = reinterpret_cast<unsigned long long*>(h->h_small());
    PMP_TRY(h, cudaMemsetAsync(least, 0xff, sizeof(*least), st));
    const double* vel = h->soa + 3 * n;  // rdata component 0 follows the positions
    k_est_dt<<<nblk(n, 256 * kEstPer), 256, 0, st>>>(vel, vel + n, vel + 2 * n, h->ids, n, 1. / g.dx[0], 1. / g.dx[1],
                                                     1. / g.dx[2], cfl, least);
    PMP_TRY(h, cudaMemcpyAsync(hl, least, sizeof(*hl), cudaMemcpyDeviceToHost, st));
    PMP_TRY(h, cudaStreamSynchronize(st));
    r = std::min(r, from_ordered(*hl));
  }
  if (max_jet_vel > 0.) {
    r = std::min(r, cfl * g.dx[0] / max_jet_vel);
  }
  *dt = r;
  return PMP_OK;
}

extern "C" int pmp_spray_derive(pmp_spray* h, const pmp_box_view* vars, int nboxes, int start_indx, int with_species,
                                void* stream)
{
  if (!h || !vars || nboxes != (int)h->boxes.size() || start_indx < 0) {
    return set_err(h, PMP_ERR_INVALID, "bad arguments to pmp_spray_derive");
  }
  if (!h->have_data || !h->have_geom) {
    return set_err(h, PMP_ERR_INVALID, "setup and geometry must be set first");
  }
  cudaSetDevice(h->device);
  pmp::quiesce(h);
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_packed(h, st);
  if (rc != PMP_OK) {
    return rc;
  }
  const int nf = h->nfuel;
  const int nvar = kSpec + ((with_species && nf > 1) ? nf : 0);
  std::vector<View32> hv(nboxes);
  std::vector<long long> prefix(nboxes + 1, 0);
  for (int b = 0; b < nboxes; ++b) {
    rc = to_view32(h, vars[b], hv[b]);
    if (rc != PMP_OK) {
      return rc;
    }
    if (vars[b].ncomp < start_indx + nvar) {
      return set_err(h, PMP_ERR_INVALID, "derive view has too few components", b);
    }
    const long long cells = (long long)(vars[b].hi[0] - vars[b].lo[0] + 1) * (vars[b].hi[1] - vars[b].lo[1] + 1) *
                            (vars[b].hi[2] - vars[b].lo[2] + 1);
    prefix[b + 1] = prefix[b] + cells;
  }
  const size_t need = sizeof(View32) * nboxes + sizeof(long long) * (nboxes + 1) + 16;
  void* sp = nullptr;
  rc = scratch(h, need, &sp);
  if (rc != PMP_OK) {
    return rc;
  }
  // {error word, views, cell prefix} in one upload
  std::vector<char> up(need, 0);
  memcpy(up.data() + 16, hv.data(), sizeof(View32) * nboxes);
  memcpy(up.data() + 16 + sizeof(View32) * nboxes, prefix.data(), sizeof(long long) * (nboxes + 1));
  int* d_err = static_cast<int*>(sp);
  View32* d_views = reinterpret_cast<View32*>(static_cast<char*>(sp) + 16);
  long long* d_prefix = reinterpret_cast<long long*>(d_views + nboxes);
  PMP_TRY(h, cudaMemcpyAsync(sp, up.data(), need, cudaMemcpyHostToDevice, st));
  const long long n = h->total;
  const pmp_geometry& g = h->geom;
  DeriveArgs A;
  memset(&A, 0, sizeof(A));
  for (int d = 0; d < 3; ++d) {
    A.pos[d] = h->soa + (long long)d * n;
    A.vel[d] = h->soa + (long long)(3 + PMP_PSTATE_VEL + d) * n;
    A.plo[d] = g.plo[d];
    A.dx[d] = g.dx[d];
    A.dxi[d] = 1. / g.dx[d];
  }
  A.T = h->soa + (long long)(3 + PMP_PSTATE_T) * n;
  A.dia = h->soa + (long long)(3 + PMP_PSTATE_DIA) * n;
  for (int f = 0; f < nf; ++f) {
    A.Y[f] = h->soa + (long long)(3 + PMP_PSTATE_Y + f) * n;
  }
  A.numdens = h->soa + (long long)(3 + PMP_PSTATE_NUMDENS(nf)) * n;
  A.film = h->soa + (long long)(3 + PMP_PSTATE_FILMHGHT(nf)) * n;
  A.id = h->ids;
  A.n = n;
  A.box_begin = h->d_box_begin;
  A.nboxes = nboxes;
  A.views = d_views;
  A.start = start_indx;
  A.species = with_species && nf > 1;
  A.nf = nf;
  for (int i = 0; i < 4 * nf; ++i) {
    A.rho_coef[i] = h->data.rho_coef[i];
  }
  A.cell_vol = g.dx[0] * g.dx[1] * g.dx[2];
  A.error = d_err;
  if (n > 0) {
    const unsigned grid = nblk(n, 128);
    switch (nf) {
      case 1:
        k_derive<1><<<grid, 128, 0, st>>>(A);
        break;
      case 2:
        k_derive<2><<<grid, 128, 0, st>>>(A);
        break;
      case 3:
        k_derive<3><<<grid, 128, 0, st>>>(A);
        break;
      default:
        k_derive<4><<<grid, 128, 0, st>>>(A);
        break;
    }
  }
  if (prefix[nboxes] > 0) {
    k_protected_divide<<<nblk(prefix[nboxes]), 256, 0, st>>>(d_views, d_prefix, nboxes, prefix[nboxes], start_indx);
  }
  int* hp = reinterpret_cast<int*>(h->h_small());
  PMP_TRY(h, cudaGetLastError());
  PMP_TRY(h, cudaMemcpyAsync(hp, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
  PMP_TRY(h, cudaStreamSynchronize(st));
  const int herr = *hp;
  if (herr != 0) {
    return set_err(h, PMP_ERR_SOURCE_BOX, "derive view does not hold a droplet's cell", -1, herr - 1);
  }
  return PMP_OK;
}

extern "C" int pmp_spray_transfer_source(pmp_spray* h, const pmp_box_view* tmp_source, const pmp_box_view* act_source,
                                         int nboxes, int source_ghosts, int act_ghosts, void* stream)
{
  if (!h || !tmp_source || !act_source || nboxes != (int)h->boxes.size() || source_ghosts < 0 || act_ghosts < 0) {
    return set_err(h, PMP_ERR_INVALID, "bad arguments to pmp_spray_transfer_source");
  }
  if (!h->have_geom || !h->have_comps || !h->have_data) {
    return set_err(h, PMP_ERR_INVALID, "setup, comps and geometry must be set first");
  }
  cudaSetDevice(h->device);
  pmp::quiesce(h);
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_box_map(h, st);
  if (rc != PMP_OK) {
    return rc;
  }
  const int g = source_ghosts;
  const int ng = std::min(act_ghosts, source_ghosts);
  std::vector<View32> ht(nboxes), ha(nboxes);
  std::vector<long long> pg(nboxes + 1, 0), pz(nboxes + 1, 0);
  int ncomp = -1;
  for (int b = 0; b < nboxes; ++b) {
    const pmp_box& bx = h->boxes[b];
    if ((rc = to_view32(h, tmp_source[b], ht[b])) != PMP_OK || (rc = to_view32(h, act_source[b], ha[b])) != PMP_OK) {
      return rc;
    }
    for (int d = 0; d < 3; ++d) {
      if (tmp_source[b].lo[d] > bx.lo[d] - g || tmp_source[b].hi[d] < bx.hi[d] + g) {
        return set_err(h, PMP_ERR_INVALID, "source view does not cover the box grown by source_ghosts", b);
      }
      if (act_source[b].lo[d] > bx.lo[d] - ng || act_source[b].hi[d] < bx.hi[d] + ng) {
        return set_err(h, PMP_ERR_INVALID, "destination view does not cover the box grown by its ghosts", b);
      }
    }
    if (ncomp < 0) {
      ncomp = tmp_source[b].ncomp;
    } else if (ncomp != tmp_source[b].ncomp) {
      return set_err(h, PMP_ERR_INVALID, "source views differ in component count", b);
    }
    auto cells = [&](int grow) {
      return (long long)(bx.hi[0] - bx.lo[0] + 1 + 2 * grow) * (bx.hi[1] - bx.lo[1] + 1 + 2 * grow) *
             (bx.hi[2] - bx.lo[2] + 1 + 2 * grow);
    };
    pg[b + 1] = pg[b] + cells(g);
    const pmp_box_view& v = tmp_source[b];
    pz[b + 1] = pz[b] + (long long)(v.hi[0] - v.lo[0] + 1) * (v.hi[1] - v.lo[1] + 1) * (v.hi[2] - v.lo[2] + 1);
  }
  const pmp_spray_comps& c = h->comps;
  AddMap M;
  memset(&M, 0, sizeof(M));
  M.same = 1;
  for (int b = 0; b < nboxes; ++b) {
    M.same = M.same && act_source[b].ncomp == tmp_source[b].ncomp;
  }
  M.mom_src = c.momSrcIndx;
  M.rho_src = c.rhoSrcIndx;
  M.eng_src = c.engSrcIndx;
  M.spec_src = c.specSrcIndx;
  M.mom = c.momIndx;
  M.rho = c.rhoIndx;
  M.eng = c.engIndx;
  M.spec = c.specIndx;
  M.nf = h->nfuel;
  for (int f = 0; f < h->nfuel; ++f) {
    M.dep[f] = h->data.dep_indx[f];
  }
  if (!M.same) {
    const int need_src = 1 + std::max({c.momSrcIndx + 2, c.rhoSrcIndx, c.engSrcIndx, c.specSrcIndx + h->nfuel - 1});
    int need_act = 1 + std::max({c.momIndx + 2, c.rhoIndx, c.engIndx});
    for (int f = 0; f < h->nfuel; ++f) {
      need_act = std::max(need_act, c.specIndx + h->data.dep_indx[f] + 1);
    }
    for (int b = 0; b < nboxes; ++b) {
      if (tmp_source[b].ncomp < need_src || act_source[b].ncomp < need_act) {
        return set_err(h, PMP_ERR_INVALID, "views lack the source or state components", b);
      }
    }
  }
  // {source views, destination views, cell prefixes, boxes} in one upload
  const size_t vb = sizeof(View32) * nboxes, xb = sizeof(long long) * (nboxes + 1), bb = sizeof(pmp_box) * nboxes;
  std::vector<char> up(2 * vb + 2 * xb + bb);
  memcpy(up.data(), ht.data(), vb);
  memcpy(up.data() + vb, ha.data(), vb);
  memcpy(up.data() + 2 * vb, pg.data(), xb);
  memcpy(up.data() + 2 * vb + xb, pz.data(), xb);
  memcpy(up.data() + 2 * vb + 2 * xb, h->boxes.data(), bb);
  void* sp = nullptr;
  if ((rc = scratch(h, up.size(), &sp)) != PMP_OK) {
    return rc;
  }
  View32* d_t = static_cast<View32*>(sp);
  View32* d_a = d_t + nboxes;
  long long* d_pg = reinterpret_cast<long long*>(d_a + nboxes);
  long long* d_pz = d_pg + nboxes + 1;
  pmp_box* d_boxes = reinterpret_cast<pmp_box*>(d_pz + nboxes + 1);
  PMP_TRY(h, cudaMemcpyAsync(sp, up.data(), up.size(), cudaMemcpyHostToDevice, st));
  const Domain D = domain_of(h);
  if (g > 0 && pg[nboxes] > 0) {
    k_sum_boundary<<<nblk(pg[nboxes]), 256, 0, st>>>(d_t, d_boxes, d_pg, nboxes, pg[nboxes], g, h->d_box_map, D, ncomp);
  }
  if (pz[nboxes] > 0) {
    k_add_reset<<<nblk(pz[nboxes]), 256, 0, st>>>(d_t, d_a, d_boxes, d_pz, nboxes, pz[nboxes], ng, M);
  }
  PMP_TRY(h, cudaGetLastError());
  PMP_TRY(h, cudaStreamSynchronize(st));
  return PMP_OK;
}

static Wrap wrap_of(const pmp_spray* h)
{
  Wrap w;
  for (int d = 0; d < 3; ++d) {
    w.lo[d] = h->geom.plo[d];
    w.hi[d] = h->geom.phi[d];
    w.dxi[d] = 1. / h->geom.dx[d];
  }
  return w;
}

// the box bounds on the host
static int read_bounds(pmp_spray* h, cudaStream_t st, const long long* d_begin, std::vector<long long>& begin)
{
  PMP_TRY(h, cudaMemcpyAsync(begin.data(), d_begin, sizeof(long long) * begin.size(), cudaMemcpyDeviceToHost, st));
  if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
    return set_err(h, PMP_ERR_CUDA, "redistribute: kernel failed");
  }
  return PMP_OK;
}

// The re-binning's keys, their sort and the box bounds (begin, host copy),
// with K-bit keys over bits [0, end_bit) and V-bit slot indices; *order: the
// sorted indices (the gather order), in sort_scratch, *d_begin the bounds.
template <typename K, typename V>
static int rebin_sort(pmp_spray* h, cudaStream_t st, long long n, int nb, int shift, int end_bit,
                      std::vector<long long>& begin, const void** order, const long long** d_bounds)
{
  size_t tbytes = 0;
  if (n > 0) {
    cub::DeviceRadixSort::SortPairs(nullptr, tbytes, (const K*)nullptr, (K*)nullptr, (const V*)nullptr, (V*)nullptr,
                                    (int)n, 0, end_bit, st);
  }
  const RebinLayout L = rebin_layout(n, nb, sizeof(K), sizeof(V), tbytes);
  const int rk = keep(h, h->sort_scratch, L.total);
  if (rk != PMP_OK) {
    return rk;
  }
  char* base = static_cast<char*>(h->sort_scratch.p);
  K* keys = reinterpret_cast<K*>(base);
  K* keys2 = reinterpret_cast<K*>(base + L.keys2);
  V* idx = reinterpret_cast<V*>(base + L.idx);
  V* perm = reinterpret_cast<V*>(base + L.perm);
  long long* d_begin = reinterpret_cast<long long*>(base + L.begin);
  pmp_box* d_boxes = reinterpret_cast<pmp_box*>(base + L.boxes);
  PMP_TRY(h, cudaMemcpyAsync(d_boxes, h->boxes.data(), sizeof(pmp_box) * nb, cudaMemcpyHostToDevice, st));
  if (n > 0) {
    k_rebin_keys<K, V, false><<<nblk(n, 256 * kRebinPer), 256, 0, st>>>(h->soa, h->soa + n, h->soa + 2 * n, h->ids, n, h->d_box_map,
                                                       domain_of(h), wrap_of(h), d_boxes, nb, shift, keys, idx, nullptr,
                                                       nullptr);
    cub::DeviceRadixSort::SortPairs(base + L.tmp, tbytes, keys, keys2, idx, perm, (int)n, 0, end_bit, st);
    k_box_bounds<K><<<nblk(nb + 1, 64), 64, 0, st>>>(keys2, n, nb, shift, d_begin);
  } else {
    PMP_TRY(h, cudaMemsetAsync(d_begin, 0, sizeof(long long) * (nb + 1), st));
  }
  *order = perm;
  *d_bounds = d_begin;
  return read_bounds(h, st, d_begin, begin);
}

// The same by counting (cell_sort.cuh); *sorted: false when a cell holds too
// many droplets, or there is no memory for the counts, and nothing was sorted.
static int rebin_count(pmp_spray* h, cudaStream_t st, long long n, int nb, int shift, long long cells,
                       std::vector<long long>& begin, const void** order, const long long** d_bounds, bool* sorted)
{
  auto up = [](size_t b) { return align256(b); };
  const CellSortLayout L = cell_sort_layout(cells, n);
  const size_t ranks = L.total + up(sizeof(unsigned) * n), bounds = ranks + up(sizeof(int) * n);
  const size_t boxes = bounds + up(sizeof(long long) * (nb + 1));
  *sorted = false;
  bool have = try_keep(h, h->sort_scratch, boxes + sizeof(pmp_box) * nb) == cudaSuccess;
  int rc = have ? count_cells(h, cells, st, &have) : PMP_OK;
  if (rc != PMP_OK || !have) {
    return rc;
  }
  char* base = static_cast<char*>(h->sort_scratch.p);
  unsigned* counts = static_cast<unsigned*>(h->counts.p);
  unsigned* keys = reinterpret_cast<unsigned*>(base + L.total);
  int* rank = reinterpret_cast<int*>(base + ranks);
  long long* d_begin = reinterpret_cast<long long*>(base + bounds);
  pmp_box* d_boxes = reinterpret_cast<pmp_box*>(base + boxes);
  PMP_TRY(h, cudaMemcpyAsync(d_boxes, h->boxes.data(), sizeof(pmp_box) * nb, cudaMemcpyHostToDevice, st));
  k_rebin_keys<unsigned, int, true><<<nblk(n, 256 * kRebinPer), 256, 0, st>>>(h->soa, h->soa + n, h->soa + 2 * n, h->ids, n, h->d_box_map,
                                                             domain_of(h), wrap_of(h), d_boxes, nb, shift, keys, rank,
                                                             counts, h->crowded());
  cell_sort(counts, cells, keys, rank, n, base, st);
  h->cell_sorts += 1;
  k_box_starts<<<nblk(nb + 1), 256, 0, st>>>(reinterpret_cast<unsigned*>(base), nb, shift, d_begin);
  rc = read_bounds(h, st, d_begin, begin);
  if (rc != PMP_OK) {
    return rc;
  }
  h->zero_cells = cells;
  *sorted = *h->crowded() == 0;
  if (!*sorted) {
    found_crowded(h);
  }
  *order = base + L.order;
  *d_bounds = d_begin;
  return PMP_OK;
}

extern "C" int pmp_spray_redistribute(pmp_spray* h, long long* removed, void* stream)
{
  if (!h) {
    return PMP_ERR_INVALID;
  }
  if (!h->have_geom) {
    return set_err(h, PMP_ERR_INVALID, "geometry must be set first");
  }
  cudaSetDevice(h->device);
  pmp::quiesce(h);
  cudaStream_t st = (cudaStream_t)stream;
  int rc = ensure_packed(h, st);
  if (rc == PMP_OK) {
    rc = ensure_box_map(h, st);
  }
  if (rc != PMP_OK) {
    return rc;
  }
  const int nb = (int)h->boxes.size();
  const long long n = h->total;
  const int nc = h->ncomp();
  // key bits: the largest box's cell count, then the box index (nb: dead)
  int shift = 0;
  for (const pmp_box& bx : h->boxes) {
    const unsigned long long cells =
      pmp::brick_key_count(bx.hi[0] - bx.lo[0] + 1, bx.hi[1] - bx.lo[1] + 1, bx.hi[2] - bx.lo[2] + 1);
    while (shift < 63 && (1ULL << shift) < cells) {
      ++shift;
    }
  }
  int end_bit = shift + 1;
  while (end_bit < 64 && (1LL << (end_bit - shift)) <= nb) {
    ++end_bit;
  }
  if (end_bit > 62 || nb >= (1 << 22)) {
    return set_err(h, PMP_ERR_INVALID, "box too large for the re-binning key");
  }
  std::vector<long long> begin(nb + 1, 0);
  const bool narrow = end_bit <= 32 && n < (1LL << 31);
  const void* order = nullptr;
  const long long* d_begin = nullptr;
  const long long cells = padded_cells(nb, shift);
  bool sorted = false;
  if (narrow && counting_pays(cells, n, h->grid_cells, kDenseRebin) && try_counting(h)) {
    rc = rebin_count(h, st, n, nb, shift, cells, begin, &order, &d_begin, &sorted);
  }
  if (rc == PMP_OK && !sorted) {
    rc = narrow ? rebin_sort<unsigned, int>(h, st, n, nb, shift, end_bit, begin, &order, &d_begin)
                : rebin_sort<unsigned long long, long long>(h, st, n, nb, shift, end_bit, begin, &order, &d_begin);
  }
  if (rc != PMP_OK) {
    return rc;
  }
  const long long live = begin[nb];
  // gather into the spare store (grown when too small), which then becomes
  // the store; the old store becomes the spare
  rc = keep(h, h->spare, store_bytes(h, std::max(live, 1LL)));
  if (rc != PMP_OK) {
    return rc;
  }
  double* soa2 = static_cast<double*>(h->spare.p);
  int* ids2 = reinterpret_cast<int*>(soa2 + (long long)nc * live);
  if (live > 0) {
    if (narrow) {
      k_gather_soa<<<nblk(live), 256, 0, st>>>(h->soa, n, h->ids, static_cast<const int*>(order), live, nc,
                                               soa2, ids2);
    } else {
      k_gather_soa<<<nblk(live), 256, 0, st>>>(h->soa, n, h->ids, static_cast<const long long*>(order), live, nc,
                                               soa2, ids2);
    }
    // each box's new order is its caller order (h->perm_b holds >= n >= live slots)
    k_rebin_perm<<<nblk(live), 256, 0, st>>>(h->perm(), d_begin, nb, live);
  }
  if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
    return set_err(h, PMP_ERR_CUDA, "redistribute: gather failed");
  }
  std::swap(h->store, h->spare);
  store_attach(h, live);
  if (removed) {
    *removed = n - live;
  }
  rc = install_rebinned(h, begin, st);
  if (rc != PMP_OK) {
    return rc;
  }
  PMP_TRY(h, cudaStreamSynchronize(st));
  return PMP_OK;
}
