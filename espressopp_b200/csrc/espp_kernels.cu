// espp_kernels.cu - sm_100a kernels of the short-range MD step.
//
//  re-binning     k_fold_bin -> k_scan_* -> k_scatter -> k_sort_cells (-> k_move)
//                 (storage::DomainDecomposition::decomposeRealParticles, one node)
//  Verlet list    k_build_block (a block per run of 32 particles of a row of cells,
//                 candidates filtered against the run's bounding box) / k_build_nl_run (one
//                 warp per run, lists of any length): FP32 test with the reference's FP64
//                 ghost-shift arithmetic near the cutoff, full per-particle list
//                 (VerletList::_rebuildUsingBuffers)
//  forces         k_force_mixed (FP32 on box-wrapped int32 coordinates, int64 2^-32
//                 fixed-point output) / k_force_fp64 (plain FP64); LJ + FENE fused
//  integrator     k_integrate: aftCalcF (Langevin, CapForce) + integrate2 of step n +
//                 integrate1 of step n+1 in one pass over the particle arrays; k_steps: every
//                 step of a small system up to the next re-sort in one launch
//  observables    FP64 energy / virial / kinetic with fixed-order block reductions
#include <math.h>
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <type_traits>

#include "espp_device.h"
#include "espp_internal.h"
#include "espp_tab.h"
#include "espp_tc.h"

namespace espp {

void make_float_table(const LJTable& t, LJPairF* f) {
  for (int k = 0; k < kMaxTypes * kMaxTypes; ++k) {
    const LJPair& p = t.p[k];
    f[k].ff1 = (float)p.ff1;
    f[k].ff2 = (float)p.ff2;
    f[k].rcsq = p.set ? (float)p.rcsq : -1.0f;
    f[k].capsq = p.caprad > 0 ? (float)(p.caprad * p.caprad) : -1.0f;
    f[k].capff = (float)p.capff;
    f[k].set = p.set;
  }
}

namespace {


// ---- Philox4x32-10 (Salmon et al., SC'11) ----------------------------------------
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    if (r > 0) {
      k0 += 0x9E3779B9u;
      k1 += 0xBB67AE85u;
    }
    uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
    uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
    c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
  }
  return c;
}

__device__ __forceinline__ void langevin_uniforms(uint64_t seed, int64_t id, int64_t step,
                                                  int phase, double u[3]) {
  uint4 c = make_uint4((uint32_t)(uint64_t)id, (uint32_t)((uint64_t)id >> 32),
                       (uint32_t)(uint64_t)step,
                       ((uint32_t)((uint64_t)step >> 32) & 0x7FFFFFFFu) |
                           ((uint32_t)phase << 31));
  uint4 r = philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  u[0] = ((double)r.x + 0.5) * (1.0 / 4294967296.0);
  u[1] = ((double)r.y + 0.5) * (1.0 / 4294967296.0);
  u[2] = ((double)r.z + 0.5) * (1.0 / 4294967296.0);
}

// ---- re-binning --------------------------------------------------------------------

// OrthorhombicBC::foldCoordinate + CellGrid::mapPositionToCellChecked/Clipped.  Bound by
// memory: positions and images go back only where a fold changed them (20.6 us, 16.3 without
// the other writes, at a million particles).
__global__ void k_fold_bin(DevView d, RebuildScratch s, int fold) {
  const ParticleArrays a = d.pa[0];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  int c[3];
  bool outside = false;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double x = a.x[(size_t)k * d.cap + i];
    if (fold) {
      double q = floor(__dmul_rn(x, d.invL[k]));
      if (!(fabs(q) < 1.0e9)) {
        outside = true;
        q = 0.0;
      }
      int tmp = (int)q;
      if (tmp != 0) {  // most particles are inside the box: nothing to write
        a.img[(size_t)k * d.cap + i] += tmp;
        x = __dsub_rn(x, __dmul_rn((double)tmp, d.L[k]));
        a.x[(size_t)k * d.cap + i] = x;
      }
    }
    double lpos = x;
    double t = __dmul_rn(lpos, d.invCellSize[k]);
    int ck = (t > -2.0e9 && t < 2.0e9) ? (int)t : (t > 0 ? d.nc[k] : -1);
    if (!(x == x)) {
      outside = true;
      ck = 0;
    }
    if (lpos < 0.0 && t <= -1.0) ck = -1;  // (int) truncates toward zero
    if (ck < 0) {
      if (fold && !(lpos >= -2.220446049250313e-16)) outside = true;
      ck = 0;
    } else if (ck >= d.nc[k]) {
      if (fold && !(x <= d.L[k] + 2.220446049250313e-16)) outside = true;
      ck = d.nc[k] - 1;
    }
    c[k] = ck;
  }
  if (outside) atomicOr(d.err, kErrOutside);
  int cell = c[0] + d.nc[0] * (c[1] + d.nc[1] * c[2]);
  s.cellOf[i] = cell;
  s.slot[i] = atomicAdd(&s.cellCount[cell], 1);
}

// Exclusive scan of the cell counts into cellStart: sums of tiles of cells, then each
// tile's scan behind the sum of the tiles before it (one tile: the second pass alone).  The
// counts are left zero for the next binning.
constexpr int kScanBlock = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanBlock * kScanItems;

__device__ __forceinline__ int block_exclusive_scan(int v, int* sm, int& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  if (lane == 31) sm[w] = x;
  __syncthreads();
  if (w == 0) {
    int y = lane < (int)(blockDim.x >> 5) ? sm[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += t;
    }
    sm[lane] = y;
  }
  __syncthreads();
  total = sm[(blockDim.x >> 5) - 1];
  const int excl = x - v + (w > 0 ? sm[w - 1] : 0);
  __syncthreads();
  return excl;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_tiles(const int32_t* __restrict__ count,
                                                            int n, int32_t* __restrict__ tile_sum) {
  __shared__ int sm[32];
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int v = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) v += (base + k < n) ? count[base + k] : 0;
  int total;
  block_exclusive_scan(v, sm, total);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_apply(int32_t* __restrict__ count, int n,
                                                            const int32_t* __restrict__ tile_sum,
                                                            int32_t* __restrict__ start) {
  __shared__ int sm[32];
  __shared__ int s_before;
  int before = 0;
  for (int t = threadIdx.x; t < (int)blockIdx.x; t += blockDim.x) before += tile_sum[t];
  int total;
  block_exclusive_scan(before, sm, total);
  if (threadIdx.x == 0) s_before = total;
  __syncthreads();
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int c[kScanItems];
  int v = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    c[k] = (base + k < n) ? count[base + k] : 0;
    if (base + k < n) count[base + k] = 0;
    v += c[k];
  }
  int run = block_exclusive_scan(v, sm, total) + s_before;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) start[base + k] = run;
    run += c[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) start[n] = run;
}

__global__ void k_scatter(DevView d, RebuildScratch s) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  s.perm[d.cellStart[s.cellOf[i]] + s.slot[i]] = i;
}

// Order inside a cell: by the Morton code of the particle's 8 x 8 x 8 sub-cell, then by
// id.  The layout is independent of the atomic arrival order above, and consecutive
// particles (the lanes of a force warp) sit close together, so their neighbour lists
// overlap and their coordinate gathers share cache lines.
__device__ __forceinline__ unsigned spread3(unsigned v) {  // bits b2 b1 b0 -> b2..b1..b0
  return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4);
}
__device__ __forceinline__ uint64_t in_cell_key(const DevView& d, const ParticleArrays& a, int v,
                                                const int (&cc)[3]) {
  unsigned q[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double f = (a.x[(size_t)i * d.cap + v] - cc[i] * d.cellSize[i]) * d.invCellSize[i];
    const int b = (int)(f * 8.0);
    q[i] = (unsigned)(b < 0 ? 0 : (b > 7 ? 7 : b));
  }
  // x in the most significant bit: a run of consecutive particles of one row of cells
  // (the Verlet build's groups) then spans a short range of x
  const uint64_t morton = spread3(q[2]) | (spread3(q[1]) << 1) | (spread3(q[0]) << 2);
  return (morton << 54) | (uint64_t)(a.id[v] - d.idMin);
}

// Row k of the other copy of the arrays from row o, with everything derived from a row:
// packed and cell-relative coordinates, cell, id map.
__device__ __forceinline__ void move_row(const DevView& d, const RebuildScratch& s,
                                         const ParticleArrays& src, const ParticleArrays& dst,
                                         int o, int k) {
  double p[3];
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    p[e] = src.x[(size_t)e * d.cap + o];
    dst.x[(size_t)e * d.cap + k] = p[e];
    dst.v[(size_t)e * d.cap + k] = src.v[(size_t)e * d.cap + o];
    dst.img[(size_t)e * d.cap + k] = src.img[(size_t)e * d.cap + o];
  }
  const int ty = src.type[o];
  const int64_t id = src.id[o];
  dst.id[k] = id;
  dst.type[k] = ty;
  dst.mass[k] = src.mass[o];
  const int cell = s.cellOf[o];
  d.pcell[k] = cell;
  d.posq[k] = fixed_coords(d, p[0], p[1], p[2], ty);
  const int cx = cell % d.nc[0], cy = (cell / d.nc[0]) % d.nc[1];
  const int cz = cell / (d.nc[0] * d.nc[1]);
  d.xrel[k] = make_float4((float)(p[0] - cx * d.cellSize[0]), (float)(p[1] - cy * d.cellSize[1]),
                          (float)(p[2] - cz * d.cellSize[2]), __int_as_float(cx));
  const int64_t off = id - d.idMin;
  if (off < 0 || off >= d.idSpan)
    atomicOr(d.err, kErrIdRange);
  else
    d.id2idx[off] = k;
}

// The last block to get here swaps the two copies of the arrays: every block has read their
// pointers by then.
__device__ __forceinline__ void swap_when_last(const DevView& d, const RebuildScratch& s,
                                               const ParticleArrays& src,
                                               const ParticleArrays& dst) {
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(s.ticket, 1u) == gridDim.x - 1) {
    *s.ticket = 0u;
    d.pa[0] = dst;
    d.pa[1] = src;
  }
}

// Sorts the cells of a block: LANES lanes a cell (a quarter warp where cells hold few
// particles) rank its particles by their keys in shared memory.  MOVE: the block's threads
// then take its rows, a contiguous run, one each, and move them: one launch in place of an
// in-cell sort, a gather, an id map and a swap, which is what a re-sort of a small system
// costs (7.5 us for 32,768 particles, 18 as four kernels).  Its registers and the sort's
// barrier leave a third of the threads in flight that a plain gather has, so large systems
// (kMoveApart) write the order and move in a kernel of its own (100 us fused, 82 apart at a
// million particles).  The ranking takes 8 us at 2,028 particles in 16 large cells, a serial
// insertion sort by one lane a cell 115.
constexpr int kSortThreads = 256;
constexpr int kSortKeys = 1024;  // particles of a block ranked in shared memory
constexpr int kMoveApart = 150000;

template <int LANES, bool MOVE>
__global__ void __launch_bounds__(kSortThreads) k_sort_cells(DevView d, RebuildScratch s) {
  constexpr int kCells = kSortThreads / LANES;
  __shared__ uint64_t s_key[kSortKeys];
  __shared__ int s_ord[kSortKeys];
  const ParticleArrays src = d.pa[0], dst = d.pa[1];
  const int w = threadIdx.x / LANES, lane = threadIdx.x % LANES;
  const int c0 = blockIdx.x * kCells, c = c0 + w;
  const int first = d.cellStart[c0], rows = d.cellStart[min(c0 + kCells, d.ncells)] - first;
  const int b = c < d.ncells ? d.cellStart[c] - first : 0;
  const int n = c < d.ncells ? d.cellStart[c + 1] - first - b : 0;
  const int cc[3] = {c % d.nc[0], (c / d.nc[0]) % d.nc[1], c / (d.nc[0] * d.nc[1])};
  const bool fits = rows <= kSortKeys;
  int* const perm = s.perm + first;
  if (fits) {
    for (int q = lane; q < n; q += LANES) s_key[b + q] = in_cell_key(d, src, perm[b + q], cc);
    __syncwarp();
    for (int q = lane; q < n; q += LANES) {
      const uint64_t key = s_key[b + q];
      int rank = 0;
      for (int m = 0; m < n; ++m) rank += s_key[b + m] < key;
      s_ord[b + rank] = perm[b + q];
    }
  } else if (lane == 0) {  // cells this full are sorted by insertion
    for (int k = b + 1; k < b + n; ++k) {
      const int v = perm[k];
      const uint64_t key = in_cell_key(d, src, v, cc);
      int m = k - 1;
      while (m >= b && in_cell_key(d, src, perm[m], cc) > key) {
        perm[m + 1] = perm[m];
        --m;
      }
      perm[m + 1] = v;
    }
  }
  __syncthreads();
  if (MOVE) {
    for (int q = threadIdx.x; q < rows; q += kSortThreads)
      move_row(d, s, src, dst, fits ? s_ord[q] : perm[q], first + q);
    swap_when_last(d, s, src, dst);
  } else if (fits) {
    for (int q = threadIdx.x; q < rows; q += kSortThreads) perm[q] = s_ord[q];
  }
}

__global__ void __launch_bounds__(kBlock, 5) k_move(DevView d, RebuildScratch s) {
  const ParticleArrays src = d.pa[0], dst = d.pa[1];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < d.n) move_row(d, s, src, dst, s.perm[k], k);
  swap_when_last(d, s, src, dst);
}

__global__ void k_posq(DevView d) {
  const ParticleArrays a = d.pa[0];
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.n) return;
  d.posq[k] = fixed_coords(d, a.x[k], a.x[(size_t)d.cap + k], a.x[2 * (size_t)d.cap + k],
                           a.type[k]);
}

// Cell-relative FP32 positions from the current coordinates and the cells of the last
// re-sort (a Verlet rebuild without re-binning, VerletList::rebuild on stale cells).
__global__ void k_xrel(DevView d) {
  const ParticleArrays a = d.pa[0];
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.n) return;
  const int cell = d.pcell[k];
  const int cx = cell % d.nc[0], cy = (cell / d.nc[0]) % d.nc[1], cz = cell / (d.nc[0] * d.nc[1]);
  d.xrel[k] = make_float4((float)(a.x[k] - cx * d.cellSize[0]),
                          (float)(a.x[(size_t)d.cap + k] - cy * d.cellSize[1]),
                          (float)(a.x[2 * (size_t)d.cap + k] - cz * d.cellSize[2]),
                          __int_as_float(cx));
}

// ---- Verlet list -------------------------------------------------------------------

// Both forms of the build test the candidates of a group of particles in FP32 on coordinates
// relative to the group's first cell, staged in shared memory ("chunks"), two candidates per
// packed f32x2 operation, every lane against its own particle.  Candidates within a band
// around (rc + skin)^2 (BuildBand) are decided, after the chunk's other partners, by the
// reference's FP64 arithmetic (exact_pair_test: d = p1 - (p2 + ghost shift),
// ((dx dx + dy dy) + dz dz), Particle.hpp:93-98, DomainDecomposition.cpp:1347-1391).  The pair
// set is therefore the reference's (VerletList.cpp:274-450), and each list is in a fixed
// order.  Lists are written in whole 32-byte sectors.
constexpr int kStageLd = 44;  // staging row: <= 7 carried + <= 32 appended; 11 x 16 B

// x-cells a group spans beyond its first one, at most: its candidate x-cells ca-h .. cb+h then
// number 32, and the FP32 coordinates stay small enough for a narrow band.
__host__ __device__ __forceinline__ int group_span(int h) { return 31 - 2 * h; }

// The FP32 test's band.  A coordinate of up to X (the edge of a group's frame) is rounded at
// most twice, the difference of two is off by at most 4 * 2^-24 X on an axis, and r^2 by
// (2 q + q^2) r^2 with q = 4 * 2^-24 |(X, Y, Z)| / r, besides 3e-7 r^2 of its own rounding.
// 2e-5 covers 31 cells as wide as the cutoff (1.5e-5); a frame of wider cells gets its own.
struct BuildBand {
  float lo, hi;   // FP32 decides outside
  float mid, hw;  // a chunk with a candidate this near to mid is looked through again
  float keepsq;   // squared distance from the group's bounding box beyond which none is a partner
};
BuildBand build_band(const DevView& d, double cutsq) {
  const int h = d.hci;
  const double X = (std::min(group_span(h), d.nc[0] - 1) + h + 1) * d.cellSize[0];
  const double Y = (h + 1) * d.cellSize[1], Z = (h + 1) * d.cellSize[2];
  const double q = 2.4e-7 * sqrt((X * X + Y * Y + Z * Z) / cutsq);
  const double eps = std::max(2e-5, 3e-7 + q * (2.0 + q));
  return {(float)(cutsq * (1.0 - eps)), (float)(cutsq * (1.0 + eps)), (float)cutsq,
          (float)(cutsq * (1.5 * eps)), (float)(cutsq * (1.0 + 5.0 * eps))};
}

// Fast tests of one chunk (nv valid candidates) against the lane's particle.  Returns
// whether any candidate came near the cutoff (a superset of the borderline band).
// STENCIL: candidate m counts only when its x-cell offset c.xo[m] lies within h cells of
// the lane's own (rel, relative to the same origin): the reference's neighbour cells when
// particles may have left the cells of the last re-sort.
template <bool SELF, bool EXCL, class Chunk, bool STENCIL = false>
__device__ __forceinline__ bool chunk_scan(const DevView& d, const Chunk& c, int nv,
                                           unsigned long long xi2, unsigned long long yi2,
                                           unsigned long long zi2, int i, int64_t idi,
                                           float lo, unsigned long long mid2, float hw,
                                           int* __restrict__ srow, int& pend, int rel = 0,
                                           int h = 1) {
  bool band = false;
#pragma unroll
  for (int m = 0; m < 32; m += 2) {
    if (m >= nv) break;
    const unsigned long long cx = *reinterpret_cast<const unsigned long long*>(&c.x[m]);
    const unsigned long long cy = *reinterpret_cast<const unsigned long long*>(&c.y[m]);
    const unsigned long long cz = *reinterpret_cast<const unsigned long long*>(&c.z[m]);
    const int2 jj = *reinterpret_cast<const int2*>(&c.j[m]);
    const unsigned long long dx = f2_sub(xi2, cx), dy = f2_sub(yi2, cy), dz = f2_sub(zi2, cz);
    const unsigned long long r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
    const unsigned long long t = f2_sub(r2, mid2);
    band |= (fabsf(f2_lo(t)) <= hw) | (fabsf(f2_hi(t)) <= hw);
    bool ina = f2_lo(r2) < lo, inb = f2_hi(r2) < lo;
    if (SELF) {
      ina &= jj.x != i;
      inb &= jj.y != i;
    }
    if constexpr (STENCIL) {
      const int2 xo = *reinterpret_cast<const int2*>(&c.xo[m]);
      ina &= (unsigned)(xo.x - rel + h) <= (unsigned)(2 * h);
      inb &= (unsigned)(xo.y - rel + h) <= (unsigned)(2 * h);
    }
    if (EXCL) {
      if (ina && is_excluded(d, idi, c.id[m])) ina = false;
      if (inb && is_excluded(d, idi, c.id[m + 1])) inb = false;
    }
    if (ina) srow[pend++] = jj.x;
    if (inb) srow[pend++] = jj.y;
  }
  return band;
}

// Writes the lane's full blocks of 8 to its list and keeps the remainder in front.
__device__ __forceinline__ void stage_flush(int* __restrict__ srow, int& pend, int& blk,
                                            int* __restrict__ nl, int i, size_t cap, int kb) {
  const int nb = pend >> 3;
  if (nb == 0) return;
  for (int b = 0; b < nb; ++b, ++blk) {
    const int4 v0 = *reinterpret_cast<const int4*>(&srow[8 * b]);
    const int4 v1 = *reinterpret_cast<const int4*>(&srow[8 * b + 4]);
    if (blk < kb) {
      int4* dst = reinterpret_cast<int4*>(nl + nl_index(8 * blk, i, cap));
      dst[0] = v0;
      dst[1] = v1;
    }
  }
  const int rem = pend & 7;
  for (int k = 0; k < rem; ++k) srow[k] = srow[8 * nb + k];
  pend = rem;
}

// ---- Verlet build, run form ---------------------------------------------------------
// One warp per 32 consecutive sorted particles, split where they change row of cells
// (cy, cz) or would span too many x-cells (group_span); lane l holds particle g + l.  A group
// spans the x-cells ca..cb of one row; its candidates are the particles of x-cells ca-h .. cb+h
// of the (2h+1)^2 rows around (cy, cz), staged in the frame of cell (ca, cy, cz).  A candidate
// farther than the cutoff from the bounding box of the group's particles cannot be a partner
// of any of them and is dropped before it takes a slot of a chunk (ballot + prefix count), so
// the 32 lanes test only survivors and no lane idles for lack of particles.
// A candidate of a farther cell (a group spans several x-cells) neither passes the test nor
// comes near the cutoff where the particles were binned at their current positions in cells
// whose edges all exceed the list cutoff by 0.1 %; elsewhere (STALE) each particle's own
// neighbour cells are enforced.
constexpr int kRunWarps = 4;

struct RunChunk {  // 64 slots: a scan takes 32, the rest waits for the next
  float x[64], y[64], z[64];
  int j[64];
  int xo[64];  // x-cell of the candidate, relative to ca
  int64_t id[64];
};

__device__ __forceinline__ float warp_fmin(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_fmax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

struct RunShared {  // one warp's
  __align__(16) int stage[32 * kStageLd];
  RunChunk chunk;
  int pre[33];  // prefix of the candidate x-cells' counts
  int st[32];   // their first sorted index
};

// Lists of the particles g + lane of the lanes in todo, by one warp.
template <bool EXCL, bool STALE>
__device__ __forceinline__ void build_run(const DevView& d, double cutsq, const BuildBand& limits,
                                          int g, unsigned todo, RunShared& sh) {
  const ParticleArrays a = d.pa[0];
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu;
  const float lo = limits.lo, hi = limits.hi, hw = limits.hw, keepsq = limits.keepsq;
  const unsigned long long mid2 = f2_pack(limits.mid, limits.mid);
  const float hx = (float)d.cellSize[0], hy = (float)d.cellSize[1], hz = (float)d.cellSize[2];
  const int nx = d.nc[0], ny = d.nc[1], nz = d.nc[2];
  const int h = d.hci, sw = 2 * h + 1;  // stencil reach and width (halfCellInt)
  const int span = group_span(h);
  const float4* __restrict__ xr = d.xrel;
  const int K = d.K;
  const size_t cap = d.cap;
  int* __restrict__ nl = d.nl;
  RunChunk& ch = sh.chunk;
  int* __restrict__ srow = &sh.stage[lane * kStageLd];
  const int ip = g + lane;
  const int mcell = (todo >> lane) & 1u ? d.pcell[ip] : 0;
  const int mcx = mcell % nx, mrow = mcell / nx;
  while (todo) {
    const int leader = __ffs(todo) - 1;
    const int row = __shfl_sync(full, mrow, leader);
    const int ca = __shfl_sync(full, mcx, leader);
    const unsigned grp = __ballot_sync(full, ((todo >> lane) & 1u) && mrow == row &&
                                                 mcx - ca <= span);
    todo &= ~grp;
    const bool own = (grp >> lane) & 1u;
    const int cb = __shfl_sync(full, mcx, 31 - __clz(grp));
    const int cy = row % ny, cz = row / ny;
    const int i = own ? ip : g + leader;
    // the lane's particle in the frame of cell (ca, cy, cz); lanes outside the group far away
    float fx = 1e18f, fy = 1e18f, fz = 1e18f;
    if (own) {
      const float4 r = xr[ip];
      fx = r.x + (float)(mcx - ca) * hx;
      fy = r.y;
      fz = r.z;
    }
    const float bxl = warp_fmin(own ? fx : 3e38f), bxh = warp_fmax(own ? fx : -3e38f);
    const float byl = warp_fmin(own ? fy : 3e38f), byh = warp_fmax(own ? fy : -3e38f);
    const float bzl = warp_fmin(own ? fz : 3e38f), bzh = warp_fmax(own ? fz : -3e38f);
    const unsigned long long xi2 = f2_pack(fx, fx), yi2 = f2_pack(fy, fy), zi2 = f2_pack(fz, fz);
    const int64_t idi = (EXCL && own) ? a.id[ip] : -3;
    const int nxs = cb - ca + sw;  // candidate x-cells ca-h .. cb+h
    int pend = 0, blk = 0;
    for (int rr = 0; rr < sw * sw; ++rr) {
      const int oz = rr / sw - h, oy = rr % sw - h;
      const int ncy = cy + oy, ncz = cz + oz;
      const int wcy = ncy < 0 ? ncy + ny : (ncy >= ny ? ncy - ny : ncy);
      const int wcz = ncz < 0 ? ncz + nz : (ncz >= nz ? ncz - nz : ncz);
      const int rb = nx * (wcy + ny * wcz);
      {
        int st = 0, ct = 0;
        if (lane < nxs) {
          int xc = ca - h + lane;
          xc += xc < 0 ? nx : (xc >= nx ? -nx : 0);
          st = d.cellStart[rb + xc];
          ct = d.cellStart[rb + xc + 1] - st;
        }
        int pre = ct;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(full, pre, o);
          if (lane >= o) pre += t;
        }
        sh.st[lane] = st;
        sh.pre[lane + 1] = pre;
        if (lane == 0) sh.pre[0] = 0;
      }
      __syncwarp();
      const int nrow = sh.pre[nxs];
      const float ofy = (float)oy * hy, ofz = (float)oz * hz;
      int fill = 0;
      for (int cb0 = 0; cb0 < nrow; cb0 += 32) {
        const int t = cb0 + lane;
        bool keep = false;
        float cx = 0.f, cy2 = 0.f, cz2 = 0.f;
        int j = 0, k = 0;
        if (t < nrow) {
          while (sh.pre[k + 1] <= t) ++k;
          j = sh.st[k] + (t - sh.pre[k]);
          const float4 rj = xr[j];
          cx = rj.x + (float)(k - h) * hx;
          cy2 = rj.y + ofy;
          cz2 = rj.z + ofz;
          const float ex = fmaxf(0.f, fmaxf(bxl - cx, cx - bxh));
          const float ey = fmaxf(0.f, fmaxf(byl - cy2, cy2 - byh));
          const float ez = fmaxf(0.f, fmaxf(bzl - cz2, cz2 - bzh));
          keep = fmaf(ez, ez, fmaf(ey, ey, ex * ex)) <= keepsq;
        }
        const unsigned km = __ballot_sync(full, keep);
        if (keep) {
          const int pos = fill + __popc(km & ((1u << lane) - 1u));
          ch.x[pos] = cx;
          ch.y[pos] = cy2;
          ch.z[pos] = cz2;
          ch.j[pos] = j;
          ch.xo[pos] = k - h;
          if (EXCL) ch.id[pos] = a.id[j];
        }
        fill += __popc(km);
        const bool last = cb0 + 32 >= nrow;
        while (fill >= 32 || (last && fill > 0)) {
          const int nv = min(fill, 32);
          // the scan reads candidates in pairs: an odd count gets a far-away partner slot
          if ((nv & 1) && lane == 0) {
            ch.x[nv] = ch.y[nv] = ch.z[nv] = -1e18f;
            ch.j[nv] = -1;
            if (EXCL) ch.id[nv] = -2;
          }
          __syncwarp();
          const bool self = oy == 0 && oz == 0;
          const bool band =
              self ? chunk_scan<true, EXCL, RunChunk, STALE>(d, ch, nv, xi2, yi2, zi2, i, idi, lo,
                                                             mid2, hw, srow, pend, mcx - ca, h)
                   : chunk_scan<false, EXCL, RunChunk, STALE>(d, ch, nv, xi2, yi2, zi2, i, idi,
                                                              lo, mid2, hw, srow, pend, mcx - ca,
                                                              h);
          if (__builtin_expect(__any_sync(full, band), 0) && own) {
            // borderline candidates of this chunk: the reference's FP64 test decides
            const int wy = ncy < 0 ? -1 : (ncy >= ny ? 1 : 0);
            const int wz = ncz < 0 ? -1 : (ncz >= nz ? 1 : 0);
            for (int m = 0; m < nv; ++m) {
              const unsigned long long dx = f2_sub(xi2, f2_pack(ch.x[m], ch.x[m]));
              const unsigned long long dy = f2_sub(yi2, f2_pack(ch.y[m], ch.y[m]));
              const unsigned long long dz = f2_sub(zi2, f2_pack(ch.z[m], ch.z[m]));
              const float r2 = f2_lo(f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx))));
              const int jm = ch.j[m];
              if (!(r2 >= lo && r2 <= hi) || jm == i) continue;
              const int xu = ca + ch.xo[m];  // the candidate's x-cell, unwrapped
              const int ox = xu - mcx;
              if (ox < -h || ox > h) continue;  // not a neighbour cell of this particle
              const int wx = xu < 0 ? -1 : (xu >= nx ? 1 : 0);
              const bool fwd = oz > 0 || (oz == 0 && (oy > 0 || (oy == 0 && ox > 0)));
              bool in = exact_pair_test(a.x, d.cap, i, jm, fwd, wx * d.L[0], wy * d.L[1],
                                        wz * d.L[2], cutsq);
              if (EXCL && in && is_excluded(d, idi, ch.id[m])) in = false;
              if (in) srow[pend++] = jm;
            }
          }
          stage_flush(srow, pend, blk, nl, i, cap, K >> 3);
          __syncwarp();
          // slots 32 .. fill-1 move to the front
          if (lane < fill - 32) {
            const int sidx = 32 + lane;
            ch.x[lane] = ch.x[sidx];
            ch.y[lane] = ch.y[sidx];
            ch.z[lane] = ch.z[sidx];
            ch.j[lane] = ch.j[sidx];
            ch.xo[lane] = ch.xo[sidx];
            if (EXCL) ch.id[lane] = ch.id[sidx];
          }
          fill -= nv;
          __syncwarp();
        }
      }
      __syncwarp();
    }
    const int total = blk * 8 + pend;
    if (own) {
      if (total > K) atomicOr(d.err, kErrNlOverflow);
      d.nn[i] = min(total, K);
      if (pend > 0) {
        for (int k = pend; k < 8; ++k) srow[k] = i;
        pend = 8;
        stage_flush(srow, pend, blk, nl, i, cap, K >> 3);
      }
    }
    const int wmax = __reduce_max_sync(full, own ? total : 0);
    if (lane == 0 && wmax > 0) atomicMax(&d.ctr->nnMax, wmax);
    __syncwarp();
  }
}

template <bool EXCL, bool STALE>
__global__ void __launch_bounds__(kRunWarps * 32) k_build_nl_run(DevView d, double cutsq,
                                                                 BuildBand limits) {
  __shared__ RunShared s_run[kRunWarps];
  const int g = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32;
  if (g >= d.n) return;
  const unsigned valid = __ballot_sync(0xffffffffu, g + (int)(threadIdx.x & 31) < d.n);
  build_run<EXCL, STALE>(d, cutsq, limits, g, valid, s_run[threadIdx.x >> 5]);
}

// ---- Verlet build, block form --------------------------------------------------------
// The run form with four warps on one run of 32 particles: lane l of every warp holds
// particle g + l, and the (2h+1)^2 rows of candidate cells are shared out among the warps
// (block_row_owner).  A row's candidates are contiguous in the sorted order but for the
// periodic wrap, so a warp streams them without a search and loads the next 32 while it tests
// the last; it compacts the survivors of the bounding-box test over all its rows before it
// scans them, keeps its partners in its own stage (transposed: entry-major, no bank conflicts)
// and the block writes the lists once, in whole blocks of 8.
// A warp alone spends about 7 cycles an instruction on this work, so a run handled by one
// warp lasts 60 us however few particles there are.  Run form / this one: 71 / 18 us at 2,028
// particles, 69 / 32 at 32,768, 163 / 129 at 241,133, 540 / 479 at a million, 2.02 / 1.88 ms at
// 4,096,000 (issue bound in both: about 320 instructions a particle here), 48 / 28 at a
// 40,000-bead melt.
constexpr int kBlockW = 4;  // warps a run
// Particles up to which two blocks share a run (SPLIT).  One block a run / two: 22 / 18 us at
// 2,028, 34 / 32 at 32,768, 129 / 135 at 241,133, 1.88 / 2.07 ms at 4,096,000.
constexpr int kBuildSplit = 100000;
// List capacity up to which the block form is used.  The capacity is 1.6 times the length
// expected from the density, and 32 more.  Run form / block form in a liquid: 81 / 36 us
// at 32,768 particles and 191 / 145 at 238,328 with lists of 100 entries (capacity 200), 90 /
// 90 and 201 / 171 with 114 (216), 110 / 110 and 242 / 243 with 150 (272; the system has
// changed to the run form).
constexpr int kBlockListMax = 224;

// Warp that takes row rr of the (2h+1)^2 rows, and its stage in entries.  One cell layer: the
// centre row, with 29 of an LJ particle's 78 partners on average and 46 at most (counted on
// 262,144 particles; about 60 where few cells make each a third wider), alone; opposite face
// rows together (19, at most 37: a particle near one is far from the other); the four corner
// rows together (10, at most 30).  With 6 blocks an SM, 240 entries a lane fill its shared
// memory.  Uneven densities and h > 1 share the rows out less evenly: a run with a warp whose
// partners outgrow its stage is built again by one warp in the run form.  A system with many
// such runs changes to that form (note_rebuilt_runs).
__device__ __forceinline__ int block_row_owner(int rr, int h) {
  return h > 1 ? rr % kBlockW : (int)((0x313202313ull >> (4 * rr)) & 15ull);
}
__host__ __device__ constexpr int block_stage_start(int w) {
  return w == 0 ? 0 : (w == 1 ? 76 : (w == 2 ? 134 : (w == 3 ? 192 : 240)));
}

struct BlockWarp {
  ulonglong2 a[32], b[32];  // candidate pairs: x0 x1, y0 y1; z0 z1, j0 j1
  int code[64];             // x-cell relative to ca << 8 | row of cells
};

// Appends j at shared address `at` when r2 < lo (and j is not the particle itself): the store
// is unconditional, only the advance is predicated, so a candidate costs three instructions
// and no branch; a slot behind the last entry holds the last candidate that was no partner.
template <bool SELF>
__device__ __forceinline__ void stage_append(uint32_t& at, int j, float r2, float lo, int ip) {
  if (SELF)
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.s32 q, %1, %4;\n\tsetp.lt.and.f32 p, %2, %3, q;\n\t"
        "st.shared.b32 [%0], %1;\n\t@p add.u32 %0, %0, 128;\n\t}"
        : "+r"(at)
        : "r"(j), "f"(r2), "f"(lo), "r"(ip)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %2, %3;\n\t"
        "st.shared.b32 [%0], %1;\n\t@p add.u32 %0, %0, 128;\n\t}"
        : "+r"(at)
        : "r"(j), "f"(r2), "f"(lo)
        : "memory");
}

// A block whose stages do not hold its lists: one warp builds them in the run form.
template <bool EXCL, bool STENCIL>
__device__ __noinline__ void rebuild_run(const DevView& d, double cutsq, const BuildBand& limits,
                                         int g, unsigned todo, int* shared) {
  build_run<EXCL, STENCIL>(d, cutsq, limits, g, todo, *reinterpret_cast<RunShared*>(shared));
}

// SPLIT: a run of several groups (row changes, or many x-cells) is shared by two blocks, one
// for the first of its groups, one (in the second half of the grid) for the others.  Where all
// blocks are resident at once the kernel lasts as long as its slowest block, and a block of two
// groups takes twice the time of one; a large grid only pays for the extra blocks.
template <bool EXCL, bool STENCIL, bool SPLIT>
__global__ void __launch_bounds__(32 * kBlockW, 6)
    k_build_block(const __grid_constant__ DevView d, double cutsq,
                  const __grid_constant__ BuildBand limits) {
  const ParticleArrays a = d.pa[0];
  constexpr int W = kBlockW;
  __shared__ __align__(16) BlockWarp s_w[W];
  __shared__ __align__(16) int s_stage[block_stage_start(W) * 32];
  static_assert(sizeof(RunShared) <= sizeof(s_stage), "the run form works in the stages");
  __shared__ int s_cnt[W][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool second = SPLIT && blockIdx.x >= gridDim.x / 2;
  const int g = (SPLIT ? (int)(blockIdx.x - (second ? gridDim.x / 2 : 0)) : (int)blockIdx.x) * 32;
  const unsigned full = 0xffffffffu;
  const float lo = limits.lo, hi = limits.hi, hw = limits.hw, keepsq = limits.keepsq;
  const unsigned long long mid2 = f2_pack(limits.mid, limits.mid);
  const float hx = (float)d.cellSize[0], hy = (float)d.cellSize[1], hz = (float)d.cellSize[2];
  const int nx = d.nc[0], ny = d.nc[1], nz = d.nc[2];
  const int h = d.hci, sw = 2 * h + 1, span = group_span(h);
  const float4* __restrict__ xr = d.xrel;
  BlockWarp& sm = s_w[w];
  float* const sa = reinterpret_cast<float*>(sm.a);
  float* const sb = reinterpret_cast<float*>(sm.b);
  const int ip = g + lane;
  const bool valid = ip < d.n;
  const float4 me = valid ? xr[ip] : make_float4(0.f, 0.f, 0.f, 0.f);
  const int mcx = __float_as_int(me.w);
  const int mrow = valid ? d.pcell[ip] - mcx : 0;  // first cell of the particle's row of cells
  const int64_t idi = (EXCL && valid) ? a.id[ip] : -3;
  const bool mayself = h > 1 || w == 0;  // the warp's rows hold the particles themselves
  // shared addresses of the lane's stage, 128 bytes an entry: first, next, and the last next
  // that leaves room for the 8 candidates tested between two checks
  const uint32_t st0 =
      (uint32_t)__cvta_generic_to_shared(s_stage + 32 * block_stage_start(w) + lane);
  const uint32_t stLast = st0 + 128u * (block_stage_start(w + 1) - block_stage_start(w) - 8);
  uint32_t at = st0;
  unsigned todo = __ballot_sync(full, valid), mine = todo;
  bool skip = second;  // the first group is the other block's
  while (todo) {
    const int leader = __ffs(todo) - 1;
    const int row = __shfl_sync(full, mrow, leader);
    const int ca = __shfl_sync(full, mcx, leader);
    const unsigned grp =
        __ballot_sync(full, ((todo >> lane) & 1u) && mrow == row && mcx - ca <= span);
    todo &= ~grp;
    if (SPLIT) {
      if (skip) {
        skip = false;
        mine &= ~grp;
        continue;
      }
      if (!second) {
        todo = 0u;
        mine = grp;
      }
    }
    const bool own = (grp >> lane) & 1u;
    const int cb = __shfl_sync(full, mcx, 31 - __clz(grp));
    const int rowOf = row / nx, cz = rowOf / ny, cy = rowOf - cz * ny;
    const int rel = mcx - ca;
    // the lane's particle in the frame of cell (ca, cy, cz); lanes outside the group far away
    const float fx = own ? me.x + (float)rel * hx : 1e18f;
    const float fy = own ? me.y : 1e18f, fz = own ? me.z : 1e18f;
    const float bxl = warp_fmin(own ? fx : 3e38f), bxh = warp_fmax(own ? fx : -3e38f);
    const float byl = warp_fmin(own ? fy : 3e38f), byh = warp_fmax(own ? fy : -3e38f);
    const float bzl = warp_fmin(own ? fz : 3e38f), bzh = warp_fmax(own ? fz : -3e38f);
    const unsigned long long xi2 = f2_pack(fx, fx), yi2 = f2_pack(fy, fy), zi2 = f2_pack(fz, fz);

    // tests the first nv candidates of the chunk (filled up to a multiple of 8) against the
    // lane's particle
    auto scan = [&](int nv, auto self) {
      float near = 3e38f;  // smallest |r^2 - cutoff^2|
      for (int m0 = 0; m0 < nv; m0 += 8) {
        // all loads before the first append: a store to the stage keeps later loads behind it
        ulonglong2 A[4], B[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          A[p] = sm.a[(m0 >> 1) + p];
          B[p] = sm.b[(m0 >> 1) + p];
        }
        unsigned long long r2p[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const unsigned long long dx = f2_sub(xi2, A[p].x), dy = f2_sub(yi2, A[p].y);
          const unsigned long long dz = f2_sub(zi2, B[p].x);
          r2p[p] = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
          const unsigned long long t = f2_sub(r2p[p], mid2);
          near = fminf(fminf(near, fabsf(f2_lo(t))), fabsf(f2_hi(t)));
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const unsigned long long r2 = r2p[p];
          const int ja = (int)(unsigned)B[p].y, jb = (int)(B[p].y >> 32);
          if constexpr (!EXCL && !STENCIL) {
            stage_append<decltype(self)::value>(at, ja, f2_lo(r2), lo, ip);
            stage_append<decltype(self)::value>(at, jb, f2_hi(r2), lo, ip);
          } else {
            bool ina = f2_lo(r2) < lo && ja != ip, inb = f2_hi(r2) < lo && jb != ip;
            if (STENCIL) {
              const int2 c = *reinterpret_cast<const int2*>(&sm.code[m0 + 2 * p]);
              ina &= (unsigned)((c.x >> 8) - rel + h) <= (unsigned)(2 * h);
              inb &= (unsigned)((c.y >> 8) - rel + h) <= (unsigned)(2 * h);
            }
            if (EXCL) {
              if (ina && is_excluded(d, idi, a.id[ja])) ina = false;
              if (inb && is_excluded(d, idi, a.id[jb])) inb = false;
            }
            stage_append<false>(at, ja, ina ? 0.f : 1.f, 0.5f, ip);
            stage_append<false>(at, jb, inb ? 0.f : 1.f, 0.5f, ip);
          }
        }
        at = min(at, stLast);
      }
      if (__builtin_expect(__any_sync(full, near <= hw), 0) && own && near <= hw) {
        // borderline candidates of this chunk: the reference's FP64 test decides
        for (int m = 0; m < nv; ++m) {
          const int q = 4 * (m >> 1) + (m & 1);
          const float x = sa[q], y = sa[q + 2], z = sb[q];
          const unsigned long long dx = f2_sub(xi2, f2_pack(x, x));
          const unsigned long long dy = f2_sub(yi2, f2_pack(y, y));
          const unsigned long long dz = f2_sub(zi2, f2_pack(z, z));
          const float r2 = f2_lo(f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx))));
          const int j = __float_as_int(sb[q + 2]), code = sm.code[m];
          if (!(r2 >= lo && r2 <= hi) || j == ip) continue;
          const int oz = (code & 255) / sw - h, oy = (code & 255) % sw - h;
          const int xu = ca + (code >> 8);  // the candidate's x-cell, unwrapped
          const int ox = xu - mcx;
          if (ox < -h || ox > h) continue;  // not a neighbour cell of this particle
          const int wx = xu < 0 ? -1 : (xu >= nx ? 1 : 0);
          const int wy = cy + oy < 0 ? -1 : (cy + oy >= ny ? 1 : 0);
          const int wz = cz + oz < 0 ? -1 : (cz + oz >= nz ? 1 : 0);
          const bool fwd = oz > 0 || (oz == 0 && (oy > 0 || (oy == 0 && ox > 0)));
          bool in = exact_pair_test(a.x, d.cap, ip, j, fwd, wx * d.L[0], wy * d.L[1],
                                    wz * d.L[2], cutsq);
          if (EXCL && in && is_excluded(d, idi, a.id[j])) in = false;
          if (in && at < stLast) stage_append<false>(at, j, 0.f, 1.f, ip);
        }
      }
    };

    // Segments: the candidates of a row of cells below, inside and above the box, each a
    // contiguous run of sorted particles; one lane looks up each.
    int fill = 0;
    const int nseg = 3 * sw * sw;
    for (int seg0 = 0; seg0 < nseg; seg0 += 32) {
      const int sg = seg0 + lane, rr = sg / 3, p = sg % 3 - 1;
      int js = 0, je = 0, code = 0;  // code: x shift of the frame, row, oz + h, oy + h
      if (sg < nseg) {
        const int oz1 = h == 1 ? rr / 3 : rr / sw, oy1 = rr - oz1 * sw;
        const int xs = max(ca - h, p * nx), xe = min(cb + h, p * nx + nx - 1);
        if (block_row_owner(rr, h) == w && xs <= xe) {
          const int ncy = cy + oy1 - h, ncz = cz + oz1 - h;
          const int wcy = ncy < 0 ? ncy + ny : (ncy >= ny ? ncy - ny : ncy);
          const int wcz = ncz < 0 ? ncz + nz : (ncz >= nz ? ncz - nz : ncz);
          const int rb = nx * (wcy + ny * wcz) - p * nx;
          js = d.cellStart[rb + xs];
          je = d.cellStart[rb + xe + 1];
          code = (p + 1) << 24 | rr << 16 | oz1 << 8 | oy1;
        }
      }
      unsigned segs = __ballot_sync(full, js < je);
      // the next round's candidates are loaded before this round's are filtered and scanned
      int nj = 0, ne = 0, nbase = 0, nrr = 0;  // next round: first, end, x shift, row
      float nofy = 0.f, nofz = 0.f;
      float4 nxt = make_float4(0.f, 0.f, 0.f, 0.f);
      auto load_round = [&](bool advance) {
        if (advance) {
          nj = ne = 0;
          if (segs) {
            const int src = __ffs(segs) - 1;
            segs &= segs - 1;
            nj = __shfl_sync(full, js, src);
            ne = __shfl_sync(full, je, src);
            const int c = __shfl_sync(full, code, src);
            nbase = ((c >> 24) - 1) * nx - ca;
            nrr = (c >> 16) & 255;
            nofz = (float)(((c >> 8) & 255) - h) * hz;
            nofy = (float)((c & 255) - h) * hy;
          }
        }
        if (nj + lane < ne) nxt = xr[nj + lane];
      };
      load_round(true);
      while (nj < ne) {
        const int cj = nj, ce = ne, cbase = nbase, crr = nrr;
        const float ofy = nofy, ofz = nofz;
        const float4 rj = nxt;
        nj += 32;
        load_round(nj >= ne);
        const int j = cj + lane;
        const int xo = __float_as_int(rj.w) + cbase;  // x-cell relative to ca
        const float cx = rj.x + (float)xo * hx, cyf = rj.y + ofy, czf = rj.z + ofz;
        const float ex = fmaxf(0.f, fmaxf(bxl - cx, cx - bxh));
        const float ey = fmaxf(0.f, fmaxf(byl - cyf, cyf - byh));
        const float ez = fmaxf(0.f, fmaxf(bzl - czf, czf - bzh));
        const bool keep = j < ce && fmaf(ez, ez, fmaf(ey, ey, ex * ex)) <= keepsq;
        const unsigned km = __ballot_sync(full, keep);
        if (keep) {
          const int pos = fill + __popc(km & ((1u << lane) - 1u));
          const int q = 4 * (pos >> 1) + (pos & 1);
          sa[q] = cx;
          sa[q + 2] = cyf;
          sb[q] = czf;
          sb[q + 2] = __int_as_float(j);
          sm.code[pos] = xo * 256 + crr;
        }
        fill += __popc(km);
        if (fill >= 32) {
          __syncwarp();
          if (mayself)
            scan(32, std::true_type{});
          else
            scan(32, std::false_type{});
          __syncwarp();
          // slots 32 .. fill-1 move to the front
          if (lane < (fill - 31) >> 1) {
            sm.a[lane] = sm.a[16 + lane];
            sm.b[lane] = sm.b[16 + lane];
          }
          if (lane < fill - 32) sm.code[lane] = sm.code[32 + lane];
          fill -= 32;
          __syncwarp();
        }
      }
    }
    if (fill > 0) {
      // far-away candidates fill the last 8
      const int pos = fill + lane;
      if (pos < ((fill + 7) & ~7)) {
        const int q = 4 * (pos >> 1) + (pos & 1);
        sa[q] = sa[q + 2] = sb[q] = -1e18f;
        sb[q + 2] = __int_as_float(-1);
        sm.code[pos] = 0;
      }
      __syncwarp();
      if (mayself)
        scan(fill, std::true_type{});
      else
        scan(fill, std::false_type{});
      __syncwarp();
    }
  }
  if (SPLIT && mine == 0u) return;  // the whole block: a run of one group
  const bool write = (mine >> lane) & 1u;
  s_cnt[w][lane] = (int)(at - st0) >> 7;
  if (__syncthreads_or(at == stLast)) {  // a stage without room left
    if (threadIdx.x == 0) atomicAdd((unsigned long long*)&d.ctr->rebuilt, 1ull);
    if (w == 0) rebuild_run<EXCL, STENCIL>(d, cutsq, limits, g, mine, s_stage);
    return;
  }
  // the lists: thread (w, lane) writes the blocks w, w + W, ... of particle g + lane
  int pre[W + 1], base[W];  // base: where entry k of the list would lie in warp u's stage
  pre[0] = 0;
#pragma unroll
  for (int u = 0; u < W; ++u) {
    pre[u + 1] = pre[u] + s_cnt[u][lane];
    base[u] = block_stage_start(u) - pre[u];
  }
  const int total = pre[W], K = d.K;
  if (write) {
    if (w == 0) {
      d.nn[ip] = min(total, K);
      if (total > K) atomicOr(d.err, kErrNlOverflow);
    }
    const int fit = min(total, K);
    for (int b = w; 8 * b < fit; b += W) {
      // padded to a multiple of 8 with the particle itself (r^2 = 0, masked by the force
      // kernels) so that blocks of 8 need no bounds checks; K is a multiple of 8
      int v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int k = 8 * b + e;
        int at = base[0];
#pragma unroll
        for (int u = 1; u < W; ++u) at = k >= pre[u] ? base[u] : at;
        v[e] = k < total ? s_stage[32 * (at + k) + lane] : ip;
      }
      int4* dst = reinterpret_cast<int4*>(d.nl + nl_index(8 * b, ip, d.cap));
      dst[0] = make_int4(v[0], v[1], v[2], v[3]);
      dst[1] = make_int4(v[4], v[5], v[6], v[7]);
    }
  }
  if (w == 0) {
    const int wmax = __reduce_max_sync(full, write ? total : 0);
    if (lane == 0 && wmax > 0) atomicMax(&d.ctr->nnMax, wmax);
  }
}

// ---- forces ------------------------------------------------------------------------

// Loads of arrays that other blocks write during the kernel (LIVE) go through the coherent
// path, others through the read-only one.
template <bool LIVE>
__device__ __forceinline__ int4 ld_pos(const int4* p) {
  if (!LIVE) return __ldg(p);
  int4 v;
  asm volatile("ld.global.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
template <bool LIVE>
__device__ __forceinline__ double ld_pos(const double* p) {
  if (!LIVE) return __ldg(p);
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}

// FP32 pair forces on box-wrapped int32 coordinates, T lanes a particle.  The minimum image
// is the 32-bit wrap of the coordinate difference.  Two entries are evaluated at once in the
// halves of packed f32x2 registers (20 instructions an entry, 31 scalar).  FP32 sums along
// the list, one for each half and, with one lane, two such pairs in turn, so that no FP32 sum
// is longer than about 40 entries of a liquid's 78; each sum, the lanes' and the bond terms are
// combined in int64 2^-32 fixed point, so the result does not depend on the order in which
// they are added.  Every lane of the warp takes part (act: the lane has a particle).
// Bound by the L1 data pipe: the 32 coordinates a warp gathers lie in 10 to 18 lines, 88 to 95 %
// of the pipe's wavefronts at a million particles, issue 39 % (53 % scalar).  With ListShare
// the lanes of a particle take adjacent entries, which share lines.  40 us at 241,133 particles
// of two types (two lanes; 44 with the lanes on blocks of their own), 9.2 at 32,768, 495 at
// 4,096,000 with one lane.  One lane runs three blocks an SM: with four, the second pair of
// sums spills (526 us).
template <int T, bool SINGLE, bool CAPPED, bool FENE, bool LIVE, class Share>
__device__ __forceinline__ void particle_force_mixed(const DevView& d, const FENEParams& fp,
                                                     const LJPairF* sP, const int4* posq, int i,
                                                     int sub, bool act, const Share& share,
                                                     long long (&F)[3]) {
  const ParticleArrays a = d.pa[0];
  const int4 pi = ld_pos<LIVE>(&posq[i]);
  const unsigned long long ux = f2_pack(d.fixUnit[0], d.fixUnit[0]);
  const unsigned long long uy = f2_pack(d.fixUnit[1], d.fixUnit[1]);
  const unsigned long long uz = f2_pack(d.fixUnit[2], d.fixUnit[2]);
  const LJPairF P = d.ljf[0];
  const unsigned long long ff1s = f2_pack(P.ff1, P.ff1), ff2s = f2_pack(-P.ff2, -P.ff2);
  const LJPairF* const row = sP + (SINGLE ? 0 : pi.w * d.ntypes);
  constexpr int S = T == 1 ? 2 : 1;  // pairs of FP32 sums
  unsigned long long f[S][3] = {};
  auto pairs = [&](const int4 pa, const int4 pb, unsigned long long (&sum)[3]) {
    const unsigned long long dx =
        f2_mul(f2_pack(wrapped_diff(pi.x, pa.x), wrapped_diff(pi.x, pb.x)), ux);
    const unsigned long long dy =
        f2_mul(f2_pack(wrapped_diff(pi.y, pa.y), wrapped_diff(pi.y, pb.y)), uy);
    const unsigned long long dz =
        f2_mul(f2_pack(wrapped_diff(pi.z, pa.z), wrapped_diff(pi.z, pb.z)), uz);
    const unsigned long long r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
    const float ra = f2_lo(r2), rb = f2_hi(r2);
    unsigned long long c1 = ff1s, c2 = ff2s;
    LJPairF Pa = P, Pb = P;
    if (!SINGLE) {
      Pa = row[pa.w];
      Pb = row[pb.w];
      c1 = f2_pack(Pa.ff1, Pb.ff1);
      c2 = f2_pack(-Pa.ff2, -Pb.ff2);
    }
    const unsigned long long ri2 = f2_pack(fast_rcp(ra), fast_rcp(rb));
    const unsigned long long ri6 = f2_mul(f2_mul(ri2, ri2), ri2);
    const unsigned long long ff = f2_mul(f2_mul(ri6, f2_fma(c1, ri6, c2)), ri2);
    float fa = f2_lo(ff), fb = f2_hi(ff);
    if (CAPPED) {
      if (ra <= Pa.capsq) fa = Pa.capff * rsqrtf(ra);
      if (rb <= Pb.capsq) fb = Pb.capff * rsqrtf(rb);
    }
    // padding entries are the particle itself: r^2 = 0
    fa = (ra > 0.f && ra <= Pa.rcsq) ? fa : 0.f;
    fb = (rb > 0.f && rb <= Pb.rcsq) ? fb : 0.f;
    const unsigned long long fab = f2_pack(fa, fb);
    sum[0] = f2_fma(dx, fab, sum[0]);
    sum[1] = f2_fma(dy, fab, sum[1]);
    sum[2] = f2_fma(dz, fab, sum[2]);
  };
  share.walk(d, i, sub, act ? d.nn[i] : 0, [&](const int (&j)[Share::ENT], auto next) {
    int4 q[Share::ENT];
#pragma unroll
    for (int u = 0; u < Share::ENT; ++u) q[u] = ld_pos<LIVE>(&posq[j[u]]);
    next();
#pragma unroll
    for (int u = 0; u < Share::ENT; u += 2) pairs(q[u], q[u + 1], f[u / 2 % S]);
  });
  long long Fx = 0, Fy = 0, Fz = 0;
#pragma unroll
  for (int u = 0; u < S; ++u) {
    Fx += to_fix2(f[u][0], d.err);
    Fy += to_fix2(f[u][1], d.err);
    Fz += to_fix2(f[u][2], d.err);
  }
  if (FENE && act) {
    // the particle's bonds, shared out among its lanes
    const int64_t off = a.id[i] - d.idMin;
    const int b0 = d.bondStart[off] + sub, b1 = d.bondStart[off + 1];
    float bx = 0.f, by = 0.f, bz = 0.f, bmax = 0.f;
    const float rmaxsq = (float)fp.rmaxsq, K = (float)fp.K, r0 = (float)fp.r0;
    for (int b = b0; b < b1; b += T) {
      const int64_t po = d.bondPartner[b] - d.idMin;
      const int j = (po >= 0 && po < d.idSpan) ? d.id2idx[po] : -1;
      if (j < 0) {
        atomicOr(d.err, kErrBondMissing);
        continue;
      }
      const int4 pj = ld_pos<LIVE>(&posq[j]);
      const float dx = wrapped_diff(pi.x, pj.x, d.fixUnit[0]);
      const float dy = wrapped_diff(pi.y, pj.y, d.fixUnit[1]);
      const float dz = wrapped_diff(pi.z, pj.z, d.fixUnit[2]);
      const float r2 = dx * dx + dy * dy + dz * dz;
      bmax = fmaxf(bmax, r2);
      if (!(r2 <= (float)fp.rcsq)) continue;
      float ff;
      if (fp.r0 > 2.220446049250313e-16) {
        const float r = sqrtf(r2);
        ff = -K * (r - r0) / (r * (1.f - ((r - r0) * (r - r0) / rmaxsq)));
      } else {
        ff = -K / (1.f - r2 / rmaxsq);
      }
      bx += dx * ff;
      by += dy * ff;
      bz += dz * ff;
    }
    if (b1 > b0) note_bond_sq(d.ctr, (double)bmax);
    Fx += to_fix(bx, d.err);
    Fy += to_fix(by, d.err);
    Fz += to_fix(bz, d.err);
  }
#pragma unroll
  for (int o = T / 2; o > 0; o >>= 1) {
    Fx += __shfl_xor_sync(0xffffffffu, Fx, o, T);
    Fy += __shfl_xor_sync(0xffffffffu, Fy, o, T);
    Fz += __shfl_xor_sync(0xffffffffu, Fz, o, T);
  }
  F[0] = Fx;
  F[1] = Fy;
  F[2] = Fz;
}

template <int T, bool SINGLE, bool CAPPED, bool FENE>
__global__ void __launch_bounds__(256, T == 1 ? 3 : 4) k_force_mixed(DevView d, FENEParams fp) {
  __shared__ LJPairF sP[kMaxTypes * kMaxTypes];
  if (!SINGLE) {
    for (int t = threadIdx.x; t < d.ntypes * d.ntypes; t += blockDim.x) sP[t] = d.ljf[t];
    __syncthreads();
  }
  const int gt = blockIdx.x * blockDim.x + threadIdx.x;
  if (T == 1 && gt >= d.n) return;
  const bool act = gt / T < d.n;
  const int i = act ? gt / T : 0;
  long long F[3];
  particle_force_mixed<T, SINGLE, CAPPED, FENE, false>(d, fp, sP, d.posq, i, gt % T, act,
                                                       ListShare<T>(), F);
  if (gt % T == 0 && act) {
#pragma unroll
    for (int c = 0; c < 3; ++c) d.ffix[c * (size_t)d.cap + i] = F[c];
  }
}

__device__ __forceinline__ double min_image(double dx, double L, double halfL) {
  if (dx < -halfL)
    dx += L;
  else if (dx > halfL)
    dx -= L;
  return dx;
}

// 1 / x for a pair's r^2 (positive, normal) from the hardware's approximate reciprocal r, which
// works on the 20 leading bits of the mantissa: with e = 1 - x r the geometric series
// 1 / x = r / (1 - e) = r (1 + e + e^2 + ...), cut after e^2 (the third-order member of the
// hyperpower iterations, Altman 1960).  The rounded quotient for all but 5 of 20,000 values of
// r^2 from 0.09 to 6.2, and its neighbour for those.  Forces with a division in its place are
// no closer to 80-bit ones (6.375e-15 with either) and take a third longer.
__device__ __forceinline__ double pair_rcp(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// Plain FP64 form of the same kernel (reference arithmetic of LennardJones.hpp:137-143
// and FENE.hpp:97-112 on minimum-image distances).  A warp whose particles all lie farther
// than wrapMargin from every face of the box has no partner across one: its differences are
// their own minimum images, bit for bit, and the 12 FP64 instructions of the comparisons
// and shifts (of 30 a pair) are skipped.  Bound by the FP64 pipe and the gathers: 186 us at a
// million particles of one type, 13 at 32,768; with a division in place of pair_rcp 251 and 17.
// With one or two lanes and one type a lane's entries go to two sums in turn: no sum is longer
// than with four lanes (error against 80-bit sums 6.374e-15, 6.377e-15 with one sum,
// 6.376e-15 with four lanes), and the chain of additions is half as long (188 us with one).
// With several types the second sum would spill (370 us, 320 with one, at a million).
// Registers: four blocks an SM with one type (203 us with three), three where the pair's
// constants are loaded per entry.
template <int T, bool SINGLE, bool CAPPED, bool FENE, bool LIVE, class Share>
__device__ __forceinline__ void particle_force_fp64(const DevView& d, const FENEParams& fp,
                                                    const double* X, int i, int sub, bool act,
                                                    const Share& share, double (&F)[3]) {
  const ParticleArrays a = d.pa[0];
  const double* Y = X + d.cap;
  const double* Z = X + 2 * (size_t)d.cap;
  const double xi = ld_pos<LIVE>(&X[i]), yi = ld_pos<LIVE>(&Y[i]), zi = ld_pos<LIVE>(&Z[i]);
  const LJPair* const row = d.lj + (SINGLE ? 0 : a.type[i] * d.ntypes);
  const double sc1 = d.lj[0].ff1, sc2 = d.lj[0].ff2, srcsq = d.lj[0].rcsq;
  constexpr int S = SINGLE && T <= 2 ? 2 : 1;  // partial sums
  double f[S][3] = {};
  auto pair = [&](double dx, double dy, double dz, int tj, double (&f)[3]) {
    const double r2 = dx * dx + dy * dy + dz * dz;
    const LJPair& P = row[SINGLE ? 0 : tj];
    const double c1 = SINGLE ? sc1 : P.ff1, c2 = SINGLE ? sc2 : P.ff2;
    // padding entries are the particle itself: r^2 = 0
    bool in = r2 > 0.0 && !(r2 > (SINGLE ? srcsq : P.rcsq));
    if (!SINGLE) in = in && P.set;
    const double ri2 = pair_rcp(r2);
    const double ri6 = ri2 * ri2 * ri2;
    double ff = ri6 * (c1 * ri6 - c2) * ri2;
    if (CAPPED && P.caprad > 0 && !(r2 > P.caprad * P.caprad)) ff = P.capff / sqrt(r2);
    if (in) {
      f[0] += dx * ff;
      f[1] += dy * ff;
      f[2] += dz * ff;
    }
  };
  auto loop = [&](auto wrap) {
    share.walk(d, i, sub, act ? d.nn[i] : 0, [&](const int (&j)[Share::ENT], auto next) {
      double xj[Share::ENT], yj[Share::ENT], zj[Share::ENT];
      int tj[Share::ENT];
#pragma unroll
      for (int u = 0; u < Share::ENT; ++u) {
        xj[u] = ld_pos<LIVE>(&X[j[u]]);
        yj[u] = ld_pos<LIVE>(&Y[j[u]]);
        zj[u] = ld_pos<LIVE>(&Z[j[u]]);
        tj[u] = SINGLE ? 0 : __ldg(&a.type[j[u]]);
      }
      next();
#pragma unroll
      for (int u = 0; u < Share::ENT; ++u) {
        double dx = xi - xj[u], dy = yi - yj[u], dz = zi - zj[u];
        if (decltype(wrap)::value) {
          dx = min_image(dx, d.L[0], d.halfL[0]);
          dy = min_image(dy, d.L[1], d.halfL[1]);
          dz = min_image(dz, d.L[2], d.halfL[2]);
        }
        pair(dx, dy, dz, tj[u], f[u % S]);
      }
    });
  };
  const double m = d.wrapMargin;
  const bool inner = xi > m && xi < d.L[0] - m && yi > m && yi < d.L[1] - m && zi > m &&
                     zi < d.L[2] - m;
  if (__all_sync(0xffffffffu, inner || !act))
    loop(std::false_type{});
  else
    loop(std::true_type{});
  double fx = f[0][0], fy = f[0][1], fz = f[0][2];
  if (S == 2) {
    fx += f[S - 1][0];
    fy += f[S - 1][1];
    fz += f[S - 1][2];
  }
  if (FENE && act) {
    // the particle's bonds, shared out among its lanes
    const int64_t off = a.id[i] - d.idMin;
    const int b0 = d.bondStart[off] + sub, b1 = d.bondStart[off + 1];
    double bmax = 0.0;
    for (int b = b0; b < b1; b += T) {
      const int64_t po = d.bondPartner[b] - d.idMin;
      const int j = (po >= 0 && po < d.idSpan) ? d.id2idx[po] : -1;
      if (j < 0) {
        atomicOr(d.err, kErrBondMissing);
        continue;
      }
      const double dx = min_image(xi - ld_pos<LIVE>(&X[j]), d.L[0], d.halfL[0]);
      const double dy = min_image(yi - ld_pos<LIVE>(&Y[j]), d.L[1], d.halfL[1]);
      const double dz = min_image(zi - ld_pos<LIVE>(&Z[j]), d.L[2], d.halfL[2]);
      const double r2 = dx * dx + dy * dy + dz * dz;
      bmax = fmax(bmax, r2);
      if (r2 > fp.rcsq) continue;
      double ff;
      if (fp.r0 > 2.220446049250313e-16) {
        const double r = sqrt(r2);
        ff = -fp.K * (r - fp.r0) / (r * (1 - ((r - fp.r0) * (r - fp.r0) / fp.rmaxsq)));
      } else {
        ff = -fp.K / (1.0 - r2 / fp.rmaxsq);
      }
      fx += dx * ff;
      fy += dy * ff;
      fz += dz * ff;
    }
    if (b1 > b0) note_bond_sq(d.ctr, bmax);
  }
#pragma unroll
  for (int o = T / 2; o > 0; o >>= 1) {
    fx += __shfl_xor_sync(0xffffffffu, fx, o, T);
    fy += __shfl_xor_sync(0xffffffffu, fy, o, T);
    fz += __shfl_xor_sync(0xffffffffu, fz, o, T);
  }
  F[0] = fx;
  F[1] = fy;
  F[2] = fz;
}

template <int T, bool SINGLE, bool CAPPED, bool FENE>
__global__ void __launch_bounds__(256, SINGLE ? 4 : 3) k_force_fp64(DevView d, FENEParams fp) {
  const int gt = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = gt / T < d.n;  // every lane stays for the vote and the shuffles
  const int i = act ? gt / T : 0;
  double F[3];
  particle_force_fp64<T, SINGLE, CAPPED, FENE, false>(d, fp, d.pa[0].x, i, gt % T, act,
                                                      ListShare<T>(), F);
  if (gt % T == 0 && act) {
#pragma unroll
    for (int c = 0; c < 3; ++c) d.f64[c * (size_t)d.cap + i] = F[c];
  }
}

// ---- integrator --------------------------------------------------------------------

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// aftCalcF (LangevinThermostat::frictionThermo, CapForce) on the pair force F of one
// particle, then integrate2 of this step and integrate1 of the next
// (VelocityVerlet.cpp:236-305), with the reference's operation order and no FMA contraction.
// F becomes the total force; returns |dx|^2 of integrate1 (0 without it).
__device__ __forceinline__ double advance(const IntegrateArgs& a, int64_t id, bool thermo, double m,
                                          double (&F)[3], double (&v)[3], double (&x)[3]) {
  if (thermo) {
    const double massf = sqrt(m);
    double u[3];
    langevin_uniforms(a.seed, id, a.step, a.phase, u);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double t1 = __dmul_rn(__dmul_rn(a.pref1, v[k]), m);
      const double t2 = __dmul_rn(__dmul_rn(a.pref2, u[k] - 0.5), massf);
      F[k] = __dadd_rn(F[k], __dadd_rn(t1, t2));
    }
  }
  if (a.capMode == 1) {
    const double capfsq = __dmul_rn(a.cap[0], a.cap[0]);
    const double fsq =
        __dadd_rn(__dadd_rn(__dmul_rn(F[0], F[0]), __dmul_rn(F[1], F[1])), __dmul_rn(F[2], F[2]));
    if (fsq > capfsq) {
      const double scaling = sqrt(capfsq / fsq);
#pragma unroll
      for (int k = 0; k < 3; ++k) F[k] = __dmul_rn(F[k], scaling);
    }
  } else if (a.capMode == 2) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (F[k] > 0 && F[k] > a.cap[k])
        F[k] = a.cap[k];
      else if (F[k] < 0 && F[k] < -a.cap[k])
        F[k] = -a.cap[k];
    }
  }
  const double dtfm = __ddiv_rn(__dmul_rn(0.5, a.dt), m);
  if (a.do_i2) {
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = __dadd_rn(v[k], __dmul_rn(dtfm, F[k]));
  }
  if (!a.do_i1) return 0.0;
  double dp[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    v[k] = __dadd_rn(v[k], __dmul_rn(dtfm, F[k]));
    dp[k] = __dmul_rn(v[k], a.dt);
    x[k] = __dadd_rn(x[k], dp[k]);
  }
  return __dadd_rn(__dadd_rn(__dmul_rn(dp[0], dp[0]), __dmul_rn(dp[1], dp[1])),
                   __dmul_rn(dp[2], dp[2]));
}

// The block's largest sq into *maxSq (bits of a non-negative double order like integers).
__device__ __forceinline__ void block_max_sq(double sq, double* smax, unsigned long long* maxSq) {
  sq = warp_max(sq);
  if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = sq;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < blockDim.x / 32 ? smax[threadIdx.x] : 0.0;
    v = warp_max(v);
    if (threadIdx.x == 0 && v > 0.0) atomicMax(maxSq, (unsigned long long)__double_as_longlong(v));
  }
}

template <bool MIXED>
__global__ void __launch_bounds__(256) k_integrate(DevView d, IntegrateArgs a) {
  const ParticleArrays P = d.pa[0];
  __shared__ double smax[kBlock / 32];
  if (a.fromCounters) {  // uniform over the grid: written by the decide kernel before
    a.step = d.ctr->step;
    a.pref1 = d.ctr->pref1;
    a.pref2 = d.ctr->pref2;
    if (d.ctr->remaining == 0) {
      a.do_i1 = 0;
      a.storeFtot = 1;
    }
  }
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double sq = 0.0;
  if (i < d.n && !(d.halo && d.halo[P.id[i] - d.idMin])) {  // halo copies stay put
    const size_t cap = d.cap;
    const double m = P.mass[i];
    double F[3], v[3], x[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      F[k] = MIXED ? (double)d.ffix[k * cap + i] * kInvFix : d.f64[k * cap + i];
      v[k] = P.v[k * cap + i];
      if (a.do_i1) x[k] = P.x[k * cap + i];
    }
    const int64_t id = a.langevin ? P.id[i] : 0;
    sq = advance(a, id, a.langevin && !(d.langExcl && d.langExcl[id - d.idMin]), m, F, v, x);
    if (a.storeFtot) {
#pragma unroll
      for (int k = 0; k < 3; ++k) d.ftot[k * cap + i] = F[k];
    }
    if (a.do_i1) {
#pragma unroll
      for (int k = 0; k < 3; ++k) P.x[k * cap + i] = x[k];
      d.posq[i] = fixed_coords(d, x[0], x[1], x[2], P.type[i]);
    }
    if (a.do_i1 || a.do_i2) {
#pragma unroll
      for (int k = 0; k < 3; ++k) P.v[k * cap + i] = v[k];
    }
  }
  if (a.do_i1) block_max_sq(sq, smax, &d.ctr->maxSq);
}

__device__ __forceinline__ int decide_core(DevCounters* c, double skinHalf) {
  const double m = __longlong_as_double((long long)c->maxSq);
  c->maxSq = 0ull;
  const double md = __dadd_rn(c->maxDist, sqrt(m));
  const int f = md > skinHalf ? 1 : 0;
  c->maxDist = f ? 0.0 : md;
  c->flag = f;
  c->resorts += f;
  return f;
}

__global__ void k_decide(DevCounters* c, double skinHalf) { decide_core(c, skinHalf); }

// First node of the captured step loop: advance the step, decide on the re-sort and
// set the IF (re-sort) and WHILE (more steps) conditionals.
__global__ void k_decide_graph(DevCounters* c, double skinHalf, cudaGraphConditionalHandle hIf,
                               cudaGraphConditionalHandle hWhile) {
  c->step += 1;
  const long long rem = c->remaining - 1;
  c->remaining = rem;
  const int f = decide_core(c, skinHalf);
  cudaGraphSetConditional(hIf, f ? 1u : 0u);
  cudaGraphSetConditional(hWhile, rem > 0 ? 1u : 0u);
}

constexpr int kBarrierTries = 1 << 21;  // about a second

// ---- steps of a small system ------------------------------------------------------------
// All steps up to the next re-sort or the end of the run in one cooperative launch.  A small
// system's step is bound by launches and by the tail of each kernel, not by its work: the
// force, integrate and decide kernels of 32,768 particles take 15 us a step, most of it
// latency.  Here the lanes that sum a particle's force also advance it, and one barrier over
// the grid ends the step; positions alternate between two buffers, so a step reads the old
// ones while it writes the new ones.  The largest displacement goes through three slots in
// turn (one being raised, one read, one cleared).  Every block takes the same decision from
// the same numbers; block 0 writes it down.
// The result is that of the separate kernels, bit for bit: the same arithmetic with the same
// lanes a particle.  A step without re-sorts takes 6.3 us at 1,728 particles and 9.6 (mixed) or
// 12.0 (FP64) at 32,768.  With re-sorts, separate kernels against this one: mixed 18.5 / 13.3 us
// a step at 8,000 particles, 24.5 / 18.9 at 32,768, 32.0 / 26.2 at 64,000; FP64 21.2 / 14.1 at
// 8,000 and 33.8 / 26.0 at 46,656.
// A step's chain of L2 round trips is its cost, so the barrier is one counter that only grows
// (the blocks arrive on it and poll it), and the thread that polled also fetches *word, the
// value every thread wants next.  passed: barriers passed so far times the grid's blocks.
__device__ __forceinline__ bool grid_barrier(StepSync* s, unsigned long long& passed,
                                             const unsigned long long* word, double& value,
                                             unsigned* err) {
  __shared__ bool s_ok;
  __shared__ unsigned long long s_word;
  passed += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    // the barriers of the block order its threads' accesses before the release here and
    // behind the acquire below
    unsigned long long now;
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(&s->count) : "memory");
    int tries = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(&s->count) : "memory");
    } while (now < passed && ++tries < kBarrierTries);
    s_ok = now >= passed;
    if (!s_ok) atomicOr(err, kErrTimeout);
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(s_word) : "l"(word) : "memory");
  }
  __syncthreads();
  value = __longlong_as_double((long long)s_word);
  return s_ok;
}

// Threads of the one block an SM runs: what the registers of the force loop allow (64 in
// FP32, 96 in FP64).
template <bool MIXED>
constexpr int kStepThreads = MIXED ? 1024 : 640;

// A lane's share of a list kept in shared memory for the whole launch, as 16-bit indices two a
// word (the step kernel's systems hold at most 65,536 particles): blocks of 8 entries as in
// ListShare, a particle's words contiguous with a stride of 52, so the lanes of a warp fall on
// different banks.  The entries come in the order of ListShare, B of them a step: a barrier
// over the grid drops the SM's L1, so a step's chain is list, coordinates, sums, and both fewer
// round trips and more gathers in flight shorten it.  Blocks beyond the stage are read from
// the list itself.
constexpr int kStepWords = 52, kStepBlocks = kStepWords / 4;

template <int T, int B>
struct StepShare {
  static constexpr int E = T == 1 ? 8 : (T == 2 ? 4 : 2);  // entries of a block a lane takes
  static constexpr int ENT = B;
  static constexpr int U = B / E;                          // blocks of one step
  static constexpr int kStride = T == 8 ? 2 : 1;
  const uint32_t* words;  // the particle's words

  template <class F>
  __device__ __forceinline__ void walk(const DevView& d, int i, int sub, int cnt, F&& f) const {
    const int nblk = (cnt + 7) >> 3, first = T == 8 ? sub >> 2 : 0;
    const int lane = T >= 4 ? (sub & 3) * 2 : sub * E;  // first entry inside a block
    for (int b = first; b < nblk; b += U * kStride) {
      int j[ENT];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = b + u * kStride;
#pragma unroll
        for (int e = 0; e < E; e += 2) {
          int j0 = i, j1 = i;
          if (k < nblk) {
            if (k < kStepBlocks) {
              const uint32_t w = words[4 * k + (lane + e) / 2];
              j0 = (int)(w & 0xffffu);
              j1 = (int)(w >> 16);
            } else {
              const int2 v = ld_list2(reinterpret_cast<const int2*>(
                  d.nl + nl_index(8 * k, i, d.cap) + lane + e));
              j0 = v.x;
              j1 = v.y;
            }
          }
          j[u * E + e] = j0;
          j[u * E + e + 1] = j1;
        }
      }
      f(j, [] {});
    }
  }
};

template <bool MIXED, int T, bool SINGLE, bool CAPPED, bool FENE>
__global__ void __launch_bounds__(kStepThreads<MIXED>, 1)
    k_steps(DevView d, FENEParams fp, IntegrateArgs a, double skinHalf, StepSync* sync,
            cudaGraphConditionalHandle hIf, cudaGraphConditionalHandle hWhile) {
  const ParticleArrays P = d.pa[0];
  // the second buffers of the positions: the re-sort's target is free between re-sorts
  double* const xAlt = d.pa[1].x;
  int4* const posqAlt = reinterpret_cast<int4*>(d.pa[1].v);
  __shared__ LJPairF sP[kMaxTypes * kMaxTypes];
  __shared__ double smax[kStepThreads<MIXED> / 32];
  if (MIXED && !SINGLE)
    for (int t = threadIdx.x; t < d.ntypes * d.ntypes; t += blockDim.x) sP[t] = d.ljf[t];
  DevCounters* const c = d.ctr;
  long long step = c->step, rem = c->remaining;
  double maxDist = c->maxDist, msq = __longlong_as_double((long long)c->maxSq);
  bool resume = c->flag != 0;  // the re-sort of this step is done: its force is next
  // between launches the counter is a multiple of the grid's blocks
  unsigned long long passed = *(volatile unsigned long long*)&sync->count;
  passed -= passed % gridDim.x;
  a.pref1 = c->pref1;
  a.pref2 = c->pref2;
  const int gt = blockIdx.x * blockDim.x + threadIdx.x, sub = gt % T;
  const size_t cap = d.cap;
  // one particle a group of T lanes (the grid covers them), its list into shared memory
  const bool act = gt / T < d.n;
  const int i = act ? gt / T : 0;
  extern __shared__ uint32_t s_list[];
  const int perBlock = blockDim.x / T, p0 = blockIdx.x * perBlock;
  for (int q = threadIdx.x; q < perBlock * kStepWords; q += blockDim.x) {
    const int p = p0 + q / kStepWords, w = q % kStepWords;
    if (p >= d.n || 2 * w >= ((d.nn[p] + 7) & ~7)) continue;
    const int2 v =
        *reinterpret_cast<const int2*>(d.nl + nl_index(8 * (w >> 2), p, cap) + 2 * (w & 3));
    s_list[q] = (uint32_t)v.x | (uint32_t)v.y << 16;
  }
  const bool thermo = a.langevin && !(d.langExcl && d.langExcl[P.id[i] - d.idMin]);
  const StepShare<T, MIXED ? 8 : (T == 1 ? 8 : 4)> share{s_list + threadIdx.x / T * kStepWords};
  bool resort = false, ok = true;
  int k = 0, slot = 0;  // steps done: the current positions are in the first buffer when even
  __syncthreads();
  while (true) {
    const int4* const posq = k & 1 ? posqAlt : d.posq;
    int4* const posqNew = k & 1 ? d.posq : posqAlt;
    const double* const X = k & 1 ? xAlt : P.x;
    double* const xNew = k & 1 ? P.x : xAlt;
    if (sub == 0) {  // under way while the step is decided; read behind the pair loop
      if (MIXED) prefetch_l1(&posq[i]);
      prefetch_l1(&P.mass[i]);
      prefetch_l1(&P.id[i]);
      prefetch_l1(&P.type[i]);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        prefetch_l1(&P.v[e * cap + i]);
        prefetch_l1(&(MIXED ? P.x : X)[e * cap + i]);
      }
    }
    if (!resume) {
      ++step;
      --rem;
      const double md = __dadd_rn(maxDist, sqrt(msq));
      resort = md > skinHalf;
      maxDist = resort ? 0.0 : md;
      if (resort) break;
    }
    resume = false;
    a.step = step;
    a.do_i1 = rem > 0 ? 1 : 0;
    double sq = 0.0;
    double F[3];
    if (MIXED) {
      long long G[3];
      particle_force_mixed<T, SINGLE, CAPPED, FENE, true>(d, fp, sP, posq, i, sub, act, share, G);
#pragma unroll
      for (int e = 0; e < 3; ++e) F[e] = (double)G[e] * kInvFix;
    } else {
      particle_force_fp64<T, SINGLE, CAPPED, FENE, true>(d, fp, X, i, sub, act, share, F);
    }
    if (sub == 0 && act) {
      double v[3], x[3];
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        v[e] = P.v[e * cap + i];
        x[e] = ld_pos<true>((MIXED ? P.x : X) + e * cap + i);
      }
      sq = advance(a, P.id[i], thermo, P.mass[i], F, v, x);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        P.v[e * cap + i] = v[e];
        if (a.do_i1) (MIXED ? P.x : xNew)[e * cap + i] = x[e];
        if (rem == 0) d.ftot[e * cap + i] = F[e];
      }
      if (MIXED && a.do_i1) posqNew[i] = fixed_coords(d, x[0], x[1], x[2], P.type[i]);
    }
    if (a.do_i1) {
      block_max_sq(sq, smax, &sync->maxSq[slot]);
      if (gt == 0) sync->maxSq[slot == 2 ? 0 : slot + 1] = 0ull;
    }
    ok = grid_barrier(sync, passed, &sync->maxSq[slot], msq, d.err);
    if (!ok || rem == 0) break;
    ++k;
    slot = slot == 2 ? 0 : slot + 1;
  }
  // behind this barrier nobody reads the counters or the slots any more
  if (resort) ok = grid_barrier(sync, passed, &sync->maxSq[slot], msq, d.err);
  const bool odd = k & 1;
  // the run's end: current positions into the first buffer (packed ones are made anew by a
  // re-sort)
  if (MIXED ? odd && !resort : odd || !resort) {
    if (act && sub == 0) {
      if (MIXED) {
        d.posq[i] = ld_pos<true>(&posqAlt[i]);
      } else {
        double x[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          x[e] = ld_pos<true>((odd ? xAlt : P.x) + e * cap + i);
          if (odd) P.x[e * cap + i] = x[e];
        }
        d.posq[i] = fixed_coords(d, x[0], x[1], x[2], P.type[i]);
      }
    }
  }
  if (gt == 0) {
    c->step = step;
    c->remaining = rem;
    c->maxDist = maxDist;
    c->maxSq = 0ull;
    c->flag = resort ? 1 : 0;
    c->resorts += resort ? 1 : 0;
    sync->maxSq[0] = sync->maxSq[1] = sync->maxSq[2] = 0ull;
    cudaGraphSetConditional(hIf, ok && resort ? 1u : 0u);
    cudaGraphSetConditional(hWhile, ok && (resort || rem > 0) ? 1u : 0u);
  }
}

// ---- observables -------------------------------------------------------------------


// LJ energy (E = 4 eps ((sig^2/r^2)^6 - (sig^2/r^2)^3) - shift, LennardJones.hpp:109-114) or
// virial r.F and its tensor (VerletListInteractionTemplate.hpp:274-331) over each listed pair
// once (j > i).  T lanes a particle (ListShare), a block of 256 threads 256 particles in T
// rounds; the minimum image is skipped where k_force_fp64 skips it.  Bound by the FP64 pipe and
// the latency of the gathers: 277 us (energy) and 321 (virial tensor) at a million particles,
// 423 with one lane that loads entry by entry.  Two lanes at every size; a call with four takes
// 49.0 us (energy) and 62.0 (virial) against 47.4 and 53.5 at 8,000 particles, 96 and 114
// against 88 and 111 at 216,000.
constexpr int kObsLanes = 2;
template <bool ENERGY, bool SINGLE>
__global__ void __launch_bounds__(kBlock, 3) k_lj_obs(DevView d, double* partials) {
  constexpr int T = kObsLanes;
  const ParticleArrays a = d.pa[0];
  const double* X = a.x;
  const double* Y = a.x + d.cap;
  const double* Z = a.x + 2 * (size_t)d.cap;
  const LJPair P0 = d.lj[0];
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  const int sub = threadIdx.x % T;
  const double m = d.wrapMargin;
  using Share = ListShare<T>;
  for (int round = 0; round < T; ++round) {
    const int i0 = blockIdx.x * kBlock + round * (kBlock / T) + threadIdx.x / T;
    const bool act = i0 < d.n && !(d.halo && is_halo(d, a.id[i0]));
    const int i = act ? i0 : 0;
    const double xi = X[i], yi = Y[i], zi = Z[i];
    const LJPair* const row = d.lj + (SINGLE ? 0 : a.type[i] * d.ntypes);
    auto loop = [&](auto wrap) {
      Share::walk(d, i, sub, act ? d.nn[i] : 0, [&](const int (&j)[Share::ENT], auto next) {
        double xj[Share::ENT], yj[Share::ENT], zj[Share::ENT];
        int tj[Share::ENT];
#pragma unroll
        for (int u = 0; u < Share::ENT; ++u) {
          xj[u] = __ldg(&X[j[u]]);
          yj[u] = __ldg(&Y[j[u]]);
          zj[u] = __ldg(&Z[j[u]]);
          tj[u] = SINGLE ? 0 : __ldg(&a.type[j[u]]);
        }
        next();
#pragma unroll
        for (int u = 0; u < Share::ENT; ++u) {
          // padding entries are the particle itself: j = i
          const bool here = d.halo ? j[u] != i && pair_counted_here(d, i, j[u], a.id[i], a.id[j[u]])
                                   : j[u] > i;
          if (!here) continue;
          double dx = xi - xj[u], dy = yi - yj[u], dz = zi - zj[u];
          if (decltype(wrap)::value) {
            dx = min_image(dx, d.L[0], d.halfL[0]);
            dy = min_image(dy, d.L[1], d.halfL[1]);
            dz = min_image(dz, d.L[2], d.halfL[2]);
          }
          const double r2 =
              __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
          const LJPair& P = SINGLE ? P0 : row[tj[u]];
          if (!P.set || r2 > P.rcsq) continue;
          if (ENERGY) {
            double ds = r2;
            if (P.caprad > 0 && !(ds > P.caprad * P.caprad)) ds = P.caprad * P.caprad;
            const double frac2 = P.ef2 * pair_rcp(ds);
            const double frac6 = __dmul_rn(__dmul_rn(frac2, frac2), frac2);
            acc[0] +=
                __dsub_rn(__dmul_rn(P.ef1, __dsub_rn(__dmul_rn(frac6, frac6), frac6)), P.shift);
          } else {
            double ff;
            if (P.caprad > 0 && !(r2 > P.caprad * P.caprad)) {
              ff = P.capff / sqrt(r2);
            } else {
              const double ri2 = pair_rcp(r2);
              const double ri6 = ri2 * ri2 * ri2;
              ff = ri6 * (P.ff1 * ri6 - P.ff2) * ri2;
            }
            const double f0 = dx * ff, f1 = dy * ff, f2 = dz * ff;
            acc[1] += dx * f0;
            acc[2] += dy * f1;
            acc[3] += dz * f2;
            acc[4] += dx * f1;
            acc[5] += dx * f2;
            acc[6] += dy * f2;
          }
        }
      });
    };
    const bool inner = xi > m && xi < d.L[0] - m && yi > m && yi < d.L[1] - m && zi > m &&
                       zi < d.L[2] - m;
    if (__all_sync(0xffffffffu, inner || !act))
      loop(std::false_type{});
    else
      loop(std::true_type{});
  }
  if (!ENERGY) acc[0] = acc[1] + acc[2] + acc[3];
  block_sum_store<7>(acc, partials);
}

// FENE energy (FENE.hpp:91-95) or virial over each bond once (partner id > own id).
__global__ void k_fene_obs(DevView d, FENEParams fp, int energy, double* partials) {
  const ParticleArrays a = d.pa[0];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  if (i < d.n && fp.on && !is_halo(d, a.id[i])) {
    const double* X = a.x;
    const double* Y = a.x + d.cap;
    const double* Z = a.x + 2 * (size_t)d.cap;
    const int64_t id = a.id[i];
    const int64_t off = id - d.idMin;
    const int b0 = d.bondStart[off], b1 = d.bondStart[off + 1];
    for (int b = b0; b < b1; ++b) {
      const int64_t pid = d.bondPartner[b];
      if (pid <= id) continue;
      const int j = d.id2idx[pid - d.idMin];
      if (j < 0) continue;
      const double dx = min_image(X[i] - X[j], d.L[0], d.halfL[0]);
      const double dy = min_image(Y[i] - Y[j], d.L[1], d.halfL[1]);
      const double dz = min_image(Z[i] - Z[j], d.L[2], d.halfL[2]);
      const double r2 =
          __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
      if (r2 > fp.rcsq) continue;
      if (energy) {
        const double q = (sqrt(r2) - fp.r0) / fp.rmax;
        acc[0] += -0.5 * fp.rmaxsq * fp.K * log(1 - q * q) - fp.shift;
      } else {
        double ff;
        if (fp.r0 > 2.220446049250313e-16) {
          const double r = sqrt(r2);
          ff = -fp.K * (r - fp.r0) / (r * (1 - ((r - fp.r0) * (r - fp.r0) / fp.rmaxsq)));
        } else {
          ff = -fp.K / (1.0 - r2 / fp.rmaxsq);
        }
        const double f0 = dx * ff, f1 = dy * ff, f2 = dz * ff;
        acc[0] += dx * f0 + dy * f1 + dz * f2;
        acc[1] += dx * f0;
        acc[2] += dy * f1;
        acc[3] += dz * f2;
        acc[4] += dx * f1;
        acc[5] += dx * f2;
        acc[6] += dy * f2;
      }
    }
  }
  block_sum_store<7>(acc, partials);
}

// ---- analysis::RadialDistrF -----------------------------------------------------------

constexpr int kRdfTile = 256;
constexpr int kRdfSmemBins = 10 * 1024;  // shared counts of a block (40 KB beside the tiles)
// Half width of the zone about a bin's edge, in bins, up to which the FP32 pass decides enough
// pairs (rdf_eps at 8192 bins: one pair in 30 lies within it, one in 250 at 1024).  FP64
// against FP32 first, 32,768 particles: 1734 / 1052 us at 2048 bins, 1755 / 1335 at 4096,
// 1785 / 1749 at 8192.
constexpr double kRdfFastEps = 0.0165;

// Bin of a pair in the reference's arithmetic (RadialDistrF.cpp:104-129): the FP64 minimum
// image (one shift per axis, its two comparisons), static_cast<int>(|d| / dr).
__device__ __forceinline__ int rdf_bin(const DevView& d, double ex, double ey, double ez,
                                       double dr) {
  double e[3] = {ex, ey, ez};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (e[k] < -d.halfL[k]) e[k] += d.L[k];
    if (e[k] > d.halfL[k]) e[k] -= d.L[k];
  }
  const double r = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(e[0], e[0]), __dmul_rn(e[1], e[1])),
                                  __dmul_rn(e[2], e[2])));
  return (int)(r / dr);
}

// Pair-distance histogram over all pairs i < j.  One block per pair of 256-particle tiles
// (upper triangle, decoded from the linear block index); counts are integers, so the
// histogram does not depend on the order of the additions.
// FAST: two partners at once in packed FP32 on the box-wrapped int32 coordinates, whose
// 32-bit difference is the minimum image; |d| / dr comes out within eps of a bin's width
// (rdf_eps; far = 1/2 - eps), and only a pair within eps of a bin's edge takes the reference's
// FP64 arithmetic, as does a block with a particle outside [-L/4, 5L/4], where one shift is not
// the minimum image.  17 instructions a pair, all of them FP32 or integer, against 40 in FP64.
// Counts go to `copies` copies of the histogram in shared memory, a lane's copy by its bank
// (no bank conflicts with 32), flushed with one global atomic per non-empty bin.
// Bound by issue: 743 us a call at 32,768 particles and 256 bins, 1,617 with FP64 for every pair.
template <bool SMEM, bool FAST>
__global__ void __launch_bounds__(kRdfTile) k_rdf(DevView d, int rdfN, int ntiles, double dr,
                                                  float far, int copies, unsigned long long* hist) {
  extern __shared__ unsigned s_hist[];
  using Coord = std::conditional_t<FAST, int, double>;
  __shared__ __align__(16) Coord sx[kRdfTile], sy[kRdfTile], sz[kRdfTile];
  // linear block index -> (bi, bj), bj >= bi, rows of the upper triangle in order
  const long long k = blockIdx.x;
  const double T = 2.0 * ntiles + 1.0;
  long long bi = (long long)((T - sqrt(T * T - 8.0 * (double)k)) * 0.5);
  auto row_start = [&](long long r) { return r * ntiles - r * (r - 1) / 2; };
  while (bi > 0 && row_start(bi) > k) --bi;
  while (bi + 1 < ntiles && row_start(bi + 1) <= k) ++bi;
  const long long bj = bi + (k - row_start(bi));
  const double* X = d.pa[0].x;
  const size_t c = d.cap;
  if (SMEM)
    for (int b = threadIdx.x; b < rdfN * copies; b += blockDim.x) s_hist[b] = 0u;
  const long long j0 = bj * kRdfTile, jt = j0 + threadIdx.x;
  const long long i = bi * kRdfTile + threadIdx.x;
  const int jn = (int)min((long long)kRdfTile, (long long)d.n - j0);
  auto in_reach = [&](long long p) {
    bool ok = true;
    for (int q = 0; q < 3; ++q) {
      const double x = X[q * c + p];
      ok = ok && x >= -0.25 * d.L[q] && x <= 1.25 * d.L[q];
    }
    return ok;
  };
  bool fast = FAST;
  if constexpr (FAST) {
    int4 q = make_int4(0, 0, 0, 0);
    bool ok = true;
    if (jt < d.n) {
      q = d.posq[jt];
      ok = in_reach(jt);
    }
    if (i < d.n) ok = ok && in_reach(i);
    sx[threadIdx.x] = q.x;
    sy[threadIdx.x] = q.y;
    sz[threadIdx.x] = q.z;
    fast = __syncthreads_and(ok) != 0;
  } else {
    if (jt < d.n) {
      sx[threadIdx.x] = X[jt];
      sy[threadIdx.x] = X[c + jt];
      sz[threadIdx.x] = X[2 * c + jt];
    }
    __syncthreads();
  }
  unsigned* const mine = s_hist + (threadIdx.x & (copies - 1));
  auto count = [&](int bin) {
    if (bin >= rdfN) return;
    if (SMEM)
      atomicAdd(mine + bin * copies, 1u);
    else
      atomicAdd(&hist[bin], 1ull);
  };
  if (i < d.n) {
    const int t0 = bi == bj ? threadIdx.x + 1 : 0;
    const double xi = X[i], yi = X[c + i], zi = X[2 * c + i];
    auto exact = [&](int t) {
      const long long j = j0 + t;
      return rdf_bin(d, xi - X[j], yi - X[c + j], zi - X[2 * c + j], dr);
    };
    if constexpr (!FAST) {
      for (int t = t0; t < jn; ++t) count(rdf_bin(d, xi - sx[t], yi - sy[t], zi - sz[t], dr));
    } else if (fast) {
      const int4 p = d.posq[i];
      const float inv = (float)(1.0 / dr);
      const float gx = d.fixUnit[0] * inv, gy = d.fixUnit[1] * inv, gz = d.fixUnit[2] * inv;
      const unsigned long long ux = f2_pack(gx, gx), uy = f2_pack(gy, gy), uz = f2_pack(gz, gz);
      const float magic = 12582912.f;  // 1.5 * 2^23: adding it rounds to an integer
      const unsigned long long half = f2_pack(0.5f, 0.5f);
      const unsigned long long mb = f2_pack(magic, magic);
      // pairs of partners t, t + 1 from an even t; an odd first or last partner masked
      for (int t = t0 & ~1; t < jn; t += 2) {
        const int2 qx = *reinterpret_cast<const int2*>(&sx[t]);
        const int2 qy = *reinterpret_cast<const int2*>(&sy[t]);
        const int2 qz = *reinterpret_cast<const int2*>(&sz[t]);
        const unsigned long long ex =
            f2_mul(f2_pack(wrapped_diff(p.x, qx.x), wrapped_diff(p.x, qx.y)), ux);
        const unsigned long long ey =
            f2_mul(f2_pack(wrapped_diff(p.y, qy.x), wrapped_diff(p.y, qy.y)), uy);
        const unsigned long long ez =
            f2_mul(f2_pack(wrapped_diff(p.z, qz.x), wrapped_diff(p.z, qz.y)), uz);
        const unsigned long long r2 = f2_fma(ez, ez, f2_fma(ey, ey, f2_mul(ex, ex)));
        const unsigned long long r = f2_pack(fast_sqrt(f2_lo(r2)), fast_sqrt(f2_hi(r2)));
        // floor(r) = round(r - 1/2) away from the integers
        const unsigned long long rh = f2_sub(r, half), y = f2_add(rh, mb);
        const unsigned long long off = f2_sub(rh, f2_sub(y, mb));  // 1/2 off at an integer r
        int ba = __float_as_int(f2_lo(y)) - 0x4B400000, bb = __float_as_int(f2_hi(y)) - 0x4B400000;
        if (fabsf(f2_lo(off)) > far) ba = exact(t);
        if (fabsf(f2_hi(off)) > far && t + 1 < jn) bb = exact(t + 1);
        if (t >= t0) count(ba);
        if (t + 1 < jn) count(bb);
      }
    } else {
      for (int t = t0; t < jn; ++t) count(exact(t));
    }
  }
  if (SMEM) {
    __syncthreads();
    for (int b = threadIdx.x; b < rdfN; b += blockDim.x) {
      unsigned n = 0u;
      for (int q = 0; q < copies; ++q) n += s_hist[b * copies + ((q + threadIdx.x) & (copies - 1))];
      if (n) atomicAdd(&hist[b], (unsigned long long)n);
    }
  }
}

__device__ __forceinline__ long long to_fix_d(double f, unsigned* err) {
  if (!(fabs(f) < 1.0e9)) atomicOr(err, kErrFixOverflow);
  return __double2ll_rn(f * 4294967296.0);
}

// ---- interaction::Cosine on a FixedTripleList ---------------------------------------

__device__ __forceinline__ double mimg_box(double d, double L, double hL) {
  // OrthorhombicBC::getMinimumImageVectorBox (src/bc/OrthorhombicBC.cpp:86-105)
  if (d < -hL)
    d += L;
  else if (d > hL)
    d -= L;
  return d;
}

__device__ __forceinline__ bool triple_dists(const DevView& d, int t, double* d12, double* d32) {
  const ParticleArrays a = d.pa[0];
  int k[3];
  for (int q = 0; q < 3; ++q) {
    const int64_t o = d.triples[3 * (size_t)t + q] - d.idMin;
    k[q] = (o >= 0 && o < d.idSpan) ? d.id2idx[o] : -1;
    if (k[q] < 0) return false;
  }
  const size_t c = d.cap;
  for (int q = 0; q < 3; ++q) {
    const double p2 = a.x[q * c + k[1]];
    d12[q] = mimg_box(a.x[q * c + k[0]] - p2, d.L[q], d.halfL[q]);
    d32[q] = mimg_box(a.x[q * c + k[2]] - p2, d.L[q], d.halfL[q]);
  }
  return true;
}

// Cosine::_computeForceRaw (Cosine.hpp:79-119) in the reference's operation order.
__device__ __forceinline__ void cosine_force(const CosineParams& P, const double* d12,
                                             const double* d32, double* f12, double* f32) {
  const double SMALL_EPSILON = 1.0E-9;
  const double d12sq = __dadd_rn(__dadd_rn(__dmul_rn(d12[0], d12[0]), __dmul_rn(d12[1], d12[1])),
                                 __dmul_rn(d12[2], d12[2]));
  const double d32sq = __dadd_rn(__dadd_rn(__dmul_rn(d32[0], d32[0]), __dmul_rn(d32[1], d32[1])),
                                 __dmul_rn(d32[2], d32[2]));
  const double m12 = sqrt(d12sq), m32 = sqrt(d32sq);
  const double dot = __dadd_rn(__dadd_rn(__dmul_rn(d12[0], d32[0]), __dmul_rn(d12[1], d32[1])),
                               __dmul_rn(d12[2], d32[2]));
  double c = dot / __dmul_rn(m12, m32);
  if (c < -1.0) c = -1.0;
  if (c > 1.0) c = 1.0;
  const double sn = sqrt(__dsub_rn(1.0, __dmul_rn(c, c)));
  const double a11 = c / d12sq, a12 = -1.0 / __dmul_rn(m12, m32), a22 = c / d32sq;
  if (sn > SMALL_EPSILON) {
    const double pre = __dsub_rn(P.Kcos_theta0, __dmul_rn(P.Ksin_theta0, c) / sn);
    for (int q = 0; q < 3; ++q) {
      f12[q] = __dmul_rn(pre, __dadd_rn(__dmul_rn(a11, d12[q]), __dmul_rn(a12, d32[q])));
      f32[q] = __dmul_rn(pre, __dadd_rn(__dmul_rn(a22, d32[q]), __dmul_rn(a12, d12[q])));
    }
  } else {
    for (int q = 0; q < 3; ++q) f12[q] = f32[q] = 0.0;
  }
}

// per triple: force12 and force32 into tripF
// TabulatedAngular::_computeForceRaw (TabulatedAngular.hpp:88-113) in the reference's
// operation order (no clamp of cos(theta), as there).
__device__ __forceinline__ void tab_angle_force(const DevView& d, const double* d12,
                                                const double* d32, double* f12, double* f32) {
  const double d12sq = __dadd_rn(__dadd_rn(__dmul_rn(d12[0], d12[0]), __dmul_rn(d12[1], d12[1])),
                                 __dmul_rn(d12[2], d12[2]));
  const double d32sq = __dadd_rn(__dadd_rn(__dmul_rn(d32[0], d32[0]), __dmul_rn(d32[1], d32[1])),
                                 __dmul_rn(d32[2], d32[2]));
  const double d1232 = __dmul_rn(sqrt(d12sq), sqrt(d32sq));
  const double dot = __dadd_rn(__dadd_rn(__dmul_rn(d12[0], d32[0]), __dmul_rn(d12[1], d32[1])),
                               __dmul_rn(d12[2], d32[2]));
  const double c = __ddiv_rn(dot, d1232);
  double a = tab_value(d.tabs[d.tabAngle], d.tabCoef, true, acos(c));
  a = __dmul_rn(a, __ddiv_rn(1.0, sqrt(__dsub_rn(1.0, __dmul_rn(c, c)))));
  const double a11 = __ddiv_rn(__dmul_rn(a, c), d12sq);
  const double a12 = __ddiv_rn(-a, d1232);
  const double a22 = __ddiv_rn(__dmul_rn(a, c), d32sq);
  for (int q = 0; q < 3; ++q) {
    f12[q] = __dadd_rn(__dmul_rn(a11, d12[q]), __dmul_rn(a12, d32[q]));
    f32[q] = __dadd_rn(__dmul_rn(a22, d32[q]), __dmul_rn(a12, d12[q]));
  }
}

// per triple: force12, force32 of Cosine and/or TabulatedAngular (summed when both act)
__global__ void k_angle_forces(DevView d) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.ntriples) return;
  double d12[3], d32[3], f12[3] = {0, 0, 0}, f32[3] = {0, 0, 0};
  if (triple_dists(d, t, d12, d32)) {
    if (d.cosine.on) cosine_force(d.cosine, d12, d32, f12, f32);
    if (d.tabAngle >= 0) {
      double g12[3], g32[3];
      tab_angle_force(d, d12, d32, g12, g32);
      for (int q = 0; q < 3; ++q) {
        f12[q] = d.cosine.on ? f12[q] + g12[q] : g12[q];
        f32[q] = d.cosine.on ? f32[q] + g32[q] : g32[q];
      }
    }
  } else {
    atomicOr(d.err, kErrBondMissing);
  }
  for (int q = 0; q < 3; ++q) {
    d.tripF[6 * (size_t)t + q] = f12[q];
    d.tripF[6 * (size_t)t + 3 + q] = f32[q];
  }
}

// per particle: p1 += force12, centre -= force12 + force32, p3 += force32
// (FixedTripleListInteractionTemplate::addForces, :183-201), in the order of the
// particle's triple list
template <bool MIXED>
__global__ void k_angle_gather(DevView d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  const int64_t off = d.pa[0].id[i] - d.idMin;
  double f[3] = {0, 0, 0};
  for (int e = d.tripStart[off]; e < d.tripStart[off + 1]; ++e) {
    const int t = d.tripEntry[e] >> 2, role = d.tripEntry[e] & 3;
    const double* F = d.tripF + 6 * (size_t)t;
    for (int q = 0; q < 3; ++q)
      f[q] += role == 0 ? F[q] : (role == 2 ? F[3 + q] : -(F[q] + F[3 + q]));
  }
  const size_t c = d.cap;
  for (int q = 0; q < 3; ++q) {
    if (MIXED)
      d.ffix[q * c + i] += to_fix_d(f[q], d.err);
    else
      d.f64[q * c + i] += f[q];
  }
}

// Energy (FixedTripleListInteractionTemplate::computeEnergy :205-275: minimum image by
// rounding, theta = acos(cos), then Cosine::_computeEnergyRaw (kind 0) or the table's
// getEnergy (kind 1)) or virial d12.f12 + d32.f32.
__global__ void k_angle_obs(DevView d, int energy, int kind, double* partials) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  if (t < d.ntriples) {
    double d12[3], d32[3];
    if (triple_dists(d, t, d12, d32)) {
      if (energy) {
        // getMinimumImageVector: subtract round(d / L) L
        const ParticleArrays a = d.pa[0];
        for (int q = 0; q < 3; ++q) {
          const int k0 = d.id2idx[d.triples[3 * (size_t)t] - d.idMin];
          const int k1 = d.id2idx[d.triples[3 * (size_t)t + 1] - d.idMin];
          const int k2 = d.id2idx[d.triples[3 * (size_t)t + 2] - d.idMin];
          const size_t c = d.cap;
          const double e12 = a.x[q * c + k0] - a.x[q * c + k1];
          const double e32 = a.x[q * c + k2] - a.x[q * c + k1];
          d12[q] = e12 - round(e12 * d.invL[q]) * d.L[q];
          d32[q] = e32 - round(e32 * d.invL[q]) * d.L[q];
        }
        const double s12 = d12[0] * d12[0] + d12[1] * d12[1] + d12[2] * d12[2];
        const double s32 = d32[0] * d32[0] + d32[1] * d32[1] + d32[2] * d32[2];
        const double cth = (d12[0] * d32[0] + d12[1] * d32[1] + d12[2] * d32[2]) /
                           (sqrt(s12) * sqrt(s32));
        acc[0] = kind == 0 ? d.cosine.K * (1.0 + cos(acos(cth) - d.cosine.theta0))
                           : tab_value(d.tabs[d.tabAngle], d.tabCoef, false, acos(cth));
      } else {
        double f12[3], f32[3];
        if (kind == 0)
          cosine_force(d.cosine, d12, d32, f12, f32);
        else
          tab_angle_force(d, d12, d32, f12, f32);
        acc[0] = d12[0] * f12[0] + d12[1] * f12[1] + d12[2] * f12[2] + d32[0] * f32[0] +
                 d32[1] * f32[1] + d32[2] * f32[2];
        acc[1] = d12[0] * f12[0] + d32[0] * f32[0];
        acc[2] = d12[1] * f12[1] + d32[1] * f32[1];
        acc[3] = d12[2] * f12[2] + d32[2] * f32[2];
        acc[4] = d12[0] * f12[1] + d32[0] * f32[1];
        acc[5] = d12[0] * f12[2] + d32[0] * f32[2];
        acc[6] = d12[1] * f12[2] + d32[1] * f32[2];
      }
    }
  }
  block_sum_store<7>(acc, partials);
}

// ---- interaction::Tabulated ---------------------------------------------------------


// Distance vector i - j under the minimum image, and its square in the reference's
// order ((dx dx + dy dy) + dz dz).
__device__ __forceinline__ double tab_dist(const DevView& d, const double* X, int i, int j,
                                           double& dx, double& dy, double& dz) {
  const size_t c = d.cap;
  dx = min_image(X[i] - X[j], d.L[0], d.halfL[0]);
  dy = min_image(X[c + i] - X[c + j], d.L[1], d.halfL[1]);
  dz = min_image(X[2 * c + i] - X[2 * c + j], d.L[2], d.halfL[2]);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Tabulated pair forces over the Verlet list (VerletListTabulated: force = dist *
// getForce(r) / r below the cutoff, Tabulated.hpp:99-115) and tabulated bond forces
// over the fixed pair list (FixedPairListTabulated), added to the forces the main pair
// kernel wrote, or written where there is none (ADD false).  kTabLanes lanes a particle share
// its list and its bonds: one lane a particle leaves 50,000 sites' chains of square root, table
// lookup and division at 340 threads an SM (36 us).  FP64 distances and table arithmetic, the
// reference's operations, in both precision modes (the mixed mode adds the sum as int64 2^-32
// fixed point).
constexpr int kTabLanes = 4;

template <bool MIXED, bool ADD>
__global__ void __launch_bounds__(256, 3) k_force_tab(DevView d) {
  const ParticleArrays a = d.pa[0];
  const int gt = blockIdx.x * blockDim.x + threadIdx.x, sub = gt % kTabLanes;
  const bool act = gt / kTabLanes < d.n;  // every lane stays for the vote and the shuffles
  const int i = act ? gt / kTabLanes : 0;
  const double* X = a.x;
  const size_t c = d.cap;
  const double xi = X[i], yi = X[c + i], zi = X[2 * c + i];
  double f[3] = {0.0, 0.0, 0.0};
  auto add = [&](const TabDesc T, double dx, double dy, double dz) {
    const double r2 =
        __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    if (r2 > T.rcsq) return r2;
    const double r = sqrt(r2);
    const double ff = tab_value(T, d.tabCoef, true, r) / r;
    f[0] += dx * ff;
    f[1] += dy * ff;
    f[2] += dz * ff;
    return r2;
  };
  if (d.tabNT > 0) {
    using Share = ListShare<kTabLanes>;
    const int ti = a.type[i];
    const int32_t* const row = ti < d.tabNT ? d.tabPair + ti * d.tabNT : nullptr;
    // one descriptor for every pair: the table's types are those of its last change, the
    // system's (the LJ table's) may be more by now
    const bool single = d.tabNT == 1 && d.ntypes == 1 && d.tabPair[0] >= 0;
    const TabDesc T0 = d.tabs[single ? d.tabPair[0] : 0];
    auto loop = [&](auto wrap, auto one) {
      constexpr bool ONE = decltype(one)::value;
      Share::walk(d, i, sub, act && row ? d.nn[i] : 0, [&](const int (&j)[Share::ENT], auto next) {
        double xj[Share::ENT], yj[Share::ENT], zj[Share::ENT];
        int tj[Share::ENT];
#pragma unroll
        for (int u = 0; u < Share::ENT; ++u) {
          xj[u] = __ldg(&X[j[u]]);
          yj[u] = __ldg(&X[c + j[u]]);
          zj[u] = __ldg(&X[2 * c + j[u]]);
          tj[u] = ONE ? 0 : __ldg(&a.type[j[u]]);
        }
        next();
#pragma unroll
        for (int u = 0; u < Share::ENT; ++u) {
          // padding entries are the particle itself
          int t = -1;
          if (ONE)
            t = j[u] != i ? 0 : -1;
          else if (j[u] != i && tj[u] < d.tabNT)
            t = row[tj[u]];
          if (t < 0) continue;
          double dx = xi - xj[u], dy = yi - yj[u], dz = zi - zj[u];
          if (decltype(wrap)::value) {
            dx = min_image(dx, d.L[0], d.halfL[0]);
            dy = min_image(dy, d.L[1], d.halfL[1]);
            dz = min_image(dz, d.L[2], d.halfL[2]);
          }
          if constexpr (ONE)
            add(T0, dx, dy, dz);
          else
            add(d.tabs[t], dx, dy, dz);
        }
      });
    };
    const double m = d.wrapMargin;
    const bool inner = xi > m && xi < d.L[0] - m && yi > m && yi < d.L[1] - m && zi > m &&
                       zi < d.L[2] - m;
    // every lane of a warp takes the same branch
    const bool in = __all_sync(0xffffffffu, inner || !act) != 0;
    if (single)
      in ? loop(std::false_type{}, std::true_type{}) : loop(std::true_type{}, std::true_type{});
    else
      in ? loop(std::false_type{}, std::false_type{}) : loop(std::true_type{}, std::false_type{});
  }
  if (act && d.tabBond >= 0 && d.bondStart) {
    const int64_t off = a.id[i] - d.idMin;
    const int b0 = d.bondStart[off] + sub, b1 = d.bondStart[off + 1];
    double bmax = 0.0;
    for (int b = b0; b < b1; b += kTabLanes) {
      const int64_t po = d.bondPartner[b] - d.idMin;
      const int j = (po >= 0 && po < d.idSpan) ? d.id2idx[po] : -1;
      if (j < 0) {
        atomicOr(d.err, kErrBondMissing);
        continue;
      }
      bmax = fmax(bmax, add(d.tabs[d.tabBond], min_image(xi - X[j], d.L[0], d.halfL[0]),
                            min_image(yi - X[c + j], d.L[1], d.halfL[1]),
                            min_image(zi - X[2 * c + j], d.L[2], d.halfL[2])));
    }
    if (b1 > b0) note_bond_sq(d.ctr, bmax);
  }
#pragma unroll
  for (int o = kTabLanes / 2; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 3; ++q) f[q] += __shfl_xor_sync(0xffffffffu, f[q], o, kTabLanes);
  if (!act || sub != 0) return;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (MIXED)
      d.ffix[q * c + i] = to_fix_d(f[q], d.err) + (ADD ? d.ffix[q * c + i] : 0ll);
    else
      d.f64[q * c + i] = ADD ? d.f64[q * c + i] + f[q] : f[q];
  }
}

// Energy (getEnergy(r) - shift below the cutoff) or virial and its tensor of the
// tabulated pair interaction (bond = 0, each Verlet pair once) or the tabulated bonds
// (bond = 1, each bond once).
__global__ void k_tab_obs(DevView d, int bond, int energy, double* partials) {
  const ParticleArrays a = d.pa[0];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  auto add = [&](int t, int j) {
    const TabDesc& T = d.tabs[t];
    double dx, dy, dz;
    const double r2 = tab_dist(d, a.x, i, j, dx, dy, dz);
    if (r2 > T.rcsq) return;
    const double r = sqrt(r2);
    if (energy) {
      acc[0] += tab_value(T, d.tabCoef, false, r) - T.shift;
    } else {
      const double ff = tab_value(T, d.tabCoef, true, r) / r;
      const double f0 = dx * ff, f1 = dy * ff, f2 = dz * ff;
      acc[0] += dx * f0 + dy * f1 + dz * f2;
      acc[1] += dx * f0;
      acc[2] += dy * f1;
      acc[3] += dz * f2;
      acc[4] += dx * f1;
      acc[5] += dx * f2;
      acc[6] += dy * f2;
    }
  };
  if (i < d.n && !is_halo(d, a.id[i])) {
    if (!bond && d.tabNT > 0) {
      const int ti = a.type[i];
      const int cnt = d.nn[i];
      for (int k = 0; k < cnt; ++k) {
        const int j = d.nl[nl_index(k, i, d.cap)];
        if (d.halo ? !pair_counted_here(d, i, j, a.id[i], a.id[j]) : j < i) continue;
        const int tj = a.type[j];
        if (ti >= d.tabNT || tj >= d.tabNT) continue;
        const int t = d.tabPair[ti * d.tabNT + tj];
        if (t >= 0) add(t, j);
      }
    } else if (bond && d.tabBond >= 0 && d.bondStart) {
      const int64_t id = a.id[i];
      const int64_t off = id - d.idMin;
      for (int b = d.bondStart[off]; b < d.bondStart[off + 1]; ++b) {
        const int64_t pid = d.bondPartner[b];
        if (pid <= id) continue;
        const int j = d.id2idx[pid - d.idMin];
        if (j >= 0) add(d.tabBond, j);
      }
    }
  }
  block_sum_store<7>(acc, partials);
}

__global__ void k_kinetic(DevView d, double* partials) {
  const ParticleArrays a = d.pa[0];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[1] = {0.0};
  if (i < d.n && !is_halo(d, a.id[i])) {
    const double vx = a.v[i], vy = a.v[(size_t)d.cap + i], vz = a.v[2 * (size_t)d.cap + i];
    acc[0] = a.mass[i] * (vx * vx + vy * vy + vz * vz);
  }
  block_sum_store<1>(acc, partials);
}

// sum m v^2 and count of the particles whose type t < 64 has bit t set in typeMask
// (Temperature::compute_real with add_type, Temperature.hpp:57-125)
__global__ void k_kinetic_types(DevView d, unsigned long long typeMask, double* partials) {
  const ParticleArrays a = d.pa[0];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[2] = {0.0, 0.0};
  if (i < d.n && !is_halo(d, a.id[i])) {
    const int t = a.type[i];
    if (t >= 0 && t < 64 && ((typeMask >> t) & 1ull)) {
      const double vx = a.v[i], vy = a.v[(size_t)d.cap + i], vz = a.v[2 * (size_t)d.cap + i];
      acc[0] = a.mass[i] * (vx * vx + vy * vy + vz * vz);
      acc[1] = 1.0;
    }
  }
  block_sum_store<2>(acc, partials);
}

// mass * Tensor(v, v) of each particle: (xx, yy, zz, xy, xz, yz), m (v_a v_b)
__global__ void k_kinetic_tensor(DevView d, double* partials) {
  const ParticleArrays a = d.pa[0];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double acc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (i < d.n && !is_halo(d, a.id[i])) {
    const double v[3] = {a.v[i], a.v[(size_t)d.cap + i], a.v[2 * (size_t)d.cap + i]};
    const double m = a.mass[i];
    acc[0] = __dmul_rn(m, __dmul_rn(v[0], v[0]));
    acc[1] = __dmul_rn(m, __dmul_rn(v[1], v[1]));
    acc[2] = __dmul_rn(m, __dmul_rn(v[2], v[2]));
    acc[3] = __dmul_rn(m, __dmul_rn(v[0], v[1]));
    acc[4] = __dmul_rn(m, __dmul_rn(v[0], v[2]));
    acc[5] = __dmul_rn(m, __dmul_rn(v[1], v[2]));
  }
  block_sum_store<6>(acc, partials);
}

__global__ void k_pair_count(DevView d, int32_t* counts) {
  const ParticleArrays a = d.pa[0];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  const int64_t idi = a.id[i];
  if (is_halo(d, idi)) {  // pairs of a halo particle are listed by the domain owning it
    counts[i] = 0;
    return;
  }
  int c = 0;
  for (int k = 0; k < d.nn[i]; ++k) c += a.id[d.nl[nl_index(k, i, d.cap)]] > idi;
  counts[i] = c;
}

__global__ void k_pair_write(DevView d, const int64_t* offsets, int64_t* out) {
  const ParticleArrays a = d.pa[0];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  const int64_t idi = a.id[i];
  if (is_halo(d, idi)) return;
  int64_t o = offsets[i];
  for (int k = 0; k < d.nn[i]; ++k) {
    const int64_t idj = a.id[d.nl[nl_index(k, i, d.cap)]];
    if (idj > idi) {
      out[2 * o] = idi;
      out[2 * o + 1] = idj;
      ++o;
    }
  }
}

// Order-independent digest of the pair set: each unordered pair once (from the particle
// with the smaller id), hashed as mix(mix(smaller id) ^ larger id) with the splitmix64
// finaliser (Steele, Lea and Flood, OOPSLA 2014); per block the count, the wrapping sum,
// the xor and the wrapping sum of a second hash.  Integer sums: the result does not
// depend on the order of the lists.
__global__ void k_pair_digest(DevView d, unsigned long long* partials) {
  const ParticleArrays a = d.pa[0];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long v[4] = {0ull, 0ull, 0ull, 0ull};
  if (i < d.n && !is_halo(d, a.id[i])) {
    const int64_t idi = a.id[i];
    const unsigned long long hi0 = digest_mix((unsigned long long)idi);
    for (int k = 0; k < d.nn[i]; ++k) {
      const int64_t idj = a.id[d.nl[nl_index(k, i, d.cap)]];
      if (idj > idi) {
        const unsigned long long h = digest_mix(hi0 ^ (unsigned long long)idj);
        v[0] += 1ull;
        v[1] += h;
        v[2] ^= h;
        v[3] += digest_mix(h);
      }
    }
  }
  digest_block_store(v, partials);
}

__global__ void k_digest_reduce(const unsigned long long* partials, int nb,
                                unsigned long long* out) {
  unsigned long long v[4] = {0ull, 0ull, 0ull, 0ull};
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    v[0] += partials[(size_t)b * 4];
    v[1] += partials[(size_t)b * 4 + 1];
    v[2] ^= partials[(size_t)b * 4 + 2];
    v[3] += partials[(size_t)b * 4 + 3];
  }
  digest_block_store(v, out);
}

// Particle state by id through the dense id map: scatter host rows into the sorted
// arrays / gather them back out (Storage::lookupRealParticle on the device).
__global__ void k_set_by_id(DevView d, int n, const int64_t* ids, const double* pos,
                            const double* vel, const int32_t* img) {
  const ParticleArrays a = d.pa[0];
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int64_t off = ids[r] - d.idMin;
  const int k = (off >= 0 && off < d.idSpan) ? d.id2idx[off] : -1;
  if (k < 0) {
    atomicOr(d.err, kErrIdRange);
    return;
  }
  for (int c = 0; c < 3; ++c) {
    if (pos) a.x[(size_t)c * d.cap + k] = pos[3 * (size_t)r + c];
    if (vel) a.v[(size_t)c * d.cap + k] = vel[3 * (size_t)r + c];
    if (img) a.img[(size_t)c * d.cap + k] = img[3 * (size_t)r + c];
  }
  if (pos)
    d.posq[k] = fixed_coords(d, a.x[k], a.x[(size_t)d.cap + k], a.x[2 * (size_t)d.cap + k],
                             a.type[k]);
}

__global__ void k_get_by_id(DevView d, int n, const int64_t* ids, double* pos, double* vel,
                            double* force, int32_t* img) {
  const ParticleArrays a = d.pa[0];
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int64_t off = ids[r] - d.idMin;
  const int k = (off >= 0 && off < d.idSpan) ? d.id2idx[off] : -1;
  if (k < 0) {
    atomicOr(d.err, kErrIdRange);
    return;
  }
  for (int c = 0; c < 3; ++c) {
    if (pos) pos[3 * (size_t)r + c] = a.x[(size_t)c * d.cap + k];
    if (vel) vel[3 * (size_t)r + c] = a.v[(size_t)c * d.cap + k];
    if (force) force[3 * (size_t)r + c] = d.ftot[(size_t)c * d.cap + k];
    if (img) img[3 * (size_t)r + c] = a.img[(size_t)c * d.cap + k];
  }
}

}  // namespace

// ---- FP32 throughput probe (the FLOP side of the step's roofline) ---------------------
// Eight independent FMA chains per thread, scalar or packed f32x2; the result is kept live
// by a store that never happens for finite inputs.
template <bool PACKED>
__global__ void __launch_bounds__(256) k_fma_probe(float* out, int iters) {
  const float b = 1.0000001f, c = 1.0e-7f;
  if (PACKED) {
    unsigned long long a[8];
    const unsigned long long bb = f2_pack(b, b), cc = f2_pack(c, c);
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = f2_pack(threadIdx.x * 1e-3f + q, q * 0.5f);
    for (int it = 0; it < iters; ++it) {
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = f2_fma(a[q], bb, cc);
    }
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) s += f2_lo(a[q]) + f2_hi(a[q]);
    if (s == -1.0f) out[blockIdx.x] = s;
  } else {
    float a[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = threadIdx.x * 1e-3f + q;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = fmaf(a[q], b, c);
    }
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) s += a[q];
    if (s == -1.0f) out[blockIdx.x] = s;
  }
}

// ---- launchers ---------------------------------------------------------------------

void launch_fold_bin(const DevView& d, RebuildScratch& s, bool fold, cudaStream_t st) {
  if (d.n > 0) k_fold_bin<<<blocks_for(d.n), kBlock, 0, st>>>(d, s, fold ? 1 : 0);
}

int scan_tiles(int ncells) { return (ncells + kScanTile - 1) / kScanTile; }

// Cell starts, then the particles into their cells' rows of the other copy of the arrays
// (swapped on the device).
void launch_sort_cells(const DevView& d, RebuildScratch& s, cudaStream_t st) {
  const int ntiles = scan_tiles(d.ncells);
  if (ntiles > 1) k_scan_tiles<<<ntiles, kScanBlock, 0, st>>>(s.cellCount, d.ncells, s.tileSum);
  k_scan_apply<<<ntiles, kScanBlock, 0, st>>>(s.cellCount, d.ncells, s.tileSum, d.cellStart);
  if (d.n == 0) return;
  k_scatter<<<blocks_for(d.n), kBlock, 0, st>>>(d, s);
  // 8 lanes a cell up to 6 particles a cell on average
  const bool few = d.n <= 6ll * d.ncells, move = d.n < kMoveApart;
  const int nb = blocks_for(d.ncells, kSortThreads / (few ? 8 : 32));
  if (few)
    move ? k_sort_cells<8, true><<<nb, kSortThreads, 0, st>>>(d, s)
         : k_sort_cells<8, false><<<nb, kSortThreads, 0, st>>>(d, s);
  else
    move ? k_sort_cells<32, true><<<nb, kSortThreads, 0, st>>>(d, s)
         : k_sort_cells<32, false><<<nb, kSortThreads, 0, st>>>(d, s);
  if (!move) k_move<<<blocks_for(d.n), kBlock, 0, st>>>(d, s);
}

int resort_launches(const DevView& d) {
  return 4 + (scan_tiles(d.ncells) > 1 ? 1 : 0) + (d.n < kMoveApart ? 0 : 1);
}

void launch_xrel(const DevView& d, cudaStream_t st) {
  if (d.n > 0) k_xrel<<<blocks_for(d.n), kBlock, 0, st>>>(d);
}

void launch_posq(const DevView& d, cudaStream_t st) {
  if (d.n > 0) k_posq<<<blocks_for(d.n), kBlock, 0, st>>>(d);
}

// Cells binned at the current positions (fresh) with edges 0.1 % above the list cutoff need
// no check of a candidate's cell (see the run form); otherwise each particle's own neighbour
// cells are enforced.  Lists of a capacity beyond kBlockListMax, and systems whose lists do not fit the
// block form's stages, take the run form, which writes its lists as it goes.
void launch_build_nl(const DevView& d, double cutsq, bool fresh, cudaStream_t st) {
  if (d.n == 0) return;
  const double rc = sqrt(cutsq) * (1.0 + 1e-3) / d.hci;
  bool stencil = !fresh;
  for (int k = 0; k < 3; ++k) stencil = stencil || d.cellSize[k] < rc;
  const bool excl = d.exclStart != nullptr;
  const BuildBand band = build_band(d, cutsq);
#define ESPP_BUILD_CASE(KERNEL, NB, NT)                                    \
  do {                                                                     \
    if (excl)                                                              \
      stencil ? KERNEL(true, true)<<<NB, NT, 0, st>>>(d, cutsq, band)      \
              : KERNEL(true, false)<<<NB, NT, 0, st>>>(d, cutsq, band);    \
    else                                                                   \
      stencil ? KERNEL(false, true)<<<NB, NT, 0, st>>>(d, cutsq, band)     \
              : KERNEL(false, false)<<<NB, NT, 0, st>>>(d, cutsq, band);   \
  } while (0)
#define ESPP_RUN(E, S) k_build_nl_run<E, S>
#define ESPP_BLOCK(E, S) k_build_block<E, S, false>
#define ESPP_BLOCK2(E, S) k_build_block<E, S, true>
  if (d.K > kBlockListMax || d.runForm)
    ESPP_BUILD_CASE(ESPP_RUN, blocks_for((long long)d.n, kRunWarps * 32), kRunWarps * 32);
  else if (d.n < kBuildSplit)
    ESPP_BUILD_CASE(ESPP_BLOCK2, 2 * blocks_for((long long)d.n, 32), 32 * kBlockW);
  else
    ESPP_BUILD_CASE(ESPP_BLOCK, blocks_for((long long)d.n, 32), 32 * kBlockW);
#undef ESPP_BUILD_CASE
#undef ESPP_RUN
#undef ESPP_BLOCK
#undef ESPP_BLOCK2
}

template <int TPP, bool MIXED>
static void force_dispatch(const DevView& d, bool single, bool capped, bool fene,
                           const FENEParams& fp, cudaStream_t st) {
  const int grid = blocks_for((long long)d.n * TPP);
#define ESPP_FORCE_CASE(S, C, F)                                                   \
  if (single == S && capped == C && fene == F) {                                   \
    if (MIXED)                                                                     \
      k_force_mixed<TPP, S, C, F><<<grid, kBlock, 0, st>>>(d, fp);                 \
    else                                                                           \
      k_force_fp64<TPP, S, C, F><<<grid, kBlock, 0, st>>>(d, fp);                  \
    return;                                                                        \
  }
  ESPP_FORCE_CASE(true, false, false)
  ESPP_FORCE_CASE(true, false, true)
  ESPP_FORCE_CASE(true, true, false)
  ESPP_FORCE_CASE(true, true, true)
  ESPP_FORCE_CASE(false, false, false)
  ESPP_FORCE_CASE(false, false, true)
  ESPP_FORCE_CASE(false, true, false)
  ESPP_FORCE_CASE(false, true, true)
#undef ESPP_FORCE_CASE
}

double measure_fp32_tflops(int nsm, cudaStream_t st) {
  const int blocks = nsm * 8, threads = 256, iters = 8192;
  float* out = nullptr;
  cudaMalloc(&out, sizeof(float) * blocks);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  double best = 0.0;
  for (int packed = 0; packed < 2; ++packed) {
    for (int rep = 0; rep < 3; ++rep) {
      cudaEventRecord(e0, st);
      if (packed)
        k_fma_probe<true><<<blocks, threads, 0, st>>>(out, iters);
      else
        k_fma_probe<false><<<blocks, threads, 0, st>>>(out, iters);
      cudaEventRecord(e1, st);
      cudaEventSynchronize(e1);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      const double flops = 2.0 * (packed ? 16.0 : 8.0) * iters * (double)blocks * threads;
      if (ms > 0.f && rep > 0) best = fmax(best, flops / (ms * 1e-3) / 1e12);
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  return best;
}

// The failure path of the tensor-core kernels, run on purpose: one CTA holds TMEM and
// waits on an mbarrier that nothing arrives on, with the same bounded wait the kernels
// use but `spins` tries; when the wait gives up it sets kErrTimeout, releases the TMEM
// and returns.  out[0] = nanoseconds spent in the wait, out[1] = 1 if it gave up.
__global__ void __launch_bounds__(32) k_wait_selftest(unsigned* err, long long spins,
                                                      unsigned long long* out) {
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_base;
  tc::tmem_alloc(tc::smem_u32(&tmem_base), 32);
  if (threadIdx.x == 0) tc::mbar_init(tc::smem_u32(&mbar));
  __syncwarp();
  tc::fence_after();
  if (threadIdx.x == 0) {
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    const bool done = tc::mbar_wait(tc::smem_u32(&mbar), 0, spins);
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    if (!done) atomicOr(err, kErrTimeout);
    out[0] = t1 - t0;
    out[1] = done ? 0ull : 1ull;
  }
  __syncwarp();
  tc::fence_before();
  tc::tmem_dealloc(tmem_base, 32);
}

void launch_wait_selftest(unsigned* err, long long spins, unsigned long long* out,
                          cudaStream_t st) {
  k_wait_selftest<<<1, 32, 0, st>>>(err, spins, out);
}

void launch_forces(const DevView& d, bool mixed, const FENEParams& fp, int tpp,
                   cudaStream_t st) {
  if (d.n == 0) return;
  const bool fene = fp.on != 0;
  switch (tpp) {
    case 2:
      mixed ? force_dispatch<2, true>(d, d.ljSingle != 0, d.ljCapped != 0, fene, fp, st)
            : force_dispatch<2, false>(d, d.ljSingle != 0, d.ljCapped != 0, fene, fp, st);
      break;
    case 4:
      mixed ? force_dispatch<4, true>(d, d.ljSingle != 0, d.ljCapped != 0, fene, fp, st)
            : force_dispatch<4, false>(d, d.ljSingle != 0, d.ljCapped != 0, fene, fp, st);
      break;
    case 8:
      mixed ? force_dispatch<8, true>(d, d.ljSingle != 0, d.ljCapped != 0, fene, fp, st)
            : force_dispatch<8, false>(d, d.ljSingle != 0, d.ljCapped != 0, fene, fp, st);
      break;
    default:
      mixed ? force_dispatch<1, true>(d, d.ljSingle != 0, d.ljCapped != 0, fene, fp, st)
            : force_dispatch<1, false>(d, d.ljSingle != 0, d.ljCapped != 0, fene, fp, st);
  }
}


void launch_integrate(const DevView& d, const IntegrateArgs& a, cudaStream_t st) {
  if (d.n == 0) return;
  if (a.mixed)
    k_integrate<true><<<blocks_for(d.n), kBlock, 0, st>>>(d, a);
  else
    k_integrate<false><<<blocks_for(d.n), kBlock, 0, st>>>(d, a);
}

void launch_decide(const DevView& d, double skinHalf, cudaStream_t st) {
  k_decide<<<1, 1, 0, st>>>(d.ctr, skinHalf);
}

void launch_decide_graph(const DevView& d, double skinHalf, cudaGraphConditionalHandle hIf,
                         cudaGraphConditionalHandle hWhile, cudaStream_t st) {
  k_decide_graph<<<1, 1, 0, st>>>(d.ctr, skinHalf, hIf, hWhile);
}

namespace {
template <bool MIXED, int T>
cudaError_t steps_dispatch(const DevView& d, const FENEParams& fp, const IntegrateArgs& a,
                           double skinHalf, StepSync* sync,
                           cudaGraphConditionalHandle hIf, cudaGraphConditionalHandle hWhile,
                           int nsm, cudaStream_t st) {
  using Kernel = void (*)(DevView, FENEParams, IntegrateArgs, double, StepSync*,
                          cudaGraphConditionalHandle, cudaGraphConditionalHandle);
  const bool single = d.ljSingle != 0, capped = d.ljCapped != 0, fene = fp.on != 0;
  Kernel f = nullptr;
#define ESPP_STEPS_CASE(S, C, F) \
  if (single == S && capped == C && fene == F) f = k_steps<MIXED, T, S, C, F>;
  ESPP_STEPS_CASE(true, false, false)
  ESPP_STEPS_CASE(true, false, true)
  ESPP_STEPS_CASE(true, true, false)
  ESPP_STEPS_CASE(true, true, true)
  ESPP_STEPS_CASE(false, false, false)
  ESPP_STEPS_CASE(false, false, true)
  ESPP_STEPS_CASE(false, true, false)
  ESPP_STEPS_CASE(false, true, true)
#undef ESPP_STEPS_CASE
  // one block an SM, as large as the particles need to fill them all
  const long long lanes = (long long)d.n * T;
  int block = (int)((lanes + nsm - 1) / nsm + 31) / 32 * 32;
  if (block < 64) block = 64;
  if (block > kStepThreads<MIXED>) return cudaErrorCooperativeLaunchTooLarge;
  const size_t smem = sizeof(uint32_t) * kStepWords * (block / T);
  cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int perSm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, f, block, smem);
  if (e != cudaSuccess) return e;
  const int grid = blocks_for(lanes, block);
  if ((long long)perSm * nsm < grid) return cudaErrorCooperativeLaunchTooLarge;
  DevView dv = d;
  FENEParams fv = fp;
  IntegrateArgs av = a;
  void* args[] = {&dv, &fv, &av, &skinHalf, &sync, &hIf, &hWhile};
  return cudaLaunchCooperativeKernel((const void*)f, dim3(grid), dim3(block), args, smem, st);
}
}  // namespace

int step_threads(bool mixed) { return mixed ? kStepThreads<true> : kStepThreads<false>; }

cudaError_t launch_steps(const DevView& d, bool mixed, const FENEParams& fp,
                         const IntegrateArgs& a, double skinHalf, StepSync* sync,
                         cudaGraphConditionalHandle hIf, cudaGraphConditionalHandle hWhile,
                         int tpp, int nsm, cudaStream_t st) {
#define ESPP_STEPS(T)                                                                        \
  return mixed ? steps_dispatch<true, T>(d, fp, a, skinHalf, sync, hIf, hWhile, nsm, st)     \
               : steps_dispatch<false, T>(d, fp, a, skinHalf, sync, hIf, hWhile, nsm, st)
  switch (tpp) {
    case 1: ESPP_STEPS(1);
    case 2: ESPP_STEPS(2);
    case 4: ESPP_STEPS(4);
    default: ESPP_STEPS(8);
  }
#undef ESPP_STEPS
}

void launch_lj_observables(const DevView& d, double* partials, int nblocks, double* out,
                           int energy, cudaStream_t st) {
#define ESPP_OBS_CASE(E, S)                          \
  if ((energy != 0) == E && (d.ljSingle != 0) == S) \
    k_lj_obs<E, S><<<nblocks, kBlock, 0, st>>>(d, partials);
  ESPP_OBS_CASE(true, true)
  ESPP_OBS_CASE(true, false)
  ESPP_OBS_CASE(false, true)
  ESPP_OBS_CASE(false, false)
#undef ESPP_OBS_CASE
  k_sum_partials<7><<<1, kSumThreads, 0, st>>>(partials, nblocks, out);
}

void launch_fene_observables(const DevView& d, const FENEParams& fp, double* partials,
                             int nblocks, double* out, int energy, cudaStream_t st) {
  k_fene_obs<<<nblocks, kBlock, 0, st>>>(d, fp, energy, partials);
  k_sum_partials<7><<<1, kSumThreads, 0, st>>>(partials, nblocks, out);
}

// Bound on the error of |d| / dr in k_rdf's FP32 arithmetic: six roundings of 6e-8 on a distance
// of up to rdfN bins, and the packed coordinates' unit of L / 2^32 an axis; at least 2e-6 rdfN.
static double rdf_eps(const DevView& d, int rdfN, double dr) {
  const double unit =
      sqrt(d.L[0] * d.L[0] + d.L[1] * d.L[1] + d.L[2] * d.L[2]) / 4294967296.0 / dr;
  return std::max(2e-6 * rdfN, 4e-7 * rdfN + 1.1 * unit);
}

void launch_rdf(const DevView& d, int rdfN, double dr, unsigned long long* hist,
                cudaStream_t st) {
  if (d.n < 2) return;
  const long long ntiles = (d.n + kRdfTile - 1) / kRdfTile;
  const long long nblocks = ntiles * (ntiles + 1) / 2;
  // as many copies of the counts as 32 KB hold, a power of two up to one a bank
  int copies = 1;
  while (copies < 32 && 2 * copies * rdfN <= 8192) copies *= 2;
  const size_t smem = sizeof(unsigned) * rdfN * copies;
  const double eps = rdf_eps(d, rdfN, dr);
  if (rdfN <= kRdfSmemBins && eps <= kRdfFastEps)
    k_rdf<true, true><<<(unsigned)nblocks, kRdfTile, smem, st>>>(d, rdfN, (int)ntiles, dr,
                                                                 (float)(0.5 - eps), copies, hist);
  else if (rdfN <= kRdfSmemBins)
    k_rdf<true, false><<<(unsigned)nblocks, kRdfTile, smem, st>>>(d, rdfN, (int)ntiles, dr, 0.f,
                                                                  copies, hist);
  else
    k_rdf<false, false><<<(unsigned)nblocks, kRdfTile, 0, st>>>(d, rdfN, (int)ntiles, dr, 0.f, 1,
                                                                hist);
}

static bool has_angles(const DevView& d) {
  return d.n > 0 && d.ntriples > 0 && (d.cosine.on || d.tabAngle >= 0);
}

void launch_angle_terms(const DevView& d, cudaStream_t st) {
  if (has_angles(d)) k_angle_forces<<<blocks_for(d.ntriples), kBlock, 0, st>>>(d);
}

void launch_angle_forces(const DevView& d, bool mixed, cudaStream_t st) {
  if (!has_angles(d)) return;
  if (mixed)
    k_angle_gather<true><<<blocks_for(d.n), kBlock, 0, st>>>(d);
  else
    k_angle_gather<false><<<blocks_for(d.n), kBlock, 0, st>>>(d);
}

void launch_angle_observables(const DevView& d, double* partials, int nblocks, double* out,
                              int energy, int kind, cudaStream_t st) {
  k_angle_obs<<<nblocks, kBlock, 0, st>>>(d, energy, kind, partials);
  k_sum_partials<7><<<1, kSumThreads, 0, st>>>(partials, nblocks, out);
}

void launch_force_tab(const DevView& d, bool mixed, bool add, cudaStream_t st) {
  if (d.n == 0 || !has_tab_forces(d)) return;
  const int nb = blocks_for((long long)d.n * kTabLanes);
  if (mixed)
    add ? k_force_tab<true, true><<<nb, kBlock, 0, st>>>(d)
        : k_force_tab<true, false><<<nb, kBlock, 0, st>>>(d);
  else
    add ? k_force_tab<false, true><<<nb, kBlock, 0, st>>>(d)
        : k_force_tab<false, false><<<nb, kBlock, 0, st>>>(d);
}

void launch_tab_observables(const DevView& d, int bond, double* partials, int nblocks,
                            double* out, int energy, cudaStream_t st) {
  k_tab_obs<<<nblocks, kBlock, 0, st>>>(d, bond, energy, partials);
  k_sum_partials<7><<<1, kSumThreads, 0, st>>>(partials, nblocks, out);
}

void launch_kinetic(const DevView& d, double* partials, int nblocks, double* out,
                    cudaStream_t st) {
  k_kinetic<<<nblocks, kBlock, 0, st>>>(d, partials);
  k_sum_partials<1><<<1, kSumThreads, 0, st>>>(partials, nblocks, out);
}

void launch_kinetic_types(const DevView& d, unsigned long long typeMask, double* partials,
                          int nblocks, double* out, cudaStream_t st) {
  k_kinetic_types<<<nblocks, kBlock, 0, st>>>(d, typeMask, partials);
  k_sum_partials<2><<<1, kSumThreads, 0, st>>>(partials, nblocks, out);
}

void launch_kinetic_tensor(const DevView& d, double* partials, int nblocks, double* out,
                           cudaStream_t st) {
  k_kinetic_tensor<<<nblocks, kBlock, 0, st>>>(d, partials);
  k_sum_partials<6><<<1, kSumThreads, 0, st>>>(partials, nblocks, out);
}

void launch_pair_count(const DevView& d, int32_t* counts, cudaStream_t st) {
  if (d.n > 0) k_pair_count<<<blocks_for(d.n), kBlock, 0, st>>>(d, counts);
}

void launch_pair_write(const DevView& d, const int64_t* offsets, int64_t* out,
                       cudaStream_t st) {
  if (d.n > 0) k_pair_write<<<blocks_for(d.n), kBlock, 0, st>>>(d, offsets, out);
}

void launch_pair_digest(const DevView& d, unsigned long long* partials, int nblocks,
                        unsigned long long* out, cudaStream_t st) {
  k_pair_digest<<<nblocks, kBlock, 0, st>>>(d, partials);
  k_digest_reduce<<<1, kBlock, 0, st>>>(partials, nblocks, out);
}

int observable_blocks(int n) { return blocks_for(n > 0 ? n : 1); }

void launch_set_by_id(const DevView& d, int n, const int64_t* ids, const double* pos,
                      const double* vel, const int32_t* img, cudaStream_t st) {
  if (n > 0) k_set_by_id<<<blocks_for(n), kBlock, 0, st>>>(d, n, ids, pos, vel, img);
}

void launch_get_by_id(const DevView& d, int n, const int64_t* ids, double* pos, double* vel,
                      double* force, int32_t* img, cudaStream_t st) {
  if (n > 0) k_get_by_id<<<blocks_for(n), kBlock, 0, st>>>(d, n, ids, pos, vel, force, img);
}

}  // namespace espp
