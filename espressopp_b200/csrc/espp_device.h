// espp_device.h - device helpers shared by the kernel files: fixed-point coordinates,
// packed FP32 arithmetic, the reference's exact pair test, fixed-order reductions and
// the pair-set digest.
#pragma once

#include <stdint.h>

#include "espp_internal.h"

namespace espp {
namespace {

constexpr int kBlock = 256;

inline int blocks_for(long long n, int b = kBlock) { return (int)((n + b - 1) / b); }

__device__ __forceinline__ int4 fixed_coords(const DevView& d, double x, double y, double z,
                                             int type) {
  // box-wrapped int32: the low 32 bits of round(x * 2^32 / L)
  long long qx = __double2ll_rn(x * d.fixScale[0]);
  long long qy = __double2ll_rn(y * d.fixScale[1]);
  long long qz = __double2ll_rn(z * d.fixScale[2]);
  return make_int4((int)(unsigned)qx, (int)(unsigned)qy, (int)(unsigned)qz, type);
}

// A halo particle is a copy of a particle that another domain of a spatial
// decomposition owns (a ghost of DomainDecomposition's frame cells, DomainDecomposition.
// cpp:1243-1391): it takes part in this domain's pairs and bonds as a partner only, is not
// integrated or thermostatted, and is skipped as the first particle of every observable.
__device__ __forceinline__ bool is_halo(const DevView& d, int64_t id) {
  return d.halo && d.halo[id - d.idMin];
}

// Pair (i, j) of a full list is counted once by the observables: by its lower sorted index
// in a system without halo particles; with halo particles, a pair of two owned particles
// by the lower index and a pair with a halo partner by the lower id, so that the domains
// of a decomposition together count every pair once.
__device__ __forceinline__ bool pair_counted_here(const DevView& d, int i, int j, int64_t idi,
                                                  int64_t idj) {
  if (!d.halo) return j > i;
  return d.halo[idj - d.idMin] ? idj > idi : j > i;
}

// FixedPairListInteractionTemplate.hpp:145-150: every force pass raises the list's
// long-time maximum bond length^2 to the longest bond it saw.  The maximum is kept as the
// bits of a non-negative double, which order like unsigned integers; the atomic is issued
// only by a thread whose bond is longer than the stored value.
__device__ __forceinline__ void note_bond_sq(DevCounters* c, double r2) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(r2);
  if (b > *(volatile unsigned long long*)&c->ltMaxBondSq) atomicMax(&c->ltMaxBondSq, b);
}

__device__ __forceinline__ float wrapped_diff(int a, int b, float unit) {
  return (float)(int)((unsigned)a - (unsigned)b) * unit;
}

__device__ __forceinline__ float wrapped_diff(int a, int b) {
  return (float)(int)((unsigned)a - (unsigned)b);
}

// 16-byte read of the Verlet list that does not allocate in L1, so that the list stream
// leaves L1 to the coordinate gathers
__device__ __forceinline__ int4 ld_list(const int4* p) {
  int4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ int2 ld_list2(const int2* p) {
  int2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.s32 {%0, %1}, [%2];"
               : "=r"(v.x), "=r"(v.y)
               : "l"(p));
  return v;
}

__device__ __forceinline__ float fast_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// A lane's share of the Verlet list when T lanes work on a particle.  The lanes of a particle
// take adjacent entries of the same block of 8 (lane s of 4: entries 2s, 2s + 1; 8 lanes: two
// blocks at a time), so the 32 coordinate gathers of a warp fall on the few cache lines that
// 32 / T particles' neighbouring partners share: 16.3 lines a gather with one lane a particle,
// 9.8 with four on adjacent entries (counted on the sorted 110,592-particle fluid).
// f(j) receives the ENT entries of one step; entries past the list are the particle itself.
template <int T>
struct ListShare {
  static constexpr int E = T == 1 ? 8 : (T == 2 ? 4 : 2);  // entries of a block a lane takes
  static constexpr int U = E == 2 ? 2 : 1;                 // blocks of one step
  static constexpr int ENT = E * U;
  static constexpr int kStride = T == 8 ? 2 : 1;           // blocks between a lane's blocks

  template <class F>
  static __device__ __forceinline__ void walk(const DevView& d, int i, int sub, int cnt, F&& f) {
    const int nblk = (cnt + 7) >> 3;
    const int first = T == 8 ? sub >> 2 : 0;
    const int* p = d.nl + nl_index(8 * first, i, d.cap) + (T >= 4 ? (sub & 3) * 2 : sub * E);
    const size_t step = (size_t)d.cap * 8 * kStride;
    int w[ENT];
    auto fetch = [&](int b) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool in = b + u * kStride < nblk;
        const int* q = p + u * step;
        if (E == 2) {
          int2 v = make_int2(i, i);
          if (in) v = ld_list2(reinterpret_cast<const int2*>(q));
          w[2 * u] = v.x;
          w[2 * u + 1] = v.y;
        } else {
#pragma unroll
          for (int h = 0; h < E / 4; ++h) {
            int4 v = make_int4(i, i, i, i);
            if (in) v = ld_list(reinterpret_cast<const int4*>(q) + h);
            w[4 * h] = v.x;
            w[4 * h + 1] = v.y;
            w[4 * h + 2] = v.z;
            w[4 * h + 3] = v.w;
          }
        }
      }
      p += U * step;
    };
    fetch(first);
    for (int b = first; b < nblk; b += U * kStride) {
      int j[ENT];
#pragma unroll
      for (int u = 0; u < ENT; ++u) j[u] = w[u];
      // the next step's entries are loaded before this step's coordinates are used
      f(j, [&] { fetch(b + U * kStride); });
    }
  }
};

__device__ __forceinline__ void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

__device__ __forceinline__ float fast_sqrt(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ bool is_excluded(const DevView& d, int64_t a, int64_t b) {
  if (!d.exclStart) return false;
  int64_t off = a - d.idMin;
  int e0 = d.exclStart[off], e1 = d.exclStart[off + 1];
  for (int e = e0; e < e1; ++e)
    if (d.exclIds[e] == b) return true;
  return false;
}

// The reference's FP64 inclusion test for one candidate pair (rarely reached: only
// candidates whose FP32 distance lies within the 2e-5 band around the cutoff).
__device__ __forceinline__ bool exact_pair_test_inl(const double* __restrict__ x, size_t cap,
                                                   int i, int j, bool fwd, double sx, double sy,
                                                   double sz, double cutsq) {
  const double xi = x[i], yi = x[cap + i], zi = x[2 * cap + i];
  const double xj = x[j], yj = x[cap + j], zj = x[2 * cap + j];
  double ex, ey, ez;
  if (fwd) {  // p1 = i, p2 = ghost of j at xj + s
    ex = __dsub_rn(xi, __dadd_rn(xj, sx));
    ey = __dsub_rn(yi, __dadd_rn(yj, sy));
    ez = __dsub_rn(zi, __dadd_rn(zj, sz));
  } else {  // p1 = j, p2 = ghost of i at xi - s
    ex = __dsub_rn(xj, __dadd_rn(xi, -sx));
    ey = __dsub_rn(yj, __dadd_rn(yi, -sy));
    ez = __dsub_rn(zj, __dadd_rn(zi, -sz));
  }
  const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez));
  return !(d2 > cutsq);
}
__device__ __noinline__ bool exact_pair_test(const double* __restrict__ x, size_t cap, int i,
                                             int j, bool fwd, double sx, double sy, double sz,
                                             double cutsq) {
  return exact_pair_test_inl(x, cap, i, j, fwd, sx, sy, sz, cutsq);
}

// Packed FP32 pairs (sm_100 f32x2 arithmetic): two particles' coordinates in one 64-bit
// register, low half first.
// The two halves form one 64-bit register pair (mov.b64 with a vector operand), so
// packing and unpacking are register moves rather than 64-bit shifts.
__device__ __forceinline__ unsigned long long f2_pack(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ unsigned long long f2_sub(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b,
                                                     unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

#pragma nv_diag_suppress 550  // the other half of the unpacked pair is not needed
__device__ __forceinline__ float f2_lo(unsigned long long v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return lo;
}
__device__ __forceinline__ float f2_hi(unsigned long long v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return hi;
}
#pragma nv_diag_default 550

__device__ __forceinline__ long long to_fix(float f, unsigned* err) {
  if (!(fabsf(f) < 1.0e9f)) atomicOr(err, kErrFixOverflow);
  return __float2ll_rn(f * 4294967296.0f);
}

// The same for a sum held in two packed partial sums, each rounded by itself: the total obeys
// the same limit, and no partial sum leaves the range.
__device__ __forceinline__ long long to_fix2(unsigned long long f, unsigned* err) {
  const float a = f2_lo(f), b = f2_hi(f);
  if (!(fabsf(a + b) < 1.0e9f) || !(fmaxf(fabsf(a), fabsf(b)) < 1.0e9f))
    atomicOr(err, kErrFixOverflow);
  return __float2ll_rn(a * 4294967296.0f) + __float2ll_rn(b * 4294967296.0f);
}

template <int NV>
__device__ void block_sum_store(double (&v)[NV], double* partials) {
  __shared__ double sm[NV][kBlock / 32];
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    double t = v[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) sm[c][threadIdx.x >> 5] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int c = 0; c < NV; ++c) {
      double t = 0.0;
      for (int w = 0; w < (int)(blockDim.x / 32); ++w) t += sm[c][w];
      partials[(size_t)blockIdx.x * NV + c] = t;
    }
  }
}

// Fixed-order sum of the block partials (one block of kSumThreads) -> out[0..NV)
constexpr int kSumThreads = 1024;
template <int NV>
__global__ void __launch_bounds__(kSumThreads) k_sum_partials(const double* __restrict__ partials,
                                                              int nblocks, double* out) {
  __shared__ double sm[NV][kSumThreads / 32];
  double acc[NV];
#pragma unroll
  for (int c = 0; c < NV; ++c) acc[c] = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += kSumThreads)
#pragma unroll
    for (int c = 0; c < NV; ++c) acc[c] += partials[(size_t)b * NV + c];
#pragma unroll
  for (int c = 0; c < NV; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if ((threadIdx.x & 31) == 0) sm[c][threadIdx.x >> 5] = acc[c];
  }
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int c = 0; c < NV; ++c) {
      double t = sm[c][threadIdx.x];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (threadIdx.x == 0) out[c] = t;
    }
  }
}

__device__ __forceinline__ unsigned long long digest_mix(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ void digest_block_store(unsigned long long (&v)[4],
                                                   unsigned long long* partials) {
  __shared__ unsigned long long sm[4][kBlock / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    v[1] += __shfl_xor_sync(0xffffffffu, v[1], o);
    v[2] ^= __shfl_xor_sync(0xffffffffu, v[2], o);
    v[3] += __shfl_xor_sync(0xffffffffu, v[3], o);
  }
  if ((threadIdx.x & 31) == 0)
    for (int c = 0; c < 4; ++c) sm[c][threadIdx.x >> 5] = v[c];
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t[4] = {0ull, 0ull, 0ull, 0ull};
    for (int w = 0; w < (int)(blockDim.x / 32); ++w) {
      t[0] += sm[0][w];
      t[1] += sm[1][w];
      t[2] ^= sm[2][w];
      t[3] += sm[3][w];
    }
    for (int c = 0; c < 4; ++c) partials[(size_t)blockIdx.x * 4 + c] = t[c];
  }
}

}  // namespace
}  // namespace espp
