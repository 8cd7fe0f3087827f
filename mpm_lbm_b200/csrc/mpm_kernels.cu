// Particle-side kernels of the coupled FSI step: MPM -> LBM projection,
// LBM -> MPM reaction transfer and the MLS-MPM substep.
//
// Reference semantics:
//   projection      src/mpm_lbm/sim/coupling/projection.py:21-97
//   penalty react.  src/mpm_lbm/sim/coupling/penalty.py:90-129
//   engineering     src/mpm_lbm/sim/coupling/moving_boundary.py:58-110
//   link-area       src/mpm_lbm/sim/coupling/link_area.py:84-193
//                   (+ link_area_accounting.py:42-148 for the area scale)
//   MPM substep     src/mpm_lbm/sim/mpm/solid.py:212-315
// Particle fields are planar ([comp][n]); the MPM grid and the lattice are
// x-fastest: node = (k * n + j) * n + i, cell = (k * ny + j) * nx + i.

#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>

#include "common.cuh"
#include "mpm_common.cuh"

namespace fsi {

// ---------------------------------------------------------- projection ----
// Float-atomic scatter of the particles vb * kPsT ..., kPsT threads: each warp
// stages its 32 particles in shared memory and takes the runs of consecutive
// particles with one base cell (neighbours in a body are neighbours in
// memory) one after the other, lane o on stencil cell o, so that a run gives
// each cell one atomic per field instead of one per particle; particles in
// random order cost no more atomics than before.  Bound by the atomics: a
// thread per particle with its own 27 x 5 (and 27 divisions) took 136 us for
// the 16-case batch, this takes 77 us.
constexpr int kPsT = 128;
enum { kPsY = 4, kPsZ = 8, kPsQ = 12, kPsN = 20 };  // record: wx0..2 base0, wy base1, wz base2, vol/cell m mv0 mv1, mv2

__device__ __forceinline__ void project_scatter_body(const LatView& L, const FsiParticles& pt,
                                                     const FsiCouplingParams& cp, float* phi, float* smass, float* svel,
                                                     int p0) {
  __shared__ float4 s_rec[kPsT * kPsN / 4];
  const int lane = threadIdx.x & 31, n = pt.n, p = p0 + threadIdx.x;
  float* const warp_rec = reinterpret_cast<float*>(s_rec) + (threadIdx.x & ~31) * kPsN;
  const bool live = p < n;
  BSpline b;
  b.base[0] = b.base[1] = b.base[2] = 0;
  __syncwarp();
  if (live) {
    const float X[3] = {pt.x[p], pt.x[n + p], pt.x[2 * n + p]};
    bspline(X, cp.inv_dx_norm, b);
    const float vol = pt.vol0[p] * fmaxf(pt.Jp[p], 0.0f), m = pt.mass[p];
    float* const r = warp_rec + lane * kPsN;
#pragma unroll
    for (int a = 0; a < 3; ++a)
      *reinterpret_cast<float4*>(r + 4 * a) = make_float4(b.w[a][0], b.w[a][1], b.w[a][2], __int_as_float(b.base[a]));
    *reinterpret_cast<float4*>(r + kPsQ) = make_float4(vol / cp.cell_volume_norm, m, m * (pt.v[p] * cp.vel_scale),
                                                       m * (pt.v[n + p] * cp.vel_scale));
    r[kPsQ + 4] = m * (pt.v[2 * n + p] * cp.vel_scale);
  }
  const int q0 = __shfl_up_sync(0xffffffffu, b.base[0], 1), q1 = __shfl_up_sync(0xffffffffu, b.base[1], 1),
            q2 = __shfl_up_sync(0xffffffffu, b.base[2], 1);
  unsigned m = __ballot_sync(0xffffffffu, live && (lane == 0 || q0 != b.base[0] || q1 != b.base[1] || q2 != b.base[2]));
  const int count = __popc(__ballot_sync(0xffffffffu, live));  // the warp's particles are its first lanes
  __syncwarp();
  const int ox = min(lane / 9, 2), oy = (lane / 3) % 3, oz = lane % 3;  // lanes 27-31 are not used
  while (m) {
    const int first = __ffs(m) - 1;
    m &= m - 1;
    const int end = m ? __ffs(m) - 1 : count;
    const float* r = warp_rec + first * kPsN;
    const int I = __float_as_int(r[3]) + ox, J = __float_as_int(r[kPsY + 3]) + oy, K = __float_as_int(r[kPsZ + 3]) + oz;
    float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    for (int i = first; i < end; ++i, r += kPsN) {
      const float w = r[ox] * r[kPsY + oy] * r[kPsZ + oz];
      const float4 t = *reinterpret_cast<const float4*>(r + kPsQ);
      acc[0] += w * t.x;
      acc[1] += w * t.y;
      acc[2] += w * t.z;
      acc[3] += w * t.w;
      acc[4] += w * r[kPsQ + 4];
    }
    if (lane < 27 && I >= 0 && I < L.nx && J >= 0 && J < L.ny && K >= 0 && K < L.nz) {
      const int64_t c = lat_cell(L, I, J, K);
      atomicAdd(phi + c, acc[0]);
      atomicAdd(smass + c, acc[1]);
#pragma unroll
      for (int a = 0; a < 3; ++a) atomicAdd(svel + a * L.pitch + c, acc[2 + a]);
    }
  }
}

__global__ void __launch_bounds__(kPsT) k_project_scatter(LatView L, FsiParticles pt, FsiCouplingParams cp, float* phi,
                                                          float* smass, float* svel) {
  project_scatter_body(L, pt, cp, phi, smass, svel, blockIdx.x * kPsT);
}

// normalize_projection (projection.py:67-91) of one cell, with the cell's
// share of the projection statistics accumulated in a
struct ProjAcc {
  double pm = 0.0, pvr = 0.0, pvc = 0.0;
  float mx = 0.f;
  int na = 0;
};

__device__ __forceinline__ void project_stat_cell(const FsiCouplingParams& cp, float raw, float cl, float m,
                                                  ProjAcc& a) {
  a.mx = fmaxf(a.mx, raw);
  a.na += cl > 1.0e-8f;
  a.pm += m;
  a.pvr += (double)raw * cp.cell_volume_norm;
  a.pvc += (double)cl * cp.cell_volume_norm;
}

__device__ __forceinline__ void project_normalize_cell(const LatView& L, const FsiCouplingParams& cp, float* phi,
                                                       float* smass, float* svel, int64_t c, ProjAcc& a) {
  const float raw = phi[c];
  const float m = smass[c];
  if (m > cp.eps_mass) {
    for (int q = 0; q < 3; ++q) svel[q * L.pitch + c] = svel[q * L.pitch + c] / m;
  } else {
    for (int q = 0; q < 3; ++q) svel[q * L.pitch + c] = 0.f;
  }
  const float cl = fminf(1.0f, fmaxf(0.0f, raw));
  phi[c] = cl;
  project_stat_cell(cp, raw, cl, m, a);
}

// the CTA's statistics into st: warp sums, then the CTA's warps in shared
// memory, then one atomic per CTA and value (an atomic per warp serialised
// tens of thousands of FP64 adds on five addresses)
__device__ __forceinline__ void project_stats_flush(ProjAcc a, FsiCouplingStats* st) {
  __shared__ double s_d[32][3];
  __shared__ float s_m[32];
  __shared__ int s_n[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  a.pm = warp_sum_d(a.pm);
  a.pvr = warp_sum_d(a.pvr);
  a.pvc = warp_sum_d(a.pvc);
  a.mx = warp_max(fmaxf(a.mx, 0.f));
  a.na = __reduce_add_sync(0xffffffffu, (unsigned)a.na);
  if (lane == 0) {
    s_d[wid][0] = a.pm;
    s_d[wid][1] = a.pvr;
    s_d[wid][2] = a.pvc;
    s_m[wid] = a.mx;
    s_n[wid] = a.na;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ProjAcc t;
    for (int w = 0; w < nw; ++w) {
      t.pm += s_d[w][0];
      t.pvr += s_d[w][1];
      t.pvc += s_d[w][2];
      t.mx = fmaxf(t.mx, s_m[w]);
      t.na += s_n[w];
    }
    if (t.pm != 0.0) atomicAdd(&st->projected_mass, t.pm);
    if (t.pvr != 0.0) atomicAdd(&st->projected_volume_raw, t.pvr);
    if (t.pvc != 0.0) atomicAdd(&st->projected_volume_clamped, t.pvc);
    if (t.mx > 0.f) atomic_max_nonneg(&st->max_phi_raw, t.mx);
    if (t.na) atomicAdd(&st->active_cell_count, t.na);
  }
}

// grid-stride over the cells (every thread of the CTA reaches the flush)
__global__ void k_project_normalize(LatView L, FsiCouplingParams cp, float* phi, float* smass, float* svel,
                                    FsiCouplingStats* st) {
  const int64_t n = (int64_t)L.nx * L.ny * L.nz;
  ProjAcc a;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x)
    project_normalize_cell(L, cp, phi, smass, svel, c, a);
  project_stats_flush(a, st);
}

// ------------------------------------- projection in particle order ----
// projection.py:39-65 adds, for particle p = 0, 1, ... and its 27 stencil
// offsets, w * vol / cell_volume, w * m and w * m * v to the cells; a serial
// run sums every cell's terms in ascending p.  Here particles are sorted by
// B-spline base cell (a counting sort over the bounding box of the base cells),
// and one warp per cell collects the ids of its <= 27 base cells, sorts them in
// registers and sums the terms in that order with IEEE FP32 adds.  The term
// arithmetic is written with explicit round-to-nearest operations, so no
// multiply-add is contracted and every term is the one a serial FP32 run
// computes.  Six launches, overlapped as far as the data allows: at the sizes of
// one coupled step most of them last 2-4 us.  None of their pointers is marked
// __restrict__: a load may not move above griddep_wait().
//
// scratch->box: [0..2] max(-base), [3..5] max(base) over the particles whose
// base cell touches the lattice (base in [-2, dim - 1] on each axis), 0x80808080
// (INT_MIN-like) in an empty box; [6] counts the finished CTAs of k_po_scan.

struct OrdBase {
  int b[3];
  float fx[3];
};

__device__ __forceinline__ OrdBase ordered_base(const FsiParticles& pt, int p, float inv_dx) {
  OrdBase o;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float Xp = __fmul_rn(pt.x[a * pt.n + p], inv_dx);
    o.b[a] = (int)__fsub_rn(Xp, 0.5f);
    o.fx[a] = __fsub_rn(Xp, (float)o.b[a]);
  }
  return o;
}

__device__ __forceinline__ bool ordered_base_touches(const LatView& L, const OrdBase& o) {
  return o.b[0] >= -2 && o.b[0] < L.nx && o.b[1] >= -2 && o.b[1] < L.ny && o.b[2] >= -2 && o.b[2] < L.nz;
}

// quadratic B-spline weight of offset d for fractional position f: the
// reference's values bit for bit (solid.py:222-230 / projection.py:45-47; its
// 1.5 - f is -(f - 1.5) exactly, and the sign cancels in the square)
__device__ __forceinline__ float ordered_w(float f, int d) {
  const float t = __fsub_rn(f, d == 0 ? 1.5f : (d == 1 ? 1.0f : 0.5f));
  return d == 1 ? __fsub_rn(0.75f, __fmul_rn(t, t)) : __fmul_rn(__fmul_rn(0.5f, t), t);
}

struct OrdBox {
  int lo[3], hi[3], ext[3];
  int64_t keys;
};

__device__ __forceinline__ OrdBox ordered_box(const int32_t* box) {
  OrdBox B;
  int64_t k = 1;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    B.lo[a] = -box[a];
    B.hi[a] = box[3 + a];
    B.ext[a] = B.hi[a] >= B.lo[a] ? B.hi[a] - B.lo[a] + 1 : 0;
    k *= B.ext[a];
  }
  B.keys = k;
  return B;
}

// the fields the gather adds to (cells without contributors keep these values:
// phi = mass = 0 and the quotient normalize_projection gives for mass 0), the
// statistics' first stat_words words and the box; one launch for five fills
__device__ __forceinline__ void fill_words(float* p, int64_t n, float v) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
  int64_t done = 0;
  if (((uintptr_t)p & 15) == 0) {
    done = n & ~(int64_t)3;
    for (int64_t i = t; i < n / 4; i += nt) reinterpret_cast<float4*>(p)[i] = make_float4(v, v, v, v);
  }
  for (int64_t i = done + t; i < n; i += nt) p[i] = v;
}

__global__ void k_po_clear(int64_t pitch, float* phi, float* smass, float* svel, float empty_vel, int32_t* stats,
                           int stat_words, int32_t* box) {
  griddep_wait();
  griddep_launch();
  if (blockIdx.x == 0) {
    if (threadIdx.x < 7) box[threadIdx.x] = threadIdx.x < 6 ? (int32_t)0x80808080 : 0;
    for (int i = threadIdx.x; i < stat_words; i += blockDim.x) stats[i] = 0;
  }
  fill_words(phi, pitch, 0.f);
  fill_words(smass, pitch, 0.f);
  fill_words(svel, 3 * pitch, empty_vel);
}

// six atomics per CTA (a warp's six each took 26 us at 196,608 particles)
__global__ void __launch_bounds__(256) k_po_box(LatView L, FsiParticles pt, float inv_dx, int32_t* box) {
  __shared__ int s_v[8][6];
  griddep_wait();
  griddep_launch();
  int v[6];
#pragma unroll
  for (int a = 0; a < 6; ++a) v[a] = INT_MIN;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < pt.n; p += (int64_t)gridDim.x * blockDim.x) {
    const OrdBase o = ordered_base(pt, (int)p, inv_dx);
    if (ordered_base_touches(L, o)) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        v[a] = max(v[a], -o.b[a]);
        v[3 + a] = max(v[3 + a], o.b[a]);
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    const int w = __reduce_max_sync(0xffffffffu, v[a]);
    if ((threadIdx.x & 31) == 0) s_v[threadIdx.x >> 5][a] = w;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    int w = s_v[0][threadIdx.x];
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) w = max(w, s_v[i][threadIdx.x]);
    if (w != INT_MIN) atomicMax(box + threadIdx.x, w);
  }
}

__device__ __forceinline__ int ordered_key(const OrdBox& B, const int b[3]) {
  return ((b[2] - B.lo[2]) * B.ext[1] + (b[1] - B.lo[1])) * B.ext[0] + (b[0] - B.lo[0]);
}

__global__ void k_po_count(LatView L, FsiParticles pt, float inv_dx, const int32_t* box, int32_t* key,
                           int32_t* count) {
  griddep_wait();
  griddep_launch();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= pt.n) return;
  const OrdBox B = ordered_box(box);
  const OrdBase o = ordered_base(pt, p, inv_dx);
  int k = -1;
  if (ordered_base_touches(L, o)) {
    k = ordered_key(B, o.b);
    atomicAdd(count + k, 1);
  }
  key[p] = k;
}

// Exclusive scan of count[0, keys] (count[keys] taken as 0) in blocks of kPoBlk
// keys: start[k] is the sum over its own block before k, except that a block's
// first entry (where that sum is 0) holds the sum over all blocks before it,
// which the last CTA to finish works out from the block totals; po_begin() adds
// the two.  One CTA walking over all keys took 51 us for a plate in a
// 256 x 128 x 128 lattice.
constexpr int kPoScanT = 1024, kPoBlk = 4 * kPoScanT;

__device__ __forceinline__ int po_begin(const int32_t* start, int k) {
  const int base = start[k & ~(kPoBlk - 1)];
  return (k & (kPoBlk - 1)) ? base + start[k] : base;
}

// inclusive scan over the CTA's kPoScanT threads; s_w: one word per warp
__device__ __forceinline__ int po_cta_scan(int v, int* s_w) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  __syncthreads();  // s_w may still be read from the call before
  if (lane == 31) s_w[wid] = v;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < kPoScanT / 32; ++w) before += w < wid ? s_w[w] : 0;
  return v + before;
}

__global__ __launch_bounds__(kPoScanT) void k_po_scan(int32_t* box, const int32_t* count, int32_t* start) {
  __shared__ int s_w[kPoScanT / 32];
  __shared__ int s_last;
  griddep_wait();
  griddep_launch();
  const int nk = (int)ordered_box(box).keys, nb = nk / kPoBlk + 1, t = threadIdx.x;
  if ((int)blockIdx.x >= nb) return;
  for (int b = blockIdx.x; b < nb; b += gridDim.x) {
    int c[4], k = b * kPoBlk + 4 * t, sum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      c[i] = k + i < nk ? count[k + i] : 0;
      sum += c[i];
    }
    const int inc = po_cta_scan(sum, s_w);
    int off = inc - sum;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (k + i <= nk && (k + i) % kPoBlk != 0) start[k + i] = off;
      off += c[i];
    }
    if (t == kPoScanT - 1) start[b * kPoBlk] = inc;  // the block's total
  }
  __threadfence();
  __syncthreads();
  if (t == 0) s_last = atomicAdd(box + 6, 1) == min(nb, (int)gridDim.x) - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  int carry = 0;
  for (int b0 = 0; b0 < nb; b0 += kPoScanT) {
    const int b = b0 + t;
    const int v = b < nb ? __ldcg(start + (int64_t)b * kPoBlk) : 0;
    const int inc = po_cta_scan(v, s_w);
    if (b < nb) start[(int64_t)b * kPoBlk] = carry + inc - v;
    __syncthreads();
    if (t == kPoScanT - 1) s_last = inc;
    __syncthreads();
    carry += s_last;
  }
}

// counts each base cell's counter back down to zero, the particles in any order
__global__ void k_po_fill(int n, const int32_t* key, const int32_t* start,
                          int32_t* count, int32_t* list) {
  griddep_wait();
  griddep_launch();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int k = key[p];
  if (k >= 0) list[po_begin(start, k) + atomicSub(count + k, 1) - 1] = p;
}

// the five terms particle p adds to the cell at offset d from its base cell
__device__ __forceinline__ void ordered_terms(const FsiParticles& pt, const FsiCouplingParams& cp, int p,
                                              const OrdBase& o, const int d[3], float t[5]) {
  const int n = pt.n;
  const float w = __fmul_rn(__fmul_rn(ordered_w(o.fx[0], d[0]), ordered_w(o.fx[1], d[1])), ordered_w(o.fx[2], d[2]));
  const float J = fmaxf(pt.Jp[p], 0.0f);
  const float cur_vol = __fmul_rn(pt.vol0[p], J);
  const float mc = __fmul_rn(w, pt.mass[p]);
  t[0] = __fdiv_rn(__fmul_rn(w, cur_vol), cp.cell_volume_norm);
  t[1] = mc;
#pragma unroll
  for (int a = 0; a < 3; ++a) t[2 + a] = __fmul_rn(mc, __fmul_rn(pt.v[a * n + p], cp.vel_scale));
}

// Ascending order of the warp's 32 E values, value r of a lane at lane * E + r
// afterwards: a bitonic network, whose steps within a lane need no shuffle.
template <int E>
__device__ __forceinline__ void po_warp_sort(int (&v)[E], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= E) {
        const bool keep_min = ((lane & (j / E)) == 0) == ((lane & (k / E)) == 0);
#pragma unroll
        for (int r = 0; r < E; ++r) {
          const int y = __shfl_xor_sync(0xffffffffu, v[r], j / E);
          v[r] = keep_min ? min(v[r], y) : max(v[r], y);
        }
      } else {
#pragma unroll
        for (int r = 0; r < E; ++r) {
          if (r & j) continue;
          const bool up = ((lane * E + r) & k) == 0;
          const int lo = min(v[r], v[r | j]), hi = max(v[r], v[r | j]);
          v[r] = up ? lo : hi;
          v[r | j] = up ? hi : lo;
        }
      }
    }
  }
}

template <int E>
__device__ __forceinline__ void po_sort_ids(int* cand, int m, int lane) {
  int v[E];
#pragma unroll
  for (int r = 0; r < E; ++r) v[r] = r * 32 + lane < m ? cand[r * 32 + lane] : INT_MAX;
  po_warp_sort<E>(v, lane);
  __syncwarp();
#pragma unroll
  for (int r = 0; r < E; ++r) cand[lane * E + r] = v[r];  // cand holds kPoCap >= 32 E words
  __syncwarp();
}

constexpr int kPoWarps = 4;
constexpr int kPoCap = 512;     // ids sorted at a time
constexpr int kPoTerms = 128;   // terms staged at a time
constexpr int kPoRow = kPoTerms + 4;

// One warp per cell: the ids of the cell's base cells into shared memory, sorted
// there, then per 128 of them the terms (lane = particle) and five serial sums
// (lane = field), normalised as normalize_projection does.  Bound by the
// latency of sort, terms and serial sums (at 64 registers, 32 warps per SM; with 96
// registers and terms unrolled by four 1.5 times slower).  Ranking every id against
// all others, and separate sort, normalise and fill passes around it, made the whole
// projection 50.7 us for a block of 8^3 cells (4,096 particles), 87.9 us for 24,576
// particles in 128 x 64 x 64 cells and 392 us for 196,608 in 256 x 128 x 128; with
// this it takes 21.6, 35.7 and 131 us.
__global__ __launch_bounds__(32 * kPoWarps, 8) void k_po_gather(LatView L, FsiParticles pt, FsiCouplingParams cp,
                                                             const int32_t* box,
                                                             const int32_t* start,
                                                             const int32_t* list, float* phi,
                                                             float* smass, float* svel,
                                                             FsiCouplingStats* st) {
  __shared__ int s_cand[kPoWarps][kPoCap];
  __shared__ float4 s_term[kPoWarps][5 * kPoRow / 4];
  griddep_wait();
  griddep_launch();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int* cand = s_cand[wid];
  float* term = reinterpret_cast<float*>(s_term[wid]);
  const OrdBox B = ordered_box(box);
  __shared__ ProjAcc s_stat[kPoWarps];  // lane 0's, out of the registers
  if (lane == 0) s_stat[wid] = ProjAcc();
  // cells reached from the box: [lo, hi + 2] clipped to the lattice
  int clo[3];
  unsigned cext[3];
  const int dims[3] = {L.nx, L.ny, L.nz};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    clo[a] = max(B.lo[a], 0);
    cext[a] = B.keys ? (unsigned)max(min(B.hi[a] + 2, dims[a] - 1) - clo[a] + 1, 0) : 0u;
  }
  const unsigned ncell = cext[0] * cext[1] * cext[2];  // <= the lattice's cells, checked against 2^31 on the host
  // lane l < 27 owns stencil offset d = (l / 9, l / 3 % 3, l % 3): base cell = cell - d
  const int d[3] = {lane / 9, (lane / 3) % 3, lane % 3};
  for (unsigned q = blockIdx.x * kPoWarps + wid; q < ncell; q += gridDim.x * kPoWarps) {
    const unsigned row = q / cext[0];
    const int ci = clo[0] + (int)(q - row * cext[0]);
    const int cj = clo[1] + (int)(row % cext[1]);
    const int ck = clo[2] + (int)(row / cext[1]);
    const int b[3] = {ci - d[0], cj - d[1], ck - d[2]};
    int s = 0, len = 0;
    if (lane < 27 && b[0] >= B.lo[0] && b[0] <= B.hi[0] && b[1] >= B.lo[1] && b[1] <= B.hi[1] && b[2] >= B.lo[2] &&
        b[2] <= B.hi[2]) {
      const int k = ordered_key(B, b);
      s = po_begin(start, k);
      len = po_begin(start, k + 1) - s;
    }
    int off = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, off, o);
      if (lane >= o) off += y;
    }
    const int K = __shfl_sync(0xffffffffu, off, 31);
    off -= len;
    if (K == 0) continue;
    float acc = 0.f;  // lane v < 5: running sum of term v
    int last = -1;    // the ids up to here are summed
    for (int done = 0, m; done < K; done += m) {
      if (K <= kPoCap) {
        m = K;
        const int longest = (int)__reduce_max_sync(0xffffffffu, (unsigned)len);
        for (int i0 = 0; i0 < longest; i0 += 8) {  // eight loads in flight
          int id[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) id[i] = i0 + i < len ? list[s + i0 + i] : 0;
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (i0 + i < len) cand[off + i0 + i] = id[i];
        }
      } else {
        // the next (at most kPoCap) ids: the largest bound with no more of
        // them in (last, bound], found by bisection over the ids
        int lo = last, hi = pt.n - 1;
        m = 0;
        while (lo < hi) {
          const int mid = lo + (hi - lo + 1) / 2;
          int cnt = 0;
          for (int l = 0; l < 27; ++l) {
            const int sl = __shfl_sync(0xffffffffu, s, l), nl = __shfl_sync(0xffffffffu, len, l);
            for (int i = lane; i < nl; i += 32) {
              const int id = list[sl + i];
              cnt += id > last && id <= mid;
            }
          }
          cnt = (int)__reduce_add_sync(0xffffffffu, (unsigned)cnt);
          if (cnt <= kPoCap) {
            lo = mid;
          } else {
            hi = mid - 1;
          }
        }
        for (int l = 0; l < 27; ++l) {
          const int sl = __shfl_sync(0xffffffffu, s, l), nl = __shfl_sync(0xffffffffu, len, l);
          for (int i0 = 0; i0 < nl; i0 += 32) {
            const int id = i0 + lane < nl ? list[sl + i0 + lane] : -1;
            const bool take = id > last && id <= lo;
            const unsigned mask = __ballot_sync(0xffffffffu, take);
            if (take) cand[m + __popc(mask & ((1u << lane) - 1u))] = id;
            m += __popc(mask);
          }
        }
        last = lo;
        if (m == 0) break;  // not reached: K ids lie in [0, n)
      }
      __syncwarp();
      if (m <= 32)
        po_sort_ids<1>(cand, m, lane);
      else if (m <= 64)
        po_sort_ids<2>(cand, m, lane);
      else if (m <= 128)
        po_sort_ids<4>(cand, m, lane);
      else if (m <= 256)
        po_sort_ids<8>(cand, m, lane);
      else
        po_sort_ids<16>(cand, m, lane);
      for (int c0 = 0; c0 < m; c0 += kPoTerms) {
        const int mc = min(kPoTerms, m - c0);
#pragma unroll 1
        for (int u = 0; u < (mc + 31) / 32; ++u) {
          const int i = u * 32 + lane;
          // lanes past the end repeat the last particle; +0 to a sum that started at +0 changes no bit
          const int p = cand[c0 + min(i, mc - 1)];
          const OrdBase o = ordered_base(pt, p, cp.inv_dx_norm);
          const int dd[3] = {ci - o.b[0], cj - o.b[1], ck - o.b[2]};
          float t[5];
          ordered_terms(pt, cp, p, o, dd, t);
#pragma unroll
          for (int v = 0; v < 5; ++v) term[v * kPoRow + i] = i < mc ? t[v] : 0.f;
        }
        __syncwarp();
        if (lane < 5) {
          const float4* row4 = reinterpret_cast<const float4*>(term + lane * kPoRow);
#pragma unroll 4
          for (int r = 0; r < (mc + 3) / 4; ++r) {
            const float4 x = row4[r];
            acc = __fadd_rn(acc, x.x);
            acc = __fadd_rn(acc, x.y);
            acc = __fadd_rn(acc, x.z);
            acc = __fadd_rn(acc, x.w);
          }
        }
        __syncwarp();
      }
    }
    const int64_t c = lat_cell(L, ci, cj, ck);
    const float m = __shfl_sync(0xffffffffu, acc, 1);
    if (lane == 0) {
      const float cl = fminf(1.0f, fmaxf(0.0f, acc));
      phi[c] = cl;
      project_stat_cell(cp, acc, cl, m, s_stat[wid]);
    } else if (lane == 1) {
      smass[c] = m;
    } else if (lane < 5) {
      svel[(lane - 2) * L.pitch + c] = m > cp.eps_mass ? acc / m : 0.f;
    }
  }
  ProjAcc stat;
  if (lane == 0) stat = s_stat[wid];
  project_stats_flush(stat, st);
}

// ------------------------------------------------------------ reaction ----
__global__ void k_reaction(LatView L, const float* hydro, const float* phi, FsiParticles pt, FsiGrid g,
                           FsiCouplingParams cp, FsiCouplingStats* st, const FsiLbmDiag* diag) {
  __shared__ float s_scale;
  if (threadIdx.x == 0) {
    float raw = 1.f;
    s_scale = cp.kind == 2 ? link_area_scale(diag, cp, &raw) : 1.0f;
    if (blockIdx.x == 0 && cp.kind == 2) {
      st->area_scale = s_scale;
      st->raw_area_scale = raw;
    }
  }
  __syncthreads();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = pt.n;
  bool act = false, gated = false;
  float pf[3] = {0.f, 0.f, 0.f}, pnorm = 0.f, gmax = 0.f;
  double gnet[3] = {0.0, 0.0, 0.0};
  if (p < n) {
    const float X[3] = {pt.x[p], pt.x[n + p], pt.x[2 * n + p]};
    BSpline b;
    bspline(X, cp.inv_dx_norm, b);
    ReactParticle r;
    reaction_particle(L, hydro, phi, cp, b, pt.Jp[p], pt.vol0[p], s_scale, r);
    for (int a = 0; a < 3; ++a) pf[a] = r.pf[a];
    act = r.act;
    gated = r.gated;
    pnorm = r.pnorm;
    const bool scatter = r.scatter;
    if (scatter) {
      const int64_t N = (int64_t)g.n * g.n * g.n;
#pragma unroll
      for (int ox = 0; ox < 3; ++ox)
#pragma unroll
        for (int oy = 0; oy < 3; ++oy)
#pragma unroll
          for (int oz = 0; oz < 3; ++oz) {
            const int I = b.base[0] + ox, Jj = b.base[1] + oy, K = b.base[2] + oz;
            if (I < 0 || I >= g.n || Jj < 0 || Jj >= g.n || K < 0 || K >= g.n) continue;
            const float w = b.w[0][ox] * b.w[1][oy] * b.w[2][oz];
            const int64_t node = ((int64_t)K * g.n + Jj) * g.n + I;
            const float c0 = w * pf[0], c1 = w * pf[1], c2 = w * pf[2];
            atomicAdd(g.f_ext + node, c0);
            atomicAdd(g.f_ext + N + node, c1);
            atomicAdd(g.f_ext + 2 * N + node, c2);
            gnet[0] += c0;
            gnet[1] += c1;
            gnet[2] += c2;
            gmax = fmaxf(gmax, sqrtf(c0 * c0 + c1 * c1 + c2 * c2));
          }
    }
  }
  // diagnostics reductions (penalty.py:202-240, moving_boundary.py:312-374)
  const int na = __popc(__ballot_sync(0xffffffffu, act));
  const float pm = warp_max(pnorm), gm = warp_max(gmax);
  double pn[3], gn[3];
  for (int a = 0; a < 3; ++a) {
    pn[a] = warp_sum_d(gated ? (double)pf[a] : 0.0);
    gn[a] = warp_sum_d(gnet[a]);
  }
  if ((threadIdx.x & 31) == 0) {
    if (na) atomicAdd(&st->active_reaction_particle_count, na);
    if (pm > 0.f) atomic_max_nonneg(&st->max_particle_reaction_norm, pm);
    if (gm > 0.f) atomic_max_nonneg(&st->max_grid_reaction_norm, gm);
    for (int a = 0; a < 3; ++a) {
      if (pn[a] != 0.0) atomicAdd(&st->net_particle_reaction[a], pn[a]);
      if (gn[a] != 0.0) atomicAdd(&st->net_grid_reaction[a], gn[a]);
    }
  }
}

// ----------------------------------------------------------------- MPM ----
// The four launches of a substep wait for one another on the device only
// (griddep_wait / griddep_launch): for a few thousand particles they last 2-7 us
// each, less than the host needs for one call of its own, so fsi_mpm_substep
// sends them together.  4,096 particles on 48^3 nodes: with three fills and three
// calls 42.6 us per substep, with this 21.8 us.
__global__ void k_grid_clear(int64_t nodes, float* v, float* m, float* f) {
  griddep_wait();
  griddep_launch();
  fill_words(v, 3 * nodes, 0.f);
  fill_words(m, nodes, 0.f);
  fill_words(f, 3 * nodes, 0.f);
}

__global__ void k_p2g(FsiParticles pt, FsiGrid g, FsiMpmParams mp) {
  griddep_wait();
  griddep_launch();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= pt.n) return;
  const int n = pt.n;
  const float X[3] = {pt.x[p], pt.x[n + p], pt.x[2 * n + p]};
  BSpline b;
  bspline(X, mp.inv_dx, b);
  P2GParticle q;
  p2g_particle(pt, p, mp, q);
  pt.Jp[p] = q.J;
  const int G = g.n;
  const int64_t N = (int64_t)G * G * G;
#pragma unroll
  for (int ox = 0; ox < 3; ++ox)
#pragma unroll
    for (int oy = 0; oy < 3; ++oy)
#pragma unroll
      for (int oz = 0; oz < 3; ++oz) {
        const int I = b.base[0] + ox, Jj = b.base[1] + oy, K = b.base[2] + oz;
        if (I < 0 || I >= G || Jj < 0 || Jj >= G || K < 0 || K >= G) continue;
        float w, mom[3];
        p2g_node(q, b, ox, oy, oz, mp.dx, w, mom);
        const int64_t node = ((int64_t)K * G + Jj) * G + I;
#pragma unroll
        for (int a = 0; a < 3; ++a) atomicAdd(g.v + a * N + node, w * mom[a]);
        atomicAdd(g.m + node, w * q.mass);
      }
}

__global__ void k_grid_update(FsiGrid g, FsiMpmParams mp) {
  griddep_wait();
  griddep_launch();
  const int G = g.n;
  const int64_t N = (int64_t)G * G * G;
  const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= N) return;
  const float m = g.m[node];
  if (!(m > 0.0f)) return;
  const float P[3] = {g.v[node], g.v[N + node], g.v[2 * N + node]};
  const float f[3] = {g.f_ext[node], g.f_ext[N + node], g.f_ext[2 * N + node]};
  float v[3];
  grid_node_velocity(P, m, f, (int)(node % G), (int)((node / G) % G), (int)(node / ((int64_t)G * G)), G, mp, v);
#pragma unroll
  for (int a = 0; a < 3; ++a) g.v[a * N + node] = v[a];
}

__global__ void k_g2p(FsiParticles pt, FsiGrid g, FsiMpmParams mp) {
  griddep_wait();
  griddep_launch();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= pt.n) return;
  const int n = pt.n;
  float X[3] = {pt.x[p], pt.x[n + p], pt.x[2 * n + p]};
  BSpline b;
  bspline(X, mp.inv_dx, b);
  const int G = g.n;
  const int64_t N = (int64_t)G * G * G;
  float nv[3] = {0.f, 0.f, 0.f}, nC[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float s4 = 4.0f * mp.inv_dx * mp.inv_dx;
#pragma unroll
  for (int ox = 0; ox < 3; ++ox)
#pragma unroll
    for (int oy = 0; oy < 3; ++oy)
#pragma unroll
      for (int oz = 0; oz < 3; ++oz) {
        const int I = b.base[0] + ox, Jj = b.base[1] + oy, K = b.base[2] + oz;
        if (I < 0 || I >= G || Jj < 0 || Jj >= G || K < 0 || K >= G) continue;
        const int64_t node = ((int64_t)K * G + Jj) * G + I;
        const float gv[3] = {g.v[node], g.v[N + node], g.v[2 * N + node]};
        g2p_node(b, ox, oy, oz, mp.dx, s4, gv, nv, nC);
      }
  g2p_finish(pt, p, mp, X, nv, nC);
}

static inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

static int check_particles(const FsiParticles* pt) {
  if (!pt) return invalid("null particles");
  if (pt->n <= 0) return invalid("n_particles must be positive");
  if (!pt->x || !pt->v || !pt->C || !pt->F || !pt->Jp || !pt->mass || !pt->vol0) return invalid("null particle field");
  return FSI_OK;
}

}  // namespace fsi

using namespace fsi;

extern "C" int fsi_project(const FsiLbmState* s, const FsiParticles* pt, const FsiCouplingParams* cp,
                           FsiCouplingStats* stats, void* stream) {
  if (!s || !cp || !stats) return invalid("null argument");
  int rc = check_particles(pt);
  if (rc) return rc;
  if (!s->phi || !s->smass || !s->svel) return invalid("projection needs phi, smass, svel");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t P = s->pitch;
  if ((rc = cuda_check(cudaMemsetAsync(s->phi, 0, sizeof(float) * P, st), "clear phi"))) return rc;
  if ((rc = cuda_check(cudaMemsetAsync(s->smass, 0, sizeof(float) * P, st), "clear smass"))) return rc;
  if ((rc = cuda_check(cudaMemsetAsync(s->svel, 0, sizeof(float) * 3 * P, st), "clear svel"))) return rc;
  if ((rc = cuda_check(cudaMemsetAsync(stats, 0, offsetof(FsiCouplingStats, active_reaction_particle_count), st),
                       "clear projection stats")))
    return rc;
  const LatView L{s->nx, s->ny, s->nz, P};
  k_project_scatter<<<nblk(pt->n, kPsT), kPsT, 0, st>>>(L, *pt, *cp, s->phi, s->smass, s->svel);
  if ((rc = launch_check("k_project_scatter"))) return rc;
  const int64_t n = (int64_t)s->nx * s->ny * s->nz;
  k_project_normalize<<<(unsigned)std::min<int64_t>(nblk(n, 256), 8LL * device_sm_count()), 256, 0, st>>>(
      L, *cp, s->phi, s->smass, s->svel, stats);
  return launch_check("k_project_normalize");
}

extern "C" int fsi_project_ordered(const FsiLbmState* s, const FsiParticles* pt, const FsiCouplingParams* cp,
                                   const FsiProjectScratch* sc, FsiCouplingStats* stats, void* stream) {
  if (!s || !cp || !sc || !stats) return invalid("null argument");
  int rc = check_particles(pt);
  if (rc) return rc;
  if (!s->phi || !s->smass || !s->svel) return invalid("projection needs phi, smass, svel");
  if (!sc->count || !sc->start || !sc->list || !sc->key || !sc->box) return invalid("null projection scratch array");
  const int64_t keys = (int64_t)(s->nx + 2) * (s->ny + 2) * (s->nz + 2);
  if (keys > INT_MAX - 1) return invalid("lattice too large for the ordered projection");
  if (sc->key_capacity < keys) return invalid("scratch key_capacity below (nx + 2) * (ny + 2) * (nz + 2)");
  if (sc->particle_capacity < pt->n) return invalid("scratch particle_capacity below the particle count");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t P = s->pitch;
  const LatView L{s->nx, s->ny, s->nz, P};
  const float inv_dx = cp->inv_dx_norm;
  const int sms = device_sm_count();
  static_assert(offsetof(FsiCouplingStats, active_reaction_particle_count) % 4 == 0, "statistics are cleared by words");
  const int stat_words = (int)(offsetof(FsiCouplingStats, active_reaction_particle_count) / 4);
  const float empty_vel = 0.0f > cp->eps_mass ? NAN : 0.0f;
  const unsigned pb = nblk(pt->n, 256);
  const unsigned clear_ctas = (unsigned)std::min<int64_t>(nblk(P, 1024), 8LL * sms);
  const unsigned scan_ctas = (unsigned)std::min<int64_t>(keys / kPoBlk + 1, 2LL * sms);
  auto launched = [&](cudaError_t e, const char* what) {
    const int r = cuda_check(e, what);
    return r ? r : launch_check(what);
  };
  if ((rc = launched(launch_pdl(k_po_clear, dim3(clear_ctas), dim3(256), 0, st, P, s->phi, s->smass, s->svel, empty_vel,
                                reinterpret_cast<int32_t*>(stats), stat_words, sc->box),
                     "k_po_clear")))
    return rc;
  if ((rc = launched(launch_pdl(k_po_box, dim3(std::min(pb, 2u * sms)), dim3(256), 0, st, L, *pt, inv_dx, sc->box), "k_po_box"))) return rc;
  if ((rc = launched(launch_pdl(k_po_count, dim3(pb), dim3(256), 0, st, L, *pt, inv_dx, sc->box, sc->key, sc->count),
                     "k_po_count")))
    return rc;
  if ((rc = launched(launch_pdl(k_po_scan, dim3(scan_ctas), dim3(kPoScanT), 0, st, sc->box, sc->count, sc->start),
                     "k_po_scan")))
    return rc;
  if ((rc = launched(launch_pdl(k_po_fill, dim3(pb), dim3(256), 0, st, pt->n, sc->key, sc->start, sc->count, sc->list),
                     "k_po_fill")))
    return rc;
  return launched(launch_pdl(k_po_gather, dim3(sms * 8), dim3(32 * kPoWarps), 0, st, L, *pt, *cp, sc->box, sc->start,
                             sc->list, s->phi, s->smass, s->svel, stats),
                  "k_po_gather");
}

extern "C" int fsi_reaction_to_grid(const FsiLbmState* s, const float* hydro, const FsiParticles* pt, const FsiGrid* g,
                                    const FsiCouplingParams* cp, FsiCouplingStats* stats, void* stream) {
  if (!s || !hydro || !g || !cp || !stats) return invalid("null argument");
  int rc = check_particles(pt);
  if (rc) return rc;
  if (cp->kind < 0 || cp->kind > 2) return invalid("reaction kind must be 0 (penalty), 1 (engineering), 2 (link-area)");
  cudaStream_t st = (cudaStream_t)stream;
  const size_t off = offsetof(FsiCouplingStats, active_reaction_particle_count);
  if ((rc = cuda_check(cudaMemsetAsync(reinterpret_cast<char*>(stats) + off, 0, sizeof(FsiCouplingStats) - off, st),
                       "clear reaction stats")))
    return rc;
  const LatView L{s->nx, s->ny, s->nz, s->pitch};
  k_reaction<<<nblk(pt->n, 128), 128, 0, st>>>(L, hydro, s->phi, *pt, *g, *cp, stats, s->diag);
  return launch_check("k_reaction");
}

// particles per CTA: one warp each while that leaves SMs without one
static int particle_threads(int n) { return (int64_t)n <= 32LL * 4 * device_sm_count() ? 32 : 128; }

static int check_grid_phase(const FsiGrid* g, const FsiMpmParams* mp) {
  return g && mp && g->n > 0 ? FSI_OK : invalid("bad grid or params");
}

static int launch_grid_clear(const FsiGrid* g, cudaStream_t st) {
  const int64_t N = (int64_t)g->n * g->n * g->n;
  const unsigned ctas = (unsigned)std::min<int64_t>(nblk(N, 512), 8LL * device_sm_count());
  const int rc = cuda_check(launch_pdl(k_grid_clear, dim3(ctas), dim3(256), 0, st, N, g->v, g->m, g->f_ext),
                            "k_grid_clear (launch)");
  return rc ? rc : launch_check("k_grid_clear");
}

static int launch_p2g(const FsiParticles* pt, const FsiGrid* g, const FsiMpmParams* mp, cudaStream_t st) {
  const int t = particle_threads(pt->n);
  const int rc = cuda_check(launch_pdl(k_p2g, dim3(nblk(pt->n, t)), dim3(t), 0, st, *pt, *g, *mp), "k_p2g (launch)");
  return rc ? rc : launch_check("k_p2g");
}

static int launch_grid_update(const FsiGrid* g, const FsiMpmParams* mp, cudaStream_t st) {
  const int64_t N = (int64_t)g->n * g->n * g->n;
  const int rc = cuda_check(launch_pdl(k_grid_update, dim3(nblk(N, 256)), dim3(256), 0, st, *g, *mp),
                            "k_grid_update (launch)");
  return rc ? rc : launch_check("k_grid_update");
}

static int launch_g2p(const FsiParticles* pt, const FsiGrid* g, const FsiMpmParams* mp, cudaStream_t st) {
  const int t = particle_threads(pt->n);
  const int rc = cuda_check(launch_pdl(k_g2p, dim3(nblk(pt->n, t)), dim3(t), 0, st, *pt, *g, *mp), "k_g2p (launch)");
  return rc ? rc : launch_check("k_g2p");
}

extern "C" int fsi_mpm_p2g(const FsiParticles* pt, const FsiGrid* g, const FsiMpmParams* mp, void* stream) {
  int rc = check_particles(pt);
  if (rc || (rc = check_grid_phase(g, mp))) return rc;
  return launch_p2g(pt, g, mp, (cudaStream_t)stream);
}

extern "C" int fsi_mpm_grid_update(const FsiGrid* g, const FsiMpmParams* mp, void* stream) {
  const int rc = check_grid_phase(g, mp);
  return rc ? rc : launch_grid_update(g, mp, (cudaStream_t)stream);
}

extern "C" int fsi_mpm_g2p(const FsiParticles* pt, const FsiGrid* g, const FsiMpmParams* mp, void* stream) {
  int rc = check_particles(pt);
  if (rc || (rc = check_grid_phase(g, mp))) return rc;
  if (!pt->fixed || !pt->fixed_x) return invalid("null fixed-particle fields");
  return launch_g2p(pt, g, mp, (cudaStream_t)stream);
}

extern "C" int fsi_mpm_substep(const FsiParticles* pt, const FsiGrid* g, const FsiMpmParams* mp, void* stream) {
  int rc = check_particles(pt);
  if (rc || (rc = check_grid_phase(g, mp))) return rc;
  if (!g->v || !g->m || !g->f_ext) return invalid("null grid field");
  if (!pt->fixed || !pt->fixed_x) return invalid("null fixed-particle fields");
  cudaStream_t st = (cudaStream_t)stream;
  if ((rc = launch_grid_clear(g, st)) || (rc = launch_p2g(pt, g, mp, st)) || (rc = launch_grid_update(g, mp, st)))
    return rc;
  return launch_g2p(pt, g, mp, st);
}

// ---- batched cases: projection (grid.y = case slot) -------------------------
namespace fsi {
namespace {

__device__ __forceinline__ LatView lat_of(const FsiBatchCase& bc) {
  return LatView{bc.lbm.nx, bc.lbm.ny, bc.lbm.nz, bc.lbm.pitch};
}

// fsi_project's clears: solid_phi, solid_mass, solid_vel and the projection
// reductions
__global__ void k_batch_project_clear(FsiBatchCase* cases) {
  const FsiBatchCase& bc = cases[blockIdx.y];
  if (!bc.active) return;
  const int64_t P = bc.lbm.pitch;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P; i += stride) {
    bc.lbm.phi[i] = 0.f;
    bc.lbm.smass[i] = 0.f;
    bc.lbm.svel[i] = 0.f;
    bc.lbm.svel[P + i] = 0.f;
    bc.lbm.svel[2 * P + i] = 0.f;
  }
  if (blockIdx.x == 0) {
    int* w = reinterpret_cast<int*>(bc.proj_stats);
    for (int i = threadIdx.x; i < (int)(offsetof(FsiCouplingStats, active_reaction_particle_count) / 4);
         i += blockDim.x)
      w[i] = 0;
  }
}

__global__ void __launch_bounds__(kPsT) k_batch_project_scatter(const FsiBatchCase* __restrict__ cases) {
  const FsiBatchCase& bc = cases[blockIdx.y];
  if (!bc.active) return;
  const LatView L = lat_of(bc);
  const FsiParticles pt = bc.pt;
  const FsiCouplingParams cp = bc.cp;
  for (int p0 = blockIdx.x * kPsT; p0 < pt.n; p0 += gridDim.x * kPsT)
    project_scatter_body(L, pt, cp, bc.lbm.phi, bc.lbm.smass, bc.lbm.svel, p0);
}

__global__ void k_batch_project_normalize(const FsiBatchCase* __restrict__ cases) {
  const FsiBatchCase& bc = cases[blockIdx.y];
  if (!bc.active) return;
  const LatView L = lat_of(bc);
  const FsiCouplingParams cp = bc.cp;
  const int64_t n = (int64_t)L.nx * L.ny * L.nz;
  ProjAcc a;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x)
    project_normalize_cell(L, cp, bc.lbm.phi, bc.lbm.smass, bc.lbm.svel, c, a);
  project_stats_flush(a, bc.proj_stats);
}

}  // namespace
}  // namespace fsi

extern "C" int fsi_batch_project(FsiBatchCase* cases, const FsiBatchDims* d, void* stream) {
  if (!cases || !d || d->n_cases <= 0 || d->n_cases > 65535 || d->max_cells <= 0 || d->max_particles <= 0)
    return invalid("bad batch arguments");
  cudaStream_t st = (cudaStream_t)stream;
  // one CTA per 128 particles and per 256 to 2,048 cells of the largest case (smaller cases' extra CTAs exit at once)
  const int64_t cap = 1 << 20;
  const unsigned gc = batch_grid((d->max_cells + 255) / 256, d->n_cases, 8, 8);
  k_batch_project_clear<<<dim3(gc, d->n_cases), 256, 0, st>>>(cases);
  int rc = launch_check("k_batch_project_clear");
  if (rc) return rc;
  const unsigned gp = (unsigned)std::min<int64_t>((d->max_particles + 127) / 128, cap);
  k_batch_project_scatter<<<dim3(gp, d->n_cases), kPsT, 0, st>>>(cases);
  if ((rc = launch_check("k_batch_project_scatter"))) return rc;
  k_batch_project_normalize<<<dim3(gc, d->n_cases), 256, 0, st>>>(cases);
  return launch_check("k_batch_project_normalize");
}
