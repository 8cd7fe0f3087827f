// Binned MPM substeps: particles sorted by 8x8x8-cell block and cut into
// chunks; one launch per substep, in which each CTA takes whole chunks
// through the G2P gather of the previous substep (grid update evaluated while
// the chunk's node box is staged), the P2G stress / reaction payload and the
// P2G scatter, summed per chunk in shared memory and added to the grid with
// one global atomic per touched node value.  Three grid buffers rotate so that
// only the boxes touched two substeps earlier are zeroed, by the launch after
// their last reader.
//
// The per-particle and per-node arithmetic is the one of the one-phase
// kernels (mpm_common.cuh) to rounding: solid.py:212-315 and the reaction transfers of
// penalty.py:90-129, moving_boundary.py:58-110, link_area.py:84-193.  The
// order of the sums differs (stencils axis by axis, per-warp tiles, then one
// global atomic per chunk and touched node value), and a node's velocity is
// its momentum plus dt times its force, times one reciprocal of its mass.

#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "common.cuh"
#include "grid_node.cuh"
#include "mpm_common.cuh"

namespace fsi {
namespace {

constexpr int kChunk = FSI_BIN_CHUNK;  // particles per chunk
constexpr int kEdge = FSI_BIN_EDGE;
// nodes of a chunk's box that are staged in shared memory: the stencils of a
// chunk of one bin span at most (8 + 2)^3 = 1000 nodes; the rest absorbs a node
// of drift since the last binning (an 11^3 box).  A wider box is read from and
// added to the grid directly.
constexpr int kTileCap = 1331;

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// bin of a particle: the cell block of its B-spline base cell (solid.py:222-223)
__device__ __forceinline__ int particle_bin(const float X[3], float inv_dx, int G, int nb) {
  int c[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float Xp = __fmul_rn(X[a], inv_dx);
    c[a] = clampi((int)(Xp - 0.5f), 0, G - 1) / kEdge;
  }
  return (c[2] * nb + c[1]) * nb + c[0];
}

__device__ __forceinline__ void bin_count_body(const FsiParticles& pt, float inv_dx, int G, int nb,
                                               int32_t* key, int32_t* count, int vb, int vg) {
  const int p = vb * blockDim.x + threadIdx.x;
  if (p >= pt.n) return;
  const int n = pt.n;
  const float X[3] = {pt.x[p], pt.x[n + p], pt.x[2 * n + p]};
  const int k = particle_bin(X, inv_dx, G, nb);
  key[p] = k;
  atomicAdd(count + k, 1);
}

__global__ void k_bin_count(FsiParticles pt, float inv_dx, int G, int nb, int32_t* key, int32_t* count) {
  griddep_wait();
  griddep_launch();
  bin_count_body(pt, inv_dx, G, nb, key, count, blockIdx.x, gridDim.x);
}

// One CTA: exclusive scan of the bin counts and of the chunks per bin, the
// chunk table, and the counts reset to zero for the next binning.  Each
// thread owns a contiguous, 4-aligned range of bins and reads it with 16-byte
// loads, so the pass costs a few memory latencies rather than one per bin.
//
// Chunks: a bin of c particles is cut into ceil(c / kChunk) chunks of equal
// size (sizes differ by at most one), so that no chunk of a few particles
// follows a full one.
__device__ __forceinline__ int4 ld_bins4(const int32_t* p, int b, int b1) {
  if (b + 4 <= b1) return *reinterpret_cast<const int4*>(p + b);
  int4 v = make_int4(0, 0, 0, 0);
  if (b < b1) v.x = p[b];
  if (b + 1 < b1) v.y = p[b + 1];
  if (b + 2 < b1) v.z = p[b + 2];
  return v;
}

__device__ __forceinline__ int chunks_of(int c) { return (c + kChunk - 1) / kChunk; }

__device__ __forceinline__ void bin_scan_body(int nbins, int32_t* count, int32_t* start, int2* chunk,
                                              int32_t* meta) {
  __shared__ int s_p[32], s_c[32];
  const int T = blockDim.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int per = ((nbins + T - 1) / T + 3) & ~3;
  const int b0 = min(tid * per, nbins), b1 = min(b0 + per, nbins);
  int ps = 0, cs = 0;
  for (int b = b0; b < b1; b += 4) {
    const int4 c = ld_bins4(count, b, b1);
    ps += c.x + c.y + c.z + c.w;
    cs += chunks_of(c.x) + chunks_of(c.y) + chunks_of(c.z) + chunks_of(c.w);
  }
  int pi = ps, ci = cs;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, pi, o), c = __shfl_up_sync(0xffffffffu, ci, o);
    if (lane >= o) {
      pi += a;
      ci += c;
    }
  }
  if (lane == 31) {
    s_p[wid] = pi;
    s_c[wid] = ci;
  }
  __syncthreads();
  if (wid == 0) {
    const int nw = T >> 5;
    const int a0 = lane < nw ? s_p[lane] : 0, c0 = lane < nw ? s_c[lane] : 0;
    int a = a0, c = c0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, c, o);
      if (lane >= o) {
        a += x;
        c += y;
      }
    }
    if (lane < nw) {
      s_p[lane] = a - a0;
      s_c[lane] = c - c0;
    }
  }
  __syncthreads();
  int po = s_p[wid] + pi - ps, co = s_c[wid] + ci - cs;
  for (int b = b0; b < b1; b += 4) {
    const int4 c4 = ld_bins4(count, b, b1);
    const int cv[4] = {c4.x, c4.y, c4.z, c4.w};
    int st[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      st[q] = po;
      const int nc = chunks_of(cv[q]);
      if (nc > 0) {
        const int sz = cv[q] / nc, rem = cv[q] - sz * nc;  // rem chunks of sz + 1, then sz
        int off = po;
        for (int i = 0; i < nc; ++i) {
          const int n = sz + (i < rem ? 1 : 0);
          chunk[co++] = make_int2(off, n);
          off += n;
        }
      }
      po += cv[q];
    }
    if (b + 4 <= b1) {
      *reinterpret_cast<int4*>(start + b) = make_int4(st[0], st[1], st[2], st[3]);
      *reinterpret_cast<int4*>(count + b) = make_int4(0, 0, 0, 0);
    } else {
      for (int q = 0; q < 4 && b + q < b1; ++q) {
        start[b + q] = st[q];
        count[b + q] = 0;
      }
    }
  }
  if (tid == T - 1) meta[0] = co;
}

__global__ __launch_bounds__(1024) void k_bin_scan(int nbins, int32_t* count, int32_t* start, int2* chunk,
                                                   int32_t* meta) {
  griddep_wait();
  griddep_launch();
  bin_scan_body(nbins, count, start, chunk, meta);
}

__device__ __forceinline__ void bin_scatter_body(int n, const int32_t* key, int32_t* cursor, int32_t* perm,
                                                 int vb, int vg) {
  const int p = vb * blockDim.x + threadIdx.x;
  if (p >= n) return;
  perm[atomicAdd(cursor + key[p], 1)] = p;
}

__global__ void k_bin_scatter(int n, const int32_t* key, int32_t* cursor, int32_t* perm) {
  griddep_wait();
  griddep_launch();
  bin_scatter_body(n, key, cursor, perm, blockIdx.x, gridDim.x);
}

// Orders the particles of each bin by B-spline base node (counting sort over
// the bin's kEdge^3 base cells; order within a cell unspecified), so that the
// chunks cut from a bin are compact slabs and particles sharing a stencil are
// adjacent.  One CTA per bin (grid-stride); the bin's range of perm is sorted
// through the same range of `tmp`.  After fsi_mpm_bin's scatter, end[b] is the
// end offset of bin b in perm (its start is end[b - 1]).
constexpr int kBinCells = kEdge * kEdge * kEdge;
constexpr int kSortT = 256;

__device__ __forceinline__ int local_base_cell(const FsiParticles& pt, int p, float inv_dx, int G) {
  int l = 0;
  for (int a = 2; a >= 0; --a) {
    const float Xp = __fmul_rn(pt.x[a * pt.n + p], inv_dx);
    l = l * kEdge + clampi((int)(Xp - 0.5f), 0, G - 1) % kEdge;
  }
  return l;
}

__device__ __forceinline__ void bin_sort_body(const FsiParticles& pt, float inv_dx, int G, int nbins,
                                              const int32_t* end, int32_t* perm,
                                              int32_t* tmp, int vb, int vg) {
  __shared__ int cnt[kBinCells];
  __shared__ int wsum[kSortT / 32];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  constexpr int PER = kBinCells / kSortT;  // counters per thread
  static_assert(kBinCells % kSortT == 0, "bin cells must be a multiple of the sort CTA");
  for (int b = vb; b < nbins; b += vg) {
    const int lo = b ? end[b - 1] : 0, hi = end[b];
    if (hi - lo < 2) continue;  // uniform over the CTA
    for (int i = t; i < kBinCells; i += kSortT) cnt[i] = 0;
    __syncthreads();
    for (int i = lo + t; i < hi; i += kSortT) atomicAdd(&cnt[local_base_cell(pt, perm[i], inv_dx, G)], 1);
    __syncthreads();
    // exclusive scan of the counters: PER per thread, then warps, then CTA
    int v[PER], sum = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      v[q] = cnt[t * PER + q];
      sum += v[q];
    }
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) wsum[wid] = inc;
    __syncthreads();
    int off = inc - sum;
    for (int w = 0; w < wid; ++w) off += wsum[w];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      cnt[t * PER + q] = off;  // becomes the cell's cursor
      off += v[q];
    }
    __syncthreads();
    for (int i = lo + t; i < hi; i += kSortT) {
      const int p = perm[i];
      tmp[lo + atomicAdd(&cnt[local_base_cell(pt, p, inv_dx, G)], 1)] = p;
    }
    __syncthreads();
    for (int i = lo + t; i < hi; i += kSortT) perm[i] = tmp[i];
    __syncthreads();
  }
}

__global__ __launch_bounds__(kSortT) void k_bin_sort(FsiParticles pt, float inv_dx, int G, int nbins,
                                                      const int32_t* end, int32_t* perm,
                                                      int32_t* tmp) {
  griddep_wait();
  griddep_launch();
  bin_sort_body(pt, inv_dx, G, nbins, end, perm, tmp, blockIdx.x, gridDim.x);
}

struct Box {
  int lo[3], ext[3];
  int vol;
};

__device__ __forceinline__ Box load_box(const int32_t* r) {
  Box b;
  unsigned v = 1;  // extents of at most 1600 nodes (see layout()): below 2^32
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b.lo[a] = r[a];
    b.ext[a] = max(r[3 + a] - r[a] + 1, 0);
    v *= (unsigned)b.ext[a];
  }
  b.vol = (int)min(v, (unsigned)INT_MAX);
  return b;
}

// quadratic B-spline weight of offset o for the fractional position f (the
// expressions of bspline())
__device__ __forceinline__ float bspline_w(float f, int o) {
  return o == 0 ? 0.5f * (1.5f - f) * (1.5f - f) : (o == 1 ? 0.75f - (f - 1.0f) * (f - 1.0f) : 0.5f * (f - 0.5f) * (f - 0.5f));
}

// G2P sums of a particle whose stencil leaves the grid, or whose chunk's node
// box does not fit the shared-memory stage (bins gone stale): a rolled loop
// over the nodes inside the grid, from the stage when stg is non-null, from
// the grid otherwise.  Three nodes' loads together instead of one's: clouds whose
// boxes have outgrown the stage (24,576 particles, bins 30 substeps old at 0.3
// cells a substep) 54 -> 41 us per substep; in the batched kernel the registers
// for it cost every substep 2 %.
// U: nodes whose loads are in flight together
template <int U>
__device__ __noinline__ void g2p_slow(const float* stg, int nv, const Box& bx, const FsiGrid& g, const FsiMpmParams& mp,
                                      const BSpline& b, float s4, float v[3], float nC[9]) {
  const int G = g.n;
  const int64_t N = (int64_t)G * G * G;
  float sv[3] = {0.f, 0.f, 0.f}, sC[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
  for (int o0 = 0; o0 < 27; o0 += U) {
    float P[U][3], f[U][3], m[U];
#pragma unroll
    for (int h = 0; h < U; ++h) {
      const int o = min(o0 + h, 26);
      const int I = clampi(b.base[0] + o / 9, 0, G - 1), J = clampi(b.base[1] + (o / 3) % 3, 0, G - 1),
                K = clampi(b.base[2] + o % 3, 0, G - 1);  // a node outside is left out below
      const int li = ((K - bx.lo[2]) * bx.ext[1] + (J - bx.lo[1])) * bx.ext[0] + (I - bx.lo[0]);
      const int64_t node = ((int64_t)K * G + J) * G + I;
      const float* const p = stg ? stg + li : g.v + node;
      const int64_t step = stg ? nv : N;
      P[h][0] = p[0];
      P[h][1] = p[step];
      P[h][2] = p[2 * step];
      m[h] = g.m[node];
      f[h][0] = g.f_ext[node];
      f[h][1] = g.f_ext[N + node];
      f[h][2] = g.f_ext[2 * N + node];
    }
#pragma unroll
    for (int h = 0; h < U; ++h) {
      const int o = o0 + h, ox = o / 9, oy = (o / 3) % 3, oz = o % 3;
      const int id[3] = {b.base[0] + ox, b.base[1] + oy, b.base[2] + oz};
      if (o >= 27 || id[0] < 0 || id[0] >= G || id[1] < 0 || id[1] >= G || id[2] < 0 || id[2] >= G) continue;
      const float w = bspline_w(b.fx[0], ox) * bspline_w(b.fx[1], oy) * bspline_w(b.fx[2], oz);
      const float d[3] = {((float)ox - b.fx[0]) * mp.dx, ((float)oy - b.fx[1]) * mp.dx,
                          ((float)oz - b.fx[2]) * mp.dx};
      if (!stg && m[h] > 0.f) {
        const NodeMass nm = node_mass(m[h]);
#pragma unroll
        for (int a = 0; a < 3; ++a) P[h][a] = grid_node_component(P[h][a], nm, f[h][a], mp.gravity[a], id[a], G, mp);
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float wg = w * P[h][a];
        sv[a] += wg;
#pragma unroll
        for (int k = 0; k < 3; ++k) sC[a * 3 + k] += wg * d[k] * s4;
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) v[a] = sv[a];
#pragma unroll
  for (int a = 0; a < 9; ++a) nC[a] = sC[a];
}

// P2G payload of a particle (shared memory), one record of kQn floats per
// particle of the chunk.  The momentum a particle gives to the stencil node
// (ox, oy, oz), m v + A d with d the node's offset, and its weight are a sum
// and a product over the axes, so the record holds per axis and offset o the
// weight and that axis' share of the momentum: the scatter adds up three of
// them per node (4 wide loads and 15 operations a particle, against 8 loads
// and 21 operations from m v, A and the offset):
//   [4 (3 a + o)] share0 share1 share2 weight   (a = 0: m v is in the share)
//   [36] mass pf0 pf1 pf2                      [40] key base0 base1 base2
// key: the index of the base node in the chunk's box (int bits), -1 when the
// stencil leaves the grid or the chunk's box is too large; base as int bits,
// modulo 3 where one or two tiles fit the box and the key is not -1.
// A record of 44 floats keeps the 128-bit stores of 8 consecutive particles
// on distinct banks.
enum { kQmass = 36, kQkey = 40, kQn = 44 };

// ---- fused substep sequence --------------------------------------------------
// M substeps in M + 1 launches (after a prologue).  Launch s, for each chunk of
// its CTA: the gather of substep s - 1 (G2P from grid buffer (s - 1) % 3, the
// new particle state written to the particle fields and kept in registers),
// then the P2G payload of substep s from that state and its scatter into
// buffer s % 3.  A chunk's particles belong to one CTA for the launch, so
// gather, payload and scatter of a chunk follow each other without any
// grid-wide synchronisation; the launch boundary is the one grid-wide step
// (every scatter of substep s is complete before any gather of it).  The
// launch also zeroes the boxes substep s - 2 recorded in buffer (s + 1) % 3,
// whose last reader (the gather of substep s - 2) ran in the launch before:
// three buffers, so that no launch zeroes a buffer that another CTA of the
// same launch still reads or writes.
//
// A CTA has one thread per particle of the chunk (four warps), which keeps the
// particle's state in registers from the gather to the payload; the scatter
// is by runs of one base node (see there).  Five CTA barriers per chunk.
//
// What bounds it: where a chunk has an SM to itself, the chain of a warp's
// dependent instructions (some 2,500 a substep at 5 cycles each) and of the
// trips to L2; where the SMs hold four, the same chains four to a scheduler, with
// a third to half of the issue slots used.  The bytes (the state of 24,576
// particles and the touched nodes) move in 1 us.  So the
// arithmetic is arranged for few instructions: no thread repeats another's
// work, the tensor-product stencils are summed axis by axis (a node costs two
// multiply-adds per value in the gather), the scatter adds three prepared
// shares per node, shared memory sees no floating-point atomic (a
// compare-and-swap loop of some 100 cycles there), the reaction's lattice box
// arrives by asynchronous copies under the stress, statistics that a later
// substep overwrites are not formed, and what does not depend on the previous
// launch is read before its end.
// One substep, before (two threads per particle, 8 warps, tile with
// shared-memory atomics) and now: 19.7 -> 12.2 us from launch to launch (4,096
// particles), 23.7 -> 18.5 us (24,576 in the benchmarked duct), 126 -> 77 us
// (196,608 there); the 16-case batch's 11 launches 1,312 -> 630-650 us.  Three
// threads per particle (12 warps, one axis each) took 13-21 us at the small sizes
// but 116 us at 196,608 particles and no less than before in a batch.
// Particles at random positions, with the reaction, at 8 / 2 / 0.5 / 0.125 per
// cell, that earlier form and this one: 24,576 particles 23 / 24 / 28 / 58 us and
// 18 / 21 / 24 / 37 us; 196,608: 105 / 129 / 183 / 359 us and
// 67 / 92 / 133 / 217 us.

// bins->meta: [0] chunks, [1 + b] records in box[b], [4] chunks scattered
// without a tile, [5 + b] buffer b holds recorded boxes not yet zeroed
enum { kMetaChunks = 0, kMetaRec = 1, kMetaOverflow = 4, kMetaDirty = 5 };
constexpr int kSeqT = kChunk;
constexpr int kSeqOcc = 4;          // resident CTAs per SM (by registers and by shared memory)
// one region for the staged node velocities (G2P, 3 per node), the reaction's
// lattice box (4 per cell) and the scatter tiles (7 values per node and copy
// with the reaction, 4 without): each is written after the last read of the one
// before it.  A compact chunk of 128 particles at 8 per cell has boxes of 120-220
// nodes, at 2 per cell 270-440, at one per two cells 440-770.
// Where four CTAs of an SM are resident: as large as leaves 60 KB of the SM's
// memory to the L1 cache, whose lines hold the loads in flight (the particle
// state, scattered when the particles are in random order).  Four tiles fit 234
// nodes with the reaction (410 without), two 468 (820), one 937 (all that are
// staged).  8,192 floats (292, 585 and 1,170 nodes), which leave 28 KB, took
// 775 us, not 633, per substep of 10^6 particles in random order, 248, not 225 us,
// in order; 105, not 87, and 70.5, not 67.5 us for 196,608 (the latter with the
// reaction); only at one particle per cell, 100, not 106 us.
constexpr int kStageFloats = 6560;
// Two CTAs per SM, for clouds of less than 48 full chunks with the reaction and
// for few box records: four tiles for 438 nodes with the reaction (768 without),
// two for 877, one for all.  4,096 particles at 8 per cell, with the reaction, on
// 32^3 and 80^3 nodes: 13.5 -> 12.1 and 12.7 -> 11.8 us per substep; a step of ten
// substeps of a plate in a 75 x 52 x 61 box (two of them) 425 -> 403 us.
constexpr int kWideStageFloats = 12288;
static_assert(kStageFloats >= 4 * kTileCap && kStageFloats % 4 == 0, "stage holds the lattice box");
constexpr size_t seq_smem(int stage) { return sizeof(float) * (stage + kQn * kChunk); }

struct SeqArgs {
  FsiParticles pt;
  FsiGrid grid[3];
  FsiMpmParams mp;
  const int32_t* perm;
  const int2* chunks;
  int32_t* meta;
  int32_t* box;        // [3][max_chunks][6]
  int64_t box_stride;  // 6 * max_chunks
  LatView L;
  const float* hydro;
  const float* phi;
  FsiCouplingParams cp;
  FsiCouplingStats* stats;  // [3]; null without the reaction transfer
  const FsiLbmDiag* diag;
  int32_t s, M;             // launch index (0..M) and substeps in the sequence
};

// quotient of a small non-negative integer (below 2^20) by an integer of which
// inv is the reciprocal (small_inv): exact, as (a + 1/2) / b is at least
// 1 / (2 b) away from an integer and the errors of inv and of the product stay
// below 4e-7 of the quotient
__device__ __forceinline__ float small_inv(int b) { return __fdividef(1.0f, (float)b); }
__device__ __forceinline__ int small_div(int a, float inv) { return (int)(((float)a + 0.5f) * inv); }

// zeroes the first nq of the seven values (momentum, mass, external force) of
// the nodes of the recorded boxes: warp w of the nw warps that share the work
// takes the records w, w + nw, ...; where there are several warps per record
// they share it, 32 nodes in turn (SHARE; in the batched kernel, whose arguments
// are in shared memory, not in constants, the registers for it cost 2 %)
template <bool SHARE = true>
__device__ __forceinline__ void zero_boxes(const FsiGrid& go, const int32_t* rec, int nrec, int w, int nw, int nq) {
  const int G = go.n;
  const int64_t N = (int64_t)G * G * G;
  const int parts = SHARE ? max(1, nw / max(nrec, 1)) : 1;
  for (int u = w; u < nrec * parts; u += nw) {
    const int r = u / parts;
    const Box bx = load_box(rec + 6 * r);
    const int e0 = bx.ext[0], e01 = e0 * bx.ext[1];
    const bool small = bx.vol < (1 << 20);  // the range of small_div
    const float i0 = small_inv(max(e0, 1)), i01 = small_inv(max(e01, 1));
    for (int li = 32 * (u - r * parts) + (threadIdx.x & 31); li < bx.vol; li += 32 * parts) {
      const int k = small ? small_div(li, i01) : li / e01, q = li - k * e01;
      const int j = small ? small_div(q, i0) : q / e0, i = q - j * e0;
      const int64_t node = ((int64_t)(k + bx.lo[2]) * G + (j + bx.lo[1])) * G + (i + bx.lo[0]);
      go.v[node] = 0.f;
      go.v[N + node] = 0.f;
      go.v[2 * N + node] = 0.f;
      go.m[node] = 0.f;
      if (nq > 4) {
        go.f_ext[node] = 0.f;
        go.f_ext[N + node] = 0.f;
        go.f_ext[2 * N + node] = 0.f;
      }
    }
  }
}

__device__ __forceinline__ void zero_reaction_stats(FsiCouplingStats* st) {
  st->active_reaction_particle_count = 0;
  st->max_particle_reaction_norm = 0.f;
  st->max_grid_reaction_norm = 0.f;
  st->area_scale = 0.f;
  st->raw_area_scale = 0.f;
  for (int a = 0; a < 3; ++a) {
    st->net_particle_reaction[a] = 0.0;
    st->net_grid_reaction[a] = 0.0;
  }
}

// grid buffer b by value (a select, not an indexed access, so that a
// SeqArgs held in registers needs no local memory)
__device__ __forceinline__ FsiGrid grid_of(const SeqArgs& A, int b) {
  return b == 0 ? A.grid[0] : (b == 1 ? A.grid[1] : A.grid[2]);
}

// zeroes every buffer with boxes left from an earlier sequence, and the
// reaction record of the first substep
__device__ __forceinline__ void seq_prologue_body(const SeqArgs& A, int vb, int vg) {
  const int nw = blockDim.x >> 5;
  for (int b = 0; b < 3; ++b)
    if (A.meta[kMetaDirty + b])
      zero_boxes(grid_of(A, b), A.box + b * A.box_stride, A.meta[kMetaRec + b], vb * nw + (threadIdx.x >> 5), vg * nw, 7);
  if (A.stats && vb == 0 && threadIdx.x == 0) zero_reaction_stats(A.stats);
}

// 4-byte asynchronous copy to a shared-memory address (zero-filled when n = 0)
__device__ __forceinline__ void copy4_async(unsigned dst, const float* src, int n) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// reaction_particle() from the chunk's lattice box staged in shared memory
// (lat[q * nv + li], q = 0..2 the force field, 3 phi; li the index in the box
// bx) for a particle whose stencil lies inside it, summed axis by axis
__device__ __forceinline__ void reaction_particle_staged(const float* __restrict__ lat, int li, int e0, int e01, int nv,
                                                         const FsiCouplingParams& cp, const BSpline& b, float Jp,
                                                         float vol0, float scale, ReactParticle& r) {
  float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    if (f == 3 && cp.kind == 0) break;
    const float* const q = lat + li + f * nv;
#pragma unroll
    for (int oz = 0; oz < 3; ++oz) {
      float t = 0.f;
#pragma unroll
      for (int oy = 0; oy < 3; ++oy) {
        const float* const x = q + oz * e01 + oy * e0;
        t += b.w[1][oy] * (b.w[0][0] * x[0] + b.w[0][1] * x[1] + b.w[0][2] * x[2]);
      }
      sum[f] += b.w[2][oz] * t;
    }
  }
  const float hs[3] = {sum[0], sum[1], sum[2]};
  reaction_from_sums(cp, hs, sum[3], Jp, vol0, scale, r);
}

// Parts that a sequence cuts its chunks into: twice as many while every part
// still has a CTA of its own (the substep then takes as long as one part) and a
// box record, up to max_split (1 where other cases fill the device)
__device__ __forceinline__ int seq_split(int nbin, int ctas, int records, int max_split) {
  int split = 1;
  while (2 * split <= max_split && nbin * split * 2 <= min(ctas, records)) split *= 2;
  return split;
}

// CTAs that take part: one per item and half as many to zero old boxes
__device__ __forceinline__ int seq_ctas_used(int items) { return items + (items >> 1) + 8; }

// Adds the momentum components a0 .. a0 + NM - 1 and the values f0 .. f0 + NF - 1 of (mass, reaction) of the payload
// records [first, last) to a tile of nv nodes and box extents e0, e0 x e1.  Lane l takes the nodes of one class of
// indices modulo 3, of which every stencil holds one: no two lanes meet in a node, so four particles go through
// together, the sums handed on in registers where they share a node (two at a time were 1-2 % faster where the SMs are
// full, 10-20 % slower where a chunk has one to itself).
template <int NM, int NF>
__device__ __forceinline__ void scatter_values(const float* sp, int first, int last, int a0, int f0, float* tile, int nv,
                                               int e0, int e01, const FsiGrid& g) {
  constexpr int NV = NM + NF, U = 4;
  const int lane = threadIdx.x & 31, G = g.n;
  const int rx = lane % 3, ry = (lane / 3) % 3, rz = min(lane / 9, 2);  // lanes 27-31 are not used
  struct Rec {
    int at;  // node in the box
    float w, val[NV];
  };
  auto read = [&](const float* r, int ox, int oy, int oz, int key) {
    const float *const x = r + 4 * ox, *const y = r + 12 + 4 * oy, *const z = r + 24 + 4 * oz;
    Rec c;
    c.at = key + oz * e01 + oy * e0 + ox;
    c.w = x[3] * y[3] * z[3];
#pragma unroll
    for (int i = 0; i < NM; ++i) c.val[i] = x[a0 + i] + y[a0 + i] + z[a0 + i];
#pragma unroll
    for (int i = 0; i < NF; ++i) c.val[NM + i] = r[kQmass + f0 + i];
    return c;
  };
  auto offset = [](int cls, int base) { return cls - base + (cls < base ? 3 : 0); };
  auto value = [&](int i) { return tile + (i < NM ? a0 + i : 3 + f0 + i - NM) * nv; };
  int lp = first;
  while (lp < last) {
    int4 head[U];
    int low = 0;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      head[k] = *reinterpret_cast<const int4*>(sp + min(lp + k, last - 1) * kQn + kQkey);
      low = min(low, head[k].x);
    }
    if (low >= 0 && lp + U <= last) {
      Rec c[U];
      float t[U][NV];
#pragma unroll
      for (int k = 0; k < U; ++k)
        c[k] = read(sp + (lp + k) * kQn, offset(rx, head[k].y), offset(ry, head[k].z), offset(rz, head[k].w), head[k].x);
#pragma unroll
      for (int k = 0; k < U; ++k)
#pragma unroll
        for (int i = 0; i < NV; ++i) t[k][i] = value(i)[c[k].at];
#pragma unroll
      for (int k = 0; k < U; ++k) {
#pragma unroll
        for (int j = 0; j < k; ++j) {
          const bool same = c[j].at == c[k].at;
#pragma unroll
          for (int i = 0; i < NV; ++i) t[k][i] = same ? t[j][i] : t[k][i];
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) t[k][i] += c[k].w * c[k].val[i];
      }
      if (lane < 27) {
#pragma unroll
        for (int k = 0; k < U; ++k)
#pragma unroll
          for (int i = 0; i < NV; ++i) value(i)[c[k].at] = t[k][i];
      }
      lp += U;
      continue;
    }
    const float* const r = sp + lp * kQn;
    const int4 h = head[0];
    if (h.x >= 0) {
      const Rec c = read(r, offset(rx, h.y), offset(ry, h.z), offset(rz, h.w), h.x);
      if (lane < 27) {
#pragma unroll
        for (int i = 0; i < NV; ++i) value(i)[c.at] += c.w * c.val[i];
      }
    } else {
      // a stencil that leaves the grid: to the grid
      const Rec c = read(r, rx, ry, rz, 0);
      const int I = h.y + rx, J = h.z + ry, K = h.w + rz;
      if (lane < 27 && I >= 0 && I < G && J >= 0 && J < G && K >= 0 && K < G) {
        const int64_t N = (int64_t)G * G * G, node = ((int64_t)K * G + J) * G + I;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int f = f0 + i - NM;  // of (mass, reaction)
          float* const dst = i < NM ? g.v + (a0 + i) * N : (f == 0 ? g.m : g.f_ext + (f - 1) * N);
          const float x = c.w * c.val[i];
          if (x != 0.f) atomicAdd(dst + node, x);
        }
      }
    }
    ++lp;
  }
}

// Boxes that only one or two tiles fit: the warps that share a tile divide the grid values between them, so that each
// adds its values of all the tile's particles, with no turns and no atomics.  Such boxes hold two particles per cell or
// fewer (sparse clouds), and nearly every particle is a run of its own there.
template <bool REACT>
__device__ __forceinline__ void scatter_shared_tiles(const float* sp, int count, int copies, float* stg, int stride,
                                                     int nv, int e0, int e01, const FsiGrid& g) {
  constexpr int NW = kSeqT / 32;
  const int wid = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < copies * stride / 4; i += kSeqT)
    reinterpret_cast<float4*>(stg)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  const int group = NW / copies, c = wid / group, m = wid % group;  // warps per tile, this one's tile and part
  const int first = c * count / copies, last = (c + 1) * count / copies;
  float* const tile = stg + c * stride;
  if (copies == 2) {
    if (REACT) {
      if (m == 0)
        scatter_values<3, 1>(sp, first, last, 0, 0, tile, nv, e0, e01, g);
      else
        scatter_values<0, 3>(sp, first, last, 0, 1, tile, nv, e0, e01, g);
    } else {
      if (m == 0)
        scatter_values<2, 0>(sp, first, last, 0, 0, tile, nv, e0, e01, g);
      else
        scatter_values<1, 1>(sp, first, last, 2, 0, tile, nv, e0, e01, g);
    }
  } else if (m < 3) {
    scatter_values<1, REACT ? 1 : 0>(sp, first, last, m, 1 + m, tile, nv, e0, e01, g);
  } else {
    scatter_values<0, 1>(sp, first, last, 0, 0, tile, nv, e0, e01, g);
  }
}

// one particle's part of the reaction diagnostics
struct ReactStats {
  int act;              // reaction not zero
  float pnorm, gnorm;   // norms of the particle's force and of its largest node share
  float pf[3], gf[3];   // force of a gated particle; force given to the grid
  float sw;             // the part of gf that reaches nodes inside the grid
};

__device__ __forceinline__ ReactStats reaction_stats(const ReactParticle& rp, const BSpline& b, int G) {
  ReactStats t = {};
  t.act = rp.act;
  t.pnorm = rp.pnorm;
  if (rp.gated)
    for (int r = 0; r < 3; ++r) t.pf[r] = rp.pf[r];
  if (rp.scatter) {
    // the sums over the particle's nodes inside the grid factorise by axis
    float mw = 1.f, n2 = 0.f;
    t.sw = 1.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      float wa = 0.f, ma = 0.f;
#pragma unroll
      for (int o = 0; o < 3; ++o) {
        const bool in = b.base[a] + o >= 0 && b.base[a] + o < G;
        wa += in ? b.w[a][o] : 0.f;
        ma = fmaxf(ma, in ? b.w[a][o] : 0.f);
      }
      t.sw *= wa;
      mw *= ma;
    }
    for (int r = 0; r < 3; ++r) {
      t.gf[r] = rp.pf[r];
      n2 += rp.pf[r] * rp.pf[r];
    }
    t.gnorm = sqrtf(n2) * mw;
  }
  return t;
}

// launch A.s of the sequence for the chunks vb, vb + vg, ... (kSeqT threads,
// seq_smem(STAGE) bytes of dynamic shared memory), launched with programmatic stream
// serialization: what is read before the wait (the chunk table, perm, mass,
// vol0, fixed) was complete before the launch before the last one, and every
// launch of the sequence waits for the one before it.
template <bool REACT, bool BATCH, int STAGE>
__device__ __forceinline__ void mpm_seq_body(const SeqArgs& A, int vb, int vg, int max_split) {
  constexpr int T = kSeqT, NW = T / 32;
  constexpr int NQ = REACT ? 7 : 4;  // grid values a substep writes
  extern __shared__ float4 seq_smem4[];
  float* const stg = reinterpret_cast<float*>(seq_smem4);  // node velocities, then the lattice box, then the tiles
  float* const sp = stg + STAGE;                           // [kChunk][kQn] P2G payload
  __shared__ int s_lo[3], s_hi[3];
  __shared__ unsigned s_start[NW];  // bit i of word w: particle 32 w + i starts a run of one base node
  __shared__ float s_scale;
  __shared__ int s_cnt[NW];
  __shared__ float s_fmax[NW][2];
  __shared__ double s_dsum[NW][6];
  const FsiParticles& pt = A.pt;
  const FsiMpmParams& mp = A.mp;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int n = pt.n;
  const int s = A.s;
  const bool do_g2p = s > 0, do_p2g = s < A.M;
  // only the record of the last substep remains: each launch zeroes the slot of the substep after its own, so that the
  // last two zero those of the two substeps before the last
  const bool do_stats = REACT && s + 1 == A.M;
  const int bg = (s + 2) % 3, bs = s % 3, bz = (s + 1) % 3;
  const int G = A.grid[0].n;
  const int64_t N = (int64_t)G * G * G;
  // work items: the chunks, each cut into `split` parts
  const int nbin = A.meta[kMetaChunks];
  const int split = seq_split(nbin, vg, (int)(A.box_stride / 6), max_split);
  const int nch = nbin * split;
  vg = min(vg, seq_ctas_used(nch));
  if (vb >= vg) return;
  // this thread's particle of the CTA's first item
  int2 ch = make_int2(0, 0);
  int p = 0, pfixed = 0;
  float pmass = 0.f, pvol0 = 0.f;
  auto load_chunk = [&](int c) {
    ch = A.chunks[c / split];
    const int part = c % split, lo = part * ch.y / split, hi = (part + 1) * ch.y / split;
    ch = make_int2(ch.x + lo, hi - lo);
    if (tid < ch.y) {
      p = A.perm[ch.x + tid];
      pfixed = pt.fixed[p];
      pmass = pt.mass[p];
      pvol0 = pt.vol0[p];
    }
  };
  if (vb < nch) load_chunk(vb);
  griddep_wait();
  griddep_launch();
  FsiCouplingStats* const st = REACT ? A.stats + bs : nullptr;
  if (vb == 0 && tid == 0) {
    if (s == 0) {  // the prologue zeroed every buffer
      A.meta[kMetaDirty + 1] = 0;
      A.meta[kMetaDirty + 2] = 0;
    }
    if (s >= 2) A.meta[kMetaDirty + bz] = 0;
    if (do_p2g) {
      A.meta[kMetaRec + bs] = nch;
      A.meta[kMetaDirty + bs] = 1;
    }
    if (REACT) zero_reaction_stats(A.stats + bz);  // the record of substep s + 1
  }
  if (REACT && do_p2g && tid == 0) {
    float raw = 1.f;
    s_scale = A.cp.kind == 2 ? link_area_scale(A.diag, A.cp, &raw) : 1.0f;
    if (vb == 0 && A.cp.kind == 2) {
      st->area_scale = s_scale;
      st->raw_area_scale = raw;
    }
  }
  // the boxes of substep s - 2: CTAs left without a chunk (fewer chunks than
  // CTAs) zero them, off the path of the CTAs that have one; with fewer than one
  // of these per 16 chunks (the boxes of parts are smaller) every CTA has a
  // share, after its own chunks: one CTA took 90 us over 278 boxes of 700 nodes,
  // 21 took 70 us over 571 of 630 (48 us shared out)
  const bool by_idle = 16 * split * (vg - nch) >= nch;
  const int zero_first = by_idle ? nch : 0;
  if (vb >= nch) {
    if (s >= 2)
      zero_boxes<!BATCH>(grid_of(A, bz), A.box + bz * A.box_stride, A.meta[kMetaRec + bz], (vb - zero_first) * NW + wid,
                 (vg - zero_first) * NW, NQ);
    return;
  }
  if (tid < 3) {
    s_lo[tid] = INT_MAX;
    s_hi[tid] = INT_MIN;
  }

  const float s4 = 4.0f * mp.inv_dx * mp.inv_dx;
  if (do_stats && lane == 0) {
    s_cnt[wid] = 0;
    s_fmax[wid][0] = s_fmax[wid][1] = 0.f;
#pragma unroll
    for (int r = 0; r < 6; ++r) s_dsum[wid][r] = 0.0;
  }
  for (int c = vb; c < nch; c += vg) {
    if (c != vb) {
      load_chunk(c);
      __syncthreads();  // the tiles of the chunk before are read
    }
    const bool live = tid < ch.y;
    const Box bg_box = load_box(A.box + bg * A.box_stride + 6 * c);  // of substep s - 1 (unused at s = 0)
    float X[3] = {0.f, 0.f, 0.f}, v[3] = {0.f, 0.f, 0.f}, C[9], F[9];
#pragma unroll
    for (int a = 0; a < 9; ++a) C[a] = F[a] = 0.f;
    if (live) {
#pragma unroll
      for (int a = 0; a < 3; ++a) X[a] = pt.x[a * n + p];
#pragma unroll
      for (int a = 0; a < 9; ++a) F[a] = pt.F[(int64_t)a * n + p];
      if (!do_g2p) {
#pragma unroll
        for (int a = 0; a < 3; ++a) v[a] = pt.v[a * n + p];
#pragma unroll
        for (int a = 0; a < 9; ++a) C[a] = pt.C[(int64_t)a * n + p];
      }
    }
    if (do_g2p) {
      // ---- G2P of substep s - 1 from buffer bg
      const FsiGrid g = grid_of(A, bg);
      const Box& bx = bg_box;
      const int nv = bx.vol <= kTileCap ? bx.vol : 0;
      const int e0 = bx.ext[0], e01 = e0 * bx.ext[1];
      {
        const float i0 = small_inv(e0), i01 = small_inv(e01);
        for (int li = tid; li < nv; li += T) {
          const int k = small_div(li, i01), r = li - k * e01, j = small_div(r, i0), i = r - j * e0;
          const int I = i + bx.lo[0], Jj = j + bx.lo[1], K = k + bx.lo[2];
          const int64_t node = ((int64_t)K * G + Jj) * G + I;
          const float m = g.m[node];
          const float P[3] = {g.v[node], g.v[N + node], g.v[2 * N + node]};
          const float f[3] = {g.f_ext[node], g.f_ext[N + node], g.f_ext[2 * N + node]};
          float u[3] = {P[0], P[1], P[2]};
          if (m > 0.0f) {
            const NodeMass nm = node_mass(m);
            u[0] = grid_node_component(P[0], nm, f[0], mp.gravity[0], I, G, mp);
            u[1] = grid_node_component(P[1], nm, f[1], mp.gravity[1], Jj, G, mp);
            u[2] = grid_node_component(P[2], nm, f[2], mp.gravity[2], K, G, mp);
          }
#pragma unroll
          for (int a = 0; a < 3; ++a) stg[a * nv + li] = u[a];
        }
      }
      __syncthreads();
      if (live) {
        BSpline b;
        bspline(X, mp.inv_dx, b);
        const bool inside = b.base[0] >= 0 && b.base[0] + 2 < G && b.base[1] >= 0 && b.base[1] + 2 < G &&
                            b.base[2] >= 0 && b.base[2] + 2 < G;
        float nC[9];
        if (nv > 0 && inside) {
          const float* const q =
              stg + ((b.base[2] - bx.lo[2]) * bx.ext[1] + (b.base[1] - bx.lo[1])) * e0 + (b.base[0] - bx.lo[0]);
          float wd[3][3];  // weight times offset from the particle
#pragma unroll
          for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int o = 0; o < 3; ++o) wd[a][o] = b.w[a][o] * (((float)o - b.fx[a]) * mp.dx);
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            float n0 = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
#pragma unroll
            for (int oz = 0; oz < 3; ++oz) {
              float t0 = 0.f, tx = 0.f, ty = 0.f;
#pragma unroll
              for (int oy = 0; oy < 3; ++oy) {
                const float* const r = q + a * nv + oz * e01 + oy * e0;
                const float s0 = b.w[0][0] * r[0] + b.w[0][1] * r[1] + b.w[0][2] * r[2];
                const float s1 = wd[0][0] * r[0] + wd[0][1] * r[1] + wd[0][2] * r[2];
                t0 += b.w[1][oy] * s0;
                tx += b.w[1][oy] * s1;
                ty += wd[1][oy] * s0;
              }
              n0 += b.w[2][oz] * t0;
              cx += b.w[2][oz] * tx;
              cy += b.w[2][oz] * ty;
              cz += wd[2][oz] * t0;
            }
            v[a] = n0;
            nC[a * 3] = cx * s4;
            nC[a * 3 + 1] = cy * s4;
            nC[a * 3 + 2] = cz * s4;
          }
        } else {
          g2p_slow<BATCH ? 1 : 3>(nv > 0 ? stg : nullptr, nv, bx, g, mp, b, s4, v, nC);
        }
        float Fo[9];
#pragma unroll
        for (int a = 0; a < 9; ++a) Fo[a] = F[a];
        g2p_state(pt, p, mp, pfixed != 0, X, v, nC, Fo, F);
#pragma unroll
        for (int a = 0; a < 9; ++a) C[a] = nC[a];
        if (!do_p2g) pt.Jp[p] = det3(F);
      }
    } else {
      __syncthreads();  // publishes the s_lo / s_hi reset
    }
    if (!do_p2g) continue;
    // the chunk's node box: smallest and largest base node per axis
    BSpline b;
    bspline(X, mp.inv_dx, b);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int lo = __reduce_min_sync(0xffffffffu, live ? b.base[r] : INT_MAX);
      const int hi = __reduce_max_sync(0xffffffffu, live ? b.base[r] : INT_MIN);
      if (lane == 0) {
        if (lo != INT_MAX) atomicMin(&s_lo[r], lo);
        if (hi != INT_MIN) atomicMax(&s_hi[r], hi);
      }
    }
    __syncthreads();  // the box of substep s is complete, the staged velocities are read
    int32_t rec[6];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      rec[r] = max(s_lo[r], 0);
      rec[3 + r] = s_hi[r] == INT_MIN ? -1 : min(min(s_hi[r], G) + 2, G - 1);
    }
    const Box bx = load_box(rec);
    const int e0 = bx.ext[0], e1 = bx.ext[1], e01 = e0 * e1;
    // staged: the lattice box fits its region; copies: scatter tiles that fit
    const bool staged = bx.vol <= kTileCap;
    const int nv = staged ? bx.vol : 0;
    const int stride = (NQ * nv + 3) & ~3;  // floats of a tile
    const int copies = !staged ? 0 : (4 * stride <= STAGE ? 4 : (2 * stride <= STAGE ? 2 : (stride <= STAGE)));
    if (tid == 0) {
      int32_t* const out = A.box + bs * A.box_stride + 6 * c;
#pragma unroll
      for (int r = 0; r < 6; ++r) out[r] = rec[r];
      if (!copies) atomicAdd(A.meta + kMetaOverflow, 1);
    }
    const float i0 = small_inv(max(e0, 1)), i01 = small_inv(max(e01, 1));
    if (REACT && staged) {
      // the chunk's lattice box (force field, phi), copied while the stress is computed
      const unsigned dst = (unsigned)__cvta_generic_to_shared(stg);
      for (int li = tid; li < nv; li += T) {
        const int k = small_div(li, i01), r = li - k * e01, j = small_div(r, i0), i = r - j * e0;
        const int I = i + bx.lo[0], Jj = j + bx.lo[1], K = k + bx.lo[2];
        const int in = I < A.L.nx && Jj < A.L.ny && K < A.L.nz ? 4 : 0;
        const int cl = in ? (K * A.L.ny + Jj) * A.L.nx + I : 0;  // below 2^31: 19 values a cell stay below 2^32
        copy4_async(dst + 4 * li, A.hydro + cl, in);
        copy4_async(dst + 4 * (nv + li), A.hydro + A.L.pitch + cl, in);
        copy4_async(dst + 4 * (2 * nv + li), A.hydro + 2 * A.L.pitch + cl, in);
        if (A.cp.kind != 0) copy4_async(dst + 4 * (3 * nv + li), A.phi + cl, in);
      }
    }
    // ---- P2G payload of substep s
    float* const rq = sp + tid * kQn;
    float J = 1.f;
    if (live) {
      P2GParticle q;
      p2g_particle_state(F, C, v, pmass, pvol0, mp, q);
      J = q.J;
      pt.Jp[p] = J;
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int o = 0; o < 3; ++o) {
          const float d = ((float)o - b.fx[a]) * mp.dx;
          float t[3];
#pragma unroll
          for (int r = 0; r < 3; ++r) t[r] = a == 0 ? q.mv[r] + q.aff[r * 3] * d : q.aff[r * 3 + a] * d;
          *reinterpret_cast<float4*>(rq + 4 * (3 * a + o)) = make_float4(t[0], t[1], t[2], b.w[a][o]);
        }
    }
    if (REACT && staged) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
    }
    ReactStats st_add = {};
    if (live) {
      const bool inside = b.base[0] >= 0 && b.base[0] + 2 < G && b.base[1] >= 0 && b.base[1] + 2 < G &&
                          b.base[2] >= 0 && b.base[2] + 2 < G;
      const int li = ((b.base[2] - bx.lo[2]) * e1 + (b.base[1] - bx.lo[1])) * e0 + (b.base[0] - bx.lo[0]);
      float pf[3] = {0.f, 0.f, 0.f};
      if (REACT) {
        ReactParticle rp;
        if (staged && inside)
          reaction_particle_staged(stg, li, e0, e01, nv, A.cp, b, J, pvol0, s_scale, rp);
        else
          reaction_particle(A.L, A.hydro, A.phi, A.cp, b, J, pvol0, s_scale, rp);
        if (rp.scatter)
          for (int r = 0; r < 3; ++r) pf[r] = rp.pf[r];
        if (do_stats) st_add = reaction_stats(rp, b, G);
      }
      *reinterpret_cast<float4*>(rq + kQmass) = make_float4(pmass, pf[0], pf[1], pf[2]);
      const bool to_tile = copies && inside, mod3 = to_tile && copies < 4;
      *reinterpret_cast<int4*>(rq + kQkey) =
          make_int4(to_tile ? li : -1, mod3 ? b.base[0] % 3 : b.base[0], mod3 ? b.base[1] % 3 : b.base[1],
                    mod3 ? b.base[2] % 3 : b.base[2]);
    }
    if (do_stats) {
      // the warp's part of the diagnostics reductions (penalty.py:202-240, moving_boundary.py:312-374)
      const int na = __reduce_add_sync(0xffffffffu, (unsigned)st_add.act);
      const float pm = warp_max(st_add.pnorm), gm = warp_max(st_add.gnorm);
      double r6[6];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        r6[r] = warp_sum_d((double)st_add.pf[r]);
        r6[3 + r] = warp_sum_d((double)st_add.gf[r] * (double)st_add.sw);
      }
      if (lane == 0) {
        s_cnt[wid] += na;
        s_fmax[wid][0] = fmaxf(s_fmax[wid][0], pm);
        s_fmax[wid][1] = fmaxf(s_fmax[wid][1], gm);
#pragma unroll
        for (int r = 0; r < 6; ++r) s_dsum[wid][r] += r6[r];
      }
    }
    {
      const int q0 = __shfl_up_sync(0xffffffffu, b.base[0], 1), q1 = __shfl_up_sync(0xffffffffu, b.base[1], 1),
                q2 = __shfl_up_sync(0xffffffffu, b.base[2], 1);
      const unsigned start = __ballot_sync(
          0xffffffffu, live && (lane == 0 || q0 != b.base[0] || q1 != b.base[1] || q2 != b.base[2]));
      if (lane == 0) s_start[wid] = start;
    }
    __syncthreads();  // payload complete, the lattice box is read
    if (tid < 3) {
      s_lo[tid] = INT_MAX;
      s_hi[tid] = INT_MIN;
    }
    // ---- P2G scatter of substep s into buffer bs, in two steps without
    // floating-point atomics in shared memory (each is a compare-and-swap loop
    // of some 100 cycles).  Particles are sorted by base node within the chunk
    // (fsi_mpm_bin), so they come in runs of one base node.
    // (1) Each warp sums its runs, one particle at a time, lane o on stencil
    // node o (lanes 27-31 are not used), and adds a run's 27 x 7 sums to its
    // own copy of the tile, or straight to the grid where no tile fits (each
    // particle of such a box has most of its nodes to itself).  Where one or
    // two copies fit, the warps take turns on them if the runs are long, and
    // divide the values between them if the runs are short: from 2.5 particles a
    // run on the turns need fewer instructions (98,304 particles at 3 per cell
    // 55.5 against 58.2 us, at 2 per cell 67.2 against 62.2 us).
    const FsiGrid g = grid_of(A, bs);
    float* const dst[7] = {g.v, g.v + N, g.v + 2 * N, g.m, g.f_ext, g.f_ext + N, g.f_ext + 2 * N};
    {
      const int ox = lane / 9, oy = (lane / 3) % 3, oz = lane % 3;
      // lanes 27-31 read offset 2 of the x axis and are not used
      const int q0 = 4 * min(ox, 2), q1 = 12 + 4 * oy, q2 = 24 + 4 * oz;
      const int node_off = oz * e01 + oy * e0 + ox;
      const int words = (ch.y + 31) >> 5;            // words of 32 particles that hold any
      const int share = words <= 1 ? NW : (words == 2 ? NW / 2 : 1);  // warps that share a word's runs
      const int word = wid / share, mine = wid % share;
      float* const tile = stg + (copies ? wid % copies : 0) * stride;
      bool shared_tiles = copies == 1 || copies == 2;
      if (shared_tiles) {
        int runs = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) runs += __popc(s_start[w]);
        shared_tiles = 5 * runs > 2 * ch.y;
      }
      if (shared_tiles) {
        scatter_shared_tiles<REACT>(sp, ch.y, copies, stg, stride, nv, e0, e01, g);
      } else if (wid < copies) {
        for (int i = lane; i < stride / 4; i += 32) reinterpret_cast<float4*>(tile)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
      }
      const int rounds = shared_tiles ? 0 : (copies ? NW / copies : 1);
      for (int round = 0; round < rounds; ++round) {
        if (round > 0) __syncthreads();
        if (copies && wid / copies != round) continue;
        unsigned m = word < words ? s_start[word] : 0u;
        const int last = min(word * 32 + 32, ch.y);
        for (int turn = 0; m; turn = turn + 1 == share ? 0 : turn + 1) {
          const int first = word * 32 + __ffs(m) - 1;
          m &= m - 1;
          const int end = m ? word * 32 + __ffs(m) - 1 : last;
          if (turn != mine) continue;
          const float* rp = sp + first * kQn;
          const int4 head = *reinterpret_cast<const int4*>(rp + kQkey);
          const int key = head.x;
          // the run's sums continue those of the tile (0 where it goes to the grid)
          float* const t = tile + (key >= 0 && lane < 27 ? key + node_off : 0);
          float acc[NQ];
#pragma unroll
          for (int q = 0; q < NQ; ++q) acc[q] = key >= 0 && lane < 27 ? t[q * nv] : 0.f;
#pragma unroll 2
          for (int lp = first; lp < end; ++lp, rp += kQn) {
            const float4 x4 = *reinterpret_cast<const float4*>(rp + q0);
            const float4 y4 = *reinterpret_cast<const float4*>(rp + q1);
            const float4 z4 = *reinterpret_cast<const float4*>(rp + q2);
            const float4 f4 = *reinterpret_cast<const float4*>(rp + kQmass);
            const float w = x4.w * y4.w * z4.w;
            acc[0] += w * (x4.x + y4.x + z4.x);
            acc[1] += w * (x4.y + y4.y + z4.y);
            acc[2] += w * (x4.z + y4.z + z4.z);
            acc[3] += w * f4.x;
            if (REACT) {
              acc[NQ - 3] += w * f4.y;
              acc[NQ - 2] += w * f4.z;
              acc[NQ - 1] += w * f4.w;
            }
          }
          if (key >= 0) {
            if (lane < 27) {
#pragma unroll
              for (int q = 0; q < NQ; ++q) t[q * nv] = acc[q];
            }
            __syncwarp();  // the next run may share nodes
          } else if (lane < 27) {
            // a stencil that leaves the grid, or a box too large: to the grid
            const int I = head.y + ox, Jj = head.z + oy, K = head.w + oz;
            if (I >= 0 && I < G && Jj >= 0 && Jj < G && K >= 0 && K < G) {
              const int64_t node = ((int64_t)K * G + Jj) * G + I;
#pragma unroll
              for (int q = 0; q < NQ; ++q)
                if (acc[q] != 0.f) atomicAdd(dst[q] + node, acc[q]);
            }
          }
        }
      }
    }
    __syncthreads();
    // (2) One thread per node of the box adds the copies' values and gives
    // each to the grid with one global atomic.
    for (int li = tid; copies && li < nv; li += T) {
      const int k = small_div(li, i01), r = li - k * e01, j = small_div(r, i0), i = r - j * e0;
      const int64_t node = ((int64_t)(k + bx.lo[2]) * G + (j + bx.lo[1])) * G + (i + bx.lo[0]);
      const float* const t = stg + li;
      float val[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) val[q] = t[q * nv];
      if (copies > 1) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) val[q] += t[stride + q * nv];
      }
      if (copies > 2) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) val[q] += t[2 * stride + q * nv] + t[3 * stride + q * nv];
      }
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (val[q] != 0.f) atomicAdd(dst[q] + node, val[q]);
    }
  }
  if (!by_idle && s >= 2)
    zero_boxes<!BATCH>(grid_of(A, bz), A.box + bz * A.box_stride, A.meta[kMetaRec + bz], vb * NW + wid, vg * NW, NQ);
  if (do_stats) {
    // the CTA's part: one global atomic per CTA and quantity
    __syncthreads();
    if (tid == 0) {
      int ca = 0;
      float m0 = 0.f, m1 = 0.f;
      double d[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      for (int w = 0; w < NW; ++w) {
        ca += s_cnt[w];
        m0 = fmaxf(m0, s_fmax[w][0]);
        m1 = fmaxf(m1, s_fmax[w][1]);
        for (int r = 0; r < 6; ++r) d[r] += s_dsum[w][r];
      }
      if (ca) atomicAdd(&st->active_reaction_particle_count, ca);
      if (m0 > 0.f) atomic_max_nonneg(&st->max_particle_reaction_norm, m0);
      if (m1 > 0.f) atomic_max_nonneg(&st->max_grid_reaction_norm, m1);
      for (int r = 0; r < 3; ++r) {
        if (d[r] != 0.0) atomicAdd(&st->net_particle_reaction[r], d[r]);
        if (d[3 + r] != 0.0) atomicAdd(&st->net_grid_reaction[r], d[3 + r]);
      }
    }
  }
}

__global__ __launch_bounds__(kSeqT) void k_mpm_seq_prologue(const __grid_constant__ SeqArgs A) {
  griddep_wait();
  griddep_launch();
  seq_prologue_body(A, blockIdx.x, gridDim.x);
}

template <bool REACT, int STAGE>
__global__ __launch_bounds__(kSeqT, kSeqOcc) void k_mpm_seq(const __grid_constant__ SeqArgs A) {
  // the launch's arguments into the constant caches while the previous launch
  // still runs (a first access after the wait costs a trip to L2)
  const int* const w = reinterpret_cast<const int*>(&A);
#pragma unroll
  for (int i = 0; i < (int)(sizeof(SeqArgs) / 4); i += 16) asm volatile("" ::"r"(w[i]));
  mpm_seq_body<REACT, false, STAGE>(A, blockIdx.x, gridDim.x, 4);
}

__global__ void k_grid_velocity(FsiGrid g, FsiMpmParams mp, float* __restrict__ out) {
  const int G = g.n;
  const int64_t N = (int64_t)G * G * G;
  const int64_t node = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= N) return;
  const float m = g.m[node];
  const float P[3] = {g.v[node], g.v[N + node], g.v[2 * N + node]};
  float v[3] = {P[0], P[1], P[2]};
  if (m > 0.0f) {
    const float f[3] = {g.f_ext[node], g.f_ext[N + node], g.f_ext[2 * N + node]};
    grid_node_velocity(P, m, f, (int)(node % G), (int)((node / G) % G), (int)(node / ((int64_t)G * G)), G, mp, v);
  }
  out[node] = v[0];
  out[N + node] = v[1];
  out[2 * N + node] = v[2];
}

int layout(int32_t n_particles, int32_t n_grid, int32_t* n_bins, int32_t* max_chunks) {
  if (n_particles <= 0 || n_grid <= 0) return invalid("n_particles and n_grid must be positive");
  if (n_grid > 1600) return invalid("n_grid above 1600 is not supported by the binned substeps");
  const int64_t nb = (n_grid + kEdge - 1) / kEdge;
  const int64_t bins = nb * nb * nb;
  const int64_t mc = ((int64_t)n_particles + kChunk - 1) / kChunk + std::min<int64_t>(n_particles, bins);
  if (bins > INT_MAX || mc > INT_MAX / 18) return invalid("grid or particle count too large for binning");
  *n_bins = (int32_t)bins;
  *max_chunks = (int32_t)mc;
  return FSI_OK;
}

int check_bins(const FsiMpmBins* bins, int32_t n_particles, int32_t n_grid) {
  if (!bins) return invalid("null bins");
  if (!bins->key || !bins->count || !bins->start || !bins->perm || !bins->chunk || !bins->box || !bins->meta)
    return invalid("null bins array");
  int32_t nb = 0, mc = 0;
  const int rc = layout(n_particles, n_grid, &nb, &mc);
  if (rc) return rc;
  if (bins->n_bins != nb) return invalid("bins->n_bins does not match the grid (see fsi_mpm_bins_layout)");
  if (bins->max_chunks < mc) return invalid("bins->max_chunks below fsi_mpm_bins_layout's capacity");
  if (((uintptr_t)bins->count | (uintptr_t)bins->start | (uintptr_t)bins->chunk) & 15)
    return invalid("bins->count, start and chunk must be 16-byte aligned");
  return FSI_OK;
}

int check_particles(const FsiParticles* pt) {
  if (!pt) return invalid("null particles");
  if (pt->n <= 0) return invalid("n_particles must be positive");
  if (!pt->x || !pt->v || !pt->C || !pt->F || !pt->Jp || !pt->mass || !pt->vol0 || !pt->fixed || !pt->fixed_x)
    return invalid("null particle field");
  return FSI_OK;
}

int check_grid(const FsiGrid* g) {
  if (!g || g->n <= 0 || !g->v || !g->m || !g->f_ext) return invalid("bad grid");
  return FSI_OK;
}

int sm_count() { return device_sm_count(); }

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

using SeqKernel = void (*)(const SeqArgs);

SeqKernel seq_kernel(bool react, bool wide) {
  return react ? (wide ? k_mpm_seq<true, kWideStageFloats> : k_mpm_seq<true, kStageFloats>)
               : (wide ? k_mpm_seq<false, kWideStageFloats> : k_mpm_seq<false, kStageFloats>);
}

// CTAs of a fused-sequence launch, one resident wave (at most one CTA per chunk), and whether their stage is the wide one
int seq_ctas(bool react, int n, int max_chunks, int* ctas, bool* wide) {
  static int occ[64][2] = {};
  int dev = 0;
  int rc = cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc) return rc;
  if (dev < 0 || dev >= 64) return invalid("device ordinal out of range");
  int& o = occ[dev][react ? 1 : 0];
  if (!o) {
    for (const bool w : {false, true})
      if ((rc = cuda_check(cudaFuncSetAttribute(seq_kernel(react, w), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)seq_smem(w ? kWideStageFloats : kStageFloats)),
                           "k_mpm_seq shared memory")))
        return rc;
    int b = 0;
    if ((rc = cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, seq_kernel(react, false), kSeqT,
                                                                       seq_smem(kStageFloats)),
                         "k_mpm_seq occupancy")))
      return rc;
    o = b > 0 ? b : 1;
  }
  // (without the reaction's three values a small cloud's tiles fit, and its chunks are cut further with four CTAs)
  *wide = max_chunks <= 2 * sm_count() || (react && n < 48 * kChunk);
  *ctas = std::max(1, std::min(max_chunks, sm_count() * (*wide ? 2 : o)));
  return FSI_OK;
}

}  // namespace
}  // namespace fsi

using namespace fsi;

extern "C" int fsi_mpm_bins_layout(int32_t n_particles, int32_t n_grid, int32_t* n_bins, int32_t* max_chunks) {
  if (!n_bins || !max_chunks) return invalid("null output");
  return layout(n_particles, n_grid, n_bins, max_chunks);
}

extern "C" int fsi_mpm_bin(const FsiParticles* pt, const FsiGrid* g, const FsiMpmParams* mp, const FsiMpmBins* bins,
                           void* stream) {
  int rc = check_particles(pt);
  if (rc) return rc;
  if (!g || g->n <= 0 || !mp) return invalid("bad grid or params");
  if ((rc = check_bins(bins, pt->n, g->n))) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const int nb = (g->n + kEdge - 1) / kEdge;
  // four launches of 3-5 us for a few thousand particles, each started while the
  // one before drains (none of their pointers is __restrict__: no load may move
  // above griddep_wait()); with the mask rebuild's launches likewise, a 32^3 FSI
  // step of 10 substeps 243 -> 226 us
  auto launched = [&](cudaError_t e, const char* what) {
    const int r = cuda_check(e, what);
    return r ? r : launch_check(what);
  };
  const dim3 pb(nblk(pt->n, 256)), t(256);
  if ((rc = launched(launch_pdl(k_bin_count, pb, t, 0, st, *pt, mp->inv_dx, g->n, nb, bins->key, bins->count),
                     "k_bin_count")))
    return rc;
  if ((rc = launched(launch_pdl(k_bin_scan, dim3(1), dim3(1024), 0, st, bins->n_bins, bins->count, bins->start,
                                reinterpret_cast<int2*>(bins->chunk), bins->meta),
                     "k_bin_scan")))
    return rc;
  if ((rc = launched(launch_pdl(k_bin_scatter, pb, t, 0, st, pt->n, bins->key, bins->start, bins->perm),
                     "k_bin_scatter")))
    return rc;
  // the bin keys are no longer needed: key[] is the sort's scratch
  return launched(launch_pdl(k_bin_sort, dim3((unsigned)std::min(bins->n_bins, sm_count() * 8)), dim3(kSortT), 0, st,
                             *pt, mp->inv_dx, g->n, bins->n_bins, bins->start, bins->perm, bins->key),
                  "k_bin_sort");
}

extern "C" int fsi_mpm_substeps_binned(const FsiParticles* pt, const FsiGrid grid[3], const FsiMpmBins* bins,
                                       const FsiMpmParams* mp, int32_t n_substeps, const FsiLbmState* s,
                                       const float* hydro, const FsiCouplingParams* cp, FsiCouplingStats stats[3],
                                       void* stream) {
  int rc = check_particles(pt);
  if (rc) return rc;
  if (!grid || !mp) return invalid("null grid or params");
  for (int b = 0; b < 3; ++b)
    if ((rc = check_grid(&grid[b]))) return rc;
  if (grid[0].n != grid[1].n || grid[0].n != grid[2].n) return invalid("the three grid buffers differ in size");
  if (n_substeps < 0) return invalid("n_substeps must be >= 0");
  if ((rc = check_bins(bins, pt->n, grid[0].n))) return rc;
  if (cp) {
    if (!s || !hydro || !stats) return invalid("reaction transfer needs the lattice state, hydro and stats");
    if (cp->kind < 0 || cp->kind > 2) return invalid("reaction kind must be 0 (penalty), 1 (engineering), 2 (link-area)");
    if (cp->kind != 0 && !s->phi) return invalid("moving-boundary reaction needs phi");
    if (cp->kind == 2 && !s->diag) return invalid("link-area reaction needs the directional reductions");
    if (cp->inv_dx_norm != mp->inv_dx)
      return invalid("binned substep needs the coupling and MPM grids to share dx (inv_dx_norm == inv_dx)");
  }
  if (n_substeps == 0) return FSI_OK;
  SeqArgs A{};
  A.pt = *pt;
  for (int b = 0; b < 3; ++b) A.grid[b] = grid[b];
  A.mp = *mp;
  A.perm = bins->perm;
  A.chunks = reinterpret_cast<const int2*>(bins->chunk);
  A.meta = bins->meta;
  A.box = bins->box;
  A.box_stride = (int64_t)6 * bins->max_chunks;
  if (cp) {
    A.L = LatView{s->nx, s->ny, s->nz, s->pitch};
    A.hydro = hydro;
    A.phi = s->phi;
    A.cp = *cp;
    A.stats = stats;
    A.diag = s->diag;
  }
  A.M = n_substeps;
  int ctas = 0;
  bool wide = false;
  if ((rc = seq_ctas(cp != nullptr, pt->n, bins->max_chunks, &ctas, &wide))) return rc;
  const size_t smem = seq_smem(wide ? kWideStageFloats : kStageFloats);
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t lerr = launch_pdl(k_mpm_seq_prologue, dim3(ctas), dim3(kSeqT), 0, st, A);
  if ((rc = cuda_check(lerr, "k_mpm_seq_prologue (launch)")) || (rc = launch_check("k_mpm_seq_prologue"))) return rc;
  for (int i = 0; i <= n_substeps; ++i) {
    A.s = i;
    lerr = launch_pdl(seq_kernel(cp != nullptr, wide), dim3(ctas), dim3(kSeqT), smem, st, A);
    if ((rc = cuda_check(lerr, "k_mpm_seq (launch)")) || (rc = launch_check("k_mpm_seq"))) return rc;
  }
  return FSI_OK;
}

extern "C" int fsi_mpm_grid_velocity(const FsiGrid* g, const FsiMpmParams* mp, float* out, void* stream) {
  int rc = check_grid(g);
  if (rc) return rc;
  if (!mp || !out) return invalid("null params or output");
  const int64_t N = (int64_t)g->n * g->n * g->n;
  k_grid_velocity<<<nblk(N, 256), 256, 0, (cudaStream_t)stream>>>(*g, *mp, out);
  return launch_check("k_grid_velocity");
}

// ---- batched cases: MPM (grid.y = case slot) --------------------------------
namespace fsi {
namespace {

// the force field the reaction transfer samples: the last LBM step's link
// forces (moving boundary, one LBM step per FSI step: the ping-pong slot the
// step wrote, now pp ^ 1) or the penalty hydro force
__device__ __forceinline__ const float* batch_hydro(const FsiBatchCase& bc) {
  if (bc.mode == FSI_BATCH_MOVING) return bc.lbm.hpp + (int64_t)(bc.ctl.pp ^ 1) * 3 * bc.lbm.pitch;
  return bc.lbm.hydro;
}

__global__ void k_batch_bin_count(const FsiBatchCase* __restrict__ cases) {
  const FsiBatchCase& bc = cases[blockIdx.y];
  if (!bc.active) return;
  const int G = bc.grid[0].n, nb = (G + kEdge - 1) / kEdge;
  const int nvb = (bc.pt.n + blockDim.x - 1) / blockDim.x;
  for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x)
    bin_count_body(bc.pt, bc.mp.inv_dx, G, nb, bc.bins.key, bc.bins.count, vb, nvb);
}

__global__ __launch_bounds__(1024) void k_batch_bin_scan(const FsiBatchCase* __restrict__ cases) {
  const FsiBatchCase& bc = cases[blockIdx.y];
  if (!bc.active) return;
  bin_scan_body(bc.bins.n_bins, bc.bins.count, bc.bins.start, reinterpret_cast<int2*>(bc.bins.chunk), bc.bins.meta);
}

__global__ void k_batch_bin_scatter(const FsiBatchCase* __restrict__ cases) {
  const FsiBatchCase& bc = cases[blockIdx.y];
  if (!bc.active) return;
  const int nvb = (bc.pt.n + blockDim.x - 1) / blockDim.x;
  for (int vb = blockIdx.x; vb < nvb; vb += gridDim.x)
    bin_scatter_body(bc.pt.n, bc.bins.key, bc.bins.start, bc.bins.perm, vb, nvb);
}

// the sequence arguments of a batched case, into shared memory by the CTA
// (read by one thread they were a chain of 60 loads)
__device__ __forceinline__ void load_batch_seq(const FsiBatchCase& bc, int s, int M, SeqArgs* A) {
  const int tid = threadIdx.x, nt = blockDim.x;
  copy_words(&A->pt, &bc.pt, sizeof(FsiParticles), tid, nt);
  copy_words(A->grid, bc.grid, 3 * sizeof(FsiGrid), tid, nt);
  copy_words(&A->mp, &bc.mp, sizeof(FsiMpmParams), tid, nt);
  copy_words(&A->cp, &bc.cp, sizeof(FsiCouplingParams), tid, nt);
  if (tid != 0) return;
  A->perm = bc.bins.perm;
  A->chunks = reinterpret_cast<const int2*>(bc.bins.chunk);
  A->meta = bc.bins.meta;
  A->box = bc.bins.box;
  A->box_stride = (int64_t)6 * bc.bins.max_chunks;
  A->L = LatView{bc.lbm.nx, bc.lbm.ny, bc.lbm.nz, bc.lbm.pitch};
  A->hydro = batch_hydro(bc);
  A->phi = bc.lbm.phi;
  A->stats = bc.react_stats;
  A->diag = bc.lbm.diag;
  A->s = s;
  A->M = M;
}

__global__ __launch_bounds__(kSeqT) void k_batch_mpm_seq_prologue(const FsiBatchCase* __restrict__ cases) {
  __shared__ SeqArgs A;
  const FsiBatchCase& bc = cases[blockIdx.y];
  if (!bc.active) return;
  load_batch_seq(bc, 0, 1, &A);
  __syncthreads();
  seq_prologue_body(A, blockIdx.x, gridDim.x);
}

// Launched with programmatic stream serialization, like k_mpm_seq: the case
// records and the bins are complete before the prologue starts.
__global__ __launch_bounds__(kSeqT, kSeqOcc) void k_batch_mpm_seq(const FsiBatchCase* __restrict__ cases, int s, int M,
                                                                  int max_split) {
  __shared__ SeqArgs A;
  const FsiBatchCase& bc = cases[blockIdx.y];
  if (!bc.active) {
    if (blockIdx.x == 0) griddep_wait();  // a launch of empty slots must not end before the one ahead of it
    return;
  }
  {
    // the grid is sized for the largest case: CTAs beyond this case's share leave before the arguments are staged
    const int nbin = bc.bins.meta[kMetaChunks];
    const int split = seq_split(nbin, gridDim.x, bc.bins.max_chunks, max_split);
    if ((int)blockIdx.x >= seq_ctas_used(nbin * split)) return;
  }
  load_batch_seq(bc, s, M, &A);
  __syncthreads();
  mpm_seq_body<true, true, kStageFloats>(A, blockIdx.x, gridDim.x, max_split);
}

__global__ __launch_bounds__(kSortT) void k_batch_bin_sort(const FsiBatchCase* __restrict__ cases) {
  const FsiBatchCase& bc = cases[blockIdx.y];
  if (!bc.active) return;
  bin_sort_body(bc.pt, bc.mp.inv_dx, bc.grid[0].n, bc.bins.n_bins, bc.bins.start, bc.bins.perm, bc.bins.key,
                blockIdx.x, gridDim.x);
}

int check_batch_mpm(const FsiBatchCase* cases, const FsiBatchDims* d) {
  if (!cases || !d) return invalid("null batch argument");
  if (d->n_cases <= 0 || d->n_cases > 65535) return invalid("n_cases must be in 1..65535");
  if (d->max_particles <= 0 || d->max_chunks <= 0 || d->max_bins <= 0) return invalid("batch MPM dims must be positive");
  return FSI_OK;
}

}  // namespace
}  // namespace fsi

extern "C" int fsi_batch_mpm_bin(FsiBatchCase* cases, const FsiBatchDims* d, void* stream) {
  int rc = check_batch_mpm(cases, d);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const dim3 g(nblk(d->max_particles, 256), d->n_cases);
  k_batch_bin_count<<<g, 256, 0, st>>>(cases);
  if ((rc = launch_check("k_batch_bin_count"))) return rc;
  k_batch_bin_scan<<<dim3(1, d->n_cases), 1024, 0, st>>>(cases);
  if ((rc = launch_check("k_batch_bin_scan"))) return rc;
  k_batch_bin_scatter<<<g, 256, 0, st>>>(cases);
  if ((rc = launch_check("k_batch_bin_scatter"))) return rc;
  k_batch_bin_sort<<<dim3((unsigned)std::min(d->max_bins, 64), d->n_cases), kSortT, 0, st>>>(cases);
  return launch_check("k_batch_bin_sort");
}

extern "C" int fsi_batch_mpm_substeps(FsiBatchCase* cases, const FsiBatchDims* d, int32_t n_substeps,
                                      void* stream) {
  int rc = check_batch_mpm(cases, d);
  if (rc) return rc;
  if (n_substeps < 0) return invalid("n_substeps must be >= 0");
  if (n_substeps == 0) return FSI_OK;
  cudaStream_t st = (cudaStream_t)stream;
  {
    // once per device (not during stream capture of a later call)
    static bool attr_set[64] = {};
    int dev = 0;
    if ((rc = cuda_check(cudaGetDevice(&dev), "cudaGetDevice"))) return rc;
    if (dev < 0 || dev >= 64) return invalid("device ordinal out of range");
    if (!attr_set[dev]) {
      if ((rc = cuda_check(cudaFuncSetAttribute(k_batch_mpm_seq, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)seq_smem(kStageFloats)),
                           "k_batch_mpm_seq shared memory")))
        return rc;
      attr_set[dev] = true;
    }
  }
  // about one CTA per chunk of the largest case (a bin's chunks hold <= 128 particles each; bins
  // partly filled add chunks): CTAs stride over the case's chunk table
  if (d->mpm_ctas < 0 || d->mpm_ctas > 65535) return invalid("FsiBatchDims.mpm_ctas must be in 0..65535");
  const unsigned gx = d->mpm_ctas > 0 ? (unsigned)d->mpm_ctas
                                      : (unsigned)std::min<int64_t>(d->max_chunks, 2 * nblk(d->max_particles, kChunk) + 8);
  const dim3 gc(gx, d->n_cases);
  k_batch_mpm_seq_prologue<<<gc, kSeqT, 0, st>>>(cases);
  if ((rc = launch_check("k_batch_mpm_seq_prologue"))) return rc;
  // chunks of all cases if each were as large as the largest, against the CTAs the device holds at once
  const int64_t chunks = (int64_t)nblk(d->max_particles, kChunk) * d->n_cases, room = (int64_t)sm_count() * kSeqOcc;
  const int max_split = chunks * 4 <= room ? 4 : (chunks * 2 <= room ? 2 : 1);
  for (int i = 0; i <= n_substeps; ++i) {
    const cudaError_t lerr = launch_pdl(k_batch_mpm_seq, gc, dim3(kSeqT), seq_smem(kStageFloats), st,
                                        (const FsiBatchCase*)cases, i, n_substeps, max_split);
    if ((rc = cuda_check(lerr, "k_batch_mpm_seq (launch)")) || (rc = launch_check("k_batch_mpm_seq"))) return rc;
  }
  return FSI_OK;
}
