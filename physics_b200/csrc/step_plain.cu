// The f64 "plain" SPH passes: bit-identical to the reference's
// FluidWorld<f64>::step (crates/phy-fluid/src/sph/world.rs:183-397).
//
// Arithmetic contract: every floating-point operation is an explicit
// round-to-nearest intrinsic in the reference's evaluation order (this file
// is also compiled with -fmad=false), division and square root are the
// IEEE-exact double operations, and each particle's neighbour reduction runs
// sequentially in the reference's visit order (27 cells, di outer / dk inner,
// ascending insertion index within a cell).  One thread forms each sum, in
// that order, so the result does not depend on scheduling and repeats
// bit-exactly.
//
// Three passes: the search finds each particle's likely neighbours on f32
// coordinates (segment_filter.cuh; nothing in range is lost), the density
// pass tests and sums them in f64 and writes the neighbour lists, and the
// force pass walks the lists.  At 1,024,000 particles they take 113, 171 and
// 305 us; a density pass that tested every candidate in f64 took 479, and the
// force pass on one array per operand 317.
//
// Two exact shortcuts are used:
//   * a candidate whose squared distance exceeds `r2_guard` (the first double
//     above h*h) is skipped before the square root: sqrt(r2) >= h follows,
//     so `r < h` is false exactly as in the reference; NaN distances are
//     never skipped by it;
//   * p_j/(rho_j*rho_j) and m_j/rho_j, which the reference evaluates per pair
//     from the same operands, are evaluated once per particle in the density
//     pass (same expression, same value).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <limits>

#include "launch.cuh"
#include "segment_filter.cuh"
#include "sph_buffers.h"

namespace phy {

namespace {

constexpr int kThreads = 128;
constexpr int kForceCtas = 4;

// Kernels<T> (crates/phy-fluid/src/kernels.rs:39-65).
__device__ __forceinline__ double poly6(const StepConsts& c, double r) {
  if (r >= c.h0) return 0.0;
  double diff = __dsub_rn(c.h0sq, __dmul_rn(r, r));
  return __dmul_rn(__dmul_rn(__dmul_rn(c.poly6_c, diff), diff), diff);
}
__device__ __forceinline__ double spiky_grad_mag(const StepConsts& c, double r) {
  if (r >= c.h0 || r <= 0.0) return 0.0;
  double diff = __dsub_rn(c.h0, r);
  return __dmul_rn(__dmul_rn(c.spiky_c, diff), diff);
}
__device__ __forceinline__ double visc_lap(const StepConsts& c, double r) {
  if (r >= c.h0) return 0.0;
  return __dmul_rn(c.lap_c, __dsub_rn(c.h0, r));
}
// nalgebra Vector3::norm_squared: (x*x + y*y) + z*z.
__device__ __forceinline__ double norm2(double x, double y, double z) {
  return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

struct PlainArgs {
  const float4* __restrict__ fpos;  // box-relative f32 position, z cell (bits)
  const uint32_t* __restrict__ sorted_cell;
  // The search's record per group of 32 slots: kSearchWords * 32 candidate
  // words, kSearchWords rows of hit words (one word per slot and row, rows of
  // `stride`), and (hit words used, lanes that walk their 27 cells
  // themselves).  The hit rows are the neighbour lists' last rows: a group's
  // hits are read before its lists are written.
  uint32_t* cand;
  uint32_t* hits;
  uint2* group;
  ParticleConsts before, now;       // constants the sort read and wrote
  double* rec0;                     // packed pair operands, three parts
  double* rec1;
  double2* rec2;
  const double* __restrict__ px;
  const double* __restrict__ py;
  const double* __restrict__ pz;
  const double* __restrict__ vx;
  const double* __restrict__ vy;
  const double* __restrict__ vz;
  const double* __restrict__ mass;
  const uint32_t* __restrict__ mat;
  const uint32_t* __restrict__ cell_start;
  double* bax;  // body_acc (nullable; zeroed after use)
  double* bay;
  double* baz;
  double* rho;
  double* p;
  double* pr2;
  double* mr;
  double* acc[3];
  double* xsph[3];
  double* mu;
  double* out_pv[6];
  uint32_t* nbr;
  uint32_t* nbr_count;
  int stride;  // column stride of nbr (the buffer capacity)
  uint32_t* flags;
  unsigned long long* counters;
  double* fv_out[3];  // nullable: raw viscous force (adjoint tape)
  double* shear_out;  // nullable: strain-rate proxy (adjoint tape)
  float cull2;        // squared f32 filter radius (plain_cull2); NaN passes every candidate
};

// The pair operands of every sorted slot in three arrays: part 0 x, y, z,
// mass (the sort's gather); part 1 vx, vy, vz, rho; part 2 p/rho^2, 1/rho
// (the density pass).  A neighbour costs one load and one sector per part
// instead of one per field, and neighbours at consecutive slots share lines.
struct d4 {
  double x, y, z, w;
};
__device__ __forceinline__ d4 load_d4(const double* p) {
  d4 v;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void store_d4(double* p, double x, double y, double z, double w) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(x), "d"(y), "d"(z), "d"(w) : "memory");
}

constexpr int kSearchWarps = 8;
constexpr int kSearchCtas = 4;
constexpr int kDensityWarps = 4;
constexpr int kDensityCtas = 8;
constexpr int kSms = 148;
constexpr int kZSpan = 6;     // z cells a warp's query segment may span
constexpr int kSlotBits = 27; // slot index bits of a candidate word; the z cell modulo 32 sits above
constexpr uint32_t kLostGroup = 0xffffffffu;  // words of a group whose step does not happen
// Queries whose 27 cells hold at most this many particles (spray, sparse
// scenes) walk them one by one instead of sharing a staged segment.
constexpr unsigned kWalkBelow = 40;
static_assert(kSearchWords % kBatchWords == 0, "whole batches per group");

// The running density sum of one query and its neighbour list.
struct Query {
  int i;
  double x, y, z;
  double rho = 0.0;
  uint32_t* list;  // the next entry
  uint32_t cnt = 0;
  unsigned pairs = 0;
};

// One candidate (slot j, position and mass b) in the reference's operations
// (world.rs:219-238); records every candidate j != i that the force loop
// will not skip on the `r >= h` test: those with r < h and those whose
// distance is NaN, which the reference's force loop does not skip either
// (world.rs:297).  Without branches: a warp's lanes meet their out-of-range
// candidates and themselves at different times.  kSame: the cutoff h is at
// most the kernel radius h0, so r < h settles the kernel's own test.
template <bool kCount, bool kSame>
__device__ __forceinline__ void density_term(const StepConsts& c, const PlainArgs& a, Query& q, bool ok, int j,
                                             const d4& b) {
  // na_distance(p_i, p_j) = |p_i - p_j| (world.rs:777-779).  A zero distance
  // skips the square root's slow path.
  const double r2 = norm2(__dsub_rn(q.x, b.x), __dsub_rn(q.y, b.y), __dsub_rn(q.z, b.z));
  const bool zero = r2 == 0.0;
  double r = __dsqrt_rn(zero ? 1.0 : r2);
  r = zero ? 0.0 : r;
  const bool in = ok && r < c.h;
  const bool listed = ok && !(r >= c.h) && j != q.i;
  double w;
  if (kSame) {
    const double diff = __dsub_rn(c.h0sq, __dmul_rn(r, r));
    w = __dmul_rn(__dmul_rn(__dmul_rn(c.poly6_c, diff), diff), diff);
  } else {
    w = poly6(c, r);
  }
  const double sum = __dadd_rn(q.rho, __dmul_rn(b.w, w));
  if (in) q.rho = sum;
  if (kCount) q.pairs += in ? 1u : 0u;
  if (listed) {
    if (q.cnt < (uint32_t)kMaxNeighbors) *q.list = (uint32_t)j;
    q.list += a.stride;
    ++q.cnt;
  }
}

// The neighbour search: for every group of 32 consecutive sorted particles,
// the candidates that may be in range of some of them, in the reference's
// visit order, and a bit per (candidate, query).
//
// What bounds the search: one thread per particle testing its ~219 candidates
// is a serial chain of dependent loads (62 us however few particles there
// are).  Here a warp owns a group; its queries of one x,y column (a segment)
// share their candidates.  Lanes load the nine runs of cells around the
// segment side by side, drop what lies out of reach of the segment's bounding
// box (432 of a 4-cell segment's candidates become ~215), and the segment
// filter marks the pairs within a slightly widened radius.  The wider radius
// only lets in candidates that the density pass's f64 test then rejects, so
// the result is the reference's bit for bit.  A group whose candidates exceed
// its record, and queries in sparse surroundings, are left to the density
// pass's own walk (PlainArgs::group).
__global__ void __launch_bounds__(kSearchWarps * 32, kSearchCtas) k_search_plain(StepConsts c, PlainArgs a) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  SegmentStage& st = reinterpret_cast<SegmentStage*>(smem)[threadIdx.x >> 5];
  const int group = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  if (group * 32 >= c.n) return;
  const int i = min(group * 32 + lane, c.n - 1);
  const float4 own = a.fpos[i];
  const uint32_t cell = a.sorted_cell[i];
  if (a.flags[0] & kFlagSortLost) {
    if (group * 32 + lane < c.n) {
      keep_particle(a.before, a.now, i);
      a.nbr_count[i] = 0;  // (a recorded step then has no lists to follow)
    }
    if (lane == 0) a.group[group] = make_uint2(kLostGroup, 0u);
    return;
  }
  const bool inside = group * 32 + lane < c.n && cell < (uint32_t)c.ncells;  // else the overflow cell
  const int bz = __float_as_int(own.w);
  const int col = (int)cell - bz;  // first cell of the column
  uint32_t* slots = a.cand + (size_t)group * (kSearchWords * 32);
  uint32_t* hits = a.hits + (size_t)group * 32 + lane;
  const bool own_slot = group * 32 + lane < c.n;
  uint32_t words = 0;
  unsigned todo = __ballot_sync(0xffffffffu, inside), walkers = 0;
  bool sparse_known = false;
  while (todo) {
    // Segment: the remaining queries of the first one's column, at most
    // kZSpan cells along z (the slots ascend in z inside a column).
    const int first = __ffs(todo) - 1;
    const int scol = __shfl_sync(0xffffffffu, col, first);
    const int z0 = __shfl_sync(0xffffffffu, bz, first);
    const bool mine = ((todo >> lane) & 1u) != 0u && col == scol && bz - z0 < kZSpan;
    const unsigned seg_lanes = __ballot_sync(0xffffffffu, mine);
    if (!sparse_known && __popc(seg_lanes) < 8) {
      // A thin segment: queries with few candidates leave the search.
      sparse_known = true;
      unsigned cand = 0;
      if (inside) {
#pragma unroll
        for (int r = 0; r < 9; ++r) {
          const int c0 = (int)cell + ((r / 3 - 1) * c.ncy + r % 3 - 1) * c.ncz - 1;
          cand += a.cell_start[c0 + 3] - a.cell_start[c0];
        }
      }
      const unsigned few = __ballot_sync(0xffffffffu, inside && cand <= kWalkBelow) & todo;
      walkers |= few;
      todo &= ~few;
      if (few) continue;
    }
    todo &= ~seg_lanes;
    const int z1 = (int)__reduce_max_sync(0xffffffffu, mine ? (unsigned)bz : (unsigned)z0);
    // Lane r < 9 holds run r (dx outer, dy inner): cells z0-1 .. z1+1.
    uint32_t rs = 0, re = 0;
    if (lane < 9) {
      const int c0 = scol + ((lane / 3 - 1) * c.ncy + lane % 3 - 1) * c.ncz + z0 - 1;
      rs = a.cell_start[c0];
      re = a.cell_start[c0 + (z1 - z0) + 3];
    }
    Segment seg = make_segment(mine, own.x, own.y, own.z, a.cull2);
    // The nine runs one after another in chunks of 32 candidates, the next
    // chunk loaded ahead; lane r holds run r's end and its slots' offset.
    const uint32_t len = re - rs;
    uint32_t stop = len;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, stop, o);
      if (lane >= o) stop += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, stop, 8);
    const uint32_t shift = rs - (stop - len);
    int run = 0;
    uint32_t at = (uint32_t)lane, j = 0;
    float4 ahead = make_float4(0.f, 0.f, 0.f, 0.f);
    auto load = [&]() {
      while (__any_sync(0xffffffffu, at >= __shfl_sync(0xffffffffu, stop, run) && run < 8))
        run += at >= __shfl_sync(0xffffffffu, stop, run) && run < 8 ? 1 : 0;
      j = at + __shfl_sync(0xffffffffu, shift, run);
      if (at < total) ahead = a.fpos[j];
    };
    load();
    uint32_t m = 0;  // staged candidates
    bool full = false;
    for (uint32_t t0 = 0;; t0 += 32u) {
      const bool more = t0 < total;
      const float cx = ahead.x - seg.ctr[0], cy = ahead.y - seg.ctr[1], cz = ahead.z - seg.ctr[2];
      const uint32_t word = ((uint32_t)__float_as_int(ahead.w) << kSlotBits) | j;  // z cell modulo 32
      const bool near = at < total && (near_segment(seg, cx, cy, cz) || seg.all);
      at += 32u;
      if (t0 + 32u < total) load();
      if (__any_sync(0xffffffffu, near && !(fabsf(cx) + fabsf(cy) + fabsf(cz) < 1e30f))) seg.all = true;
      const unsigned nm = __ballot_sync(0xffffffffu, near);
      const uint32_t add = (uint32_t)__popc(nm);
      if (m + add > (uint32_t)kBatch || !more) {
        filter_batch(st, m, seg);
        const uint32_t w1 = (m + 31u) >> 5;
        if (own_slot)
          for (uint32_t w = 0; w < w1; ++w) hits[(size_t)(words + w) * a.stride] = mine ? st.hits[w][lane] : 0u;
        __syncwarp();
        words += w1;
        m = 0;
      }
      if (!more) break;
      if (words + ((m + add + 31u) >> 5) > (uint32_t)kSearchWords) {
        full = true;  // uniform
        break;
      }
      if (near) {
        const uint32_t k = m + (uint32_t)__popc(nm & ((1u << lane) - 1u));
        stage_candidate(st, k, cx, cy, cz);
        slots[words * 32u + k] = word;
      }
      m += add;
    }
    if (full) {
      walkers = __ballot_sync(0xffffffffu, inside);
      words = 0;
      break;
    }
  }
  if (lane == 0) a.group[group] = make_uint2(words, walkers);
}

// Walks the set bits of a lane's hits in candidate order.
struct HitWalk {
  const uint32_t* hits;  // this lane's column of words, a sentinel word last
  uint32_t row = 0, mask = 0, end;
  __device__ __forceinline__ HitWalk(const uint32_t* h, uint32_t words) : hits(h), end(32u * words) {}
  // The next candidate; `end` after the last (then not to be called again).
  __device__ __forceinline__ uint32_t next() {
    while (mask == 0u) mask = hits[32u * row++];
    const uint32_t k = 32u * row - 33u + (uint32_t)__ffs(mask);
    mask &= mask - 1u;
    return k;
  }
};

struct DensityStage {
  uint32_t hits[kSearchWords + 1][32];
  uint32_t slot[kSearchWords * 32];
};

// compute_density_pressure (world.rs:204-246): the reference's f64 operations
// over the candidates the search kept, in its order, one lane per particle.
// Issue-bound: ~33 candidates of ~80 instructions, a third of them f64.
template <bool kCount, bool kSame>
__global__ void __launch_bounds__(kDensityWarps * 32, kDensityCtas) k_density_plain(StepConsts c, PlainArgs a) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  DensityStage& st = reinterpret_cast<DensityStage*>(smem)[threadIdx.x >> 5];
  const int group = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  if (group * 32 >= c.n) return;
  const int i = group * 32 + lane;
  const bool valid = i < c.n;
  const int ii = valid ? i : c.n - 1;
  const uint2 rec = a.group[group];
  if (rec.x == kLostGroup) return;
  {
    const uint32_t* slots = a.cand + (size_t)group * (kSearchWords * 32) + lane;
    const uint32_t* hits = a.hits + ii;
#pragma unroll 4
    for (uint32_t w = 0; w < rec.x; ++w) {
      st.hits[w][lane] = valid ? hits[(size_t)w * a.stride] : 0u;
      st.slot[w * 32u + lane] = slots[w * 32u];
    }
    st.hits[rec.x][lane] = 1u;
  }
  const uint32_t cell = a.sorted_cell[ii];
  const uint32_t bz = (uint32_t)__float_as_int(a.fpos[ii].w);
  Query q;
  q.i = ii;
  q.x = a.px[ii];
  q.y = a.py[ii];
  q.z = a.pz[ii];
  q.list = a.nbr + ii;
  __syncwarp();
  constexpr uint32_t kMask = (1u << kSlotBits) - 1u;
  HitWalk walk(&st.hits[0][lane], rec.x);
  struct Hit {
    uint32_t k, w;
    d4 b;
  };
  // The next hit's position is loaded while this one is computed.
  auto fetch = [&](Hit& h) {
    h.k = walk.next();
    if (h.k < walk.end) {
      h.w = st.slot[h.k];
      h.b = load_d4(a.rec0 + (size_t)(h.w & kMask) * 4);
    }
  };
  // Only the query's own 27 cells count (a segment's candidates cover the
  // cells of all its queries): a candidate's z cell, kept modulo 32 in its
  // word, is at most one from the query's.
  auto term = [&](const Hit& h) {
    const bool ok = (((h.w >> kSlotBits) - bz + 1u) & 31u) <= 2u;
    density_term<kCount, kSame>(c, a, q, ok, (int)(h.w & kMask), h.b);
  };
  Hit h0, h1;
  fetch(h0);
  while (h0.k < walk.end) {
    fetch(h1);
    term(h0);
    if (h1.k >= walk.end) break;
    fetch(h0);
    term(h1);
  }
  const bool inside = valid && cell < (uint32_t)c.ncells;
  if ((rec.y >> lane) & 1u) {
    uint32_t s[9], e[9];
#pragma unroll
    for (int r = 0; r < 9; ++r) {
      const int c0 = (int)cell + ((r / 3 - 1) * c.ncy + r % 3 - 1) * c.ncz - 1;
      s[r] = a.cell_start[c0];
      e[r] = a.cell_start[c0 + 3];
    }
    // One loop over the nine runs, so lanes with short runs do not wait at
    // each run for the longest.
    uint32_t j = 0, stop = 0;
    int r = 0;
    for (;;) {
      while (j >= stop && r < 9) {
#pragma unroll
        for (int u = 0; u < 9; ++u)
          if (u == r) {
            j = s[u];
            stop = e[u];
          }
        ++r;
      }
      if (j >= stop) break;
      density_term<kCount, kSame>(c, a, q, true, (int)j, load_d4(a.rec0 + (size_t)j * 4));
      ++j;
    }
  }
  unsigned cand = 0;
  if (kCount && inside) {
    for (int r = 0; r < 9; ++r) {
      const int c0 = (int)cell + ((r / 3 - 1) * c.ncy + r % 3 - 1) * c.ncz - 1;
      cand += a.cell_start[c0 + 3] - a.cell_start[c0];
    }
  }
  if (valid) {
    const double rho = q.rho;
    a.nbr_count[i] = q.cnt;
    const double over = __dsub_rn(rho, c.rest);
    const double pr = over > 0.0 ? __dmul_rn(c.stiff, over) : 0.0;
    const double pr2 = __ddiv_rn(pr, __dmul_rn(rho, rho));
    const double mr = __ddiv_rn(a.mass[i], rho);
    a.rho[i] = rho;
    a.p[i] = pr;
    a.pr2[i] = pr2;
    a.mr[i] = mr;
    store_d4(a.rec1 + (size_t)i * 4, a.vx[i], a.vy[i], a.vz[i], rho);
    a.rec2[i] = make_double2(pr2, __drcp_rn(rho));
    // The force pass divides through reciprocals; densities whose reciprocal
    // leaves the safe range send it to plain divisions.
    if (inside && !(rho > 1e-100 && rho < 1e100)) atomicOr(a.flags + 1, 1u);
  }
  if (kCount) {
    const unsigned wc = __reduce_add_sync(0xffffffffu, cand);
    const unsigned wp = __reduce_add_sync(0xffffffffu, q.pairs);
    if (lane == 0) {
      atomicAdd(&a.counters[0], (unsigned long long)wc);
      atomicAdd(&a.counters[1], (unsigned long long)wp);
    }
  }
}

// a / b given y = 1/b rounded to nearest: q = a y is within an ulp of the
// quotient, its remainder is exact in one FMA, and the corrected quotient is
// the correctly rounded one (Markstein, IBM J. Res. Dev. 34(1), 1990),
// provided nothing under- or overflows on the way: the sort's gather
// (plain_safe) and the density pass set flags[1] otherwise.  The sign
// of a zero quotient may differ, which no sum starting at +0 can show.
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const double q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(-q, b, a), y, q);
}

struct PairTerms {
  double fpx, fpy, fpz, fvx, fvy, fvz, xsx, xsy, xsz, shear;
};

// One neighbour of compute_forces' loop body (world.rs:291-316), in the
// reference's expression order; false when the loop skips it.  kShear = false
// leaves out the shear sum (StepConsts::shear_live: every reachable visc_n is
// 1, so mu never reads it).  kFast: the quotients by r and rho_j are formed
// from one reciprocal each (div_by).
struct Neighbour {
  d4 p, v;
  double2 s;
};
__device__ __forceinline__ Neighbour load_neighbour(const PlainArgs& a, uint32_t j) {
  Neighbour b;
  b.p = load_d4(a.rec0 + (size_t)j * 4);
  b.v = load_d4(a.rec1 + (size_t)j * 4);
  b.s = a.rec2[j];
  return b;
}

template <bool kShear, bool kFast>
__device__ __forceinline__ bool plain_pair(const StepConsts& c, const Neighbour& b, double xi, double yi, double zi,
                                           double vxi, double vyi, double vzi, double m_i, double pr2_i,
                                           PairTerms& t) {
  const d4 &pj = b.p, &vj = b.v;
  const double2 sj = b.s;
  // d = pos[j] - p_i; r = |d|; skip r >= h or r <= 0 (world.rs:295-299).
  const double dx = __dsub_rn(pj.x, xi);
  const double dy = __dsub_rn(pj.y, yi);
  const double dz = __dsub_rn(pj.z, zi);
  const double r2 = norm2(dx, dy, dz);
  if (r2 > c.r2_guard) return false;
  const double r = __dsqrt_rn(r2);
  if (r >= c.h || r <= 0.0) return false;
  const double rho_j = vj.w;
  const double m_j = pj.w;
  const double mm = __dmul_rn(m_i, m_j);
  // f_press += (d / r) * (coef * grad)   (world.rs:303-306)
  const double grad = spiky_grad_mag(c, r);
  const double coef = __dmul_rn(mm, __dadd_rn(pr2_i, sj.x));
  const double cg = __dmul_rn(coef, grad);
  double ux, uy, uz, mq, mr_j;
  if (kFast) {
    const double y = __drcp_rn(r);
    ux = div_by(dx, r, y);
    uy = div_by(dy, r, y);
    uz = div_by(dz, r, y);
    mq = div_by(mm, rho_j, sj.y);
    mr_j = div_by(m_j, rho_j, sj.y);
  } else {
    ux = __ddiv_rn(dx, r);
    uy = __ddiv_rn(dy, r);
    uz = __ddiv_rn(dz, r);
    mq = __ddiv_rn(mm, rho_j);
    mr_j = __ddiv_rn(m_j, rho_j);
  }
  t.fpx = __dmul_rn(ux, cg);
  t.fpy = __dmul_rn(uy, cg);
  t.fpz = __dmul_rn(uz, cg);
  // f_visc_raw += (v_j - v_i) * (m_i * m_j / rho_j * lap)   (308-309)
  const double dvx = __dsub_rn(vj.x, vxi);
  const double dvy = __dsub_rn(vj.y, vyi);
  const double dvz = __dsub_rn(vj.z, vzi);
  const double vf = __dmul_rn(mq, visc_lap(c, r));
  t.fvx = __dmul_rn(dvx, vf);
  t.fvy = __dmul_rn(dvy, vf);
  t.fvz = __dmul_rn(dvz, vf);
  // xsph += (v_j - v_i) * (m_j / rho_j * w)   (311-312)
  const double xw = __dmul_rn(mr_j, poly6(c, r));
  t.xsx = __dmul_rn(dvx, xw);
  t.xsy = __dmul_rn(dvy, xw);
  t.xsz = __dmul_rn(dvz, xw);
  // shear += |v_j - v_i| / (r + 1e-4) * (m_j / rho_j)   (314-315)
  if (kShear) {
    const double dvn = __dsqrt_rn(norm2(dvx, dvy, dvz));
    t.shear = __dmul_rn(__ddiv_rn(dvn, __dadd_rn(r, 1e-4)), mr_j);
  }
  return true;
}

struct PlainAcc {
  double fpx = 0.0, fpy = 0.0, fpz = 0.0;
  double fvx = 0.0, fvy = 0.0, fvz = 0.0;
  double xsx = 0.0, xsy = 0.0, xsz = 0.0;
  double shear = 0.0;
};

template <bool kShear>
__device__ __forceinline__ void add_terms(PlainAcc& q, const PairTerms& t) {
  q.fpx = __dadd_rn(q.fpx, t.fpx);
  q.fpy = __dadd_rn(q.fpy, t.fpy);
  q.fpz = __dadd_rn(q.fpz, t.fpz);
  q.fvx = __dadd_rn(q.fvx, t.fvx);
  q.fvy = __dadd_rn(q.fvy, t.fvy);
  q.fvz = __dadd_rn(q.fvz, t.fvz);
  q.xsx = __dadd_rn(q.xsx, t.xsx);
  q.xsy = __dadd_rn(q.xsy, t.xsy);
  q.xsz = __dadd_rn(q.xsz, t.xsz);
  if (kShear) q.shear = __dadd_rn(q.shear, t.shear);
}

// mu_eff, acc, integrate and bounds of particle i (world.rs:319-397).
__device__ __forceinline__ void finish_plain(const StepConsts& c, const PlainArgs& a, int i, const PlainAcc& q) {
  const double rho_i = a.rho[i];
  // Power-law effective viscosity (world.rs:319-327).
  const uint32_t m = a.mat[i];
  const int midx = (int)m < c.n_visc_k ? (int)m : 0;
  double kc, nn;
  material_coeffs(c, midx, kc, nn);
  const double ex = __dsub_rn(nn, 1.0);
  const double sreg = q.shear > c.shear_min ? q.shear : c.shear_min;
  const double mu = __dmul_rn(kc, ex == 0.0 ? 1.0 : pow(sreg, ex));
  // acc = (f_press + f_visc_raw * mu) / rho_i if rho_i > 0 (329-336).
  double ax = 0.0, ay = 0.0, az = 0.0;
  if (rho_i > 0.0) {
    ax = __ddiv_rn(__dadd_rn(q.fpx, __dmul_rn(q.fvx, mu)), rho_i);
    ay = __ddiv_rn(__dadd_rn(q.fpy, __dmul_rn(q.fvy, mu)), rho_i);
    az = __ddiv_rn(__dadd_rn(q.fpz, __dmul_rn(q.fvz, mu)), rho_i);
  }
  a.acc[0][i] = ax;
  a.acc[1][i] = ay;
  a.acc[2][i] = az;
  a.xsph[0][i] = q.xsx;
  a.xsph[1][i] = q.xsy;
  a.xsph[2][i] = q.xsz;
  a.mu[i] = mu;
  if (a.shear_out) {
    a.fv_out[0][i] = q.fvx;
    a.fv_out[1][i] = q.fvy;
    a.fv_out[2][i] = q.fvz;
    a.shear_out[i] = q.shear;
  }
  // integrate (352-363): a = (acc + g) + body_acc; v += a dt; v += xsph eps; x += v dt.
  double bx = 0.0, by = 0.0, bz = 0.0;
  if (a.bax) {
    bx = a.bax[i];
    by = a.bay[i];
    bz = a.baz[i];
    a.bax[i] = 0.0;
    a.bay[i] = 0.0;
    a.baz[i] = 0.0;
  }
  double p3[3] = {a.px[i], a.py[i], a.pz[i]};
  double v3[3] = {a.vx[i], a.vy[i], a.vz[i]};
  const double acc3[3] = {ax, ay, az};
  const double xs3[3] = {q.xsx, q.xsy, q.xsz};
  const double b3[3] = {bx, by, bz};
  bool finite = true;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double ak = __dadd_rn(__dadd_rn(acc3[k], c.g[k]), b3[k]);
    double v = __dadd_rn(v3[k], __dmul_rn(ak, c.dt));
    v = __dadd_rn(v, __dmul_rn(xs3[k], c.xsph_eps));
    double x = __dadd_rn(p3[k], __dmul_rn(v, c.dt));
    // enforce_bounds: clamp and reflect with damping.
    if (x < c.lo[k]) {
      x = c.lo[k];
      v = __dmul_rn(-v, c.damp);
    } else if (x > c.hi[k]) {
      x = c.hi[k];
      v = __dmul_rn(-v, c.damp);
    }
    finite = finite && isfinite(x) && isfinite(v);
    p3[k] = x;
    v3[k] = v;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    a.out_pv[k][i] = p3[k];
    a.out_pv[3 + k][i] = v3[k];
  }
  if (!finite) atomicOr(a.flags, kFlagNonFinite);
}

// The pair sums of one particle, `kG` lanes each (its lanes are consecutive;
// lane s of the group takes every kG-th listed neighbour).  With kG > 1 each
// round's terms go through the warp's buffer and lane s adds components s,
// s + kG, .. of the round's neighbours in list order, so every sum runs in
// the reference's order whatever kG is.
template <int kG, bool kShear, bool kFast>
__device__ __forceinline__ PlainAcc plain_sums(const StepConsts& c, const PlainArgs& a, int i, bool valid, int lane,
                                               double* buf) {
  constexpr int kComp = kShear ? 10 : 9;
  const d4 pi = load_d4(a.rec0 + (size_t)i * 4);
  const d4 vi = load_d4(a.rec1 + (size_t)i * 4);
  const double pr2_i = a.pr2[i];
  PlainAcc q;
  const uint32_t cnt = valid ? a.nbr_count[i] : 0u;
  const bool listed = cnt <= (uint32_t)kMaxNeighbors;
  const uint32_t* lst = a.nbr + i;
  if (kG == 1) {
    if (listed) {
      // Two entries ahead the index is loaded, one ahead the operands.
      uint32_t j = cnt > 1 ? lst[a.stride] : 0u;
      Neighbour nb{};
      if (cnt) nb = load_neighbour(a, lst[0]);
#pragma unroll 2
      for (uint32_t k = 0; k < cnt; ++k) {
        const Neighbour b = nb;
        if (k + 1 < cnt) nb = load_neighbour(a, j);
        if (k + 2 < cnt) j = lst[(size_t)(k + 2) * a.stride];
        PairTerms t;
        if (plain_pair<kShear, kFast>(c, b, pi.x, pi.y, pi.z, vi.x, vi.y, vi.z, pi.w, pr2_i, t))
          add_terms<kShear>(q, t);
      }
    }
  } else {
    const int s = lane % kG, g = lane / kG;
    constexpr int kMine = (kComp + kG - 1) / kG;  // components this lane sums
    double sum[kMine];
#pragma unroll
    for (int u = 0; u < kMine; ++u) sum[u] = 0.0;
    const uint32_t rounds = __reduce_max_sync(0xffffffffu, listed ? (cnt + kG - 1) / kG : 0u);
    uint32_t k = (uint32_t)s;
    uint32_t j = listed && k < cnt ? lst[(size_t)k * a.stride] : 0u;
    for (uint32_t r = 0; r < rounds; ++r) {
      const bool on = listed && k < cnt;
      const uint32_t jc = j;
      k += kG;
      if (listed && k < cnt) j = lst[(size_t)k * a.stride];
      PairTerms t{};
      if (on) {
        PairTerms f;
        if (plain_pair<kShear, kFast>(c, load_neighbour(a, jc), pi.x, pi.y, pi.z, vi.x, vi.y, vi.z, pi.w, pr2_i, f)) t = f;
      }
      // A skipped neighbour adds +0, which changes no sum (none is ever -0).
      const double v[10] = {t.fpx, t.fpy, t.fpz, t.fvx, t.fvy, t.fvz, t.xsx, t.xsy, t.xsz, t.shear};
#pragma unroll
      for (int u = 0; u < kComp; ++u) buf[u * 32 + lane] = v[u];
      __syncwarp();
#pragma unroll
      for (int u = 0; u < kMine; ++u) {
        const int comp = u * kG + s;
        if (comp < kComp) {
          const double2* src = reinterpret_cast<const double2*>(buf + comp * 32 + g * kG);
#pragma unroll
          for (int p = 0; p < kG / 2; ++p) {
            const double2 d = src[p];
            sum[u] = __dadd_rn(sum[u], d.x);
            sum[u] = __dadd_rn(sum[u], d.y);
          }
        }
      }
      __syncwarp();
    }
    // Component comp of the group sits in lane comp % kG.
    double all[10];
#pragma unroll
    for (int comp = 0; comp < kComp; ++comp)
      all[comp] = __shfl_sync(0xffffffffu, sum[comp / kG], (lane / kG) * kG + comp % kG);
    q.fpx = all[0];
    q.fpy = all[1];
    q.fpz = all[2];
    q.fvx = all[3];
    q.fvy = all[4];
    q.fvz = all[5];
    q.xsx = all[6];
    q.xsy = all[7];
    q.xsz = all[8];
    if (kShear) q.shear = all[9];
  }
  if (valid && !listed && (kG == 1 || lane % kG == 0)) {
    // List overflow: rescan the 27 cells (interior: a count needs a search).
    const long long kx = key_axis(pi.x, c.inv_cell);
    const long long ky = key_axis(pi.y, c.inv_cell);
    const long long kz = key_axis(pi.z, c.inv_cell);
    const int base = cell_linear(c, kx - 1, ky - 1, kz - 1);
    for (int di = 0; di < 3; ++di) {
      for (int dj = 0; dj < 3; ++dj) {
        const int c0 = base + (di * c.ncy + dj) * c.ncz;
        const int s0 = (int)a.cell_start[c0], e0 = (int)a.cell_start[c0 + 3];
        for (int j = s0; j < e0; ++j) {
          PairTerms t;
          if (j != i &&
              plain_pair<kShear, kFast>(c, load_neighbour(a, (uint32_t)j), pi.x, pi.y, pi.z, vi.x, vi.y, vi.z, pi.w, pr2_i, t))
            add_terms<kShear>(q, t);
        }
      }
    }
  }
  return q;
}

// compute_forces (world.rs:252-347) fused with integrate (352-363) and
// enforce_bounds (366-397).  The neighbours come from the density pass's list
// (same visit order); a particle whose list overflowed rescans its 27 cells.
template <int kG, bool kShear>
__global__ void __launch_bounds__(kThreads, kForceCtas) k_force_plain(StepConsts c, PlainArgs a) {
  after_previous();
  __shared__ __align__(16) double s_buf[kG == 1 ? 1 : kThreads / 32][kG == 1 ? 1 : (kShear ? 10 : 9) * 32];
  const int lane = threadIdx.x & 31;
  const int i = (blockIdx.x * kThreads + (int)threadIdx.x) / kG;
  const bool valid = i < c.n;
  if (kG == 1 && !valid) return;
  const int ii = valid ? i : c.n - 1;
  double* buf = s_buf[kG == 1 ? 0 : threadIdx.x >> 5];
  const uint2 flags = *reinterpret_cast<const uint2*>(a.flags);  // uniform
  if (flags.x & kFlagSortLost) return;
  const bool fast = flags.y == 0u && c.h < 1e100;
  const PlainAcc q = fast ? plain_sums<kG, kShear, true>(c, a, ii, valid, lane, buf)
                          : plain_sums<kG, kShear, false>(c, a, ii, valid, lane, buf);
  if (valid && (kG == 1 || lane % kG == 0)) finish_plain(c, a, i, q);
}

// Particles below which the force pass gives each particle four lanes.
constexpr int kLanesBelow = 16384;

// Squared radius of the density pass's f32 filter: the cutoff h widened by
// the rounding of the box-relative f32 coordinates (2^-24 of the box's extent
// each, two per axis and three axes: below extent 2^-21) and of the f32
// distance.  Extents or cutoffs whose squares leave f32's normal range pass
// every candidate.
static float plain_cull2(const StepConsts& c) {
  const double extent = (double)std::max(c.ncx, std::max(c.ncy, c.ncz)) * c.h0;
  const double r = c.h * (1.0 + 0x1p-18) + extent * 0x1p-21;
  const double r2 = r * r * (1.0 + 0x1p-20);
  if (!(r2 > 1e-30 && r2 < 1e30 && c.h > 0.0)) return std::numeric_limits<float>::quiet_NaN();
  return std::nextafter((float)r2, std::numeric_limits<float>::infinity());
}

}  // namespace

void launch_plain_passes(const StepConsts& c, DevBuffers& b, cudaStream_t s, const PassEvents& ev) {
  const ParticleConsts& pc = b.pc[b.cur];
  PlainArgs a;
  a.fpos = reinterpret_cast<const float4*>(b.rec + (size_t)kPlainRec * b.capacity);
  a.sorted_cell = b.sorted_cell;
  a.cand = reinterpret_cast<uint32_t*>(b.stage);
  a.hits = b.nbr + (size_t)(kMaxNeighbors - kSearchWords) * b.capacity;
  a.group = reinterpret_cast<uint2*>(b.rec + plain_group_offset(b.capacity));
  a.rec0 = b.rec;
  a.rec1 = b.rec + 4 * (size_t)b.capacity;
  a.rec2 = reinterpret_cast<double2*>(b.rec + 8 * (size_t)b.capacity);
  a.cull2 = plain_cull2(c);
  a.before = b.pc[b.cur ^ 1];
  a.now = pc;
  a.px = b.pv0[0];
  a.py = b.pv0[1];
  a.pz = b.pv0[2];
  a.vx = b.pv0[3];
  a.vy = b.pv0[4];
  a.vz = b.pv0[5];
  a.mass = pc.mass;
  a.mat = pc.mat;
  a.cell_start = b.cell_start;
  a.bax = b.has_ba ? pc.ba[0] : nullptr;
  a.bay = b.has_ba ? pc.ba[1] : nullptr;
  a.baz = b.has_ba ? pc.ba[2] : nullptr;
  a.rho = b.rho;
  a.p = b.p;
  a.pr2 = b.pr2;
  a.mr = b.mr;
  for (int k = 0; k < 3; ++k) {
    a.acc[k] = b.acc[k];
    a.xsph[k] = b.xsph[k];
  }
  a.mu = b.mu;
  for (int k = 0; k < 6; ++k) a.out_pv[k] = b.pv1[k];
  a.nbr = b.nbr;
  a.nbr_count = b.nbr_count;
  a.stride = b.capacity;
  a.flags = b.flags;
  a.counters = b.counters;
  for (int k = 0; k < 3; ++k) a.fv_out[k] = b.tape_fv[k];
  a.shear_out = b.tape_shear;
  if (ev.after_prep) cudaEventRecord(ev.after_prep, s);
  const int groups = (c.n + 31) / 32;
  // Few groups spread over the SMs one warp each before they share one.
  const int spread = std::max(1, groups / kSms);
  const bool overlap = c.n < kOverlapBelow;
  const int sw = std::min(kSearchWarps, spread), dw = std::min(kDensityWarps, spread);
  launch_after(overlap, k_search_plain, (groups + sw - 1) / sw, sw * 32, sw * sizeof(SegmentStage), s, c, a);
  const bool same = c.h <= c.h0;
  auto density = a.counters ? (same ? k_density_plain<true, true> : k_density_plain<true, false>)
                            : (same ? k_density_plain<false, true> : k_density_plain<false, false>);
  launch_after(overlap, density, (groups + dw - 1) / dw, dw * 32, dw * sizeof(DensityStage), s, c, a);
  if (ev.after_density) cudaEventRecord(ev.after_density, s);
  const int lanes = c.n < kLanesBelow ? 4 : 1;
  auto force = lanes == 4 ? (c.shear_live ? k_force_plain<4, true> : k_force_plain<4, false>)
                          : (c.shear_live ? k_force_plain<1, true> : k_force_plain<1, false>);
  launch_after(overlap, force, (int)(((long long)c.n * lanes + kThreads - 1) / kThreads), kThreads, 0, s, c, a);
}

}  // namespace phy
