// The neighbour filter a warp shares between its queries: which of up to
// kBatch staged candidates may lie within a cutoff of each of 32 queries.
//
// What bounds the pair search is the number of instructions per tested pair:
// ~215 candidates per query at rest density, of which ~31 are in range.  The
// squared distances of 32 queries and 32 candidates are a small contraction,
// |q|^2 + |c|^2 - 2 q.c, so the tensor cores form them: one mma.sync (16
// queries x 8 candidates, TF32 operands, f32 sums) replaces 128 separate
// distance computations, and a lane only shifts the results' signs together
// (tcgen05 tiles of 128 rows would need all queries of a CTA to share their
// candidates).  TF32 rounds the operands to 11 bits, so the radius is widened
// by a bound of that error, computed per segment from its extent (about 1.6%
// of r^2 for a segment of 4 cells): every candidate in range passes, a few
// outside do too, and the caller tests the survivors exactly.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace phy {

// max(a, b) that keeps a NaN operand.
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// Order-preserving map of f32 to u32 and back (NaN bounds come out as NaN).
__device__ __forceinline__ uint32_t ord_bits(float x) {
  const uint32_t b = __float_as_uint(x);
  return b ^ ((uint32_t)((int32_t)b >> 31) | 0x80000000u);
}
__device__ __forceinline__ float ord_float(uint32_t u) {
  return __uint_as_float(u ^ (((u >> 31) - 1u) | 0x80000000u));
}

constexpr int kBatch = 256;              // staged candidates
constexpr int kBatchWords = kBatch / 32;

// One warp's staging.  Bit k of hits[w][q]: candidate 32 w + k may be in
// range of query q.  The operand array is laid out so that a lane's four
// column operands of a 32-candidate word are one 16-byte load and the four
// result bytes of a word land where the bit order needs them: candidate k of
// a word is column 2 (k >> 3) + (k & 1) of tile (k >> 1) & 3.
struct SegmentStage {
  float b[kBatchWords][4][8][4];  // [word][x, y, z, |c|^2][column][tile]
  uint32_t hits[kBatchWords][32];
};

struct Segment {
  float ctr[3], half[3];  // bounding box of the queries: centre and half extents
  float box2;             // squared reach of the box test
  uint32_t a[2][4];       // row operands (two tiles of 16 queries)
  bool all;               // no finite filter: every candidate passes
};

// Round to TF32 (to nearest in magnitude; the hardware drops the low bits).
__device__ __forceinline__ uint32_t tf32(float x) { return __float_as_uint(x) + 0x1000u; }

// The segment of the queries (x, y, z) of the lanes with `mine` set, within a
// squared radius cull2 of f32 distances (NaN: everything passes).
__device__ __forceinline__ Segment make_segment(bool mine, float x, float y, float z, float cull2) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  Segment s;
  const float p[3] = {x, y, z};
  float reach = sqrtf(cull2) * 1.0001f, qr[3], most = 0.f, cross = 0.f, far2 = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint32_t u = ord_bits(p[k]);
    const float lo = ord_float(__reduce_min_sync(0xffffffffu, mine ? u : 0xffffffffu));
    const float hi = ord_float(__reduce_max_sync(0xffffffffu, mine ? u : 0u));
    s.ctr[k] = 0.5f * lo + 0.5f * hi;
    s.half[k] = max_nan(hi - s.ctr[k], s.ctr[k] - lo) * 1.000001f;
    qr[k] = p[k] - s.ctr[k];
    most = max_nan(most, s.half[k]);
    cross += s.half[k] * (s.half[k] + reach);
    far2 += (s.half[k] + reach) * (s.half[k] + reach);
  }
  const float wide = reach + most * 0x1p-20f;
  s.box2 = wide * wide * 1.0001f;
  // TF32 operands: 2^-11 of each factor of 2 q.c and of |c|^2; f32 sums.
  const float margin = 0x1.1p-9f * cross + 0x1.1p-11f * far2 + 0x1p-17f * far2;
  const float q2 = qr[0] * qr[0] + qr[1] * qr[1] + qr[2] * qr[2];
  const float v = q2 - (cull2 + margin);
  s.all = !(fabsf(far2) < 1e30f && cull2 > 1e-30f);
  const float vhi = __uint_as_float(tf32(v) & 0xffffe000u);
  const uint32_t vlo = tf32(v - vhi);
  const uint32_t one = __float_as_uint(1.0f);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int src = 8 * r + g;
    const float rx = __shfl_sync(0xffffffffu, qr[0], src), ry = __shfl_sync(0xffffffffu, qr[1], src),
                rz = __shfl_sync(0xffffffffu, qr[2], src);
    const uint32_t h = __shfl_sync(0xffffffffu, __float_as_uint(vhi), src), l = __shfl_sync(0xffffffffu, vlo, src);
    s.a[r >> 1][r & 1] = t == 3 ? one : tf32(-2.0f * (t == 0 ? rx : t == 1 ? ry : rz));
    s.a[r >> 1][2 + (r & 1)] = t == 0 ? h : t == 1 ? l : 0u;
  }
  return s;
}

// Whether a candidate (centred coordinates) may be in reach of some query.
__device__ __forceinline__ bool near_segment(const Segment& s, float cx, float cy, float cz) {
  const float gx = max_nan(fabsf(cx) - s.half[0], 0.f);
  const float gy = max_nan(fabsf(cy) - s.half[1], 0.f);
  const float gz = max_nan(fabsf(cz) - s.half[2], 0.f);
  return !(fmaf(gz, gz, fmaf(gy, gy, gx * gx)) >= s.box2);
}

__device__ __forceinline__ void stage_candidate(SegmentStage& st, uint32_t k, float cx, float cy, float cz) {
  const uint32_t u = k & 31u;
  float* b = &st.b[k >> 5][0][2 * (u >> 3) + (u & 1u)][(u >> 1) & 3u];
  b[0] = __uint_as_float(tf32(cx));
  b[32] = __uint_as_float(tf32(cy));
  b[64] = __uint_as_float(tf32(cz));
  b[96] = __uint_as_float(tf32(fmaf(cz, cz, fmaf(cy, cy, cx * cx))));
}

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}

// Fills hits[w][q] for the m staged candidates (all lanes; candidates and
// hits are exchanged through the warp's shared memory).
__device__ __forceinline__ void filter_batch(SegmentStage& st, uint32_t m, const Segment& s) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t b1 = t < 2 ? __float_as_uint(1.0f) : 0u;
  uint8_t* out = reinterpret_cast<uint8_t*>(st.hits) + lane;  // byte t of query g's word
  __syncwarp();
#pragma unroll 2
  for (uint32_t w = 0; 32u * w < m; ++w) {
    const float4 b = *reinterpret_cast<const float4*>(&st.b[w][t][g][0]);
    const uint32_t col[4] = {__float_as_uint(b.x), __float_as_uint(b.y), __float_as_uint(b.z), __float_as_uint(b.w)};
    uint32_t acc[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int tile = 3; tile >= 0; --tile) {
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        float d[4];
        mma_tf32(d, s.a[mt], col[tile], b1);
        acc[2 * mt] = __funnelshift_l(__float_as_uint(d[1]), acc[2 * mt], 1);
        acc[2 * mt] = __funnelshift_l(__float_as_uint(d[0]), acc[2 * mt], 1);
        acc[2 * mt + 1] = __funnelshift_l(__float_as_uint(d[3]), acc[2 * mt + 1], 1);
        acc[2 * mt + 1] = __funnelshift_l(__float_as_uint(d[2]), acc[2 * mt + 1], 1);
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) out[128 * w + 32 * r] = (uint8_t)(s.all ? 0xffu : acc[r]);
  }
  // Slots past the batch hold stale candidates.
  __syncwarp();
  if (m & 31u) st.hits[m >> 5][lane] &= (1u << (m & 31u)) - 1u;
}

}  // namespace phy
