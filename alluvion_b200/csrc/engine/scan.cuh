// scan.cuh -- the distance tests of the candidate scans (neighbor build,
// sampling): which of up to 32 consecutive sorted slots lie closer than h.
#pragma once

#include "common.cuh"

namespace alb {

// Spare entries after the n sorted positions that the scans read: they load
// candidates in rounds of up to 8 and may read past a row's last candidate
// (the extra bits are masked off), so every sorted-position buffer passed to
// them holds n + kSortedPad entries.
constexpr uint32_t kSortedPad = 8;

// Sorted positions once more, as three arrays of `ld` entries (x, y, z;
// 16-byte aligned, kSortedPad spare entries each); null where no scan reads
// them (double, periodic y).
template <class TF>
struct ScanSoa {
  TF* p = nullptr;
  size_t ld = 0;
  __device__ __forceinline__ void put(uint32_t s, vec3<TF> x) const {
    if (!p) return;
    p[s] = x.x;
    p[ld + s] = x.y;
    p[2 * ld + s] = x.z;
  }
};
inline size_t scan_soa_ld(size_t n) { return (n + kSortedPad + 3) / 4 * 4; }

namespace {

// Candidates tested per round (loads issued together; measured on B200 for
// the scalar tests, per build at 8,388,608 / 1,048,576 particles: 2.79 / 0.354
// ms at 8, 2.84 / 0.358 at 4, 2.89 / 0.370 at 2, and 3.18 / 0.381 for a
// branch per candidate).
constexpr uint32_t kScan = 8;
static_assert(32 % kScan == 0 && kScan <= kSortedPad,
              "scan rounds must tile 32 and stay in the pad");
// Packed scans (float, not periodic) start at multiples of four slots, for their
// 16-byte loads; the scalar ones at the row's first slot, because the slots
// before it cost them up to a round of eight per row (1,331,000 particles in
// double, neighbor update without rows: 829 us aligned, 692 us so).
template <class TF, bool WR>
constexpr bool packed_scan() {
  return sizeof(TF) == 4 && !WR;
}
template <class TF, bool WR>
__device__ __forceinline__ uint32_t scan_start(uint32_t b) {
  return packed_scan<TF, WR>() ? b / 4 * 4 : b;
}

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Bit 31 - k of the result: candidate t0 + k (k < m <= 32, t0 a multiple of four
// in packed scans) is closer than h to xi, by the rounded operations of pdist2.
// The other bits are 0.
//
// The scans are bound by instruction issue (ncu).  In float, two candidates
// share each packed operation and eight share six 16-byte loads; the sign of
// |d|^2 - h^2 (exact: the subtraction underflows gradually) is the accept
// bit and enters the mask by one funnel shift: about 7 instructions per
// candidate instead of 12.  Build at 8,388,608 / 1,048,576 particles:
// 2,457 / 325 us with the scalar tests, 2,034 / 275 us now (B200).
template <bool WR, class TF>
__device__ __forceinline__ uint32_t accept_bits(const Cn<TF>& c, vec3<TF> xi,
                                                const vec4<TF>* __restrict__ xs,
                                                const ScanSoa<TF>& soa, uint32_t t0, uint32_t m) {
  uint32_t acc = 0;
  if constexpr (packed_scan<TF, WR>()) {
    const unsigned long long nx = pack2(-xi.x, -xi.x), ny = pack2(-xi.y, -xi.y),
                             nz = pack2(-xi.z, -xi.z);
    const float* px = soa.p + t0;
    for (uint32_t q = 0; q < m; q += kScan) {
      ulonglong2 x[2], y[2], z[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        x[u] = __ldg(reinterpret_cast<const ulonglong2*>(px + q + 4 * u));
        y[u] = __ldg(reinterpret_cast<const ulonglong2*>(px + soa.ld + q + 4 * u));
        z[u] = __ldg(reinterpret_cast<const ulonglong2*>(px + 2 * soa.ld + q + 4 * u));
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const unsigned long long dx = add2(u & 1 ? x[u / 2].y : x[u / 2].x, nx),
                                 dy = add2(u & 1 ? y[u / 2].y : y[u / 2].x, ny),
                                 dz = add2(u & 1 ? z[u / 2].y : z[u / 2].x, nz);
        // The sums by scalar additions: nvcc 12.9 contracts a packed product
        // and a packed sum although both say .rn, which moved single
        // candidates across h.  A scalar __fadd_rn is never contracted by its
        // definition; that it holds for a packed product as well rests on the
        // exact list tests (test_config2_neighbor_lists_bit_exact and
        // test_lists_at_group_and_round_edges): run them with a new toolkit.
        const float2 sx = unpack2(mul2(dx, dx)), sy = unpack2(mul2(dy, dy)),
                     sz = unpack2(mul2(dz, dz));
        const float ea = __fsub_rn(__fadd_rn(__fadd_rn(sx.x, sy.x), sz.x), c.h2);
        const float eb = __fsub_rn(__fadd_rn(__fadd_rn(sx.y, sy.y), sz.y), c.h2);
        acc = __funnelshift_l(__float_as_uint(ea), acc, 1);
        acc = __funnelshift_l(__float_as_uint(eb), acc, 1);
      }
    }
    acc <<= 32u - (m + kScan - 1) / kScan * kScan;
  } else {
    for (uint32_t q = 0; q < m; q += kScan) {
      vec3<TF> xj[kScan];
#pragma unroll
      for (uint32_t u = 0; u < kScan; ++u) xj[u] = xyz(__ldg(xs + t0 + q + u));
      uint32_t bits = 0;
#pragma unroll
      for (uint32_t u = 0; u < kScan; ++u) bits |= uint32_t(pdist2(c, xi, xj[u]) < c.h2) << u;
      acc |= bits << q;
    }
    acc = __brev(acc);
  }
  return m < 32 ? acc & ~(0xffffffffu >> m) : acc;
}

// accept_bits of the part of row [b, e) in the chunk of 32 slots at t0
// (t0 <= b in the first chunk only).
template <bool WR, class TF>
__device__ __forceinline__ uint32_t row_bits(const Cn<TF>& c, vec3<TF> xi,
                                             const vec4<TF>* __restrict__ xs,
                                             const ScanSoa<TF>& soa, uint32_t t0, uint32_t b,
                                             uint32_t e) {
  const uint32_t acc = accept_bits<WR>(c, xi, xs, soa, t0, min(e - t0, 32u));
  return t0 < b ? acc & (0xffffffffu >> (b - t0)) : acc;
}

}  // namespace

}  // namespace alb
