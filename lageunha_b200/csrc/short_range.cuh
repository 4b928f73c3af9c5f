// The short-range pair law of the tree walk (tree.cu) and the cube geometry it
// shares with the search for groups (fof.cu).
#pragma once
#include <string.h>

#include "engine_internal.cuh"

namespace tpm {

TPM_D float wrapf(uint32_t a, uint32_t b, float cpu) { return (float)(int32_t)(a - b) * cpu; }

constexpr int kLogSmemF4 = (kLogEntries + 2) / 2;  // the log-spaced table, in float4s

// The law at s = r^2 + kLogR2Floor (cells^2) from the table indexed by the
// float bits of s: the exponent and the top kLogMantissa mantissa bits pick
// the bin, whose line in s gives the value, so neither a square root nor a
// conversion is needed, and s >= 2^-20 needs no lower clamp. tlb is the
// table's shared address with the base entry kLogBase folded in (s >= 2^-20
// keeps the entry >= 0; the clamp keeps it in range).
TPM_D float law_at(float s, uint32_t tlb) {
  uint32_t kk = min(__float_as_uint(s) >> kLogShift, (uint32_t)(kLogBase + kLogEntries));
  float2 c;
  asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(c.x), "=f"(c.y) : "r"(tlb + (kk << 3)));
  return fmaf(c.y, s, c.x);
}

// The law at s with every pair beyond the cut reading one shared entry: the
// bin index is clamped at kcut (the first bin from which the Gaussian law's
// table is zero; for the reference law the bin of rsphere^2, whose value the
// per-pair test then discards), so the lanes with such pairs all load one
// address, a broadcast, and the warp's gather spreads over the banks of the
// pairs inside the cut only. Same value as law_at with the cut applied.
TPM_D float law_clamped(float s, uint32_t tlb, uint32_t kcut) {
  uint32_t kk = min(__float_as_uint(s) >> kLogShift, kcut);
  float2 c;
  asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(c.x), "=f"(c.y) : "r"(tlb + (kk << 3)));
  return fmaf(c.y, s, c.x);
}

// One source against this lane's target: the reference's AddPar
// (OST/ost.ver2.c:279-293) without the mass factor. The source comes negated
// (nsx = -x), so dx = tx + nsx is the IEEE difference tx - x. The target
// itself (r = 0) lands in bin 0 with a zero separation, adding nothing.
// kHardCut: the per-pair cut of the reference law, tested as s <= rsphere^2
// (a cut 2^-20 cells^2 inside r^2 <= rsphere^2); the Gaussian law's table is
// zero from the cut on and needs no test.
template <bool kHardCut>
TPM_D void pp_one(float nsx, float nsy, float nsz, float tx, float ty, float tz, float rs2, uint32_t kcut,
                  uint32_t tlb, float &ax, float &ay, float &az) {
  float dx = tx + nsx, dy = ty + nsy, dz = tz + nsz;
  float r2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, kLogR2Floor)));
  float f = law_clamped(r2, tlb, kcut);
  if (kHardCut) f = r2 <= rs2 ? f : 0.f;
  ax = fmaf(dx, f, ax);
  ay = fmaf(dy, f, ay);
  az = fmaf(dz, f, az);
}

// Two sources against this lane's target, the separations, r^2 and the
// accumulation as packed fp32x2 operations (sm_100 add/fma on register
// pairs): each half is the IEEE fp32 operation pp_one does, in the same
// order, so the sums are the same bits as two pp_one calls into the halves.
template <bool kHardCut>
TPM_D void pp_two(float2 nsx, float2 nsy, float2 nsz, float2 tx, float2 ty, float2 tz, float rs2, uint32_t kcut,
                  uint32_t tlb, float2 &ax, float2 &ay, float2 &az) {
  float2 dx = __fadd2_rn(tx, nsx), dy = __fadd2_rn(ty, nsy), dz = __fadd2_rn(tz, nsz);
  float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, make_float2(kLogR2Floor, kLogR2Floor))));
  float2 f = make_float2(law_clamped(r2.x, tlb, kcut), law_clamped(r2.y, tlb, kcut));
  if (kHardCut) {
    f.x = r2.x <= rs2 ? f.x : 0.f;
    f.y = r2.y <= rs2 ? f.y : 0.f;
  }
  ax = __ffma2_rn(dx, f, ax);
  ay = __ffma2_rn(dy, f, ay);
  az = __ffma2_rn(dz, f, az);
}

// The bin every pair beyond the cut reads: for the reference law the bin of
// rsphere^2 (the per-pair test discards its value), for the Gaussian law the
// first bin of the table's zero tail.
inline uint32_t law_cut_bin(const LawTable &law, float rs2) {
  if (!law.hard_cut) return law.cut_bits >> kLogShift;
  uint32_t b;
  memcpy(&b, &rs2, 4);
  return b >> kLogShift;
}

// The 4-cell cubes along one axis of an n-cell periodic box whose cells meet
// [lo, hi] (cells, unwrapped): run[0..1] = first cube and count of the first
// run, run[2..3] of the second (empty unless [lo, hi] wraps past n). Both
// runs together list each cube once; an interval of n cells or more lists
// every cube.
TPM_D void axis_runs(float lo, float hi, int n, int run[4]) {
  const int ncube = (n + 3) >> 2;
  const float fn = (float)n;
  run[0] = 0;
  run[1] = ncube;
  run[2] = 0;
  run[3] = 0;
  if (hi - lo >= fn) return;
  float lw = lo - fn * floorf(lo / fn);
  if (lw >= fn) lw = 0.f;
  if (lw < 0.f) lw = 0.f;
  float hw = lw + (hi - lo);
  int a = min((int)(lw * 0.25f), ncube - 1);
  if (hw < fn) {
    int b = min((int)(hw * 0.25f), ncube - 1);
    run[0] = a;
    run[1] = b - a + 1;
    return;
  }
  int b = min((int)((hw - fn) * 0.25f), ncube - 1);
  if (b >= a) return;  // the runs meet: every cube
  run[0] = a;
  run[1] = ncube - a;
  run[2] = 0;
  run[3] = b + 1;
}

}  // namespace tpm
