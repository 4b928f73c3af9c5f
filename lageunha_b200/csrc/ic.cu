// Zel'dovich initial conditions (sm_100a).
//
// Reference: PMSeedForce (Cosmos/CosmosIC/PMSeedForce.c:293-399) draws, mode
// by mode over the half-complex mesh (z outer, y, kx inner), two Gaussian
// deviates per mode inside the Nyquist sphere from Numerical Recipes' gasdev
// on ran3 (Cosmos/CosmosIC/nr.c:317-384), scaled by the amplitude
// pamp*bpower(rk)/rk^2, and completes the kx = 0 plane by complex conjugates.
// Zeldovich (Cosmos/CosmosIC/Zeldovich.c:14-100) takes that spectrum back to
// real space, adds the local non-Gaussian terms fNL, gNL, returns to k space
// and forms the displacement field psi = FFT^-1[i 2 pi k phi_k] / N^3.
// Set_Particle_Zeld (MakeParticle.c:149-212, with Zeld_GetVR of
// cosmosic.h:202) makes one particle per lattice point with velocity
// vamp * (vamp * psi) and, with positions stored as offsets (XYZDBL,
// cosmosic.h:272-301), offset pfact * velocity.
//
// ran3 is the subtractive generator x_t = x_{t-55} - x_{t-24} mod 10^9 and
// gasdev the polar Box-Muller method, whose rejections make the count of
// ran3 values per mode irregular. Here the stream is cut into chunks of
// kTrialsPerChunk Box-Muller trials; the state at each chunk start comes
// from powers of x modulo the recurrence's polynomial x^55 + x^31 - 1 (mod
// 10^9), so every chunk is generated by its own thread. A first pass counts
// each chunk's accepted trials, a scan gives their ranks, a second pass writes
// the accepted pairs in stream order. A mode's rank among the drawing modes
// follows from per-row counts (the drawing modes of a row are a prefix in
// kx) and a scan over the rows; mode m takes accepted pair m. The float
// arithmetic of ran3, gasdev and the scaling follows the reference's C
// expressions operation by operation.
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>

#include "tpm_engine.h"
#include "engine_internal.cuh"

using namespace tpm;

namespace {

constexpr uint64_t kMBig = 1000000000ull;
constexpr int64_t kMSeed = 161803398;
constexpr int kLag = 55;
constexpr int kRounds = 2;                     // rounds of 2 x 55 ran3 values per generator thread
constexpr int kChunkLen = 2 * kLag * kRounds;  // ran3 values per chunk, two per Box-Muller trial
constexpr int kTrialsPerChunk = kChunkLen / 2;
constexpr int kRadix = 32;                     // chunk starts per start of the level above
constexpr int kLevels = 4;                     // levels of chunk starts, kRadix apart

#define IC_CK(x)                                                                         \
  do {                                                                                   \
    cudaError_t e_ = (x);                                                                \
    if (e_ != cudaSuccess) {                                                             \
      snprintf(msg, sizeof(msg), "%s: %s", #x, cudaGetErrorString(e_));                  \
      rc = TPM_E_CUDA;                                                                   \
      goto done;                                                                         \
    }                                                                                    \
  } while (0)

// ran3's state after its initialisation (nr.c:325-345), as the history
// x_{-54..0}: x_{t} sits in slot t + 54, so x_1 = x_{-54} - x_{-23}.
__global__ void k_ran3_init(int64_t idum, uint32_t *state) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  int64_t ma[56];
  int64_t mj = kMSeed - (idum < 0 ? -idum : idum);
  mj %= (int64_t)kMBig;
  ma[55] = mj;
  int64_t mk = 1;
  for (int i = 1; i <= 54; i++) {
    int ii = (21 * i) % 55;
    ma[ii] = mk;
    mk = mj - mk;
    if (mk < 0) mk += (int64_t)kMBig;
    mj = ma[ii];
  }
  for (int k = 1; k <= 4; k++)
    for (int i = 1; i <= 55; i++) {
      ma[i] -= ma[1 + (i + 30) % 55];
      if (ma[i] < 0) ma[i] += (int64_t)kMBig;
    }
  for (int s = 1; s <= 55; s++) state[s - 1] = (uint32_t)ma[s];
}

// Sum of 55 products a_k b_(k stride) mod 10^9, a and b below 10^9: sixteen
// products fit 64 bits beside a reduced remainder.
__device__ __forceinline__ uint32_t dot_mod(const uint32_t *a, const uint32_t *b) {
  uint64_t acc = 0;
#pragma unroll
  for (int k = 0; k < kLag; k++) {
    acc += (uint64_t)a[k] * b[k];
    if (k % 16 == 15) acc %= kMBig;
  }
  return (uint32_t)(acc % kMBig);
}

// c <- c^2 (or c x with `times_x`) modulo p(x) = x^55 + x^31 - 1 and 10^9, by
// one block of at least 128 threads; w is scratch of 2 * 55 words.
__device__ void poly_step(uint32_t *c, uint32_t *w, bool times_x) {
  const int t = threadIdx.x;
  if (times_x) {
    // x^55 = 1 - x^31
    uint32_t lead = c[kLag - 1], v = 0;
    if (t < kLag) {
      v = t == 0 ? lead : c[t - 1];
      if (t == 31) v = v >= lead ? v - lead : v + (uint32_t)kMBig - lead;
    }
    __syncthreads();
    if (t < kLag) c[t] = v;
    __syncthreads();
    return;
  }
  if (t < 2 * kLag - 1) {
    const int lo = t < kLag ? 0 : t - (kLag - 1), hi = t < kLag ? t : kLag - 1;
    uint64_t acc = 0;
    for (int k = lo; k <= hi; k++) {
      acc += (uint64_t)c[k] * c[t - k];
      if ((k & 15) == 15) acc %= kMBig;
    }
    w[t] = (uint32_t)(acc % kMBig);
  }
  __syncthreads();
  // x^(55 + i) = x^i - x^(31 + i): degrees 79..108 fold into 24..53 and
  // 55..84, then 55..84 into 0..29 and 31..60, then 55..60
  const int top[3] = {2 * kLag - 2, 84, 60}, bottom[3] = {79, 61, 55};
  for (int r = 0; r < 3; r++) {
    uint32_t v = 0;
    const int d = bottom[r] + t;
    const bool on = d <= top[r];
    if (on) {
      v = w[d];
      w[d] = 0u;
    }
    __syncthreads();
    if (on) {
      uint32_t a = w[d - 55] + v;
      w[d - 55] = a >= (uint32_t)kMBig ? a - (uint32_t)kMBig : a;
    }
    __syncthreads();
    if (on) {
      uint32_t a = w[d - 24];
      w[d - 24] = a >= v ? a - v : a + (uint32_t)kMBig - v;
    }
    __syncthreads();
  }
  if (t < kLag) c[t] = w[t];
  __syncthreads();
}

// jump[l] = x^(kChunkLen kRadix^l) modulo p, l < kLevels: the state kChunkLen
// kRadix^l values on is each x_t = sum_k jump[l][k] x_(t' + k).
__global__ void __launch_bounds__(128) k_ran3_jumps(uint32_t *jump) {
  __shared__ uint32_t c[kLag], w[2 * kLag];
  const int t = threadIdx.x;
  if (t < kLag) c[t] = t == 0 ? 1u : 0u;
  __syncthreads();
  for (int bit = 30; bit >= 0; bit--) {
    if ((kChunkLen >> (bit + 1)) != 0) poly_step(c, w, false);
    if ((kChunkLen >> bit) & 1) poly_step(c, w, true);
  }
  for (int l = 0; l < kLevels; l++) {
    if (t < kLag) jump[l * kLag + t] = c[t];
    for (int r = 1; r < kRadix; r <<= 1) poly_step(c, w, false);
  }
}

// The states of one level from those of the level above: block j fills the
// states kRadix * j + i, i < kRadix (and below `count`), by repeated jumps from
// state j of `above`. The top level has one block that fills them all.
__global__ void __launch_bounds__(64) k_ran3_level(const uint32_t *above, const uint32_t *jump, int64_t count,
                                                   int per_block, uint32_t *out) {
  __shared__ uint32_t x[2 * kLag], c[kLag];
  const int t = threadIdx.x;
  const int64_t j = blockIdx.x;
  if (t < kLag) {
    x[t] = above[j * kLag + t];
    c[t] = jump[t];
  }
  __syncthreads();
  for (int i = 0; i < per_block; i++) {
    const int64_t s = j * per_block + i;
    if (s >= count) break;
    if (t < kLag) out[s * kLag + t] = x[t];
    if (i + 1 == per_block || s + 1 == count) break;
    // the next 54 values, 24 at a time (x_(t+55) = x_t - x_(t+31))
    for (int b = 0; b < kLag - 1; b += 24) {
      if (t < 24 && b + t < kLag - 1) {
        uint32_t p = x[b + t], q = x[b + t + 31];
        x[b + t + kLag] = p >= q ? p - q : p + (uint32_t)kMBig - q;
      }
      __syncthreads();
    }
    uint32_t v = 0;
    if (t < kLag) v = dot_mod(c, x + t);
    __syncthreads();
    if (t < kLag) x[t] = v;
    __syncthreads();
  }
}

// ran3's float: (float)(mj * (1.0 / MBIG)) (nr.c:351).
__device__ __forceinline__ float ran3_float(uint32_t mj) {
  return __double2float_rn(__dmul_rn((double)mj, 1.0 / (double)kMBig));
}

// One polar Box-Muller trial of gasdev (nr.c:361-384): the pair (v1, v2),
// accepted when 0 < v1^2 + v2^2 < 1.
__device__ __forceinline__ bool gasdev_trial(uint32_t m1, uint32_t m2, float2 &out) {
  float v1 = __double2float_rn(__dsub_rn(__dmul_rn(2.0, (double)ran3_float(m1)), 1.0));
  float v2 = __double2float_rn(__dsub_rn(__dmul_rn(2.0, (double)ran3_float(m2)), 1.0));
  float rsq = __fadd_rn(__fmul_rn(v1, v1), __fmul_rn(v2, v2));
  out = make_float2(v1, v2);
  return !(rsq >= 1.0f || rsq == 0.0f);
}

// The deviates of an accepted pair in the order gasdev returns them (v2*fac
// first, then the saved v1*fac).
__device__ __forceinline__ float2 gasdev_pair(float2 v) {
  float rsq = __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y));
  double d = (double)rsq;
  float fac = __double2float_rn(sqrt(__ddiv_rn(__dmul_rn(-2.0, log(d)), d)));
  return make_float2(__fmul_rn(v.y, fac), __fmul_rn(v.x, fac));
}

// Generator threads: chunk c runs kTrialsPerChunk trials from its start state.
// The first pass counts the accepted trials; the second writes their pairs at
// their rank (kept only below `need`); whoever reads a pair turns it into
// deviates. The lagged state stays in registers: a round of 110 values runs
// through the 55 of it twice with constant indices. Bound by the latency of
// one thread's chain, so a chunk is short (110 trials; with 1024 and the state
// indexed at run time the two passes took 977 us for the 256^3 noise).
template <bool kWrite>
__global__ void __launch_bounds__(64) k_ran3_trials(const uint32_t *starts, int64_t nchunks, uint32_t *counts,
                                                    const uint32_t *offs, const uint32_t *bsum, float2 *acc,
                                                    int64_t need) {
  int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= nchunks) return;
  uint32_t v[kLag];
#pragma unroll
  for (int i = 0; i < kLag; i++) v[i] = starts[c * kLag + i];
  uint32_t cnt = 0;
  const int64_t base = kWrite ? (int64_t)offs[c] + bsum[c / 4096] : 0;
  for (int r = 0; r < kRounds; r++) {
    uint32_t m1 = 0;
#pragma unroll
    for (int q = 0; q < 2 * kLag; q++) {
      const int i = q % kLag;
      const uint32_t a = v[i], b = v[(i + 31) % kLag];
      const uint32_t x = a >= b ? a - b : a + (uint32_t)kMBig - b;
      v[i] = x;
      if (q & 1) {
        float2 g;
        if (gasdev_trial(m1, x, g)) {
          if (kWrite && base + cnt < need) acc[base + cnt] = g;
          cnt++;
        }
      } else {
        m1 = x;
      }
    }
  }
  if (!kWrite) counts[c] = cnt;
}

__device__ __forceinline__ int wrap_freq(int j, int n) { return j > n / 2 ? j - n : j; }

// Largest i >= 0 with i^2 <= r (r >= 0).
__device__ __forceinline__ int isqrt_floor(int64_t r) {
  int64_t i = (int64_t)sqrt((double)r);
  while (i * i > r) i--;
  while ((i + 1) * (i + 1) <= r) i++;
  return (int)i;
}

// Drawing modes per (z, y) row: kx in [i0, imax] with 0 < k^2 <= (n/2)^2.
__global__ void k_row_counts(int n, uint32_t *cnt) {
  int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (row >= (int64_t)n * n) return;
  int j = (int)(row % n), k = (int)(row / n);
  int ky = wrap_freq(j, n), kz = wrap_freq(k, n);
  int64_t knyq = n / 2;
  int64_t r = knyq * knyq - (int64_t)ky * ky - (int64_t)kz * kz;
  uint32_t c = 0;
  if (r >= 0) {
    int imax = isqrt_floor(r);
    if (imax > n / 2) imax = n / 2;
    int i0 = (ky == 0 && kz == 0) ? 1 : 0;
    c = imax >= i0 ? (uint32_t)(imax - i0 + 1) : 0u;
  }
  cnt[row] = c;
}

// The noise spectrum [z][y][hx]: mode of rank m takes accepted pair m,
// scaled by the amplitude of its k^2 (unit amplitude without a table).
__global__ void k_fill_noise(int n, int hx, const uint32_t *rowoff, const uint32_t *bsum, const float2 *acc,
                             const float *velpot, float2 *spec) {
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    const int j = row % n, k = row / n;
    for (int i = threadIdx.x; i < hx; i += blockDim.x) {
      const int64_t e = (int64_t)row * hx + i;
      int ky = wrap_freq(j, n), kz = wrap_freq(k, n);
      int64_t knyq = n / 2;
      int64_t xksq = (int64_t)i * i + (int64_t)ky * ky + (int64_t)kz * kz;
      float2 v = make_float2(0.f, 0.f);
      if (xksq != 0 && xksq <= knyq * knyq) {
        int i0 = (ky == 0 && kz == 0) ? 1 : 0;
        int64_t rank = (int64_t)rowoff[row] + bsum[row / 4096] + (i - i0);
        float2 g = gasdev_pair(acc[rank]);
        if (velpot) {
          float a = velpot[xksq];
          v = make_float2(__fmul_rn(a, g.x), __fmul_rn(a, g.y));
        } else {
          v = g;
        }
      }
      spec[e] = v;
    }
  }
}

// The kx = 0 plane's conjugate completion (PMSeedForce.c:355-396): for
// 0 < k < n/2 the column (j, k), j != n/2, is copied conjugated to
// ((n - j) mod n, n - k); on k = 0 the columns 0 < j < n/2 go to (n - j, 0).
__global__ void k_conjugate_plane(int n, int hx, float2 *spec) {
  int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= (int64_t)n * n) return;
  int j = (int)(e % n), k = (int)(e / n);
  int dj = -1, dk = -1;
  if (k >= 1 && k < n / 2 && j != n / 2) {
    dj = (n - j) % n;
    dk = n - k;
  } else if (k == 0 && j >= 1 && j < n / 2) {
    dj = n - j;
    dk = 0;
  }
  if (dj < 0) return;
  float2 v = spec[((int64_t)k * n + j) * hx];
  spec[((int64_t)dk * n + dj) * hx] = make_float2(v.x, -v.y);
}

// phi = c2r * 1/N^3 (Zeldovich.c:36): float(float * double).
__device__ __forceinline__ float interior(const float *pad, const MeshGeom g, int x, int y, int z, double rincube) {
  float v = pad[(int64_t)(x + kGhost) + (int64_t)g.px * ((y + kGhost) + (int64_t)g.py * (z + kGhost))];
  return __double2float_rn(__dmul_rn((double)v, rincube));
}

// Sum and sum of squares of phi in FP64 (Zeldovich.c:41-56).
__global__ void k_phi_moments(const float *pad, MeshGeom g, double rincube, double *sums) {
  int n = g.n;
  double s1 = 0, s2 = 0;
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    for (int x = threadIdx.x; x < n; x += blockDim.x) {
      const int y = row % n, z = row / n;
      float f = interior(pad, g, x, y, z, rincube);
      s1 += (double)f;
      s2 += (double)__fmul_rn(f, f);  // the reference squares in float
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_down_sync(0xffffffffu, s1, o);
    s2 += __shfl_down_sync(0xffffffffu, s2, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&sums[0], s1);
    atomicAdd(&sums[1], s2);
  }
}

// phi += fNL (phi^2 - sigma^2) + gNL (phi^3 - 3 sigma^2 phi) (Zeldovich.c:57-61),
// in FP64 as the reference's mixed float/double expression evaluates it.
__global__ void k_phi_nongauss(const float *pad, MeshGeom g, double rincube, const double *sums, float fnl,
                               float gnl, float *real) {
  int n = g.n;
  double mean = sums[0] * rincube;
  double sd = sqrt(sums[1] * rincube - mean * mean);
  double s2 = sd * sd;
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    for (int x = threadIdx.x; x < n; x += blockDim.x) {
      const int64_t e = (int64_t)row * n + x;
      const int y = row % n, z = row / n;
      float d = interior(pad, g, x, y, z, rincube);
      float d2 = __fmul_rn(d, d);
      double t1 = __dmul_rn((double)fnl, __dsub_rn((double)d2, s2));
      double t2 = __dmul_rn((double)gnl, __dsub_rn((double)__fmul_rn(d2, d),
                                                   __dmul_rn(__dmul_rn(__dmul_rn(3.0, sd), sd), (double)d)));
      real[e] = __double2float_rn(__dadd_rn((double)d, __dadd_rn(t1, t2)));
    }
  }
}

// One displacement component's spectrum i 2 pi k_a phi_k for kx < n/2
// (Zeldovich.c:66-88); the kx = n/2 plane is zero.
__global__ void k_psi_spec(int n, int hx, const float2 *phik, int axis, float2 *out) {
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    const int j = row % n, k = row / n;
    for (int i = threadIdx.x; i < hx; i += blockDim.x) {
      const int64_t e = (int64_t)row * hx + i;
      float2 v = make_float2(0.f, 0.f);
      if (i < n / 2) {
        const float twopi = (float)(2 * M_PI);
        float ka;
        if (axis == 0) {
          ka = (float)i;
        } else {
          float kk = (float)(axis == 1 ? j : k);
          ka = kk > (float)(n / 2) ? kk - (float)n : kk;
        }
        float2 p = phik[e];
        v = make_float2(__fmul_rn(__fmul_rn(-twopi, ka), p.y), __fmul_rn(__fmul_rn(twopi, ka), p.x));
      }
      out[e] = v;
    }
  }
}

struct DmRecord {
  uint64_t indx;
  float x, y, z, vx, vy, vz;
};

// Particle records, one per lattice point in the order z, y, x: index
// i + N (j + N k); component a of velocity vamp * (vamp * psi) and of offset
// pfact * velocity (cosmosic.h:202-214, MakeParticle.c:181-195,
// cosmosic.h:285-288). Each thread writes a whole record: three passes that
// wrote one component each took 692 us at 256^3, on partial sectors.
__global__ void k_records(const float *px, const float *py, const float *pz, MeshGeom g, double rincube, float vamp,
                          float pfact, DmRecord *rec) {
  int n = g.n;
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    for (int x = threadIdx.x; x < n; x += blockDim.x) {
      const int y = row % n, z = row / n;
      const float *pads[3] = {px, py, pz};
      DmRecord o;
      o.indx = (uint64_t)((int64_t)row * n + x);
      float vel[3];
#pragma unroll
      for (int a = 0; a < 3; a++) vel[a] = __fmul_rn(vamp, __fmul_rn(vamp, interior(pads[a], g, x, y, z, rincube)));
      o.x = __fmul_rn(pfact, vel[0]);
      o.y = __fmul_rn(pfact, vel[1]);
      o.z = __fmul_rn(pfact, vel[2]);
      o.vx = vel[0];
      o.vy = vel[1];
      o.vz = vel[2];
      rec[(int64_t)row * n + x] = o;
    }
  }
}

// ---- second order (TwoLPT.c:259-535)
__device__ __forceinline__ float axis_freq(int axis, int i, int j, int k, int n) {
  return axis == 0 ? (float)i : (float)wrap_freq(axis == 1 ? j : k, n);
}

// -4 pi^2 k_a k_b phi_k, as ((-fourpi2 * k_a) * k_b) * phi in float, for
// every kx <= n/2 (TwoLPT.c:340-500 takes the pairs (x,x), (y,y), (z,z),
// (y,x), (z,x), (z,y) in that factor order).
__global__ void k_hessian_spec(int n, int hx, const float2 *phik, int a, int b, float2 *out) {
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    const int j = row % n, k = row / n;
    for (int i = threadIdx.x; i < hx; i += blockDim.x) {
      const int64_t e = (int64_t)row * hx + i;
      const float twopi = (float)(2 * M_PI);
      const float fourpi2 = __fmul_rn(twopi, twopi);
      float f = __fmul_rn(__fmul_rn(-fourpi2, axis_freq(a, i, j, k, n)), axis_freq(b, i, j, k, n));
      float2 p = phik[e];
      out[e] = make_float2(__fmul_rn(f, p.x), __fmul_rn(f, p.y));
    }
  }
}

// phi2 (=, +=, -=) w_a w_b / N^6 (TwoLPT.c:367-505): float product, then
// double scale and sum, stored as float.
__global__ void k_2lpt_acc(const float *pa, const float *pb, MeshGeom g, double sq, int mode, float *phi2) {
  int n = g.n;
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    for (int x = threadIdx.x; x < n; x += blockDim.x) {
      const int64_t e = (int64_t)row * n + x;
      const int y = row % n, z = row / n;
      int64_t off = (int64_t)(x + kGhost) + (int64_t)g.px * ((y + kGhost) + (int64_t)g.py * (z + kGhost));
      double d = __dmul_rn((double)__fmul_rn(pa[off], pb[off]), sq);
      if (mode == 0)
        phi2[e] = __double2float_rn(d);
      else if (mode == 1)
        phi2[e] = __double2float_rn(__dadd_rn((double)phi2[e], d));
      else
        phi2[e] = __double2float_rn(__dsub_rn((double)phi2[e], d));
    }
  }
}

// phi2_k /= -(k^2) 4 pi^2, zero at k = 0 (TwoLPT.c:510-533).
__global__ void k_inv_laplace(int n, int hx, float2 *s) {
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    const int j = row % n, k = row / n;
    for (int i = threadIdx.x; i < hx; i += blockDim.x) {
      const int64_t e = (int64_t)row * hx + i;
      int ky = wrap_freq(j, n), kz = wrap_freq(k, n);
      const float twopi = (float)(2 * M_PI);
      const float fourpi2 = __fmul_rn(twopi, twopi);
      int64_t k2 = (int64_t)i * i + (int64_t)ky * ky + (int64_t)kz * kz;
      double wave2 = (double)__fmul_rn((float)(-k2), fourpi2);
      float2 v = s[e];
      if (wave2 < 0.0) {
        double inv = 1.0 / wave2;
        v = make_float2(__double2float_rn(__dmul_rn((double)v.x, inv)), __double2float_rn(__dmul_rn((double)v.y, inv)));
      } else {
        v = make_float2(0.f, 0.f);
      }
      s[e] = v;
    }
  }
}

// TwoLPT's conversion of the velocity potential to the real potential and
// back (TwoLPT.c:288-289, 333-334): each padded row's first n floats times
// `factor` (the kx = n/2 element of an even row is left as it is).
__global__ void k_scale_rows(float2 *spec, int n, int hx, double factor) {
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    for (int i = threadIdx.x; i < hx; i += blockDim.x) {
      const int64_t e = (int64_t)row * hx + i;
      float2 v = spec[e];
      if (2 * i < n) v.x = __double2float_rn(__dmul_rn((double)v.x, factor));
      if (2 * i + 1 < n) v.y = __double2float_rn(__dmul_rn((double)v.y, factor));
      spec[e] = v;
    }
  }
}

// TwoLPT's non-Gaussian terms (TwoLPT.c:298-331): phi += fzc fNL (phi^2 -
// sigma^2) + gzc gNL (phi^3 - 3 sigma^2 phi) in FP64, fzc = 1/growth/amax,
// gzc = fzc^2.
__global__ void k_phi_nongauss_2lpt(const float *pad, MeshGeom g, double rincube, const double *sums, float fnl,
                                    float gnl, double fzc, double gzc, float *real) {
  int n = g.n;
  double mean = sums[0] * rincube;
  double sd = sqrt(sums[1] * rincube - mean * mean);
  double s2 = __dmul_rn(sd, sd);
  double three_s2 = __dmul_rn(__dmul_rn(3.0, sd), sd);
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    for (int x = threadIdx.x; x < n; x += blockDim.x) {
      const int64_t e = (int64_t)row * n + x;
      const int y = row % n, z = row / n;
      double d = (double)interior(pad, g, x, y, z, rincube);
      double d2 = __dmul_rn(d, d);
      double t1 = __dmul_rn(__dmul_rn(fzc, (double)fnl), __dsub_rn(d2, s2));
      double t2 = __dmul_rn(__dmul_rn(gzc, (double)gnl), __dsub_rn(__dmul_rn(d2, d), __dmul_rn(three_s2, d)));
      real[e] = __double2float_rn(__dadd_rn(d, __dadd_rn(t1, t2)));
    }
  }
}

// One component's spectrum of the combined potential a1 phi1 + a2 phi2 and
// its derivative along `axis` for every kx <= n/2 (TwoLPT_GetVR,
// cosmosic.h:147-149, and selfdiffphi, TwoLPT.c:58-112).
__global__ void k_grad_combined(int n, int hx, const float2 *s1, const float2 *s2, float a1, float a2, int axis,
                                float2 *out) {
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    const int j = row % n, k = row / n;
    for (int i = threadIdx.x; i < hx; i += blockDim.x) {
      const int64_t e = (int64_t)row * hx + i;
      float2 p = s1[e], q = s2[e];
      float re = __fadd_rn(__fmul_rn(a1, p.x), __fmul_rn(a2, q.x));
      float im = __fadd_rn(__fmul_rn(a1, p.y), __fmul_rn(a2, q.y));
      const float twopi = (float)(2 * M_PI);
      float ka = axis_freq(axis, i, j, k, n);
      out[e] = make_float2(__fmul_rn(__fmul_rn(-twopi, ka), im), __fmul_rn(__fmul_rn(twopi, ka), re));
    }
  }
}

// Second-order records: the velocities (which = 0) or the offsets (which = 1)
// of the three components, the fields times 1/N^3 (selfdiffphi,
// TwoLPT.c:133-134; Set_Particle_2LPT_Vel and TwoLPTPosAssign,
// MakeParticle.c:12-77 and cosmosic.h:236-271).
__global__ void k_records_2lpt(const float *px, const float *py, const float *pz, MeshGeom g, double rincube, int which,
                               DmRecord *rec) {
  int n = g.n;
  for (int row = blockIdx.x; row < n * n; row += gridDim.x) {
    for (int x = threadIdx.x; x < n; x += blockDim.x) {
      const int y = row % n, z = row / n;
      const float fx = interior(px, g, x, y, z, rincube), fy = interior(py, g, x, y, z, rincube),
                  fz = interior(pz, g, x, y, z, rincube);
      const int64_t e = (int64_t)row * n + x;
      DmRecord &o = rec[e];
      if (which == 0) {
        o.vx = fx;
        o.vy = fy;
        o.vz = fz;
      } else {
        o.indx = (uint64_t)e;
        o.x = fx;
        o.y = fy;
        o.z = fz;
      }
    }
  }
}

int grid_for_n(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  return (int)(b < 1 ? 1 : b);
}

int ic_fail(int code, const char *m) {
  set_last_error(m);
  return code;
}

// Buffers laid out one after another in one piece of memory.
struct Layout {
  static constexpr int kMax = 32;
  void **at[kMax];
  size_t off[kMax], total = 0;
  int count = 0;
  template <class T>
  void add(T **p, size_t bytes) {
    at[count] = reinterpret_cast<void **>(p);
    off[count++] = total;
    total += (bytes + 255) / 256 * 256;
  }
  void place(char *base) const {
    for (int i = 0; i < count; i++) *at[i] = base + off[i];
  }
};

// The device buffers of one call, carved from one allocation: a call makes up
// to twenty-five of them, and a cudaMalloc and cudaFree for each took as long
// as the kernels (4 ms at 256^3). The noise's scratch, read no more once the
// spectrum is filled, lies over the meshes that are written after that.
struct Carve : Layout {
  char *base = nullptr;
  Layout noise, meshes;
  char *over = nullptr;  // both of them
  cudaError_t commit() {
    add(&over, meshes.total > noise.total ? meshes.total : noise.total);
    cudaError_t e = cudaMalloc(reinterpret_cast<void **>(&base), total);
    if (e != cudaSuccess) return e;
    place(base);
    noise.place(over);
    meshes.place(over);
    return e;
  }
  ~Carve() { cudaFree(base); }
};

// Scratch of the noise stream.
struct Noise {
  int64_t modes = 0, nlev[kLevels] = {};  // drawing modes; chunk starts per level
  uint32_t *x0, *jump, *lev[kLevels], *counts, *offs, *bsum, *total, *rowcnt, *rowoff, *rbsum;
  float2 *acc;
  float *velpot = nullptr;
};

// Sizes the stream and registers its buffers.
void noise_plan(const tpm_ic_params *p, Noise &w, Carve &mem) {
  const int n = p->n;
  const int64_t knyq = n / 2, rows = (int64_t)n * n;
  // drawing modes: for each |kz| and |ky| the kx with 0 < k^2 <= (n/2)^2; the
  // largest kx falls as |ky| grows
  auto times = [&](int64_t k) { return k == 0 || 2 * k == n ? 1 : 2; };  // rows of this |k|
  for (int64_t kz = 0; kz <= knyq; kz++) {
    int64_t im = knyq;
    for (int64_t ky = 0; ky <= knyq; ky++) {
      int64_t r = knyq * knyq - ky * ky - kz * kz;
      if (r < 0) break;
      while (im * im > r) im--;
      int64_t i0 = (ky == 0 && kz == 0) ? 1 : 0;
      if (im >= i0) w.modes += (im - i0 + 1) * times(ky) * times(kz);
    }
  }
  // trials: the acceptance rate is pi/4; 3% and 4096 trials of margin
  int64_t trials = (int64_t)((double)w.modes * (4.0 / M_PI) * 1.03) + 4096;
  w.nlev[0] = (trials + kTrialsPerChunk - 1) / kTrialsPerChunk;
  for (int l = 1; l < kLevels; l++) w.nlev[l] = (w.nlev[l - 1] + kRadix - 1) / kRadix;
  const int64_t nb = (w.nlev[0] + 4095) / 4096, rnb = (rows + 4095) / 4096;
  mem.noise.add(&w.x0, sizeof(uint32_t) * kLag);
  mem.noise.add(&w.jump, sizeof(uint32_t) * kLag * kLevels);
  for (int l = 0; l < kLevels; l++) mem.noise.add(&w.lev[l], sizeof(uint32_t) * kLag * w.nlev[l]);
  mem.noise.add(&w.counts, sizeof(uint32_t) * w.nlev[0]);
  mem.noise.add(&w.offs, sizeof(uint32_t) * w.nlev[0]);
  mem.noise.add(&w.bsum, sizeof(uint32_t) * (nb + 1));
  mem.add(&w.total, sizeof(uint32_t) * 2);  // read at the end
  mem.noise.add(&w.rowcnt, sizeof(uint32_t) * rows);
  mem.noise.add(&w.rowoff, sizeof(uint32_t) * rows);
  mem.noise.add(&w.rbsum, sizeof(uint32_t) * (rnb + 1));
  mem.noise.add(&w.acc, sizeof(float2) * (w.modes > 0 ? w.modes : 1));
  if (p->iseed < 0) mem.noise.add(&w.velpot, sizeof(float) * (size_t)(knyq * knyq + 1));
}

int row_grid(int n) { return n * n < 148 * 16 ? n * n : 148 * 16; }

// The noise spectrum on the device (spec: n*n*hx float2); noise_check after the
// stream has finished says whether the stream was long enough.
cudaError_t noise_enqueue(const tpm_ic_params *p, const Noise &w, float2 *spec, cudaStream_t st) {
  const int n = p->n, hx = n / 2 + 1;
  const int64_t rows = (int64_t)n * n, knyq = n / 2, nchunks = w.nlev[0];
  if (p->iseed < 0) {
    cudaError_t e = cudaMemcpyAsync(w.velpot, p->velpot, sizeof(float) * (size_t)(knyq * knyq + 1),
                                    cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
  }
  // the reference runs its unit-amplitude path (ISEED >= 0) with seed -1
  k_ran3_init<<<1, 32, 0, st>>>(p->iseed >= 0 ? -1 : p->iseed, w.x0);
  k_ran3_jumps<<<1, 128, 0, st>>>(w.jump);
  k_ran3_level<<<1, 64, 0, st>>>(w.x0, w.jump + (kLevels - 1) * kLag, w.nlev[kLevels - 1], (int)w.nlev[kLevels - 1],
                                 w.lev[kLevels - 1]);
  for (int l = kLevels - 2; l >= 0; l--)
    k_ran3_level<<<(unsigned)w.nlev[l + 1], 64, 0, st>>>(w.lev[l + 1], w.jump + l * kLag, w.nlev[l], kRadix, w.lev[l]);
  k_ran3_trials<false><<<grid_for_n(nchunks, 64), 64, 0, st>>>(w.lev[0], nchunks, w.counts, nullptr, nullptr, nullptr,
                                                               0);
  scan_u32(w.counts, w.offs, nchunks, w.bsum, w.total, st);
  k_ran3_trials<true><<<grid_for_n(nchunks, 64), 64, 0, st>>>(w.lev[0], nchunks, nullptr, w.offs, w.bsum, w.acc,
                                                              w.modes);
  // mode ranks
  k_row_counts<<<grid_for_n(rows, 256), 256, 0, st>>>(n, w.rowcnt);
  scan_u32(w.rowcnt, w.rowoff, rows, w.rbsum, w.total + 1, st);
  k_fill_noise<<<row_grid(n), 128, 0, st>>>(n, hx, w.rowoff, w.rbsum, w.acc, w.velpot, spec);
  k_conjugate_plane<<<grid_for_n(rows, 256), 256, 0, st>>>(n, hx, spec);
  return cudaGetLastError();
}

// Waits for the stream; an error code and its message where the trials ran out.
int noise_check(const Noise &w, cudaStream_t st, char *msg, size_t len) {
  uint32_t accepted = 0;
  cudaError_t e = cudaMemcpyAsync(&accepted, w.total, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    snprintf(msg, len, "initial conditions: %s", cudaGetErrorString(e));
    return TPM_E_CUDA;
  }
  if ((int64_t)accepted < w.modes) {
    snprintf(msg, len, "noise stream too short: %u accepted trials for %lld modes", accepted, (long long)w.modes);
    return TPM_E_CUDA;
  }
  return 0;
}

int check_ic_params(const tpm_ic_params *p) {
  if (!p) return ic_fail(TPM_E_ARG, "params is NULL");
  if (p->n < 8 || p->n > 1024) return ic_fail(TPM_E_ARG, "n outside [8, 1024]");
  int m = p->n;
  while (m % 2 == 0) m /= 2;
  while (m % 3 == 0) m /= 3;
  while (m % 5 == 0) m /= 5;
  if (m != 1) return ic_fail(TPM_E_ARG, "n must be a product of 2, 3 and 5");
  if (p->iseed < 0 && !p->velpot) return ic_fail(TPM_E_ARG, "a negative seed needs the amplitude table");
  return 0;
}

}  // namespace

extern "C" {

int tpm_ic_noise(const tpm_ic_params *p, float *spec, int mem) {
  int rc = check_ic_params(p);
  if (rc) return rc;
  if (!spec) return ic_fail(TPM_E_ARG, "spec is NULL");
  if (cudaSetDevice(p->device) != cudaSuccess) return ic_fail(TPM_E_CUDA, "cudaSetDevice failed");
  char msg[256] = {0};
  int64_t elems = (int64_t)p->n * p->n * (p->n / 2 + 1);
  cudaStream_t st = nullptr;
  float2 *d = reinterpret_cast<float2 *>(spec);
  Noise noise;
  Carve buf;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess)
    return ic_fail(TPM_E_CUDA, "cudaStreamCreate failed");
  noise_plan(p, noise, buf);
  if (mem != TPM_MEM_DEVICE) buf.add(&d, sizeof(float2) * elems);
  if (buf.commit() != cudaSuccess) {
    cudaStreamDestroy(st);
    return ic_fail(TPM_E_NOMEM, "cudaMalloc failed");
  }
  IC_CK(noise_enqueue(p, noise, d, st));
  if (mem != TPM_MEM_DEVICE) IC_CK(cudaMemcpyAsync(spec, d, sizeof(float2) * elems, cudaMemcpyDeviceToHost, st));
  rc = noise_check(noise, st, msg, sizeof(msg));
done:
  if (rc) set_last_error(msg);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return rc;
}

int tpm_ic_zeldovich(const tpm_ic_params *p, void *records, int mem) {
  int rc = check_ic_params(p);
  if (rc) return rc;
  if (!records) return ic_fail(TPM_E_ARG, "records is NULL");
  if (cudaSetDevice(p->device) != cudaSuccess) return ic_fail(TPM_E_CUDA, "cudaSetDevice failed");
  char msg[256] = {0};
  MeshGeom g = make_geom(p->n);
  int n = p->n;
  int64_t cells = (int64_t)n * n * n;
  int64_t elems = g.spec_elems;
  double rincube = 1. / (double)n / (double)n / (double)n;
  cudaStream_t st = nullptr;
  FftPlan plan;
  float2 *phik = nullptr, *work = nullptr, *tw = nullptr, *spec = nullptr;
  float *pad[3] = {nullptr, nullptr, nullptr}, *real = nullptr;
  double *sums = nullptr;
  DmRecord *rec = reinterpret_cast<DmRecord *>(records);
  const size_t pad_bytes = sizeof(float) * g.px * g.py * g.pz;
  Noise noise;
  Carve buf;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess)
    return ic_fail(TPM_E_CUDA, "cudaStreamCreate failed");
  noise_plan(p, noise, buf);
  buf.add(&phik, sizeof(float2) * elems);
  for (int a = 0; a < 3; a++) buf.meshes.add(&pad[a], a < 2 ? pad_bytes : std::max(pad_bytes, sizeof(float2) * elems));
  buf.add(&sums, sizeof(double) * 2);
  buf.add(&tw, sizeof(float2) * fft_twiddles(n));
  if (mem != TPM_MEM_DEVICE) buf.add(&rec, sizeof(DmRecord) * cells);
  IC_CK(buf.commit());
  IC_CK(fft_plan_in(plan, n, tw, st));
  IC_CK(noise_enqueue(p, noise, phik, st));
  // back to real space, the local terms, and forward again (Zeldovich.c:35-63);
  // with fNL = gNL = 0 the round trip still matters: it keeps only the
  // Hermitian part of the noise on the kx = 0 and kx = n/2 planes, whose
  // conjugate completion (PMSeedForce.c:355-396) leaves the ky = n/2 and
  // kz = n/2 lines as drawn
  real = pad[1];  // free until the displacements
  work = reinterpret_cast<float2 *>(pad[2]);  // free until the last of them
  IC_CK(cudaMemsetAsync(sums, 0, sizeof(double) * 2, st));
  fft_inverse(g, plan, phik, pad[0], st);
  k_phi_moments<<<row_grid(n), 128, 0, st>>>(pad[0], g, rincube, sums);
  k_phi_nongauss<<<row_grid(n), 128, 0, st>>>(pad[0], g, rincube, sums, p->fnl, p->gnl, real);
  fft_forward(g, plan, real, phik, st);
  for (int a = 0; a < 3; a++) {
    // the last component takes phi_k's place, whose memory it may overwrite
    spec = a < 2 ? work : phik;
    k_psi_spec<<<row_grid(n), 128, 0, st>>>(n, g.hx, phik, a, spec);
    fft_inverse(g, plan, spec, pad[a], st);
  }
  k_records<<<row_grid(n), 128, 0, st>>>(pad[0], pad[1], pad[2], g, rincube, p->vamp, p->pfact, rec);
  IC_CK(cudaGetLastError());
  if (mem != TPM_MEM_DEVICE) IC_CK(cudaMemcpyAsync(records, rec, sizeof(DmRecord) * cells, cudaMemcpyDeviceToHost, st));
  rc = noise_check(noise, st, msg, sizeof(msg));
done:
  if (rc) set_last_error(msg);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return rc;
}

int tpm_ic_2lpt(const tpm_ic_params *p, void *records, int mem) {
  int rc = check_ic_params(p);
  if (rc) return rc;
  if (!records) return ic_fail(TPM_E_ARG, "records is NULL");
  const bool nongauss = p->fnl != 0.f || p->gnl != 0.f;
  if (nongauss && !(p->boxsize > 0.f && p->omep > 0.f && p->amax > 0.f && p->growth > 0.f))
    return ic_fail(TPM_E_ARG, "fnl/gnl need boxsize, omep, amax and growth > 0");
  if (cudaSetDevice(p->device) != cudaSuccess) return ic_fail(TPM_E_CUDA, "cudaSetDevice failed");
  char msg[256] = {0};
  MeshGeom g = make_geom(p->n);
  int n = p->n;
  int64_t cells = (int64_t)n * n * n;
  int64_t elems = g.spec_elems;
  double rincube = 1. / (double)n / (double)n / (double)n;
  double sq = rincube * rincube;
  const int rg = row_grid(n);
  // the pairs of TwoLPT.c:340-505: (a, b, pad slot, accumulation)
  const int pairs[7][4] = {{0, 0, 0, -1}, {1, 1, 1, 0}, {2, 2, 1, 1}, {1, 1, 0, 1},
                           {1, 0, 0, 2},  {2, 0, 0, 2}, {2, 1, 0, 2}};
  cudaStream_t st = nullptr;
  FftPlan plan;
  float2 *s1 = nullptr, *s2 = nullptr, *work = nullptr, *tw = nullptr;
  float *pad[3] = {nullptr, nullptr, nullptr}, *phi2 = nullptr;
  double *sums = nullptr;
  DmRecord *rec = reinterpret_cast<DmRecord *>(records);
  const size_t pad_bytes = sizeof(float) * g.px * g.py * g.pz;
  // offsets: AI NX damp (TwoLPTmain.c:211-213), with pfact = AI NX
  const float amp[2][2] = {{p->vamp, p->vamp2}, {p->pfact * p->damp1, p->pfact * p->damp2}};
  Noise noise;
  Carve buf;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess)
    return ic_fail(TPM_E_CUDA, "cudaStreamCreate failed");
  noise_plan(p, noise, buf);
  buf.add(&s1, sizeof(float2) * elems);
  buf.add(&s2, sizeof(float2) * elems);
  buf.add(&work, sizeof(float2) * elems);
  for (int a = 0; a < 3; a++) buf.meshes.add(&pad[a], pad_bytes);
  buf.add(&sums, sizeof(double) * 2);
  buf.add(&tw, sizeof(float2) * fft_twiddles(n));
  if (mem != TPM_MEM_DEVICE) buf.add(&rec, sizeof(DmRecord) * cells);
  IC_CK(buf.commit());
  phi2 = pad[2];  // the source, until the displacements
  IC_CK(fft_plan_in(plan, n, tw, st));
  IC_CK(noise_enqueue(p, noise, s1, st));
  if (nongauss) {
    // to the real potential, the local terms, and back (TwoLPT.c:284-335)
    const double cvel = 2.99792458E5;
    double x = (double)(100.f * p->boxsize) / cvel;
    double vp2rp = 1.5 * pow(x, 2) * (double)p->omep * (double)p->amax;
    double fzc = 1. / (double)p->growth / (double)p->amax;
    double gzc = fzc * fzc;
    IC_CK(cudaMemsetAsync(sums, 0, sizeof(double) * 2, st));
    k_scale_rows<<<rg, 128, 0, st>>>(s1, n, g.hx, vp2rp);
    fft_inverse(g, plan, s1, pad[0], st);
    k_phi_moments<<<rg, 128, 0, st>>>(pad[0], g, rincube, sums);
    k_phi_nongauss_2lpt<<<rg, 128, 0, st>>>(pad[0], g, rincube, sums, p->fnl, p->gnl, fzc, gzc, pad[1]);
    fft_forward(g, plan, pad[1], s1, st);
    k_scale_rows<<<rg, 128, 0, st>>>(s1, n, g.hx, 1.0 / vp2rp);
  }
  // the second-order source sum_{a<b} phi,aa phi,bb - phi,ab^2 in real space
  for (int q = 0; q < 7; q++) {
    k_hessian_spec<<<rg, 128, 0, st>>>(n, g.hx, s1, pairs[q][0], pairs[q][1], work);
    fft_inverse(g, plan, work, pad[pairs[q][2]], st);
    int mode = pairs[q][3];
    if (mode == 0)
      k_2lpt_acc<<<rg, 128, 0, st>>>(pad[0], pad[1], g, sq, 0, phi2);
    else if (mode == 1)
      k_2lpt_acc<<<rg, 128, 0, st>>>(pad[0], pad[1], g, sq, 1, phi2);
    else if (mode == 2)
      k_2lpt_acc<<<rg, 128, 0, st>>>(pad[0], pad[0], g, sq, 2, phi2);
  }
  fft_forward(g, plan, phi2, s2, st);
  k_inv_laplace<<<rg, 128, 0, st>>>(n, g.hx, s2);
  for (int which = 0; which < 2; which++) {
    for (int a = 0; a < 3; a++) {
      k_grad_combined<<<rg, 128, 0, st>>>(n, g.hx, s1, s2, amp[which][0], amp[which][1], a, work);
      fft_inverse(g, plan, work, pad[a], st);
    }
    k_records_2lpt<<<rg, 128, 0, st>>>(pad[0], pad[1], pad[2], g, rincube, which, rec);
  }
  IC_CK(cudaGetLastError());
  if (mem != TPM_MEM_DEVICE) IC_CK(cudaMemcpyAsync(records, rec, sizeof(DmRecord) * cells, cudaMemcpyDeviceToHost, st));
  rc = noise_check(noise, st, msg, sizeof(msg));
done:
  if (rc) set_last_error(msg);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return rc;
}

}  // extern "C"
