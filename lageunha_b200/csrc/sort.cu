// Morton-key particle sort (sm_100a).
//
// The reference orders particles spatially with a chaining mesh of
// CellWidth = 4 cells and head-inserted linked lists (Cosmos/BasicCell.c:10-42,
// BasicCell.h:33-63) and then builds one octree per bucket
// (OST/ost.ver2.c:36-196). Here every particle gets a 39-bit Morton key of its
// quantised cell coordinate (13 bits per axis: ceil(log2 N) cell bits plus
// sub-cell bits) and the (key, index) pairs are sorted by a stable LSD radix
// sort with 8-bit digits. Ties keep the input order, so the permutation is
// the stable argsort of the keys and is bit-exact against a CPU recomputation.
//
// A force evaluation sorts in single-sweep passes (sweep_sort): the digit
// counts of all five passes come from one read of the positions, each pass
// places its tiles by looking back at its predecessors' counts, and carries 8
// bytes per particle: the 7 bits of the first pass are not needed again, the
// rest of the key fits 32 bits, and the full keys of the sorted particles are
// recomputed when their positions are gathered. radix_sort_pairs (a histogram
// and a scan per pass, 64-bit keys) remains for callers without scratch for
// the look-back (tpm_morton_order_noalloc) and for 2^30 particles and more.
#include "engine_internal.cuh"
#include "lookback.h"

namespace tpm {

__global__ void k_make_keys(const uint32_t *__restrict__ pos, int64_t np, uint32_t n, int sub_bits,
                            uint64_t *__restrict__ key, uint32_t *__restrict__ val) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t qx = quantize(pos[3 * i + 0], n, sub_bits);
    uint32_t qy = quantize(pos[3 * i + 1], n, sub_bits);
    uint32_t qz = quantize(pos[3 * i + 2], n, sub_bits);
    key[i] = morton3(qx, qy, qz);
    val[i] = (uint32_t)i;
  }
}

void launch_make_keys(const uint32_t *pos, int64_t np, uint32_t n, int sub_bits, uint64_t *key,
                      uint32_t *val, cudaStream_t st) {
  int blocks = (int)((np + 255) / 256);
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (blocks < 1) blocks = 1;
  k_make_keys<<<blocks, 256, 0, st>>>(pos, np, n, sub_bits, key, val);
}

int64_t sort_tiles(int64_t np) { return (np + kSortTile - 1) / kSortTile; }

// Per-tile digit histogram; hist is digit-major: hist[d * ntiles + tile].
__global__ void __launch_bounds__(kSortThreads) k_radix_hist(const uint64_t *__restrict__ key,
                                                             int64_t np, int shift,
                                                             uint32_t *__restrict__ hist,
                                                             int64_t ntiles) {
  __shared__ uint32_t cnt[8][256];
  int tid = threadIdx.x, warp = tid >> 5;
  for (int i = tid; i < 8 * 256; i += kSortThreads) (&cnt[0][0])[i] = 0;
  __syncthreads();
  int64_t base = blockIdx.x * (int64_t)kSortTile;
#pragma unroll
  for (int r = 0; r < kSortItems; r++) {
    int64_t i = base + r * kSortThreads + tid;
    if (i < np) {
      uint32_t d = (uint32_t)(key[i] >> shift) & 0xffu;
      atomicAdd(&cnt[warp][d], 1u);
    }
  }
  __syncthreads();
  for (int d = tid; d < 256; d += kSortThreads) {
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) s += cnt[w][d];
    hist[(int64_t)d * ntiles + blockIdx.x] = s;
  }
}

// One block per digit: exclusive scan of hist[d][0..ntiles) in place and the
// digit total.
__global__ void __launch_bounds__(1024) k_radix_scan_digit(uint32_t *__restrict__ hist, int64_t ntiles,
                                                           uint32_t *__restrict__ dtotal) {
  __shared__ uint32_t wsum[32];
  __shared__ uint32_t carry;
  uint32_t *h = hist + (int64_t)blockIdx.x * ntiles;
  int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < ntiles; base += 1024) {
    int64_t i = base + tid;
    uint32_t v = i < ntiles ? h[i] : 0u;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t s = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      wsum[lane] = s;  // inclusive
    }
    __syncthreads();
    uint32_t before = carry + (warp ? wsum[warp - 1] : 0u) + x - v;
    if (i < ntiles) h[i] = before;
    __syncthreads();
    if (tid == 0) carry += wsum[31];
    __syncthreads();
  }
  if (tid == 0) dtotal[blockIdx.x] = carry;
}

// Stable scatter of one tile of kSortTile items. Warp w owns the contiguous
// items [w*256, (w+1)*256) of the tile and ranks them in chunks of 32 against
// its own running digit counts (no block barrier per chunk); a prefix over the
// warps and over the digits then gives every item its place in the tile
// sorted by digit, which is written to shared memory. The tile is finally
// written out in that order, so each digit's run goes to consecutive global
// addresses. Items of equal digit keep their input order (chunks in order,
// lanes in order, warps in order), so the pass is a stable sort.
// Four blocks per SM: the ranking is a chain through each warp's digit
// counters (eight chunks), so the scatter is latency-bound and the tile is
// kept at 2048 items (39 KB of shared memory, each lane's 8 keys and values in
// 64 registers) for more resident warps; 4096-item tiles at three blocks per
// SM took 6% longer per sort.
constexpr int kScatterWarps = kSortThreads / 32;
constexpr int kWarpItems = kSortTile / kScatterWarps;
__global__ void __launch_bounds__(kSortThreads, 4) k_radix_scatter(
    const uint64_t *__restrict__ kin, const uint32_t *__restrict__ vin, uint64_t *__restrict__ kout,
    uint32_t *__restrict__ vout, int64_t np, int shift, const uint32_t *__restrict__ hist,
    const uint32_t *__restrict__ dtotal, int64_t ntiles) {
  extern __shared__ __align__(16) unsigned char sc_smem[];
  uint64_t *sk = reinterpret_cast<uint64_t *>(sc_smem);                 // [kSortTile] keys in digit order
  uint32_t *sv = reinterpret_cast<uint32_t *>(sk + kSortTile);          // [kSortTile] values
  uint16_t *rk = reinterpret_cast<uint16_t *>(sv + kSortTile);          // [kSortTile] rank in warp's digit
  uint32_t(*wc)[256] = reinterpret_cast<uint32_t(*)[256]>(rk + kSortTile);  // [warps][256]
  __shared__ uint32_t lstart[256];  // first slot of each digit in the tile
  __shared__ uint32_t gbase[256];   // global slot of each digit's first item of this tile
  __shared__ uint32_t ws[kScatterWarps];
  int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kScatterWarps * 256; i += kSortThreads) (&wc[0][0])[i] = 0;
  __syncthreads();
  const int64_t tbase = blockIdx.x * (int64_t)kSortTile;
  const uint32_t lanemask_lt = (1u << lane) - 1u;
  // this lane's items of the warp's segment, all loaded before any is ranked
  constexpr int kChunks = kWarpItems / 32;
  uint64_t kr[kChunks];
  uint32_t vr[kChunks];
#pragma unroll
  for (int c = 0; c < kChunks; c++) {
    int64_t i = tbase + warp * kWarpItems + c * 32 + lane;
    kr[c] = i < np ? kin[i] : 0ull;
    vr[c] = i < np ? vin[i] : 0u;
  }
  // ---- ranks inside each warp's segment
#pragma unroll
  for (int c = 0; c < kChunks; c++) {
    int j = warp * kWarpItems + c * 32 + lane;
    int64_t i = tbase + j;
    bool valid = i < np;
    uint32_t d = valid ? (uint32_t)(kr[c] >> shift) & 0xffu : 0x100u;
    uint32_t peers = __match_any_sync(0xffffffffu, d);
    uint32_t prev = valid ? wc[warp][d] : 0u;
    __syncwarp();
    if (valid && (peers & lanemask_lt) == 0) wc[warp][d] = prev + __popc(peers);
    __syncwarp();
    rk[j] = (uint16_t)(prev + __popc(peers & lanemask_lt));
  }
  __syncthreads();
  // ---- per digit: prefix over the warps, the tile's count, and its global base
  uint32_t cnt;
  {
    int d = tid;
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kScatterWarps; w++) {
      uint32_t t = wc[w][d];
      wc[w][d] = run;
      run += t;
    }
    cnt = run;
    // exclusive scans over the 256 digits: tile counts and global digit totals
    uint32_t x = cnt, g = dtotal[d];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      uint32_t h = __shfl_up_sync(0xffffffffu, g, o);
      if (lane >= o) {
        x += y;
        g += h;
      }
    }
    if (lane == 31) ws[warp] = x;
    __shared__ uint32_t wg[kScatterWarps];
    if (lane == 31) wg[warp] = g;
    __syncthreads();
    uint32_t px = 0, pg = 0;
    for (int w = 0; w < warp; w++) {
      px += ws[w];
      pg += wg[w];
    }
    lstart[d] = px + x - cnt;
    gbase[d] = pg + g - dtotal[d] + hist[(int64_t)d * ntiles + blockIdx.x];
  }
  __syncthreads();
  // ---- place every item at its slot of the tile sorted by digit
#pragma unroll
  for (int c = 0; c < kChunks; c++) {
    int j = warp * kWarpItems + c * 32 + lane;
    int64_t i = tbase + j;
    if (i < np) {
      uint64_t k = kr[c];
      uint32_t d = (uint32_t)(k >> shift) & 0xffu;
      uint32_t slot = lstart[d] + wc[warp][d] + rk[j];
      sk[slot] = k;
      sv[slot] = vr[c];
    }
  }
  __syncthreads();
  // ---- write out: consecutive slots of a digit go to consecutive addresses
  int64_t nt = np - tbase < kSortTile ? np - tbase : kSortTile;
  for (int j = tid; j < nt; j += kSortThreads) {
    uint64_t k = sk[j];
    uint32_t d = (uint32_t)(k >> shift) & 0xffu;
    uint32_t g = gbase[d] + ((uint32_t)j - lstart[d]);
    kout[g] = k;
    vout[g] = sv[j];
  }
}

constexpr size_t kScatterSmem = (size_t)kSortTile * (8 + 4 + 2) + sizeof(uint32_t) * kScatterWarps * 256;

void radix_sort_pairs(uint64_t **key, uint32_t **val, uint64_t *key_alt, uint32_t *val_alt,
                      int64_t np, int nbits, SortScratch &scr, cudaStream_t st, int64_t *launches) {
  int64_t ntiles = sort_tiles(np);
  if (np <= 1) return;
  uint64_t *kin = *key, *kout = key_alt;
  uint32_t *vin = *val, *vout = val_alt;
  // the cap is an attribute of the function on the current device: raised on
  // every call, so contexts and threads on any device get it
  cudaFuncSetAttribute(k_radix_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScatterSmem);
  for (int shift = 0; shift < nbits; shift += 8) {
    k_radix_hist<<<(unsigned)ntiles, kSortThreads, 0, st>>>(kin, np, shift, scr.hist, ntiles);
    k_radix_scan_digit<<<256, 1024, 0, st>>>(scr.hist, ntiles, scr.dtotal);
    k_radix_scatter<<<(unsigned)ntiles, kSortThreads, kScatterSmem, st>>>(kin, vin, kout, vout, np, shift,
                                                                          scr.hist, scr.dtotal, ntiles);
    if (launches) *launches += 3;
    uint64_t *tk = kin;
    kin = kout;
    kout = tk;
    uint32_t *tv = vin;
    vin = vout;
    vout = tv;
  }
  *key = kin;
  *val = vin;
}

// ------------------------------------------------------------ single sweep
constexpr int kSweepThreads = 512;
constexpr int kSweepWarps = kSweepThreads / 32;
constexpr int kSweepItems = 8;
constexpr int kSweepTile = kSweepThreads * kSweepItems;
constexpr int kSweepPasses = 5;
constexpr int kLowBits = kKeyBits - 32;  // sorted by the first pass and dropped
// words before the tile states: the digit counts of every pass and the passes'
// tile tickets
constexpr int kSweepHead = kSweepPasses * 256 + 8;
// looks at its predecessors' words after which a tile counts their items itself
constexpr uint32_t kSweepLooks = 1u << 22;

int64_t sweep_words(int64_t np) { return kSweepHead + 256 * kSweepPasses * ((np + kSweepTile - 1) / kSweepTile); }

// Bits 0-9 of v at every third bit.
TPM_D uint32_t spread10(uint32_t v) {
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  return (v | (v << 2)) & 0x09249249u;
}

// Bits 10-12 of v at every third bit.
TPM_D uint32_t spread_top(uint32_t v) {
  v >>= 10;
  return (v | (v << 2) | (v << 4)) & 0x49u;
}

// morton3 of the particle's quantised coordinates in 32-bit halves: the low 30
// bits and the 9 above them.
TPM_D void key_halves(const uint32_t *__restrict__ pos, int64_t i, uint32_t n, int sub_bits, uint32_t &lo,
                      uint32_t &hi) {
  static_assert(kAxisBits == 13, "10 low and 3 high bits per axis");
  const uint32_t x = quantize(pos[3 * i + 0], n, sub_bits), y = quantize(pos[3 * i + 1], n, sub_bits),
                 z = quantize(pos[3 * i + 2], n, sub_bits);
  lo = spread10(x) | (spread10(y) << 1) | (spread10(z) << 2);
  hi = spread_top(x) | (spread_top(y) << 1) | (spread_top(z) << 2);
}

TPM_D uint64_t key_of(const uint32_t *__restrict__ pos, int64_t i, uint32_t n, int sub_bits) {
  uint32_t lo, hi;
  key_halves(pos, i, n, sub_bits, lo, hi);
  return (uint64_t)hi << 30 | lo;
}

// Digit counts of all passes: counts[pass * 256 + digit].
__global__ void __launch_bounds__(512) k_sweep_count(const uint32_t *__restrict__ pos, int64_t np, uint32_t n,
                                                     int sub_bits, uint32_t *__restrict__ counts) {
  __shared__ uint32_t h[4][kSweepPasses * 256];  // four copies: warps of one copy seldom meet
  for (int i = threadIdx.x; i < 4 * kSweepPasses * 256; i += blockDim.x) (&h[0][0])[i] = 0u;
  __syncthreads();
  uint32_t *mine = h[(threadIdx.x >> 5) & 3];
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t lo, hi;
    key_halves(pos, i, n, sub_bits, lo, hi);
    atomicAdd(&mine[lo & ((1u << kLowBits) - 1u)], 1u);
    hi = hi << (30 - kLowBits) | lo >> kLowBits;
#pragma unroll
    for (int p = 1; p < kSweepPasses; p++) atomicAdd(&mine[p * 256 + ((hi >> (8 * (p - 1))) & 0xffu)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kSweepPasses * 256; i += blockDim.x) {
    uint32_t v = h[0][i] + h[1][i] + h[2][i] + h[3][i];
    if (v) atomicAdd(&counts[i], v);
  }
}

// The items of a full tile, from item i0 on, with digit d of the first pass and
// of the others.
__device__ __noinline__ uint32_t count_low_digit(const uint32_t *pos, int64_t i0, uint32_t n, int sub_bits, uint32_t d) {
  uint32_t c = 0;
  for (int64_t i = i0; i < i0 + kSweepTile; i++) {
    uint32_t lo, hi;
    key_halves(pos, i, n, sub_bits, lo, hi);
    c += (lo & ((1u << kLowBits) - 1u)) == d ? 1u : 0u;
  }
  return c;
}
__device__ __noinline__ uint32_t count_digit(const uint32_t *key, int64_t i0, int shift, uint32_t d) {
  uint32_t c = 0;
  for (int64_t i = i0; i < i0 + kSweepTile; i++) c += ((key[i] >> shift) & 0xffu) == d ? 1u : 0u;
  return c;
}

// One pass over one tile of kSweepTile items. kFirst: the items are the
// particles in the caller's order, the digit the key's low bits; else (key,
// index) pairs with the digit at `shift` of the 32-bit key. kLast: the keys are
// not written.
//
// Ranks: warp w owns 256 consecutive items. For each chunk of 32 the first lane
// of every digit adds the digit's lanes to the warp's counter, and the old
// values are read back after all chunks have issued theirs, so the chain of a
// counter's updates runs at the shared memory's rate and not at its latency.
// Tiles take their numbers in the order in which they start, so a tile's
// predecessors are running or done when it looks back at them, and every wait
// ends; should one be stalled all the same, its items are counted instead, so the
// pass has one result.
template <bool kFirst, bool kLast>
__global__ void __launch_bounds__(kSweepThreads, 2)
    k_sweep_pass(const uint32_t *__restrict__ pos, const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin,
                 uint32_t *__restrict__ kout, uint32_t *__restrict__ vout, int64_t np, uint32_t n, int sub_bits,
                 int shift, const uint32_t *__restrict__ counts, uint32_t *__restrict__ ticket,
                 uint32_t *__restrict__ state) {
  extern __shared__ __align__(16) uint32_t sw_smem[];
  uint32_t *sk = sw_smem, *sv = sk + kSweepTile;                          // the tile in digit order
  uint32_t(*wc)[256] = reinterpret_cast<uint32_t(*)[256]>(sv + kSweepTile);  // [warps][256]
  __shared__ uint32_t lstart[256], gbase[256], ws[8], wg[8], tile_sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) tile_sh = atomicAdd(ticket, 1u);
  for (int i = tid; i < kSweepWarps * 256; i += kSweepThreads) (&wc[0][0])[i] = 0u;
  __syncthreads();
  const int64_t tile = tile_sh, tbase = tile * kSweepTile;
  const uint32_t lt = (1u << lane) - 1u;
  const int64_t i0 = tbase + warp * (kSweepItems * 32) + lane;
  // who: this lane's digit << 16 (kNoItem past the last particle), the first
  // lane of the digit << 8 and this lane's rank among its lanes; later the
  // digit and the rank within the warp's items of it
  constexpr uint32_t kNoItem = 0x100u;
  uint32_t k[kSweepItems], v[kSweepItems], who[kSweepItems], old[kSweepItems];
#pragma unroll
  for (int c = 0; c < kSweepItems; c++) {
    const int64_t i = i0 + 32 * c;
    const bool ok = i < np;
    k[c] = v[c] = 0u;
    who[c] = kNoItem;
    if (kFirst) {
      if (ok) {
        uint32_t lo, hi;
        key_halves(pos, i, n, sub_bits, lo, hi);
        k[c] = hi << (30 - kLowBits) | lo >> kLowBits;
        v[c] = (uint32_t)i;
        who[c] = lo & ((1u << kLowBits) - 1u);
      }
    } else if (ok) {
      k[c] = kin[i];
      v[c] = vin[i];
      who[c] = (k[c] >> shift) & 0xffu;
    }
  }
#pragma unroll
  for (int c = 0; c < kSweepItems; c++) {
    // the lanes with this lane's digit, by one vote per bit (a match
    // instruction is slower: 197 us for the pass over 16.8 million pairs)
    const uint32_t d = who[c];
    uint32_t same = __ballot_sync(0xffffffffu, d != kNoItem);
    if (d == kNoItem) same = ~same;
#pragma unroll
    for (int b = 0; b < (kFirst ? kLowBits : 8); b++) {
      const bool bit = (d >> b) & 1u;
      const uint32_t with = __ballot_sync(0xffffffffu, bit);
      same &= bit ? with : ~with;
    }
    who[c] = d << 16 | (uint32_t)(__ffs(same) - 1) << 8 | (uint32_t)__popc(same & lt);
    old[c] = 0u;
    if (d != kNoItem && (same & lt) == 0) old[c] = atomicAdd(&wc[warp][d], (uint32_t)__popc(same));
    __syncwarp();
  }
#pragma unroll
  for (int c = 0; c < kSweepItems; c++) {
    const uint32_t at = __shfl_sync(0xffffffffu, old[c], (int)(who[c] >> 8) & 31);
    who[c] = (who[c] & 0xffff0000u) | (at + (who[c] & 0xffu));
  }
  __syncthreads();
  // ---- per digit: prefix over the warps, the tile's count, its place
  if (tid < 256) {
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kSweepWarps; w++) {
      uint32_t t = wc[w][tid];
      wc[w][tid] = run;
      run += t;
    }
    uint32_t *mine = state + tile * 256 + tid;
    // the count travels with its flag in one word, so no fence is needed
    *reinterpret_cast<volatile uint32_t *>(mine) = run | (tile == 0 ? kAll : kOwn);
    uint32_t x = run, g = counts[tid];
    const uint32_t total = g;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      uint32_t z = __shfl_up_sync(0xffffffffu, g, o);
      if (lane >= o) {
        x += y;
        g += z;
      }
    }
    if (lane == 31) {
      ws[warp] = x;
      wg[warp] = g;
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    uint32_t px = 0, pg = 0;
    for (int w = 0; w < warp; w++) {
      px += ws[w];
      pg += wg[w];
    }
    lstart[tid] = px + x - run;
    const uint32_t before = items_before(
        tile, kSweepLooks,
        [&](int64_t t) { return *reinterpret_cast<const volatile uint32_t *>(state + t * 256 + tid); },
        [&](int64_t t) {  // a tile with tiles after it is full
          return kFirst ? count_low_digit(pos, t * kSweepTile, n, sub_bits, (uint32_t)tid)
                        : count_digit(kin, t * kSweepTile, shift, (uint32_t)tid);
        });
    if (tile > 0) *reinterpret_cast<volatile uint32_t *>(mine) = (before + run) | kAll;
    gbase[tid] = pg + g - total + before;
  }
  __syncthreads();
  // ---- place every item at its slot of the tile sorted by digit
#pragma unroll
  for (int c = 0; c < kSweepItems; c++) {
    const uint32_t d = who[c] >> 16;
    if (d != kNoItem) {
      const uint32_t slot = lstart[d] + wc[warp][d] + (who[c] & 0xffffu);
      sk[slot] = k[c];
      sv[slot] = v[c];
      if (kFirst) reinterpret_cast<uint8_t *>(wc + kSweepWarps)[slot] = (uint8_t)d;
    }
  }
  __syncthreads();
  // ---- write out: consecutive slots of a digit go to consecutive addresses
  const int nt = (int)(np - tbase < kSweepTile ? np - tbase : kSweepTile);
#pragma unroll
  for (int c = 0; c < kSweepItems; c++) {
    const int j = tid + c * kSweepThreads;
    if (j < nt) {
      const uint32_t kk = sk[j];
      const uint32_t dd = kFirst ? reinterpret_cast<uint8_t *>(wc + kSweepWarps)[j] : (kk >> shift) & 0xffu;
      const uint32_t g = gbase[dd] + ((uint32_t)j - lstart[dd]);
      if (!kLast) kout[g] = kk;
      vout[g] = sv[j];
    }
  }
}

constexpr size_t kSweepSmem = sizeof(uint32_t) * (2 * kSweepTile + kSweepWarps * 256);
constexpr size_t kSweepSmemFirst = kSweepSmem + kSweepTile;

bool sweep_sorts(int64_t np) { return np < (int64_t)kOwn; }

uint32_t *sweep_sort(const uint32_t *pos, int64_t np, uint32_t n, int sub_bits, uint32_t *key32, uint32_t *val,
                     uint32_t *val_alt, uint32_t *scratch, cudaStream_t st, int64_t *launches) {
  const int64_t ntiles = (np + kSweepTile - 1) / kSweepTile;
  uint32_t *counts = scratch, *tickets = scratch + kSweepPasses * 256, *state = scratch + kSweepHead;
  uint32_t *ka = key32, *kb = key32 + np;
  // an attribute of the function on the current device: set on every call, so
  // contexts and threads on any device get it
  cudaFuncSetAttribute(k_sweep_pass<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSweepSmemFirst);
  cudaFuncSetAttribute(k_sweep_pass<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSweepSmem);
  cudaFuncSetAttribute(k_sweep_pass<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSweepSmem);
  cudaMemsetAsync(scratch, 0, sizeof(uint32_t) * sweep_words(np), st);
  int blocks = (int)((np + 2047) / 2048);
  if (blocks > 148 * 4) blocks = 148 * 4;
  k_sweep_count<<<blocks, 512, 0, st>>>(pos, np, n, sub_bits, counts);
  k_sweep_pass<true, false><<<(unsigned)ntiles, kSweepThreads, kSweepSmemFirst, st>>>(
      pos, nullptr, nullptr, ka, val, np, n, sub_bits, 0, counts, tickets, state);
  uint32_t *vi = val, *vo = val_alt;
  for (int p = 1; p < kSweepPasses; p++) {
    uint32_t *stp = state + (int64_t)p * 256 * ntiles;
    if (p < kSweepPasses - 1)
      k_sweep_pass<false, false><<<(unsigned)ntiles, kSweepThreads, kSweepSmem, st>>>(
          pos, ka, vi, kb, vo, np, n, sub_bits, 8 * (p - 1), counts + p * 256, tickets + p, stp);
    else
      k_sweep_pass<false, true><<<(unsigned)ntiles, kSweepThreads, kSweepSmem, st>>>(
          pos, ka, vi, kb, vo, np, n, sub_bits, 8 * (p - 1), counts + p * 256, tickets + p, stp);
    uint32_t *t = ka;
    ka = kb;
    kb = t;
    t = vi;
    vi = vo;
    vo = t;
  }
  if (launches) *launches += 1 + kSweepPasses;
  return vi;
}

// The entries (cube of sorted particle i - 1, cube of i] of the range table of
// the 4-cell cubes start at i. Where the mesh is no power of two or particles
// are sparse, runs of empty entries are long (thousands): those are written by
// the whole warp. Called by whole warps; t < tp where there is nothing to
// write.
TPM_D void range_entries(int64_t tp, int64_t t, int64_t i, uint32_t *__restrict__ start) {
  const int lane = threadIdx.x & 31;
  const bool longrun = t - tp > 8;
  if (!longrun)
    for (int64_t q = tp + 1; q <= t; q++) start[q] = (uint32_t)i;
  unsigned m = __ballot_sync(0xffffffffu, longrun);
  while (m) {
    const int src = __ffs(m) - 1;
    m &= m - 1;
    const int64_t a = __shfl_sync(0xffffffffu, tp, src), b = __shfl_sync(0xffffffffu, t, src);
    for (int64_t q = a + 1 + lane; q <= b; q += 32) start[q] = (uint32_t)(i - lane + src);
  }
}

// The sorted particles: their positions, full keys and the range table of the
// cubes key >> shift (ntable of them).
__global__ void __launch_bounds__(256) k_gather_pos(const uint32_t *__restrict__ pos, const uint32_t *__restrict__ perm,
                                                    int64_t np, uint32_t n, int sub_bits, uint32_t *__restrict__ spos,
                                                    uint64_t *__restrict__ skey, int shift, uint32_t ntable,
                                                    uint32_t *__restrict__ start) {
  const int lane = threadIdx.x & 31;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); i0 <= np;
       i0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = i0 + lane;
    uint64_t k = (uint64_t)ntable << shift;
    if (i < np) {
      int64_t p = perm[i];
      const uint32_t u[3] = {pos[3 * p + 0], pos[3 * p + 1], pos[3 * p + 2]};
      k = key_of(u, 0, n, sub_bits);
      spos[3 * i + 0] = u[0];
      spos[3 * i + 1] = u[1];
      spos[3 * i + 2] = u[2];
      skey[i] = k;
    }
    int64_t t = (int64_t)(k >> shift);
    int64_t tp = __shfl_up_sync(0xffffffffu, t, 1);
    if (lane == 0) tp = i > 0 && i <= np ? (int64_t)(key_of(pos, perm[i - 1], n, sub_bits) >> shift) : -1;
    if (i > np) t = tp;
    range_entries(tp, t, i, start);
  }
}

void launch_gather_pos(const uint32_t *pos, const uint32_t *perm, int64_t np, uint32_t n, int sub_bits, uint32_t *spos,
                       uint64_t *skey, int shift, uint32_t ntable, uint32_t *start, cudaStream_t st) {
  int blocks = (int)((np + 256) / 256);
  if (blocks > 148 * 32) blocks = 148 * 32;
  k_gather_pos<<<blocks, 256, 0, st>>>(pos, perm, np, n, sub_bits, spos, skey, shift, ntable, start);
}

__global__ void k_range_table(const uint64_t *__restrict__ key, int64_t np, int shift,
                              uint32_t ntable, uint32_t *__restrict__ start) {
  const int lane = threadIdx.x & 31;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); i0 <= np;
       i0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = i0 + lane;
    int64_t t = -1, tp = -1;
    if (i <= np) {
      t = i < np ? (int64_t)(key[i] >> shift) : (int64_t)ntable;
      tp = i > 0 ? (int64_t)(key[i - 1] >> shift) : -1;
    }
    range_entries(tp, t, i, start);
  }
}

void launch_range_table(const uint64_t *key, int64_t np, int shift, uint32_t ntable, uint32_t *start,
                        cudaStream_t st) {
  int blocks = (int)((np + 256) / 256);
  if (blocks > 148 * 32) blocks = 148 * 32;
  k_range_table<<<blocks, 256, 0, st>>>(key, np, shift, ntable, start);
}

}  // namespace tpm
